// one_f.cu -- the FP32 one-launch stage (every configuration and RK mode).
#include "one_tu.cuh"

template struct chswe::OneTU<float>;
