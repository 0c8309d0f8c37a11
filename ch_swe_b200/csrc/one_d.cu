// one_d.cu -- the FP64 one-launch stage (every configuration and RK mode).
#include "one_tu.cuh"

template struct chswe::OneTU<double>;
