// advone_f.cu -- the FP32 vector kernels of the advective operator (every configuration).
#include "advone_tu.cuh"

template struct chswe::AdvOneTU<float>;
