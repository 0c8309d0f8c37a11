// advone_d.cu -- the FP64 vector kernels of the advective operator (every configuration).
#include "advone_tu.cuh"

template struct chswe::AdvOneTU<double>;
