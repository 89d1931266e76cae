// spns_len.cu -- the pass kernels of one FFT length (SPNS_LEN) in one precision
// (SPNS_T, table name suffix SPNS_P); the Makefile compiles it once per pair.
#include "len_launch.cuh"

#define SPNS_CAT2(a, b, c, d) a##b##c##d
#define SPNS_CAT(a, b, c, d) SPNS_CAT2(a, b, c, d)
extern const LenTable SPNS_CAT(spns_len_, SPNS_P, _, SPNS_LEN) = LenLaunch<SPNS_T>::table<SPNS_LEN>();
