// rfmf_anneal_i32.cu -- the sweep kernels with int32 gains (max weighted degree
// above 127): rfmf_anneal.cu compiled a second time, beside the int8 ones.
#define RFMF_GAIN_BYTES 4
#include "rfmf_anneal.cu"
