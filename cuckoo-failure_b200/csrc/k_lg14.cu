// Instantiation of the per-prime kernel (primes below 2^50) for transform length 2^14.
#include "kernel_lg.cuh"

cfb::KInfo cf_kinfo_lg14() { return cfb::kinfo<14>(); }
