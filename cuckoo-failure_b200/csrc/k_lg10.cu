// Instantiation of the per-prime kernel (primes below 2^50) for transform length 2^10.
#include "kernel_lg.cuh"

cfb::KInfo cf_kinfo_lg10() { return cfb::kinfo<10>(); }
cfb::KInfo cf_kinfo_lg10_few() { return cfb::kinfo<10, false, true>(); }
