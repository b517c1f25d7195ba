// Instantiation of the per-prime kernel for primes below 2^62 at transform length 2^14, in a unit of its
// own for its assembler options (build.py).
#include "kernel_lg.cuh"

cfb::KInfo cf_kinfo_lg14_w() { return cfb::kinfo<14, true>(); }
