// K2 and K5 for contexts of at most 7 ciphertext primes
#include "k5_kernels.cuh"

template void k2_launch_m<1>(const DevConsts&, const uint64_t*, uint64_t*, int, cudaStream_t);
template void bconv_mma_launch_m<1>(const DevConsts&, bool, const uint64_t*, uint64_t*, int, cudaStream_t);
template void k5_launch_m<1>(const DevConsts&, int, const MulScratch&, uint64_t*, int, cudaStream_t);
template void k2_mixed_launch_m<1>(const Groups&, const LaunchShape&, bool, int, const MulScratch&, cudaStream_t);
template void k5_mixed_launch_m<1>(const Groups&, const LaunchShape&, bool, int, const MulScratch&, cudaStream_t);
template void k2_launch_m<2>(const DevConsts&, const uint64_t*, uint64_t*, int, cudaStream_t);
template void bconv_mma_launch_m<2>(const DevConsts&, bool, const uint64_t*, uint64_t*, int, cudaStream_t);
template void k5_launch_m<2>(const DevConsts&, int, const MulScratch&, uint64_t*, int, cudaStream_t);
template void k2_mixed_launch_m<2>(const Groups&, const LaunchShape&, bool, int, const MulScratch&, cudaStream_t);
template void k5_mixed_launch_m<2>(const Groups&, const LaunchShape&, bool, int, const MulScratch&, cudaStream_t);
