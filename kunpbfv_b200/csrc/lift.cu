// libkbfv: the key-switch digit lift of the multiply, relinearisation and
// Galois key switches (kernels in lift.cuh).
#include "lift.cuh"

void lift_launch(const DevConsts& dc, uint64_t* sd2, int count, cudaStream_t st) {
    lift_launch_any(LiftJob{dc, sd2}, dc.mm_lift_stride, count * dc.dnum, dc.logn, dc.alpha, dc.shape.k5_threads, st);
}
void lift_mixed_launch(const Groups& G, const DevConsts& top, uint64_t* sd2, int count, cudaStream_t st) {
    lift_launch_any(MixedLiftJob{G, sd2}, G.lift_table, count * G.top_dnum, G.logn, top.alpha, top.shape.k5_threads, st);
}
