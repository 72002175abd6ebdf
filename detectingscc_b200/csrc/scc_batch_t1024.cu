// The batched kernel with CTAs of 1024 threads.
#include "scc_batch_kernel.cuh"

void *sccb_batch_kernel_1024(bool hong, bool cl) { return batch_kernel<1024>(hong, cl); }
