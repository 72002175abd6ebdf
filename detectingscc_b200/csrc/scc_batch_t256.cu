// The batched kernel with CTAs of 256 threads.
#include "scc_batch_kernel.cuh"

void *sccb_batch_kernel_256(bool hong, bool cl) { return batch_kernel<256>(hong, cl); }
