// The batched kernel with CTAs of 128 threads.
#include "scc_batch_kernel.cuh"

void *sccb_batch_kernel_128(bool hong, bool cl) { return batch_kernel<128>(hong, cl); }
