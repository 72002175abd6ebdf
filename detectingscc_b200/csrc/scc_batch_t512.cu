// The batched kernel with CTAs of 512 threads.
#include "scc_batch_kernel.cuh"

void *sccb_batch_kernel_512(bool hong, bool cl) { return batch_kernel<512>(hong, cl); }
