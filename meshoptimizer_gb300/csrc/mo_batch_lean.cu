// mo_batch_lean.cu - the batch kernel for positions-only batches, 16-bit ids.
#include "mo_batch_kernel.cuh"

namespace mogpu
{

BatchKernel batchKernelLean(int threads)
{
	return threads == 128 ? kBatch<128, false, unsigned short> : (threads == 512 ? kBatch<512, false, unsigned short> : kBatch<256, false, unsigned short>);
}

} // namespace mogpu
