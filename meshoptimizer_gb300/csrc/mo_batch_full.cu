// mo_batch_full.cu - the batch kernel with every option, 16-bit ids.
#include "mo_batch_kernel.cuh"

namespace mogpu
{

BatchKernel batchKernelFull(int threads)
{
	return threads == 128 ? kBatch<128, true, unsigned short> : (threads == 512 ? kBatch<512, true, unsigned short> : kBatch<256, true, unsigned short>);
}

} // namespace mogpu
