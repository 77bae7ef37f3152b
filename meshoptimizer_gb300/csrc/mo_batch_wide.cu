// mo_batch_wide.cu - the batch kernel for meshes whose ids need 32 bits.
#include "mo_batch_kernel.cuh"

namespace mogpu
{

BatchKernel batchKernelWide(bool full)
{
	return full ? kBatch<512, true, unsigned int> : kBatch<512, false, unsigned int>;
}

} // namespace mogpu
