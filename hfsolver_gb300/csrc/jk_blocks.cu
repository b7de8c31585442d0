// The light and middle tiers of the block Fock-build kernel (jk_blocks.cuh); the
// heavy tier is in jk_blocks_d.cu, so that they compile in parallel.
#include "internal.h"
#include "jk_blocks.cuh"

namespace hfgpu {

void launch_digest_heavy(const DigestLaunch& l, cudaStream_t s);  // jk_blocks_d.cu

void launch_digest_tier(int tier, const DigestLaunch& l, cudaStream_t s)
{
    if (tier == 0)
        digest_kernel<0><<<l.nblocks, DIGEST_BLOCK, 0, s>>>(l);
    else if (tier == 1)
        digest_kernel<1><<<l.nblocks, DIGEST_BLOCK, 0, s>>>(l);
    else
        launch_digest_heavy(l, s);
    count_launch();
    HF_CUDA(cudaGetLastError());
}

}  // namespace hfgpu
