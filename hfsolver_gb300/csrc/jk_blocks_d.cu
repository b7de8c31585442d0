// The heavy tier (kets dp and dd) of the block Fock-build kernel (jk_blocks.cuh).
#include "jk_blocks.cuh"

namespace hfgpu {

void launch_digest_heavy(const DigestLaunch& l, cudaStream_t s)
{
    digest_kernel<2><<<l.nblocks, DIGEST_BLOCK, 0, s>>>(l);
}

}  // namespace hfgpu
