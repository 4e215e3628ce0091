// Block-level pieces of batch inversion (Montgomery's simultaneous inversion): one
// inversion for the threads of a block. Used by the Fr vector operations' batch inverse
// (zkb_fr.cu) and by the MSM's affine bucket tree (zkb_msm_tree.cuh).
#pragma once
#include "zkb_field.cuh"

namespace zkb {

// The inverse of every thread's v with one inversion per block of NW warps (one zero among them makes every
// result of the block zero, as the inverse of zero is; the Fr operations' flag covers the other blocks): products up a
// binary tree (butterfly shuffles in the warp, then the warps' products in warp 0), the inversion of the
// total by warp 0's lanes alike, and down again, a child's inverse being its parent's times its
// sibling's product: 2 (5 + log2 NW) products in a row. (Two exclusive scans took 30.) sw: 2 NW elements;
// every thread of the block must call it.
template <class P, int NW>
__device__ __forceinline__ Fe<P> block_inverse(const Fe<P>& v, Fe<P>* sw) {
  static_assert(NW == 8, "three levels across warps");
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  auto up = [&](Fe<P>& p, int d) {
    Fe<P> y;
#pragma unroll
    for (int k = 0; k < P::N; k++) y.v[k] = __shfl_xor_sync(0xffffffffu, p.v[k], d);
    p = fe_mul(p, y);
    return y;
  };
  Fe<P> sib[5], p = v;
#pragma unroll
  for (int l = 0; l < 5; l++) sib[l] = up(p, 1 << l);
  if (lane == 0) sw[wid] = p;
  __syncthreads();
  if (wid == 0) {
    Fe<P> q = sw[lane & (NW - 1)], s2[3];
#pragma unroll
    for (int l = 0; l < 3; l++) s2[l] = up(q, 1 << l);
    q = fe_inv(q);
#pragma unroll
    for (int l = 2; l >= 0; l--) q = fe_mul(q, s2[l]);
    if (lane < NW) sw[NW + lane] = q;
  }
  __syncthreads();
  Fe<P> inv = sw[NW + wid];
#pragma unroll
  for (int l = 4; l >= 0; l--) inv = fe_mul(inv, sib[l]);
  return inv;
}

}  // namespace zkb
