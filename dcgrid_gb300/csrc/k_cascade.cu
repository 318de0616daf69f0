// k_cascade.cu — pressure solves of one level with the iterate kept on chip:
// small levels (dense or sparse) by one thread-block cluster per simulation.
//
// The cascade's levels differ by orders of magnitude: a few blocks at the
// coarsest level, millions of cells at a dense fine one. The grid-wide
// cooperative sweep of k_fluid.cu pays a grid barrier per sweep, which is all
// a small level costs; here such levels exchange their halos through
// distributed shared memory and a cluster barrier.
#include <algorithm>

#include "dcg_kernels.h"

namespace dcg {

// ------------------------------------------------------------ small levels
// One cluster of C CTAs relaxes one level of one simulation: CTA r holds the
// blocks [r nbc, (r + 1) nbc) of the level (nbc = ceil(blocks / C)) in shared
// memory, two planes of 64 cells per block (p and p~, as the ping-pong buffers
// of the sweeps), and writes both back to global memory once, after the last
// sweep. A lane owns one subblock (2^3 cells) of a block for the whole solve,
// a warp four blocks per group and up to CL_KG groups; the lane keeps its
// cells' alpha * div in registers, and on each axis one of its
// two outer neighbours lies in its own block and the other across one face,
// so three addresses describe its halo, in its own CTA's shared memory or,
// through the cluster window, in another's. One cluster barrier per sweep.
// A block is stored as [cell x bit][subblock][cell y, z bits], so that the
// eight lanes of a block read any x quad of their neighbours in 128
// contiguous bytes, and the y neighbours of cell x bit 1 lie 128 bytes behind
// those of bit 0; behind it, every subblock's four cells on the block's z
// faces once more as a quad (z neighbours inside the block are shuffled).
// Halo values that no block of the CTA holds as they are needed go through a
// halo area of the block, one place per lane, axis and plane: constants from
// coarser blocks (both planes, copied once per launch), another CTA's values
// (pulled by the lane before each sweep) and the compat quirk's cells (written
// by the lane after each sweep). The sweep proper then has one form.
// What bounds it: the latency chain of one group (about 700 cycles) while a
// warp has one and the level one CTA; the cluster barrier with its release
// fence and the reads of other SMs (about 0.5 us) beyond; the shared-memory
// pipe when a warp has two groups (about 16 wavefronts per block and sweep).
// Microseconds per sweep, grid-wide cooperative solve -> this: 8 blocks 3.2 ->
// 0.36, 128 blocks 3.2 -> 0.97, 1024 blocks 3.6 -> 1.40, 2048 blocks 4.2 ->
// 2.08. Two groups per warp are the limit: three spill registers, and larger
// levels have work for the whole GPU.
constexpr int CL_WARPS = 16, CL_KG = 2, CL_BLOCKS = 4 * CL_WARPS * CL_KG;
// halo area of a block: x quads, y rows and z quads, each value at the place
// (modulo 128 bytes) that it has in the neighbouring block, so that the lanes
// reading blocks and those reading halo areas use different banks
constexpr uint32_t CL_BLK = 384, CL_ZF = 256;  // bytes of a block, its z quads
constexpr uint32_t CL_HALO = 512, CL_HY = 128, CL_HZ = 384;
constexpr uint32_t CL_PLANE = CL_BLOCKS * (CL_BLK + CL_HALO);  // bytes of one plane
constexpr uint32_t CL_SMEM = 2 * CL_PLANE;

// shared-memory accesses at a 32-bit address and a constant offset
template <uint32_t OFF> __device__ __forceinline__ float4 lds4(uint32_t a) {
  float4 v;
  asm volatile("ld.shared.v4.f32 {%0, %1, %2, %3}, [%4+%5];"
               : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w)
               : "r"(a), "n"(OFF));
  return v;
}
template <uint32_t OFF> __device__ __forceinline__ float2 lds2(uint32_t a) {
  float2 v;
  asm volatile("ld.shared.v2.f32 {%0, %1}, [%2+%3];" : "=f"(v.x), "=f"(v.y) : "r"(a), "n"(OFF));
  return v;
}
__device__ __forceinline__ float lds1(uint32_t a) {
  float v;
  asm volatile("ld.shared.f32 %0, [%1];" : "=f"(v) : "r"(a));
  return v;
}
template <uint32_t OFF> __device__ __forceinline__ void sts4(uint32_t a, float4 v) {
  asm volatile("st.shared.v4.f32 [%4+%5], {%0, %1, %2, %3};" ::"f"(v.x), "f"(v.y), "f"(v.z), "f"(v.w), "r"(a), "n"(OFF)
               : "memory");
}
template <uint32_t OFF> __device__ __forceinline__ void sts2(uint32_t a, float2 v) {
  asm volatile("st.shared.v2.f32 [%2+%3], {%0, %1};" ::"f"(v.x), "f"(v.y), "r"(a), "n"(OFF) : "memory");
}
__device__ __forceinline__ void sts1(uint32_t a, float v) {
  asm volatile("st.shared.f32 [%0], %1;" ::"r"(a), "f"(v) : "memory");
}
// through the cluster window (the address may name another CTA's memory)
template <uint32_t OFF> __device__ __forceinline__ float4 ldc4(uint32_t a) {
  float4 v;
  asm volatile("ld.shared::cluster.v4.f32 {%0, %1, %2, %3}, [%4+%5];"
               : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w)
               : "r"(a), "n"(OFF));
  return v;
}
template <uint32_t OFF> __device__ __forceinline__ float2 ldc2(uint32_t a) {
  float2 v;
  asm volatile("ld.shared::cluster.v2.f32 {%0, %1}, [%2+%3];" : "=f"(v.x), "=f"(v.y) : "r"(a), "n"(OFF));
  return v;
}
__device__ __forceinline__ uint32_t map_rank(uint32_t a, uint32_t rank) {
  uint32_t r;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(a), "r"(rank));
  return r;
}
__device__ __forceinline__ void cluster_sync(unsigned csize) {
  if (csize == 1) {
    __syncthreads();
  } else {
    asm volatile("barrier.cluster.arrive.release;" ::: "memory");
    asm volatile("barrier.cluster.wait.acquire;" ::: "memory");
  }
}
__device__ __forceinline__ float2 lo2(float4 v) { return make_float2(v.x, v.y); }
__device__ __forceinline__ float2 hi2(float4 v) { return make_float2(v.z, v.w); }

// kinds of a lane's halo on one axis (4 bits per axis)
constexpr uint32_t H_REMOTE = 1, H_QUIRK = 2;
// float index of a cell (its local coordinates in the block) in the stored block
__host__ __device__ constexpr uint32_t cl_at(int x, int y, int z) {
  return (uint32_t)((x & 1) * 32 + ((x >> 1) * 4 + (y >> 1) * 2 + (z >> 1)) * 4 + (y & 1) * 2 + (z & 1));
}

// what a lane keeps of one group's block for the whole solve
struct ClLane {
  uint32_t aL, aR, aD, aU, aZ;  // shared addresses of its outer neighbours (z: across the block face), plane p
  uint32_t rx, ry, rz;              // its halo in another CTA (cluster addresses)
  uint32_t halo;                    // its block's halo area, plane p
  uint32_t kinds;
  float2 nad[4];                    // -alpha * div, z pairs of the cells (cell x, y bits)
};

// the compat quirk's halo of the lane (cells of its own block at `blk`, places
// packed in qk) into its halo places at `halo`, one plane
__device__ __noinline__ void cl_quirk(uint32_t blk, uint32_t halo, uint32_t kinds, int sub, const uint32_t *qk) {
  auto cell = [&](int a, int q) { return lds1(blk + 4u * ((qk[a] >> (8 * q)) & 255u)); };
  if (kinds & H_QUIRK)
    sts4<0>(halo + 16u * (sub ^ 4), make_float4(cell(0, 0), cell(0, 1), cell(0, 2), cell(0, 3)));
  if (kinds & (H_QUIRK << 4))
    for (int q = 0; q < 4; q++) sts1(halo + CL_HY + 128u * (q >> 1) + 16u * (sub ^ 2) + (sub & 2 ? 0u : 8u) + 4u * (q & 1), cell(1, q));
  if (kinds & (H_QUIRK << 8))
    sts4<CL_HZ>(halo + 16u * (sub ^ 1), make_float4(cell(2, 0), cell(2, 1), cell(2, 2), cell(2, 3)));
}

// One sweep of one group's blocks, plane PAR to the other.
template <int PAR>
__device__ __forceinline__ void cl_sweep(const ClLane &g, uint32_t own, bool on, int sub, unsigned flags,
                                         const uint32_t *qk) {
  constexpr uint32_t PO = PAR * CL_PLANE, PN = (PAR ^ 1) * CL_PLANE;
  if (flags & H_REMOTE) {  // uniform in the warp
    if (g.kinds & H_REMOTE) sts4<PO>(g.halo + 16u * (sub ^ 4), ldc4<PO>(g.rx));
    if (g.kinds & (H_REMOTE << 4)) {
      const float2 a = ldc2<PO>(g.ry), b = ldc2<PO + 128>(g.ry);
      const uint32_t to = g.halo + 16u * (sub ^ 2) + (sub & 2 ? 0u : 8u);
      sts2<PO + CL_HY>(to, a);
      sts2<PO + CL_HY + 128>(to, b);
    }
    if (g.kinds & (H_REMOTE << 8)) sts4<PO + CL_HZ>(g.halo + 16u * (sub ^ 1), ldc4<PO>(g.rz));
  }
  const float4 pa = lds4<PO>(own), pb = lds4<PO + 128>(own);
  const float2 p[4] = {lo2(pa), hi2(pa), lo2(pb), hi2(pb)};
  const float4 L = lds4<PO>(g.aL), R = lds4<PO>(g.aR);
  const float2 D0 = lds2<PO>(g.aD), D1 = lds2<PO + 128>(g.aD), U0 = lds2<PO>(g.aU), U1 = lds2<PO + 128>(g.aU);
  const float4 h = lds4<PO>(g.aZ);
  // z neighbours of the cells (x, y) = 00, 01, 10, 11: across the block's face,
  // and inside the block in the next lane
  const bool z = sub & 1;
  const float hz[4] = {h.x, h.y, h.z, h.w};
  float bk[4], fw[4];
#pragma unroll
  for (int q = 0; q < 4; q++) {
    const float t = __shfl_xor_sync(0xffffffffu, z ? p[q].x : p[q].y, 1);
    bk[q] = z ? t : hz[q];
    fw[q] = z ? hz[q] : t;
  }
  // per pair: L + R + D + U, then cell z = 0 adds (behind, z = 1) and cell z =
  // 1 adds (z = 0, in front), then - alpha div: the order of the scalar sweep
  float2 sum[4];
  sum[0] = __fadd2_rn(__fadd2_rn(__fadd2_rn(lo2(L), p[2]), D0), p[1]);
  sum[1] = __fadd2_rn(__fadd2_rn(__fadd2_rn(hi2(L), p[3]), p[0]), U0);
  sum[2] = __fadd2_rn(__fadd2_rn(__fadd2_rn(p[0], lo2(R)), D1), p[3]);
  sum[3] = __fadd2_rn(__fadd2_rn(__fadd2_rn(p[1], hi2(R)), p[2]), U1);
#pragma unroll
  for (int q = 0; q < 4; q++) {
    sum[q].x = sum[q].x + bk[q] + p[q].y;
    sum[q].y = sum[q].y + p[q].x + fw[q];
    sum[q] = __fadd2_rn(sum[q], g.nad[q]);
  }
  div6_pairs(sum);
  if (on) {
    sts4<PN>(own, make_float4(sum[0].x, sum[0].y, sum[1].x, sum[1].y));
    sts4<PN + 128>(own, make_float4(sum[2].x, sum[2].y, sum[3].x, sum[3].y));
    sts4<PN + CL_ZF>(own, make_float4(z ? sum[0].y : sum[0].x, z ? sum[1].y : sum[1].x, z ? sum[2].y : sum[2].x,
                                      z ? sum[3].y : sum[3].x));
  }
  if (flags & H_QUIRK) {
    __syncwarp();  // the block's new cells are stored
    if (g.kinds & (0x111u * H_QUIRK)) cl_quirk(own - 16u * sub + PN, g.halo + PN, g.kinds, sub, qk);
  }
}

// Fills a group's blocks into plane p (prolonged from the parent level when
// asked) and their halo areas, and the lane's record. b: the lane's block, at
// place i of the CTA (lanes without a block take the group's first one, on =
// false). Out of line: the sweeps need the registers.
struct ClLevel {
  long long off;
  int nblk, nbc, prolong, quirk;
  uint32_t sm0, rank;
  float alpha;
};
__device__ __noinline__ void cl_setup(const Dev &D, const ClLevel &l, uint32_t b, int i, bool on, const uint32_t *qk,
                                      ClLane &g) {
  const int sub = threadIdx.x & 7, sx = (sub >> 2) & 1, sy = (sub >> 1) & 1, sz = sub & 1;
  const int4 bp = D.pos[b];
  const uint32_t base = l.sm0 + CL_BLK * i;
  g.halo = l.sm0 + CL_BLOCKS * CL_BLK + CL_HALO * i;
  const size_t cell = (size_t)b * BV + 8 * sub;
  const float4 da = __ldcg(reinterpret_cast<const float4 *>(D.div + cell)),
               dc = __ldcg(reinterpret_cast<const float4 *>(D.div + cell) + 1);
  g.nad[0] = make_float2(-(l.alpha * da.x), -(l.alpha * da.y));
  g.nad[1] = make_float2(-(l.alpha * da.z), -(l.alpha * da.w));
  g.nad[2] = make_float2(-(l.alpha * dc.x), -(l.alpha * dc.y));
  g.nad[3] = make_float2(-(l.alpha * dc.z), -(l.alpha * dc.w));
  if (on) {
    const uint32_t to = base + 16u * sub;
    sts4<0>(to, __ldcg(reinterpret_cast<const float4 *>(D.p + cell)));
    sts4<128>(to, __ldcg(reinterpret_cast<const float4 *>(D.p + cell) + 1));
    if (l.prolong && D.parent[b] != NONE)
      for (int q = 0; q < 8; q++) {
        float t = 0.f;
        prolong_value(D, b, 8 * sub + q, t);
        sts1(to + 128u * (q >> 2) + 4u * (q & 3), t);
      }
    for (int q = 0; q < 4; q++)
      sts1(to + CL_ZF + 4u * q, lds1(to + 128u * (q >> 1) + 8u * (q & 1) + 4u * sz));
  }
  __syncwarp();  // the quirk reads other lanes' cells
  uint32_t kd = 0, at[3], far[3];
  for (int a = 0; a < 3; a++) {
    far[a] = base;
    const bool high = (a == 0 ? sx : a == 1 ? sy : sz) != 0;
    const int dir = a == 0 ? (high ? 22 : 4) : a == 1 ? (high ? 16 : 10) : (high ? 14 : 12);
    const uint32_t e = D.nbr[27u * b + dir];
    const uint32_t place = g.halo + (a == 0 ? 16u * (sub ^ 4) : a == 1 ? CL_HY + 16u * (sub ^ 2) + (sy ? 0u : 8u) : CL_HZ + 16u * (sub ^ 1));
    at[a] = place;
    if (e == OUT) {
      if (l.quirk) {
        kd |= H_QUIRK << (4 * a);
      } else {  // the lane's own outer cells
        at[a] = base + 16u * sub + (a == 0 ? (sx ? 128u : 0u) : a == 1 ? (sy ? 8u : 0u) : CL_ZF);
      }
      continue;
    }
    const uint32_t nb = e & NBR_MASK;
    const int lc = (int)(e >> 28);
    const long long li = (long long)nb - l.off;
    if (lc == 0 && li >= 0 && li < l.nblk) {
      const uint32_t r = (uint32_t)li / (uint32_t)l.nbc, i2 = (uint32_t)li - r * (uint32_t)l.nbc;
      const uint32_t there = l.sm0 + CL_BLK * i2 + (a == 0 ? 16u * (sub ^ 4) + (sx ? 0u : 128u)
                                                  : a == 1 ? 16u * (sub ^ 2) + (sy ? 0u : 8u) : CL_ZF + 16u * (sub ^ 1));
      if (r == l.rank) {
        at[a] = there;
      } else {
        kd |= H_REMOTE << (4 * a);
        far[a] = map_rank(there, r);
      }
      continue;
    }
    // constant during the solve: cells of a coarser block (injection)
    if (on)
      for (int q = 0; q < 4; q++) {
        const int u = q >> 1, v = q & 1;
        const int x = a == 0 ? (high ? 4 : -1) : 2 * sx + u;
        const int y = a == 1 ? (high ? 4 : -1) : 2 * sy + (a == 0 ? u : v);
        const int z = a == 2 ? (high ? 4 : -1) : 2 * sz + v;
        const size_t c = (size_t)nb * BV + local_of(((bp.x + x) >> lc) & 3, ((bp.y + y) >> lc) & 3, ((bp.z + z) >> lc) & 3);
        const uint32_t to = place + (a == 1 ? 128u * u + 4u * v : 8u * u + 4u * v);
        sts1(to, __ldcg(D.p + c));
        sts1(to + CL_PLANE, __ldcg(D.pt + c));
      }
  }
  g.kinds = on ? kd : 0u;  // lanes without a block repeat the group's first one and store nothing
  if (g.kinds & (0x111u * H_QUIRK)) cl_quirk(base, g.halo, g.kinds, sub, qk);
  // the outer neighbours that lie in the own block
  const uint32_t ix = base + 16u * (sub ^ 4) + (sx ? 128u : 0u), iy = base + 16u * (sub ^ 2) + (sy ? 8u : 0u);
  g.aL = sx ? ix : at[0];
  g.aR = sx ? at[0] : ix;
  g.aD = sy ? iy : at[1];
  g.aU = sy ? at[1] : iy;
  g.aZ = at[2];
  g.rx = far[0];
  g.ry = far[1];
  g.rz = far[2];
}

__global__ void __launch_bounds__(32 * CL_WARPS, 1) k_cluster_solve(const __grid_constant__ ClusterSolve P) {
  extern __shared__ __align__(128) float sm[];
  const unsigned C = (unsigned)P.csize, rank = blockIdx.x % C, m = blockIdx.x / C;
  const Dev &D = P.d[m];
  const int w = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int sub = lane & 7, sx = (sub >> 2) & 1, sy = (sub >> 1) & 1, sz = sub & 1;
  const unsigned full = 0xffffffffu;
  const uint32_t sm0 = (uint32_t)__cvta_generic_to_shared(sm);
  // places of the compat quirk's cells for the lane's halo on each axis
  uint32_t qk[3] = {0u, 0u, 0u};
#pragma unroll
  for (int q = 0; q < 4; q++) {
    const int u = q >> 1, r = q & 1;
    qk[0] |= cl_at(sx ? 0 : 1, (2 * sy + u + 1) & 3, (2 * sz + r + 1) & 3) << (8 * q);
    qk[1] |= cl_at((2 * sx + u + 1) & 3, sy ? 0 : 1, (2 * sz + r + 1) & 3) << (8 * q);
    qk[2] |= cl_at((2 * sx + u + 1) & 3, (2 * sy + r + 1) & 3, sz ? 0 : 1) << (8 * q);
  }
  for (int lev = P.hi[m]; lev >= P.lo[m]; lev--) {
    const int nblk = (int)min(__ldcg(D.load + lev), (long long)D.g.budget[lev]);
    if (nblk <= 0 || nblk > P.limit) continue;  // uniform in the cluster
    // a level of at most one group per warp stays in the first CTA: its sweeps
    // need no cluster barrier
    const unsigned Ce = nblk <= 4 * CL_WARPS ? 1u : C;
    const int nbc = (nblk + (int)Ce - 1) / (int)Ce;
    const int first = (int)rank * nbc, mine = max(0, min(nbc, nblk - first));
    const long long off = D.g.off[lev];
    const int sc = 1 << lev;
    const ClLevel lv = {off, nblk, nbc, P.prolong && lev < D.g.levels - 1, D.g.ref_compat && lev < D.g.sparse, sm0, rank,
                        (float)(sc * sc) * D.ph.dx * D.ph.dx};
    ClLane g[CL_KG];
    unsigned flags[CL_KG];  // halo kinds of any lane of the group, axes merged
#pragma unroll
    for (int k = 0; k < CL_KG; k++) {
      flags[k] = 0;
      const int i0 = 4 * (k * CL_WARPS + w);
      if (i0 >= mine) break;  // warp-uniform
      const int i = i0 + (lane >> 3) < mine ? i0 + (lane >> 3) : i0;
      ClLane r;
      cl_setup(D, lv, (uint32_t)(off + first + i), i, i == i0 + (lane >> 3), qk, r);
      g[k] = r;
      const unsigned all = __reduce_or_sync(full, r.kinds);
      flags[k] = (all | all >> 4 | all >> 8) & 15u;
    }
    cluster_sync(C);
    const uint32_t own = sm0 + CL_BLK * (4 * w + (lane >> 3)) + 16u * sub;
    const int sweeps = rank < Ce ? P.sweeps : 0;  // even
#pragma unroll 1
    for (int it = 0; it < sweeps; it += 2) {
#pragma unroll
      for (int k = 0; k < CL_KG; k++) {
        const int i0 = 4 * (k * CL_WARPS + w);
        if (i0 >= mine) break;  // warp-uniform
        cl_sweep<0>(g[k], own + 4 * CL_BLK * CL_WARPS * k, i0 + (lane >> 3) < mine, sub, flags[k], qk);
      }
      cluster_sync(Ce);
#pragma unroll
      for (int k = 0; k < CL_KG; k++) {
        const int i0 = 4 * (k * CL_WARPS + w);
        if (i0 >= mine) break;
        cl_sweep<1>(g[k], own + 4 * CL_BLK * CL_WARPS * k, i0 + (lane >> 3) < mine, sub, flags[k], qk);
      }
      cluster_sync(Ce);
    }
    // both planes back to global memory, and visible to the cluster's next level
#pragma unroll 1
    for (int i = 4 * w + (lane >> 3); i < mine; i += 4 * CL_WARPS) {
      const size_t cell = (size_t)(off + first + i) * BV + 8 * sub;
      const uint32_t at = sm0 + CL_BLK * i + 16u * sub;
      reinterpret_cast<float4 *>(D.p + cell)[0] = lds4<0>(at);
      reinterpret_cast<float4 *>(D.p + cell)[1] = lds4<128>(at);
      if (P.sweeps > 0) {
        reinterpret_cast<float4 *>(D.pt + cell)[0] = lds4<CL_PLANE>(at);
        reinterpret_cast<float4 *>(D.pt + cell)[1] = lds4<CL_PLANE + 128>(at);
      }
    }
    __threadfence();
    cluster_sync(C);
  }
}

// Largest cluster the device can hold for k_cluster_solve: 16 (with the
// non-portable opt-in), 8, or 0
int cluster_solve_size() {
  if (cudaFuncSetAttribute(k_cluster_solve, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)CL_SMEM) != cudaSuccess) {
    cudaGetLastError();
    return 0;
  }
  for (int c : {16, 8}) {
    if (c > 8 && cudaFuncSetAttribute(k_cluster_solve, cudaFuncAttributeNonPortableClusterSizeAllowed, 1) != cudaSuccess) {
      cudaGetLastError();
      continue;
    }
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)c);
    cfg.blockDim = dim3(32 * CL_WARPS);
    cfg.dynamicSmemBytes = CL_SMEM;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = (unsigned)c;
    attr[0].val.clusterDim.y = attr[0].val.clusterDim.z = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    int n = 0;
    if (cudaOccupancyMaxActiveClusters(&n, k_cluster_solve, &cfg) == cudaSuccess && n > 0) return c;
    cudaGetLastError();
  }
  return 0;
}
// The levels that go to a cluster: one group of blocks per warp. The second
// group is for launches of many members, whose clusters are smaller: alone, a
// level that needs it is faster with the whole GPU (us per sweep: 1830 sparse
// blocks 3.3 here, 2.0 in the resident solve, 1728 full ones 2.0 and 1.85; of
// 1024 full blocks 1.4 and 1.8).
long long cluster_solve_blocks(int csize) { return (long long)csize * CL_WARPS * 4; }

// max_blocks: the largest level of the launch. CTAs per cluster: about one
// group of blocks per warp, but no more than the clusters of all members fit
// the GPU at once while the blocks fit the smaller cluster.
void launch_cluster_solve(ClusterSolve &P, int max_csize, long long max_blocks, int sms, cudaStream_t st) {
  int c = 1;
  while (c < max_csize && (long long)c * CL_WARPS * 4 < max_blocks) c *= 2;
  while (c > 1 && P.n * c > sms && (long long)(c / 2) * CL_BLOCKS >= max_blocks) c /= 2;
  P.csize = c;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3((unsigned)(P.n * c));
  cfg.blockDim = dim3(32 * CL_WARPS);
  cfg.dynamicSmemBytes = CL_SMEM;
  cfg.stream = st;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = (unsigned)c;
  attr[0].val.clusterDim.y = attr[0].val.clusterDim.z = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  cudaLaunchKernelEx(&cfg, k_cluster_solve, P);
}

}  // namespace dcg
