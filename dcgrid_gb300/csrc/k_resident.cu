// k_resident.cu — one level's Jacobi sweeps, and their transpose, with the
// level's cells kept in registers: for levels too large for a cluster and
// small enough for the registers of the chip (256 blocks per SM).
//
// Half a warp holds a block, a lane the quad of cells 4h .. 4h+3 of it (two
// along y by two along z at one x). A sweep reads only the block's face halo
// from memory, the previous sweep's values of other warps: one float4 per lane
// on an x face, one float2 and two words per lane for its y and z face;
// neighbours inside the block come from warp shuffles. Sweeps are separated by
// grid barriers, so the launch is cooperative, one CTA per SM. What bounds a
// sweep is the barrier (1.4 us) and one round trip to L2, from some 16000
// blocks on the shuffles and the halo's sectors. Copying blocks and halos to
// shared tiles in every sweep (k_level_solve_batch, which larger levels need)
// took 3.1 us per sweep of 4096 blocks, 3.9 of 8192 and 7.7 of 32768; here they
// take 2.0, 2.4 and 5.8. A cluster (k_cascade.cu) takes 1.4 for 1024 blocks and
// 2.05 for 2048, here 1.8 and 1.9 and a launch: the line lies where a cluster
// has one group of blocks per warp, 1024.
#include "dcg_dev.cuh"
#include "dcg_kernels.h"

namespace dcg {

constexpr int RS_WARPS = 16;  // warps per CTA; block pairs per warp: K

// how a quad reads the halo of a face: as stored by the neighbour block (or by
// the block itself, at the domain's boundary), one coarser cell for all, or by
// the cells that the reference's refresh takes there in compat mode; SLOW and
// QUIRK: some quad of the warp has a coarser neighbour or such a boundary
enum : uint32_t {
  RS_X = 1u, RS_XC = 2u, RS_XQ = 4u, RS_YC = 8u, RS_YQ = 16u, RS_ZC = 32u, RS_SLOW = 64u, RS_QUIRK = 128u
};

struct Quad {
  float v[4];  // its cells: (y, z), (y, z+1), (y+1, z), (y+1, z+1)
  uint32_t x, fl;
};
// what a sweep needs of a quad besides: where its faces' halos and its own
// first cell are (arena cells; own ~0u: no block), and alpha * div
struct QuadRest {
  uint32_t y, z0, z1, own;
  float ad[4];
};
// With up to two pairs per warp in registers, with more in shared memory.
template <int K> struct Rests {
  static constexpr bool kShared = K > 2;
  static constexpr size_t kBytes = kShared ? (size_t)K * RS_WARPS * 32 * sizeof(QuadRest) : 0;
  QuadRest r[kShared ? 1 : K];
  uint4 *s;
  __device__ Rests() {
    extern __shared__ __align__(16) uint4 s_rest[];  // [k][index word, ad][thread]
    s = s_rest + threadIdx.x;
  }
  __device__ __forceinline__ void put(int k, const QuadRest &q) {
    if constexpr (kShared) {
      s[2 * k * RS_WARPS * 32] = make_uint4(q.y, q.z0, q.z1, q.own);
      s[(2 * k + 1) * RS_WARPS * 32] = make_uint4(__float_as_uint(q.ad[0]), __float_as_uint(q.ad[1]),
                                                  __float_as_uint(q.ad[2]), __float_as_uint(q.ad[3]));
    } else {
      r[k] = q;
    }
  }
  __device__ __forceinline__ uint4 at(int k) const {
    if constexpr (kShared) return s[2 * k * RS_WARPS * 32];
    else return make_uint4(r[k].y, r[k].z0, r[k].z1, r[k].own);
  }
  __device__ __forceinline__ float4 ad(int k) const {
    if constexpr (kShared) {
      const uint4 a = s[(2 * k + 1) * RS_WARPS * 32];
      return make_float4(__uint_as_float(a.x), __uint_as_float(a.y), __uint_as_float(a.z), __uint_as_float(a.w));
    } else {
      return make_float4(r[k].ad[0], r[k].ad[1], r[k].ad[2], r[k].ad[3]);
    }
  }
};

__device__ __forceinline__ void rs_faces(const Dev &D, uint32_t b, uint32_t a, int h, Quad &q, QuadRest &r) {
  const int4 bp = D.pos[b];
  const int x1 = (h >> 3) & 1, y1 = (h >> 2) & 1, z1 = (h >> 1) & 1, x0 = h & 1;
  const int x = 2 * x1 + x0, y = 2 * y1, z = 2 * z1;  // of the quad's first cell in the block
  const bool quirk = D.g.ref_compat && bp.w < D.g.sparse;
  const uint32_t base = a + b * (uint32_t)BV;
  q.fl = 0u;
  // a halo cell at a coarser level: the cell of `nb` that covers (cx, cy, cz)
  auto coarse = [&](uint32_t e, int cx, int cy, int cz) {
    const int k = (int)(e >> 28);
    return a + (e & NBR_MASK) * (uint32_t)BV + (uint32_t)local_of((cx >> k) & 3, (cy >> k) & 3, (cz >> k) & 3);
  };
  q.x = base;
  if (x0 == x1) {
    q.fl |= RS_X;
    const uint32_t e = D.nbr[27u * b + (x1 ? 22 : 4)];
    if (e == OUT) {
      if (quirk) q.fl |= RS_XQ;
      else q.x = base + 4 * h;
    } else if ((e >> 28) == 0u) {
      q.x = a + (e & NBR_MASK) * (uint32_t)BV + 4u * (uint32_t)(h ^ 9);
    } else {
      q.fl |= RS_XC;
      q.x = coarse(e, bp.x + (x1 ? 4 : -1), bp.y + y, bp.z + z);
    }
  }
  const uint32_t ey = D.nbr[27u * b + (y1 ? 16 : 10)];
  r.y = base;
  if (ey == OUT) {
    if (quirk) q.fl |= RS_YQ;
    else r.y = base + 4 * h + 2 * y1;
  } else if ((ey >> 28) == 0u) {
    r.y = a + (ey & NBR_MASK) * (uint32_t)BV + 4u * (uint32_t)(h ^ 4) + (y1 ? 0u : 2u);
  } else {
    q.fl |= RS_YC;
    r.y = coarse(ey, bp.x + x, bp.y + (y1 ? 4 : -1), bp.z + z);
  }
  const uint32_t ez = D.nbr[27u * b + (z1 ? 14 : 12)];
  if (ez == OUT) {
    if (quirk) {
      const int qz = z1 ? 0 : 1;
      r.z0 = base + local_of((x + 1) & 3, (y + 1) & 3, qz);
      r.z1 = base + local_of((x + 1) & 3, (y + 2) & 3, qz);
    } else {
      r.z0 = base + 4 * h + z1;
      r.z1 = r.z0 + 2;
    }
  } else if ((ez >> 28) == 0u) {
    r.z0 = a + (ez & NBR_MASK) * (uint32_t)BV + 4u * (uint32_t)(h ^ 2) + (z1 ? 0u : 1u);
    r.z1 = r.z0 + 2;
  } else {
    q.fl |= RS_ZC;
    r.z0 = r.z1 = coarse(ez, bp.x + x, bp.y + y, bp.z + (z1 ? 4 : -1));
  }
}

struct Halo {
  float4 x;
  float2 y;
  float z0, z1;
};

// The halo values of a quad as loaded: on a face to a coarser block the aligned
// vector that holds the coarser cell (rs_fix picks it when the loads are due).
// Loads go to L2: the planes are rewritten by other SMs within the launch.
__device__ __forceinline__ void rs_load(const float *__restrict__ src, const Quad &q, const uint4 &r, Halo &o) {
  o.x = make_float4(0.f, 0.f, 0.f, 0.f);
  if ((q.fl & (RS_X | RS_XQ)) == RS_X) o.x = __ldcg(reinterpret_cast<const float4 *>(src + (q.x & ~3u)));
  if (!(q.fl & RS_YQ)) o.y = __ldcg(reinterpret_cast<const float2 *>(src + (r.x & ~1u)));
  o.z0 = __ldcg(src + r.y);
  o.z1 = __ldcg(src + r.z);
}
// ADJ: a coarser neighbour contributes nothing. The compat boundary's cells on
// x and y faces are the block's own, shifted by one along every axis: they
// come from the lanes that hold them (a second load into the same registers
// would wait for the first: 1283 blocks 2.46 us per sweep, with shuffles 1.92).
template <bool ADJ> __device__ __forceinline__ void rs_fix(const Quad &q, const uint4 &r, int h, Halo &o) {
  if (q.fl & RS_QUIRK) {  // uniform in the warp
    const unsigned all = 0xffffffffu;
    const int top = threadIdx.x & 16, x1 = h & 8, y1 = h & 4, z1 = h & 2, x0 = h & 1;
    // x face: (1 or 0, y + 1 or y + 2, z + 1 or z + 2), modulo 4
    const int fx = top | (x0 ^ 1);
    const float a = __shfl_sync(all, q.v[3], fx | y1 | z1), b = __shfl_sync(all, q.v[2], fx | y1 | (z1 ^ 2)),
                c = __shfl_sync(all, q.v[1], fx | (y1 ^ 4) | z1), d = __shfl_sync(all, q.v[0], fx | (y1 ^ 4) | (z1 ^ 2));
    // y face: (x + 1, 1 or 0, z + 1 or z + 2)
    const int fy = top | (x0 ? x1 ^ 8 : x1) | (x0 ^ 1);
    const float e0 = __shfl_sync(all, q.v[1], fy | z1), e1 = __shfl_sync(all, q.v[3], fy | z1),
                f0 = __shfl_sync(all, q.v[0], fy | (z1 ^ 2)), f1 = __shfl_sync(all, q.v[2], fy | (z1 ^ 2));
    if (q.fl & RS_XQ) o.x = make_float4(a, b, c, d);
    if (q.fl & RS_YQ) o.y = make_float2(y1 ? e0 : e1, y1 ? f0 : f1);
  }
  if (!(q.fl & RS_SLOW)) return;  // uniform in the warp
  if (q.fl & RS_XC) {
    const float a = q.x & 1u ? o.x.y : o.x.x, b = q.x & 1u ? o.x.w : o.x.z, c = ADJ ? 0.f : q.x & 2u ? b : a;
    o.x = make_float4(c, c, c, c);
  }
  if (q.fl & RS_YC) {
    const float c = ADJ ? 0.f : r.x & 1u ? o.y.y : o.y.x;
    o.y = make_float2(c, c);
  }
  if (ADJ && (q.fl & RS_ZC)) o.z0 = o.z1 = 0.f;
}

// The sums of a quad's six neighbours in the order of k_jacobi (L, R, D, U, B,
// F), as pairs along z; every lane of the warp takes part.
__device__ __forceinline__ void rs_sums(const Quad &q, const Halo &hv, int h, float2 (&s)[2]) {
  const unsigned all = 0xffffffffu;
  const bool x0 = h & 1, y1 = h & 4, z1 = h & 2, xf = q.fl & RS_X;
  float n[4], f[4];  // the x neighbours of the other parity: next to the quad in its subblock, and across
#pragma unroll
  for (int i = 0; i < 4; i++) {
    n[i] = __shfl_xor_sync(all, q.v[i], 1);
    f[i] = __shfl_xor_sync(all, q.v[i], 9);
  }
  if (xf) {
    f[0] = hv.x.x;
    f[1] = hv.x.y;
    f[2] = hv.x.z;
    f[3] = hv.x.w;
  }
  // across y: the row of the quad on the other side of the block's middle, or the halo
  const float ya = __shfl_xor_sync(all, y1 ? q.v[0] : q.v[2], 4), yb = __shfl_xor_sync(all, y1 ? q.v[1] : q.v[3], 4);
  const float2 yo = make_float2(ya, yb);
  const float2 dn = y1 ? yo : hv.y, up = y1 ? hv.y : yo;
  const float za = __shfl_xor_sync(all, z1 ? q.v[0] : q.v[1], 2), zb = __shfl_xor_sync(all, z1 ? q.v[2] : q.v[3], 2);
  const float2 r0 = make_float2(q.v[0], q.v[1]), r1 = make_float2(q.v[2], q.v[3]);
#pragma unroll
  for (int r = 0; r < 2; r++) {
    const float2 nn = make_float2(n[2 * r], n[2 * r + 1]), ff = make_float2(f[2 * r], f[2 * r + 1]);
    const float zo = r ? zb : za, zh = r ? hv.z1 : hv.z0;
    float2 t = __fadd2_rn(x0 ? nn : ff, x0 ? ff : nn);
    t = __fadd2_rn(t, r ? r0 : dn);
    t = __fadd2_rn(t, r ? up : r1);
    t = __fadd2_rn(t, make_float2(z1 ? zo : zh, r ? r1.x : r0.x));
    s[r] = __fadd2_rn(t, make_float2(r ? r1.y : r0.y, z1 ? zh : zo));
  }
}

// a lane without a block reads the planes' first cells, which nothing uses
__device__ __forceinline__ void rs_flags(Quad &q) {
  if (__any_sync(0xffffffffu, q.fl & (RS_XC | RS_YC | RS_ZC))) q.fl |= RS_SLOW;
  if (__any_sync(0xffffffffu, q.fl & (RS_XQ | RS_YQ))) q.fl |= RS_QUIRK;
}

// s_end[m]: the blocks of members 0..m
template <int K>
__device__ __forceinline__ void rs_solve(const SolveBatch &P, const long long *s_end, long long total, int sweeps,
                                         GridBarrier &bar) {
  const int t = threadIdx.x, h = t & 15;
  const int warps = blockDim.x >> 5;
  Quad q[K];
  Rests<K> rest;
  int pairs = 0;  // of the warp
#pragma unroll
  for (int k = 0; k < K; k++) {
    const long long pair = (long long)(k * warps + (t >> 5)) * gridDim.x + blockIdx.x;
    const long long g = 2 * pair + ((t >> 4) & 1);
    if (2 * pair < total) pairs = k + 1;
    QuadRest r = {0u, 0u, 0u, ~0u, {0.f, 0.f, 0.f, 0.f}};
    q[k] = {{0.f, 0.f, 0.f, 0.f}, 0u, 0u};
    if (g < total) {
      int m = 0;
      while (g >= s_end[m]) m++;
      const Dev &D = P.d[m];
      const int lev = P.lev[m];
      const uint32_t b = (uint32_t)(D.g.off[lev] + g - (m ? s_end[m - 1] : 0)), a = (uint32_t)P.arena[m];
      rs_faces(D, b, a, h, q[k], r);
      r.own = a + b * (uint32_t)BV + 4u * h;
      float4 v = __ldcg(reinterpret_cast<const float4 *>(P.p + r.own));
      const float4 dv = *reinterpret_cast<const float4 *>(P.div + r.own);
      if (P.prolong && lev < D.g.levels - 1) {
        prolong_value(D, b, 4 * h, v.x);
        prolong_value(D, b, 4 * h + 1, v.y);
        prolong_value(D, b, 4 * h + 2, v.z);
        prolong_value(D, b, 4 * h + 3, v.w);
        *reinterpret_cast<float4 *>(P.p + r.own) = v;
      }
      const int sc = 1 << lev;
      const float alpha = (float)(sc * sc) * D.ph.dx * D.ph.dx;
      q[k].v[0] = v.x;
      q[k].v[1] = v.y;
      q[k].v[2] = v.z;
      q[k].v[3] = v.w;
      r.ad[0] = __fmul_rn(alpha, dv.x);
      r.ad[1] = __fmul_rn(alpha, dv.y);
      r.ad[2] = __fmul_rn(alpha, dv.z);
      r.ad[3] = __fmul_rn(alpha, dv.w);
    }
    rest.put(k, r);
    rs_flags(q[k]);
  }
  for (int it = 0; it < sweeps; it++) {
    bar.sync();  // the prolongation, then the previous sweep, of every CTA
    const float *src = (it & 1) ? P.pt : P.p;
    float *dst = (it & 1) ? P.p : P.pt;
    Halo hv, next;  // two pairs' halos in flight: more do not fit the registers
    rs_load(src, q[0], rest.at(0), hv);
#pragma unroll
    for (int k = 0; k < K; k++) {
      if (k >= pairs) break;
      if (k + 1 < K && k + 1 < pairs) rs_load(src, q[k + 1 < K ? k + 1 : k], rest.at(k + 1 < K ? k + 1 : k), next);
      const uint4 r = rest.at(k);
      const float4 ad = rest.ad(k);
      float2 s[2];
      rs_fix<false>(q[k], r, h, hv);
      rs_sums(q[k], hv, h, s);
      s[0] = __fadd2_rn(s[0], make_float2(-ad.x, -ad.y));
      s[1] = __fadd2_rn(s[1], make_float2(-ad.z, -ad.w));
      div6_pairs(s);
      q[k].v[0] = s[0].x;
      q[k].v[1] = s[0].y;
      q[k].v[2] = s[1].x;
      q[k].v[3] = s[1].y;
      if (r.w != ~0u) *reinterpret_cast<float4 *>(dst + r.w) = make_float4(s[0].x, s[0].y, s[1].x, s[1].y);
      hv = next;
    }
  }
}

// One kernel for every number of pairs per warp: the host knows the budgets
// only, and a level far below its budget would pay for pairs that it has not
// (6891 of 17952 blocks: 2.56 us per sweep with four pairs, 2.42 with two).
__global__ void __launch_bounds__(RS_WARPS * 32, 1) k_resident_solve(const __grid_constant__ SolveBatch P, int sweeps) {
  __shared__ long long s_end[BMAX];
  if (threadIdx.x == 0) {
    long long acc = 0;
    for (int m = 0; m < P.n; m++) {
      if (P.lev[m] >= 0) {
        const long long load = __ldcg(P.d[m].load + P.lev[m]);
        if (load > P.cl_max[m]) acc += load;
      }
      s_end[m] = acc;
    }
  }
  __syncthreads();
  const long long total = s_end[P.n - 1];
  const long long one = (long long)gridDim.x * (blockDim.x >> 5) * 2;  // blocks at one pair per warp
  // the cluster solve took every level, or the general solve will: the same in every CTA
  if (total == 0 || total > 8 * one) return;
  GridBarrier bar(P.bar, P.err, gridDim.x);
  if (total <= one) rs_solve<1>(P, s_end, total, sweeps, bar);
  else if (total <= 2 * one) rs_solve<2>(P, s_end, total, sweeps, bar);
  else if (total <= 4 * one) rs_solve<4>(P, s_end, total, sweeps, bar);
  else rs_solve<8>(P, s_end, total, sweeps, bar);
}

// The sweeps of one level transposed (k_adj_jacobi for each, last to first).
// On the level itself the neighbour relation is symmetric, so the transpose is
// a sweep over the adjoint without a source, a gather in place of six atomics
// per cell. What a sweep hands to coarser cells and to the divergence is its
// own adjoint over six, to the same cells in every sweep of one parity: two
// sums per cell collect it, and it is added once, at the end. (A launch per
// sweep with seven atomics per cell took 9 us for 3456 blocks.)
template <int K>
__global__ void __launch_bounds__(RS_WARPS * 32, 1)
    k_resident_adjoint(const __grid_constant__ Dev D, int level, int sweeps, float *lp0, float *lp1, float *ld) {
  const int t = threadIdx.x, h = t & 15;
  const long long total = D.load[level];
  if (total == 0) return;
  GridBarrier bar(D.bar, D.err, gridDim.x);
  const int warps = blockDim.x >> 5;
  const float *first = ((sweeps - 1) & 1) ? lp0 : lp1;  // what the last sweep wrote
  const float *other = ((sweeps - 1) & 1) ? lp1 : lp0;  // what it read: the finer levels' share of it
  Quad q[K];
  Rests<K> rest;
  int pairs = 0;
  float even[K][4], odd[K][4];  // sums of the adjoints that even and odd sweeps pass on
#pragma unroll
  for (int k = 0; k < K; k++) {
    const long long pair = (long long)(k * warps + (t >> 5)) * gridDim.x + blockIdx.x;
    const long long g = 2 * pair + ((t >> 4) & 1);
    if (2 * pair < total) pairs = k + 1;
    QuadRest r = {0u, 0u, 0u, ~0u, {0.f, 0.f, 0.f, 0.f}};
    q[k] = {{0.f, 0.f, 0.f, 0.f}, 0u, 0u};
    float4 v = make_float4(0.f, 0.f, 0.f, 0.f), o = v;
    if (g < total) {
      const uint32_t b = (uint32_t)(D.g.off[level] + g);
      rs_faces(D, b, 0u, h, q[k], r);
      r.own = b * (uint32_t)BV + 4u * h;
      v = __ldcg(reinterpret_cast<const float4 *>(first + r.own));
      o = __ldcg(reinterpret_cast<const float4 *>(other + r.own));
    }
    q[k].v[0] = v.x;
    q[k].v[1] = v.y;
    q[k].v[2] = v.z;
    q[k].v[3] = v.w;
    r.ad[0] = o.x;
    r.ad[1] = o.y;
    r.ad[2] = o.z;
    r.ad[3] = o.w;
#pragma unroll
    for (int i = 0; i < 4; i++) even[k][i] = odd[k][i] = 0.f;
    rest.put(k, r);
    rs_flags(q[k]);
  }
  for (int it = sweeps - 1; it >= 0; it--) {
    const float *src = (it & 1) ? lp0 : lp1;
    float *dst = (it & 1) ? lp1 : lp0;
    // every CTA has its own cells' share of `other` before a sweep overwrites
    // them, and later the previous sweep's results
    bar.sync();
#pragma unroll
    for (int k = 0; k < K; k++) {
      if (k >= pairs) break;
      const uint4 r = rest.at(k);
      Halo hv;
      rs_load(src, q[k], r, hv);
      rs_fix<true>(q[k], r, h, hv);
      float2 s[2];
      rs_sums(q[k], hv, h, s);
      div6_pairs(s);
      const float n[4] = {s[0].x, s[0].y, s[1].x, s[1].y};
#pragma unroll
      for (int i = 0; i < 4; i++) {
        if (it & 1) odd[k][i] += q[k].v[i];
        else even[k][i] += q[k].v[i];
        q[k].v[i] = n[i];
      }
      if (it == sweeps - 1) {
        const float4 o = rest.ad(k);
        q[k].v[0] += o.x;
        q[k].v[1] += o.y;
        q[k].v[2] += o.z;
        q[k].v[3] += o.w;
      }
      if (r.w != ~0u)
        *reinterpret_cast<float4 *>(dst + r.w) = make_float4(q[k].v[0], q[k].v[1], q[k].v[2], q[k].v[3]);
    }
  }
  const int sc = 1 << level;
  const float alpha = (float)(sc * sc) * D.ph.dx * D.ph.dx;
#pragma unroll
  for (int k = 0; k < K; k++) {
    const uint4 r = rest.at(k);
    if (r.w == ~0u) continue;
    float *l = ld + r.w;
#pragma unroll
    for (int i = 0; i < 4; i++) {
      even[k][i] = div6(even[k][i]);
      odd[k][i] = div6(odd[k][i]);
      l[i] += -alpha * (even[k][i] + odd[k][i]);
    }
    auto add = [&](uint32_t cell, float e, float o) {
      if (e != 0.f) atomicAdd(lp0 + cell, e);
      if (o != 0.f) atomicAdd(lp1 + cell, o);
    };
    const int yr = (h & 4) ? 2 : 0, zr = (h & 2) ? 1 : 0;  // the row and the column at the quad's y and z face
    if (q[k].fl & RS_XC)
      add(q[k].x, even[k][0] + even[k][1] + even[k][2] + even[k][3], odd[k][0] + odd[k][1] + odd[k][2] + odd[k][3]);
    if (q[k].fl & RS_YC)
      add(r.x, yr ? even[k][2] + even[k][3] : even[k][0] + even[k][1],
          yr ? odd[k][2] + odd[k][3] : odd[k][0] + odd[k][1]);
    if (q[k].fl & RS_ZC)
      add(r.y, zr ? even[k][1] + even[k][3] : even[k][0] + even[k][2],
          zr ? odd[k][1] + odd[k][3] : odd[k][0] + odd[k][2]);
  }
}

template <int K, class Kernel, class... Args>
static bool resident_launch(Kernel kernel, long long blocks, int sms, cudaStream_t st, const Args &...args) {
  const size_t smem = Rests<K>::kBytes;
  int occ = 0;
  // a device that refuses the launch has the other solvers: no error is left
  // behind, but one of an earlier launch is not cleared with it
  if (cudaPeekAtLastError() != cudaSuccess) return false;
  auto ok = [](cudaError_t e) {
    if (e != cudaSuccess) cudaGetLastError();
    return e == cudaSuccess;
  };
  if (smem > 48 * 1024 &&
      !ok(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem)))
    return false;
  if (!ok(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&occ, kernel, RS_WARPS * 32, smem)) || occ < 1) return false;
  // as many warps as hold the blocks in one pair each, up to the CTA's limit
  const long long pairs = (blocks + 1) / 2, warps = (pairs + sms - 1) / sms;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3((unsigned)sms);
  cfg.blockDim = dim3(32u * (unsigned)(warps < 1 ? 1 : warps < RS_WARPS ? warps : RS_WARPS));
  cfg.dynamicSmemBytes = smem;
  cfg.stream = st;
  cudaLaunchAttribute attr;
  attr.id = cudaLaunchAttributeCooperative;
  attr.val.cooperative = 1;
  cfg.attrs = &attr;
  cfg.numAttrs = 1;
  return ok(cudaLaunchKernelEx(&cfg, kernel, args...));
}
// blocks that CTAs with k pairs per warp hold
static long long resident_blocks(int sms, int k) { return (long long)sms * RS_WARPS * k * 2; }
long long resident_solve_blocks(int sms) { return resident_blocks(sms, 8); }

bool launch_resident_solve(SolveBatch &P, int sweeps, int sms, cudaStream_t st) {
  long long blocks = 0, always = 0;  // budgets, and those of levels allocated in full
  for (int m = 0; m < P.n; m++) {
    const Geom &g = P.d[m].g;
    if (P.lev[m] < 0) continue;
    blocks += g.budget[P.lev[m]];
    if (g.budget[P.lev[m]] == g.full[P.lev[m]]) always += g.budget[P.lev[m]];
  }
  const long long most = resident_solve_blocks(sms);
  P.res_max = 0;
  if (sweeps <= 0 || always > most) return false;
  const bool done = resident_launch<8>(k_resident_solve, blocks, sms, st, P, sweeps);
  if (done && blocks > most) P.res_max = most;
  return done && blocks <= most;
}
bool launch_resident_adjoint(const Dev &D, int level, int sweeps, float *lp0, float *lp1, float *ld, int sms,
                             cudaStream_t st) {
  const long long blocks = D.g.budget[level];
  // the compat mode's boundary cells of the sparse levels break the symmetry
  if (sweeps <= 0 || blocks > resident_blocks(sms, 4) || (D.g.ref_compat && level < D.g.sparse)) return false;
  if (blocks <= resident_blocks(sms, 1))
    return resident_launch<1>(k_resident_adjoint<1>, blocks, sms, st, D, level, sweeps, lp0, lp1, ld);
  if (blocks <= resident_blocks(sms, 2))
    return resident_launch<2>(k_resident_adjoint<2>, blocks, sms, st, D, level, sweeps, lp0, lp1, ld);
  return resident_launch<4>(k_resident_adjoint<4>, blocks, sms, st, D, level, sweeps, lp0, lp1, ld);
}

}  // namespace dcg
