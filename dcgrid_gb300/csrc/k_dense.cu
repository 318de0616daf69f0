// k_dense.cu — Jacobi sweeps of a dense level (a whole box of cells in a linear
// layout), several sweeps per pass over memory.
//
// A level whose budget covers its block grid is allocated in full, in raster
// order, for as long as the simulation lives, so its cells form a dense box.
// One sweep of it per pass moves 12 bytes per cell and resolves every block's
// neighbours; here a pass reads the iterate and the right-hand side once,
// relaxes T times on the way through the chip and writes the result: 12 / T
// bytes per cell and sweep, neighbours from registers and shared memory.
// The uniform grid's mip levels are dense boxes as they are; an adaptive
// level is copied into a linear box first (with its prolongation) and the
// last pass writes the block layout again.
#include <algorithm>
#include <cmath>
#include <type_traits>

#include "dcg_kernels.h"

namespace dcg {

// ------------------------------------------------------------ the pass
// Box of A (contiguous) x B x M cells. A CTA takes a tile of nq quads (four
// cells along A) by nr row pairs (along B), one thread per quad and row pair,
// and marches along M. At step s a thread computes, for every sweep i = 1..T,
// its cells of plane s - i from planes s - i - 1, s - i and s - i + 1 of sweep
// i - 1, the last of which it has just made: sweep i runs one plane behind
// sweep i - 1, and one barrier per step serves all T sweeps. Neighbours along
// A inside the quad are registers, across quads shuffles, along B rows of the
// sweep's plane in shared memory (double buffered; the place that a step
// overwrites still holds the thread's own plane before, which is read back
// instead of kept in registers). Tiles overlap by T cells (whole quads along
// A), chunks of M by 2 T planes: those cells are computed twice, nothing is
// exchanged. The loads are asynchronous copies of the thread's own cells, one
// step ahead.
// Boundaries as in k_jacobi: a neighbour outside the box is the cell itself.
// The order of the sum is the layout's: an adaptive level marches along x (x,
// y, z neighbours = M, B, A), the uniform grid along z (A, B, M).
// What bounds it: the shared-memory pipe (about 46 wavefronts per warp, step
// and sweep of 256 cells; L1 80 % busy over a pass of 256^3 cells, issue 31 %)
// and the chain of T sweeps inside a step. T = 4 in 512 threads of 116 registers;
// measured slower: T = 3 in 640 threads (17.8 against 15.1 ms for 100 sweeps
// of 512^3; 14.7 now), T = 2 in 768 (17.9), the planes before kept in registers
// for every sweep (spills, 21 ms) or for three of four (15.6). Against one sweep
// per pass over memory (grid-wide cooperative solve, 3.3 TB/s): 48.7 ms.
template <int T> __host__ __device__ constexpr int dn_threads() { return T == 2 ? 640 : 512; }
template <int T> __host__ __device__ constexpr uint32_t dn_plane() { return dn_threads<T>() * 32; }  // bytes of a tile plane
template <int T> __host__ __device__ constexpr uint32_t dn_smem() { return (3 + 2 * (T - 1) + T + 1) * dn_plane<T>(); }

__device__ __forceinline__ void dn_copy16(uint32_t to, const float *from) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(to), "l"(from) : "memory");
}
__device__ __forceinline__ void dn_copy4(uint32_t to, const float *from) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"(to), "l"(from) : "memory");
}

// UNI: the uniform grid's order of the sum, right-hand side div (times
// alpha here); else the adaptive order, right-hand side -alpha div. EDGE: A
// not a multiple of 4, rows not 16-byte aligned, or B odd.
template <int T, bool UNI, bool EDGE>
__global__ void __launch_bounds__(dn_threads<T>(), 1) k_dense_pass(const __grid_constant__ DensePass P) {
  constexpr uint32_t PL = dn_plane<T>();
  extern __shared__ __align__(128) char sm[];
  int k = 0;
  while (k + 1 < P.n && (int)blockIdx.x >= P.end[k]) k++;
  const DenseLevel &V = P.l[k];
  const int item = (int)blockIdx.x - (k ? P.end[k - 1] : 0);
  constexpr int HP = T / 2;  // row pairs of overlap
  const int nq = V.nq, nr = V.nr, A = V.A, B = V.B, M = V.M;
  const int ia = item % V.ta, ib = (item / V.ta) % V.tb, ic = item / (V.ta * V.tb);
  const int c0 = ic * V.clen, c1 = min(M, c0 + V.clen);
  const int t = threadIdx.x, lane = t & 31;
  const int r = t / nq, q = t - r * nq;
  const bool live = r < nr;  // the other threads only keep the barriers
  const int a0 = 4 * (ia * (nq - 2) + q), b0 = 2 * (ib * (nr - 2 * HP) + r);
  const bool act = live && a0 < A && b0 < B, act1 = act && b0 + 1 < B;
  const bool out = act && (ia == 0 || q > 0) && (ia == V.ta - 1 || q < nq - 1) && (ib == 0 || r >= HP) &&
                   (ib == V.tb - 1 || r < nr - HP);
  // shared memory: ring of the input's planes (3), two planes per inner sweep,
  // ring of the right-hand side's planes (T + 1); me: the thread's first row
  constexpr uint32_t LEV = 3 * PL, RHS = LEV + 2 * (T - 1) * PL;
  const uint32_t row = 16u * nq, me = live ? 2 * r * row + 16u * q : 0u, me1 = me + row;
  char *const s0 = sm + me, *const s1 = sm + me1;
  const char *const sd = sm + ((!live || r == 0 || b0 == 0) ? me : me - row);              // the row below the pair
  const char *const su = sm + ((!live || r == nr - 1 || b0 + 2 >= B) ? me1 : me1 + row);  // and the one above
  // the cells left and right of the quad: the next lane's, except at the ends
  // of a warp and of the box (the cell itself)
  const bool first = a0 == 0, last = a0 + 4 >= A;
  const bool fixl = live && (first || (lane == 0 && q > 0)), fixr = live && (last || (lane == 31 && q < nq - 1));
  const int dl = first ? 0 : -4, dr = last ? 12 : 16;
  const int tail = A - 1 - a0;             // EDGE: place of the row's last cell, if in the quad
  const bool last0 = EDGE && b0 + 1 == B;  // EDGE: the pair's first row is the last one
  auto ld = [](const char *p) { return *reinterpret_cast<const float4 *>(p); };
  auto ld1 = [](const char *p) { return *reinterpret_cast<const float *>(p); };
  for (uint32_t o = 16u * t; o < dn_smem<T>(); o += 16u * dn_threads<T>())
    *reinterpret_cast<float4 *>(sm + o) = make_float4(0.f, 0.f, 0.f, 0.f);
  const size_t plane = (size_t)A * B;
  auto copy = [&](const char *to, const float *g) {  // the thread's rows of a plane, to: its first row's place
    const uint32_t o = (uint32_t)__cvta_generic_to_shared(to);
    if (!EDGE) {
      if (act) {
        dn_copy16(o, g);
        if (act1) dn_copy16(o + row, g + A);
      }
    } else {
#pragma unroll
      for (int e = 0; e < 4; e++)
        if (act && a0 + e < A) {
          dn_copy4(o + 4u * e, g + e);
          if (act1) dn_copy4(o + row + 4u * e, g + A + e);
        }
    }
  };
  const int mlo = max(0, c0 - T), mload = min(M, c1 + T), shi = c1 - 1 + T;
  const size_t at0 = (size_t)mlo * plane + (size_t)b0 * A + a0;
  const float *gin = V.in + at0, *grh = V.rhs + at0;  // planes s + 1 (after the first copy) and s
  __syncthreads();
  // Places of the tile outside the box are never copied to, and nothing inside
  // reads them: ones, which the sweeps keep near one. Zeros sent their warps
  // through the division's component-wise test in every sweep (us per sweep of
  // 39936 blocks, whose tiles overhang: 11.9, with ones 9.4).
  if (live)
    for (int k = 0; k < 24; k++) {
      const int j = k & 1, e = (k >> 1) & 3;
      if (a0 + e >= A || b0 + j >= B) *reinterpret_cast<float *>(s0 + (k >> 3) * PL + j * row + 4 * e) = 1.f;
    }
  __syncthreads();
  if (!V.zero) copy(s0, gin);
  gin += plane;
  asm volatile("cp.async.commit_group;" ::: "memory");
  // the thread's rows: sweep i's newest plane, and for the first KW sweeps the
  // plane before it (the others read theirs back)
  constexpr int KW = T == 4 ? 1 : 2;
  float4 X[T][2], W[KW][2];
#pragma unroll
  for (int j = 0; j < 2; j++) {
#pragma unroll
    for (int i = 0; i < T; i++) X[i][j] = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
    for (int i = 0; i < KW; i++) W[i][j] = make_float4(0.f, 0.f, 0.f, 0.f);
  }
  uint32_t o0 = 0, oprev = 2 * PL, orh = 0;  // ring places of planes s, s - 1; right-hand side of plane s
  auto step = [&](auto par_, auto edge_, int s) {
    constexpr int PAR = decltype(par_)::value;
    constexpr bool EM = decltype(edge_)::value;
    const uint32_t third = 3 * PL - o0 - oprev;  // plane s + 1 goes where plane s - 2 was
    if (s + 1 < mload && !V.zero) copy(s0 + third, gin);
    if (s < mload) copy(s0 + RHS + orh, grh);
    gin += plane;
    grh += plane;
    asm volatile("cp.async.commit_group;" ::: "memory");
    asm volatile("cp.async.wait_group 1;" ::: "memory");  // plane s and right-hand side s - 1 of this thread are here
    float4 n0 = ld(s0 + o0), n1 = ld(s1 + o0);
    float4 f0, f1, g0, g1;  // sweeps T and T - 1: planes s - T and s - T + 1
#pragma unroll
    for (int i = 1; i <= T; i++) {
      const int n = s - i;
      const float4 c0v = X[i - 1][0], c1v = X[i - 1][1];
      float4 r0 = make_float4(0.f, 0.f, 0.f, 0.f), r1 = r0;
      if (!EM || (n >= mlo && n < M)) {
        const uint32_t buf = i == 1 ? oprev : LEV + (2 * (i - 2) + (PAR ^ 1)) * PL;
        const float4 dv = ld(sd + buf), uv = ld(su + buf);
        const uint32_t od = RHS + (orh >= i * PL ? orh - i * PL : orh + (T + 1 - i) * PL);
        const float4 h0 = ld(s0 + od), h1 = ld(s1 + od);
        float l0 = __shfl_up_sync(0xffffffffu, c0v.w, 1), l1 = __shfl_up_sync(0xffffffffu, c1v.w, 1);
        float e0 = __shfl_down_sync(0xffffffffu, c0v.x, 1), e1 = __shfl_down_sync(0xffffffffu, c1v.x, 1);
        if (fixl) l0 = ld1(s0 + buf + dl), l1 = ld1(s1 + buf + dl);
        if (fixr) e0 = ld1(s0 + buf + dr), e1 = ld1(s1 + buf + dr);
        // planes n - 1 (of an inner sweep: where this step puts plane n + 1) and n + 1
        float4 m0, m1, q0 = n0, q1 = n1;
        if (i <= KW) m0 = W[i <= KW ? i - 1 : 0][0], m1 = W[i <= KW ? i - 1 : 0][1];
        else m0 = ld(s0 + LEV + (2 * (i - 2) + PAR) * PL), m1 = ld(s1 + LEV + (2 * (i - 2) + PAR) * PL);
        if (EM) {
          if (n == 0) m0 = c0v, m1 = c1v;
          if (n == M - 1) q0 = c0v, q1 = c1v;
        }
        auto relax = [&](float4 c, float4 m, float4 qn, float4 d, float4 u, float l, float e, float4 h) -> float4 {
          float4 la = make_float4(l, c.x, c.y, c.z), ra = make_float4(c.y, c.z, c.w, e);
          if (EDGE) {  // the row ends inside the quad
            if (tail == 0) ra.x = c.x;
            if (tail == 1) ra.y = c.y;
            if (tail == 2) ra.z = c.z;
          }
          float2 sx, sy;
          if (UNI) {
            sx = make_float2(la.x + ra.x, la.y + ra.y);
            sy = make_float2(la.z + ra.z, la.w + ra.w);
          } else {
            sx = __fadd2_rn(make_float2(m.x, m.y), make_float2(qn.x, qn.y));
            sy = __fadd2_rn(make_float2(m.z, m.w), make_float2(qn.z, qn.w));
          }
          sx = __fadd2_rn(__fadd2_rn(sx, make_float2(d.x, d.y)), make_float2(u.x, u.y));
          sy = __fadd2_rn(__fadd2_rn(sy, make_float2(d.z, d.w)), make_float2(u.z, u.w));
          if (UNI) {
            sx = __fadd2_rn(__fadd2_rn(sx, make_float2(m.x, m.y)), make_float2(qn.x, qn.y));
            sy = __fadd2_rn(__fadd2_rn(sy, make_float2(m.z, m.w)), make_float2(qn.z, qn.w));
            // scalar products: a packed product and the packed sum behind it come
            // out fused (measured), although both are asked for rounded
            sx = __fadd2_rn(sx, make_float2(__fmul_rn(V.nalpha, h.x), __fmul_rn(V.nalpha, h.y)));
            sy = __fadd2_rn(sy, make_float2(__fmul_rn(V.nalpha, h.z), __fmul_rn(V.nalpha, h.w)));
          } else {
            sx.x = sx.x + la.x + ra.x;
            sx.y = sx.y + la.y + ra.y;
            sy.x = sy.x + la.z + ra.z;
            sy.y = sy.y + la.w + ra.w;
            sx = __fadd2_rn(sx, make_float2(h.x, h.y));
            sy = __fadd2_rn(sy, make_float2(h.z, h.w));
          }
          return make_float4(sx.x, sx.y, sy.x, sy.y);
        };
        float4 up0 = c1v;
        if (EDGE && last0) up0 = c0v;
        r0 = relax(c0v, m0, q0, dv, up0, l0, e0, h0);
        r1 = relax(c1v, m1, q1, c0v, uv, l1, e1, h1);
        float2 x[4] = {make_float2(r0.x, r0.y), make_float2(r0.z, r0.w), make_float2(r1.x, r1.y), make_float2(r1.z, r1.w)};
        div6_pairs(x);
        r0 = make_float4(x[0].x, x[0].y, x[1].x, x[1].y);
        r1 = make_float4(x[2].x, x[2].y, x[3].x, x[3].y);
      }
      if (i > 1 && live) {  // sweep i - 1's plane s - i + 1 for the rows beside (the input's planes are there already)
        *reinterpret_cast<float4 *>(s0 + LEV + (2 * (i - 2) + PAR) * PL) = n0;
        *reinterpret_cast<float4 *>(s1 + LEV + (2 * (i - 2) + PAR) * PL) = n1;
      }
      if (i <= KW) W[i <= KW ? i - 1 : 0][0] = c0v, W[i <= KW ? i - 1 : 0][1] = c1v;
      X[i - 1][0] = n0;
      X[i - 1][1] = n1;
      if (i == T) g0 = n0, g1 = n1, f0 = r0, f1 = r1;
      n0 = r0;
      n1 = r1;
    }
    auto store = [&](float *o, int m, float4 v0, float4 v1) {
      if (V.blocks) {  // block layout: cells z and z + 1 of a pair, 8 cells further the next pair
#pragma unroll
        for (int j = 0; j < 2; j++) {
          const int y = b0 + j;
          const size_t b = ((size_t)(m >> 2) * V.rb + (y >> 2)) * V.ra + (a0 >> 2);
          float2 *p = reinterpret_cast<float2 *>(o + b * BV + local_of(m & 3, y & 3, 0));
          const float4 v = j ? v1 : v0;
          p[0] = make_float2(v.x, v.y);
          p[4] = make_float2(v.z, v.w);
        }
      } else {
        float *p = o + (size_t)m * plane + (size_t)b0 * A + a0;
        if (!EDGE) {
          *reinterpret_cast<float4 *>(p) = v0;
          *reinterpret_cast<float4 *>(p + A) = v1;
        } else {
          const float w0[4] = {v0.x, v0.y, v0.z, v0.w}, w1[4] = {v1.x, v1.y, v1.z, v1.w};
#pragma unroll
          for (int e = 0; e < 4; e++)
            if (a0 + e < A) {
              p[e] = w0[e];
              if (act1) p[A + e] = w1[e];
            }
        }
      }
    };
    if (out) {
      if (s - T >= c0) store(V.out, s - T, f0, f1);
      if (V.out2 && s - T + 1 >= c0 && s - T + 1 < c1) store(V.out2, s - T + 1, g0, g1);
    }
    __syncthreads();
    oprev = o0;
    o0 = third;
    orh = orh == T * PL ? 0u : orh + PL;
  };
  const std::integral_constant<int, 0> even{};
  const std::integral_constant<int, 1> odd{};
  int s = mlo;
#pragma unroll 1
  for (; s < shi; s += 2) {
    if (s > mlo + T && s + 1 < M) {
      step(even, std::false_type{}, s);
      step(odd, std::false_type{}, s + 1);
    } else {
      step(even, std::true_type{}, s);
      step(odd, std::true_type{}, s + 1);
    }
  }
  if (s == shi) step(even, std::true_type{}, s);
}

// ------------------------------------------------------------ adaptive levels
// Linear copies of a dense adaptive level, index (x Y + y) Z + z: the iterate
// (the prolongation of the parent level, dense too, or the present p) and
// -alpha div. One thread per subblock: its eight cells share one coarse cell
// and its 26 neighbours. Out-of-domain coarse neighbours as apron_cell maps
// them: the cell clamped to the parent's own block on every axis.
__global__ void __launch_bounds__(256) k_dense_load(const __grid_constant__ DenseCopy P) {
  int k = 0;
  while (k + 1 < P.n && (int)blockIdx.x >= P.end[k]) k++;
  const DenseCopyLevel &V = P.l[k];
  const int X2 = V.X / 2, Y2 = V.Y / 2, Z2 = V.Z / 2;
  const long long i = (long long)((int)blockIdx.x - (k ? P.end[k - 1] : 0)) * 256 + threadIdx.x;
  if (i >= (long long)X2 * Y2 * Z2) return;
  const int z2 = (int)(i % Z2), y2 = (int)((i / Z2) % Y2), x2 = (int)(i / ((long long)Z2 * Y2));
  const size_t b = ((size_t)(x2 >> 1) * (V.Y / 4) + (y2 >> 1)) * (V.Z / 4) + (z2 >> 1);
  const size_t cell = b * BV + 8 * (((x2 & 1) << 2) | ((y2 & 1) << 1) | (z2 & 1));
  float v[8];
  if (V.coarse) {
    const int ry = Y2 / 4, rz = Z2 / 4;
    auto at = [&](int dx, int dy, int dz) -> float {
      int x = x2 + dx, y = y2 + dy, z = z2 + dz;
      if (x < 0 || y < 0 || z < 0 || x >= X2 || y >= Y2 || z >= Z2) {
        x = clampi(x, x2 & ~3, x2 | 3);
        y = clampi(y, y2 & ~3, y2 | 3);
        z = clampi(z, z2 & ~3, z2 | 3);
      }
      return V.coarse[(((size_t)(x >> 2) * ry + (y >> 2)) * rz + (z >> 2)) * BV + local_of(x & 3, y & 3, z & 3)];
    };
    float c[27];
#pragma unroll
    for (int j = 0; j < 27; j++) c[j] = at(j / 9 - 1, (j / 3) % 3 - 1, j % 3 - 1);
#pragma unroll
    for (int j = 0; j < 8; j++) {
      const int dx = (j & 4) ? 9 : -9, dy = (j & 2) ? 3 : -3, dz = (j & 1) ? 1 : -1;
      v[j] = (27.f * c[13] + 9.f * (c[13 + dz] + c[13 + dy] + c[13 + dx]) +
              3.f * (c[13 + dy + dz] + c[13 + dx + dz] + c[13 + dx + dy]) + c[13 + dx + dy + dz]) / 64.f;
    }
  } else {
    const float4 a = *reinterpret_cast<const float4 *>(V.p + cell), c = *reinterpret_cast<const float4 *>(V.p + cell + 4);
    v[0] = a.x; v[1] = a.y; v[2] = a.z; v[3] = a.w; v[4] = c.x; v[5] = c.y; v[6] = c.z; v[7] = c.w;
  }
  const float4 a = *reinterpret_cast<const float4 *>(V.div + cell), c = *reinterpret_cast<const float4 *>(V.div + cell + 4);
  const float d[8] = {a.x, a.y, a.z, a.w, c.x, c.y, c.z, c.w};
#pragma unroll
  for (int j = 0; j < 4; j++) {
    const size_t o = ((size_t)(2 * x2 + (j >> 1)) * V.Y + 2 * y2 + (j & 1)) * V.Z + 2 * z2;
    *reinterpret_cast<float2 *>(V.lin + o) = make_float2(v[2 * j], v[2 * j + 1]);
    *reinterpret_cast<float2 *>(V.rhs + o) = make_float2(-(V.alpha * d[2 * j]), -(V.alpha * d[2 * j + 1]));
  }
}

// ------------------------------------------------------------ host
// Tiles and chunks of a pass over the levels of one launch: the tile shapes
// and the chunk length that give the shortest schedule of CTAs, one per SM,
// when a step costs a fixed part and a part per warp. Smaller tiles and
// shorter chunks repeat more cells but occupy more SMs.
static double dn_step_cost(int threads) { return 0.3 + 0.7 * (double)((threads + 31) / 32 * 32) / 512; }
static void dn_tile(DenseLevel &l, int hp, int threads) {
  auto tiles = [](int n, int w, int halo) { return n <= w ? 1 : (n - w + w - 2 * halo - 1) / (w - 2 * halo) + 1; };
  const int a4 = (l.A + 3) / 4, b2 = (l.B + 1) / 2;
  double best = 1e300;
  for (int ta = 1; ta <= a4; ta++) {
    const int nq = ta == 1 ? a4 : (a4 - 2 + ta - 1) / ta + 2;
    if (ta > 1 && nq < 4) break;
    const int most = std::min(b2, threads / nq);
    if (most < b2 && most < 2 * hp + 1) continue;
    const int tb = tiles(b2, most, hp), nr = tb == 1 ? b2 : (b2 - 2 * hp + tb - 1) / tb + 2 * hp;
    const int tq = tiles(a4, nq, 1);
    const double w = (double)tq * tb * dn_step_cost(nq * nr);
    if (w < best) {
      best = w;
      l.nq = nq;
      l.nr = nr;
      l.ta = tq;
      l.tb = tb;
    }
  }
}
static void dn_plan(DensePass &P, int T, int sms) {
  int most = 0;
  for (int i = 0; i < P.n; i++) most = std::max(most, P.l[i].M);
  double best = 1e300;
  DenseLevel pick[BMAX];
  for (int threads = T == 2 ? dn_threads<2>() : dn_threads<4>(); threads >= 64; threads /= 2) {
    DenseLevel l[BMAX];
    for (int i = 0; i < P.n; i++) {
      l[i] = P.l[i];
      dn_tile(l[i], T / 2, threads);
    }
    if (std::any_of(l, l + P.n, [](const DenseLevel &v) { return v.nq == 0; })) break;
    for (int len = 2;; len += std::max(1, len / 8)) {
      const int clen = std::min(len, most);
      double work = 0, longest = 0;
      for (int i = 0; i < P.n; i++) {
        const double cost = (std::min(l[i].M, clen) + 2.0 * T) * dn_step_cost(l[i].nq * l[i].nr);
        work += cost * l[i].ta * l[i].tb * ((l[i].M + clen - 1) / clen);
        longest = std::max(longest, cost);
        l[i].clen = clen;
      }
      const double total = longest * std::ceil(work / longest / sms);  // waves of about equal items
      if (total < best) {
        best = total;
        std::copy(l, l + P.n, pick);
      }
      if (clen == most) break;
    }
  }
  int e = 0;
  for (int i = 0; i < P.n; i++) {
    P.l[i] = pick[i];
    e += P.l[i].ta * P.l[i].tb * ((P.l[i].M + P.l[i].clen - 1) / P.l[i].clen);
    P.end[i] = e;
  }
}

// The opt-in to this much shared memory belongs to the current device, so every
// launch asks for it; a refusal is left to the caller's launch check.
template <int T, bool UNI, bool EDGE> static void dn_launch(const DensePass &P, cudaStream_t st) {
  if (cudaFuncSetAttribute(k_dense_pass<T, UNI, EDGE>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)dn_smem<T>()) ==
      cudaSuccess)
    k_dense_pass<T, UNI, EDGE><<<(unsigned)P.end[P.n - 1], dn_threads<T>(), dn_smem<T>(), st>>>(P);
}

// sweeps (even, > 0) of the levels: src -> dst with dst2 = the iterate before
// the last, over the scratch boxes x0 (which may hold src) and x1
void launch_dense_sweeps(const DenseSweep *v, int n, int sweeps, bool uniform, int sms, cudaStream_t st) {
  DensePass P4{}, P2{};
  bool edge = false;
  for (int i = 0; i < n; i++) {
    DenseLevel l{};
    l.A = v[i].A; l.B = v[i].B; l.M = v[i].M;
    l.rhs = v[i].rhs;
    l.nalpha = v[i].nalpha;
    l.ra = v[i].A / 4; l.rb = v[i].B / 4;
    P4.l[i] = P2.l[i] = l;
    edge |= v[i].A % 4 != 0 || v[i].B % 2 != 0;
    for (const void *p : {(const void *)v[i].src, (const void *)v[i].rhs, (const void *)v[i].dst, (const void *)v[i].dst2})
      edge |= !v[i].blocks && ((uintptr_t)p & 15) != 0;
  }
  P4.n = P2.n = n;
  const int n4 = sweeps / 4, total = n4 + (sweeps % 4) / 2;
  if (n4) dn_plan(P4, 4, sms);
  if (total > n4) dn_plan(P2, 2, sms);
  for (int pass = 0; pass < total; pass++) {
    DensePass &P = pass < n4 ? P4 : P2;
    const bool lastp = pass == total - 1;
    for (int i = 0; i < n; i++) {
      DenseLevel &l = P.l[i];
      l.in = pass == 0 ? v[i].src : (pass & 1) ? v[i].x1 : v[i].x0;
      l.zero = pass == 0 && v[i].zero;
      l.out = lastp ? v[i].dst : (pass & 1) ? v[i].x0 : v[i].x1;
      l.out2 = lastp ? v[i].dst2 : nullptr;
      l.blocks = lastp && v[i].blocks;
    }
    if (pass < n4) {
      if (uniform) edge ? dn_launch<4, true, true>(P, st) : dn_launch<4, true, false>(P, st);
      else dn_launch<4, false, false>(P, st);
    } else {
      if (uniform) edge ? dn_launch<2, true, true>(P, st) : dn_launch<2, true, false>(P, st);
      else dn_launch<2, false, false>(P, st);
    }
  }
}

// one dense level per member: linear copies, sweeps, results in the block layout
void launch_dense_solve(const Dev *d, const int *lev, int n, int prolong, int sweeps, int sms, cudaStream_t st) {
  for (int g = 0; g < n; g += BMAX) {
    DenseCopy C{};
    DenseSweep v[BMAX];
    C.n = std::min(BMAX, n - g);
    long long e = 0;
    for (int i = 0; i < C.n; i++) {
      const Dev &D = d[g + i];
      const int l = lev[g + i];
      const size_t o = (size_t)D.g.off[l] * BV;
      DenseCopyLevel &c = C.l[i];
      c.X = 4 * D.g.rx[l]; c.Y = 4 * D.g.ry[l]; c.Z = 4 * D.g.rz[l];
      c.p = D.p + o;
      c.coarse = prolong && l < D.g.levels - 1 ? D.p + (size_t)D.g.off[l + 1] * BV : nullptr;
      c.div = D.div + o;
      c.lin = D.tv[0] + o;
      c.rhs = D.tv[2] + o;
      const int sc = 1 << l;
      c.alpha = (float)(sc * sc) * D.ph.dx * D.ph.dx;
      e += ((long long)(c.X / 2) * (c.Y / 2) * (c.Z / 2) + 255) / 256;
      C.end[i] = (int)e;
      v[i] = DenseSweep{c.Z, c.Y, c.X, c.lin, c.rhs, D.tv[0] + o, D.tv[1] + o, D.p + o, D.pt + o, 0.f, false, true};
    }
    k_dense_load<<<(unsigned)e, 256, 0, st>>>(C);
    launch_dense_sweeps(v, C.n, sweeps, false, sms, st);
  }
}

}  // namespace dcg
