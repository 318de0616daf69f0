// k_uniform.cu — the uniform-grid step (the reference's FluidSimulationUniform,
// src/uniformgrid/*.cu): dense x-fastest fields with a mip-mapped
// pressure / divergence / fluidity pyramid. One thread per cell; a CTA covers
// 2^sx cells along x by 256 / 2^sx along y of one z plane, the shape that
// wastes least of a row (u_cell, u_launch). The CTA's place costs two
// divisions that are uniform in the CTA; with one 64-bit division per thread
// and coordinate, index arithmetic was most of the light kernels' time (a
// Jacobi sweep of 64^3 cells 7.7 us, now 5.6, of 128^3 18 and 8.2).
#include "dcg_kernels.h"

namespace dcg {

__device__ inline size_t uidx(const UDev &U, int x, int y, int z) {
  return ((size_t)z * U.gy + y) * U.gx + x;
}
// mipmapIdx (src/utils/grid_math.cuh:41-52)
__device__ inline size_t umip(const UDev &U, int x, int y, int z, int level) {
  const int s = 1 << level;
  return (size_t)U.mip_off[level] + ((size_t)z * (U.gy / s) + y) * (U.gx / s) + x;
}

// the thread's cell of a w x h x d box, its linear index in i; false outside
__device__ __forceinline__ bool u_cell(int w, int h, int sx, int &x, int &y, int &z, size_t &i) {
  const unsigned tx = (unsigned)(w + (1 << sx) - 1) >> sx, ty = (unsigned)(h + (256 >> sx) - 1) >> (8 - sx);
  const unsigned r = blockIdx.x / tx, bx = blockIdx.x - r * tx;
  z = (int)(r / ty);
  const unsigned by = r - (unsigned)z * ty;
  x = (int)((bx << sx) + (threadIdx.x & ((1u << sx) - 1u)));
  y = (int)((by << (8 - sx)) + (threadIdx.x >> sx));
  i = ((size_t)z * h + y) * w + x;
  return x < w && y < h;
}

// k_uniform_set_solidity_ratio (uniformgrid_structure.cu:23-31)
__global__ void __launch_bounds__(256) k_u_fluidity(UDev U, int sx, int level) {
  const int s = 1 << level;
  int x, y, z;
  size_t i;
  if (u_cell(U.gx / s, U.gy / s, sx, x, y, z, i)) U.w[(size_t)U.mip_off[level] + i] = fluidity(U.g, U.ph, x, y, z, s);
}

__global__ void __launch_bounds__(256) k_u_sources(UDev U, int sx) {
  int x, y, z;
  size_t i;
  if (!u_cell(U.gx, U.gy, sx, x, y, z, i)) return;
  if (in_source(U.ph, x, y, z, 1))
    for (int k = 0; k < U.nq; k++) U.q[k][i] = src_value_at(U.ph, k, x, y, z, 0);
}

// Back-traced samples (INIT_SAMPLE, uniformgrid_fluid.cu:7-48) of NF fields:
// trilinear weights times fluidity, renormalised, corners summed in order
// (corner bits x, y, z); zero where the weights vanish. Boxes that touch the
// boundary, where corners are clamped and bc(field, value, x, y, z) applies,
// go out of line; inside, a corner pair along x is two neighbouring floats of
// one of four rows, and an address costs one addition per row and field (with
// clamped 64-bit indices per corner the two advections took 2.5 times the
// instructions).
template <int NF> struct UVals {
  float v[NF];
};
template <int NF, class BC>
__device__ __noinline__ UVals<NF> u_interp_edge(const UDev &U, const float *const (&f)[NF], float x, float y, float z, BC bc) {
  const float xf = floorf(x), yf = floorf(y), zf = floorf(z);
  const int x0 = (int)xf, y0 = (int)yf, z0 = (int)zf, x1 = x0 + 1, y1 = y0 + 1, z1 = z0 + 1;
  const float dx = x - xf, dy = y - yf, dz = z - zf;
  const float Dx = 1.f - dx, Dy = 1.f - dy, Dz = 1.f - dz;
  const int xs[2] = {clampi(x0, 0, U.gx - 1), clampi(x1, 0, U.gx - 1)},
            ys[2] = {clampi(y0, 0, U.gy - 1), clampi(y1, 0, U.gy - 1)},
            zs[2] = {clampi(z0, 0, U.gz - 1), clampi(z1, 0, U.gz - 1)};
  size_t row[4];  // (y, z) bits
#pragma unroll
  for (int c = 0; c < 4; c++) row[c] = uidx(U, 0, ys[c >> 1], zs[c & 1]);
  float wt[8], wAcc = 0.f;
#pragma unroll
  for (int c = 0; c < 8; c++) {
    wt[c] = U.w[row[c & 3] + xs[c >> 2]] * ((c & 4) ? dx : Dx) * ((c & 2) ? dy : Dy) * ((c & 1) ? dz : Dz);
    wAcc = c == 0 ? wt[0] : wAcc + wt[c];
  }
  const float wInv = 1.f / wAcc;
  UVals<NF> o;
#pragma unroll
  for (int k = 0; k < NF; k++) o.v[k] = 0.f;
  if (wAcc < 1e-6f) return o;
#pragma unroll
  for (int c = 0; c < 8; c++) {
    float v[NF];
#pragma unroll
    for (int k = 0; k < NF; k++) v[k] = f[k][row[c & 3] + xs[c >> 2]];
    bc(v, (c & 4) ? x1 : x0, (c & 2) ? y1 : y0, (c & 1) ? z1 : z0);
    const float w = wt[c] * wInv;
#pragma unroll
    for (int k = 0; k < NF; k++) o.v[k] = c == 0 ? v[k] * w : o.v[k] + v[k] * w;
  }
  return o;
}
template <int NF, class BC>
__device__ __forceinline__ void u_interp(const UDev &U, const float *const (&f)[NF], float px, float py, float pz,
                                         float (&o)[NF], BC bc) {
  const float x = px - 0.5f, y = py - 0.5f, z = pz - 0.5f;
  const float xf = floorf(x), yf = floorf(y), zf = floorf(z);
  const int x0 = (int)xf, y0 = (int)yf, z0 = (int)zf;
  if (!(x0 >= 0 && y0 >= 0 && z0 >= 0 && x0 < U.gx - 1 && y0 < U.gy - 1 && z0 < U.gz - 1)) {
    const UVals<NF> e = u_interp_edge<NF>(U, f, x, y, z, bc);
#pragma unroll
    for (int k = 0; k < NF; k++) o[k] = e.v[k];
    return;
  }
  const float dx = x - xf, dy = y - yf, dz = z - zf;
  const float Dx = 1.f - dx, Dy = 1.f - dy, Dz = 1.f - dz;
  size_t row[4];  // (y, z) bits
  row[0] = uidx(U, x0, y0, z0);
  row[2] = row[0] + U.gx;
  row[1] = row[0] + (size_t)U.gx * U.gy;
  row[3] = row[1] + U.gx;
  float wt[8];
#pragma unroll
  for (int c = 0; c < 8; c++)
    wt[c] = U.w[row[c & 3] + (c >> 2)] * ((c & 4) ? dx : Dx) * ((c & 2) ? dy : Dy) * ((c & 1) ? dz : Dz);
  const float wAcc = wt[0] + wt[1] + wt[2] + wt[3] + wt[4] + wt[5] + wt[6] + wt[7];
  const float wInv = 1.f / wAcc;
#pragma unroll
  for (int c = 0; c < 8; c++) wt[c] = wt[c] * wInv;
  const bool none = wAcc < 1e-6f;
#pragma unroll
  for (int k = 0; k < NF; k++) {
    float a = 0.f;
#pragma unroll
    for (int c = 0; c < 8; c++) {
      const float v = f[k][row[c & 3] + (c >> 2)];
      a = c == 0 ? v * wt[0] : a + v * wt[c];
    }
    o[k] = none ? 0.f : a;
  }
}

// k_uniform_advect_velocity (uniformgrid_fluid.cu:88-96) + buoyancy extension
__global__ void __launch_bounds__(256) k_u_advect_velocity(const __grid_constant__ UDev U, int sx) {
  int x, y, z;
  size_t i;
  if (!u_cell(U.gx, U.gy, sx, x, y, z, i)) return;
  const float px = ((float)x + 0.5f) - U.v[0][i] * U.ph.dt * U.ph.rdx;
  const float py = ((float)y + 0.5f) - U.v[1][i] * U.ph.dt * U.ph.rdx;
  const float pz = ((float)z + 0.5f) - U.v[2][i] * U.ph.dt * U.ph.rdx;
  const float *const f[3] = {U.v[0], U.v[1], U.v[2]};
  float o[3];
  u_interp(U, f, px, py, pz, o, [&U](float *v, int cx, int cy, int cz) {
    vel_bc(U.g, U.ph, v[0], v[1], v[2], cx, cy, cz, 1);
  });
  if (U.ph.buoy_a != 0.f || U.ph.buoy_b != 0.f) {
    float b = -U.ph.buoy_a * U.q[0][i];
    if (U.nq > 1) b = b + U.ph.buoy_b * (U.q[1][i] - U.ph.t_amb);
    o[1] = o[1] + U.ph.dt * b;
  }
  U.tv[0][i] = o[0];
  U.tv[1][i] = o[1];
  U.tv[2][i] = o[2];
}

// indices of a cell's six neighbours, the cell itself outside the domain
struct UNb {
  size_t l, r, d, u, b, f;
};
__device__ __forceinline__ UNb u_neighbours(size_t i, int x, int y, int z, int w, int h, int d) {
  const size_t wh = (size_t)w * h;
  return {x > 0 ? i - 1 : i,         x < w - 1 ? i + 1 : i,  y > 0 ? i - w : i, y < h - 1 ? i + w : i,
          z > 0 ? i - wh : i, z < d - 1 ? i + wh : i};
}
// k_uniform_apply_pressure (uniformgrid_fluid.cu:239-260) of one cell
__device__ __forceinline__ void u_project(const UDev &U, size_t i, int x, int y, int z, float &v0, float &v1, float &v2) {
  const UNb n = u_neighbours(i, x, y, z, U.gx, U.gy, U.gz);
  const float alpha = 0.5f * U.ph.rdx;
  const float *P = U.p, *W = U.w;
  const float pc = P[i];
  v0 = U.v[0][i] - alpha * (W[n.r] * (P[n.r] - pc) + W[n.l] * (pc - P[n.l]));
  v1 = U.v[1][i] - alpha * (W[n.u] * (P[n.u] - pc) + W[n.d] * (pc - P[n.d]));
  v2 = U.v[2][i] - alpha * (W[n.f] * (P[n.f] - pc) + W[n.b] * (pc - P[n.b]));
}

// k_uniform_advect_density (uniformgrid_fluid.cu:98-105) + sources. APPLY: the
// pressure application of the same step first, in the same pass: the scalar
// advection reads no velocity but its own cell's, so the results are those of
// the two one after the other.
__device__ __noinline__ void u_source(const UDev &U, size_t i, int x, int y, int z) {
  for (int k = 0; k < U.nq; k++) U.tq[k][i] = src_value_at(U.ph, k, x, y, z, 0);
}
template <bool APPLY, int NQ> __global__ void __launch_bounds__(256) k_u_advect_scalars(const __grid_constant__ UDev U, int sx) {
  int x, y, z;
  size_t i;
  if (!u_cell(U.gx, U.gy, sx, x, y, z, i)) return;
  float v0, v1, v2;
  if (APPLY) {
    u_project(U, i, x, y, z, v0, v1, v2);
    U.v[0][i] = v0;
    U.v[1][i] = v1;
    U.v[2][i] = v2;
  } else {
    v0 = U.v[0][i];
    v1 = U.v[1][i];
    v2 = U.v[2][i];
  }
  if (in_source(U.ph, x, y, z, 1)) {
    u_source(U, i, x, y, z);
    return;
  }
  const float px = ((float)x + 0.5f) - v0 * U.ph.dt * U.ph.rdx;
  const float py = ((float)y + 0.5f) - v1 * U.ph.dt * U.ph.rdx;
  const float pz = ((float)z + 0.5f) - v2 * U.ph.dt * U.ph.rdx;
  const float *f[NQ];
#pragma unroll
  for (int k = 0; k < NQ; k++) f[k] = U.q[k];
  float o[NQ];
  u_interp<NQ>(U, f, px, py, pz, o, [&U](float *v, int cx, int cy, int cz) {
#pragma unroll
    for (int k = 0; k < NQ; k++) v[k] = q_bc(U.g, U.ph, v[k], k, cx, cy, cz, 1);
  });
  if (U.ph.em_n > 0) o[0] = o[0] + U.ph.dt * emission_at(U.g, U.ph, x, y, z, 1);
#pragma unroll
  for (int k = 0; k < NQ; k++) U.tq[k][i] = o[k];
}

// k_uniform_calc_divergence (uniformgrid_fluid.cu:107-132)
__global__ void __launch_bounds__(256) k_u_divergence(UDev U, int sx) {
  int x, y, z;
  size_t i;
  if (!u_cell(U.gx, U.gy, sx, x, y, z, i)) return;
  const UNb n = u_neighbours(i, x, y, z, U.gx, U.gy, U.gz);
  U.p[i] = 0.f;
  U.pt[i] = 0.f;
  float vl = U.v[0][n.l], vr = U.v[0][n.r], vd = U.v[1][n.d], vu = U.v[1][n.u], vb = U.v[2][n.b], vf = U.v[2][n.f];
  if (x == 0) vl = vel_bc1(U.g, U.ph, vl, 0, x - 1, y, z, 1);
  if (x == U.gx - 1) vr = vel_bc1(U.g, U.ph, vr, 0, x + 1, y, z, 1);
  if (y == 0) vd = vel_bc1(U.g, U.ph, vd, 1, x, y - 1, z, 1);
  if (y == U.gy - 1) vu = vel_bc1(U.g, U.ph, vu, 1, x, y + 1, z, 1);
  if (z == 0) vb = vel_bc1(U.g, U.ph, vb, 2, x, y, z - 1, 1);
  if (z == U.gz - 1) vf = vel_bc1(U.g, U.ph, vf, 2, x, y, z + 1, 1);
  const float *W = U.w;
  U.div[i] = 0.5f * U.ph.rdx * (W[n.r] * vr - W[n.l] * vl + W[n.u] * vu - W[n.d] * vd + W[n.f] * vf - W[n.b] * vb);
}

// k_uniform_restrict (uniformgrid_fluid.cu:134-160)
__global__ void __launch_bounds__(256) k_u_restrict(UDev U, int sx, int level) {
  const int s = 1 << level, cs = s / 2;
  int x, y, z;
  size_t i;
  if (!u_cell(U.gx / s, U.gy / s, sx, x, y, z, i)) return;
  const int wc = U.gx / cs, hc = U.gy / cs;
  const size_t idx = (size_t)U.mip_off[level] + i;
  const size_t i000 = umip(U, 2 * x, 2 * y, 2 * z, level - 1);
  const size_t i001 = i000 + 1, i010 = i000 + wc, i011 = i010 + 1;
  const size_t i100 = i000 + (size_t)wc * hc, i101 = i100 + 1, i110 = i100 + wc, i111 = i110 + 1;
  U.p[idx] = 0.f;
  U.pt[idx] = 0.f;
  const float *V = U.div;
  U.div[idx] = 0.125f * (V[i000] + V[i001] + V[i010] + V[i011] + V[i100] + V[i101] + V[i110] + V[i111]);
}

// calcPressure / k_uniform_jacobi(_inv) (uniformgrid_fluid.cu:162-204)
__global__ void __launch_bounds__(256) k_u_jacobi(UDev U, int sx, int level, const float *__restrict__ src,
                                                  float *__restrict__ dst) {
  const int s = 1 << level;
  const int w = U.gx / s, h = U.gy / s, d = U.gz / s;
  int x, y, z;
  size_t i;
  if (!u_cell(w, h, sx, x, y, z, i)) return;
  i += (size_t)U.mip_off[level];
  const UNb n = u_neighbours(i, x, y, z, w, h, d);
  const float alpha = U.ph.dx * U.ph.dx * (float)s * (float)s;
  dst[i] = div6(src[n.l] + src[n.r] + src[n.d] + src[n.u] + src[n.b] + src[n.f] - alpha * U.div[i]);
}

// k_uniform_prolongate (uniformgrid_fluid.cu:206-237): one cell, index i of its level
__device__ inline float u_prolong(const UDev &U, int level, int x, int y, int z) {
  const int s = 1 << level;
  const int w = U.gx / s, h = U.gy / s, d = U.gz / s;
  const size_t i000 = umip(U, x / 2, y / 2, z / 2, level + 1);
  const int sx = (x == 0 || x == w - 1) ? 0 : 2 * (x % 2) - 1;
  const int sy = (y == 0 || y == h - 1) ? 0 : 2 * (y % 2) - 1;
  const int sz = (z == 0 || z == d - 1) ? 0 : 2 * (z % 2) - 1;
  const size_t i001 = i000 + sx;
  const size_t i010 = i000 + (long long)sy * w / 2;
  const size_t i011 = i010 + sx;
  const size_t i100 = i000 + (long long)sz * (w / 2) * (h / 2);
  const size_t i101 = i100 + sx;
  const size_t i110 = i100 + (long long)sy * (w / 2);
  const size_t i111 = i110 + sx;
  const float *P = U.p;
  return (27.f * P[i000] + 9.f * (P[i001] + P[i010] + P[i100]) + 3.f * (P[i011] + P[i101] + P[i110]) + P[i111]) / 64.f;
}
__global__ void __launch_bounds__(256) k_u_prolongate(UDev U, int sx, int level, float *out) {
  const int s = 1 << level;
  int x, y, z;
  size_t i;
  if (u_cell(U.gx / s, U.gy / s, sx, x, y, z, i)) out[i] = u_prolong(U, level, x, y, z);
}

// Small mip levels hi..lo (coarse to fine, each of at most SB_CELLS cells) by
// one CTA, a level's prolongation and all its sweeps in shared memory (two
// planes); a thread keeps its cells' right-hand sides and the faces of the box
// on which they lie in registers. One launch and a CTA barrier per sweep
// instead of a launch per sweep (2.3 us inside a graph, 4.1 us launched).
// Bound by the issue rate of one SM: about 0.15 us per sweep and 1024 cells;
// larger levels are faster with the whole GPU.
constexpr int SB_THREADS = 1024, SB_K = 8, SB_CELLS = SB_K * SB_THREADS;
constexpr int SB_SMEM = SB_CELLS * 8;
__global__ void __launch_bounds__(SB_THREADS, 1) k_u_small(UDev U, int hi, int lo, int sweeps_hi, int sweeps) {
  extern __shared__ __align__(16) float sb[];
  for (int level = hi; level >= lo; level--) {
    const int s = 1 << level;
    const int w = U.gx / s, h = U.gy / s, d = U.gz / s, wh = w * h, n = wh * d;
    const size_t off = (size_t)U.mip_off[level];
    const float alpha = U.ph.dx * U.ph.dx * (float)s * (float)s;
    const bool top = level == U.levels - 1;
    const int todo = level == hi ? sweeps_hi : sweeps;
    float ad[SB_K];
    unsigned face[SB_K];
#pragma unroll
    for (int k = 0; k < SB_K; k++) {
      const int i = threadIdx.x + k * SB_THREADS;
      if (i >= n) break;
      const int z = i / wh, y = (i - z * wh) / w, x = i - z * wh - y * w;
      face[k] = (unsigned)((x == 0) | (x == w - 1) << 1 | (y == 0) << 2 | (y == h - 1) << 3 | (z == 0) << 4 |
                           (z == d - 1) << 5);
      ad[k] = alpha * U.div[off + i];
      sb[i] = top ? 0.f : u_prolong(U, level, x, y, z);
      sb[SB_CELLS + i] = 0.f;
    }
    for (int it = 0; it < todo; it++) {
      const float *src = sb + (it & 1) * SB_CELLS;
      float *dst = sb + ((it & 1) ^ 1) * SB_CELLS;
      __syncthreads();
#pragma unroll
      for (int k = 0; k < SB_K; k++) {
        const int i = threadIdx.x + k * SB_THREADS;
        if (i >= n) break;
        const unsigned f = face[k];
        const float *c = src + i;
        const float l = c[(f & 1u) ? 0 : -1], r = c[(f & 2u) ? 0 : 1], dn = c[(f & 4u) ? 0 : -w],
                    up = c[(f & 8u) ? 0 : w], bk = c[(f & 16u) ? 0 : -wh], fw = c[(f & 32u) ? 0 : wh];
        dst[i] = div6(l + r + dn + up + bk + fw - ad[k]);
      }
    }
    __syncthreads();
    for (int i = threadIdx.x; i < n; i += SB_THREADS) {
      U.p[off + i] = sb[i];  // an even number of sweeps
      if (todo > 0) U.pt[off + i] = sb[SB_CELLS + i];
    }
    __syncthreads();  // the next level's prolongation reads p
  }
}

// k_uniform_apply_pressure (uniformgrid_fluid.cu:239-260)
__global__ void __launch_bounds__(256) k_u_apply_pressure(UDev U, int sx) {
  int x, y, z;
  size_t i;
  if (!u_cell(U.gx, U.gy, sx, x, y, z, i)) return;
  float v0, v1, v2;
  u_project(U, i, x, y, z, v0, v1, v2);
  U.v[0][i] = v0;
  U.v[1][i] = v1;
  U.v[2][i] = v2;
}

__global__ void __launch_bounds__(256) k_u_noise(UDev U, int sx, unsigned long long seed, float amp) {
  int x, y, z;
  size_t i;
  if (!u_cell(U.gx, U.gy, sx, x, y, z, i)) return;
  for (int d = 0; d < 3; d++) U.v[d][i] = U.v[d][i] + amp * noise_unit(seed, x, y, z, 0, d);
}

// k_uniform_debug_stats (uniformgrid_structure.cu:33-43): sum rho * w.
__global__ void __launch_bounds__(256) k_u_stats(UDev U) {
  const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  double m = 0.0;
  if (i < U.nc) m = (double)U.q[0][i] * (double)U.w[i];
  for (int o = 16; o > 0; o >>= 1) m += __shfl_xor_sync(0xffffffffu, m, o);
  if ((threadIdx.x & 31) == 0 && m != 0.0) atomicAdd(&U.red[1], m);
}

static unsigned ugrid(long long n) { return (unsigned)((n + 255) / 256); }
static long long ucells(const UDev &U, int level) {
  const int s = 1 << level;
  return (long long)(U.gx / s) * (U.gy / s) * (U.gz / s);
}
// launches a cell kernel over a mip level with the CTA shape (32, 16 or 8 cells
// along x) that covers its planes with the fewest threads, wide rows first
template <class K, class... Args>
static void u_launch(K kernel, const UDev &U, int level, cudaStream_t st, Args... args) {
  const long long w = U.gx >> level, h = U.gy >> level, d = U.gz >> level;
  auto ctas = [&](int sx) { return ((w + (1 << sx) - 1) >> sx) * ((h + (256 >> sx) - 1) >> (8 - sx)); };
  int sx = 5;
  for (int k = 4; k >= 3; k--)
    if (10 * ctas(k) < 9 * ctas(sx)) sx = k;
  kernel<<<(unsigned)(ctas(sx) * d), 256, 0, st>>>(U, sx, args...);
}

void launch_u_fluidity(const UDev &U, cudaStream_t st) {
  for (int l = 0; l < U.levels; l++) u_launch(k_u_fluidity, U, l, st, l);
}
void launch_u_sources(const UDev &U, cudaStream_t st) { u_launch(k_u_sources, U, 0, st); }
void launch_u_advect_velocity(const UDev &U, cudaStream_t st) { u_launch(k_u_advect_velocity, U, 0, st); }
void launch_u_advect_scalars(const UDev &U, bool apply, cudaStream_t st) {
  if (U.nq == 3) u_launch(apply ? k_u_advect_scalars<true, 3> : k_u_advect_scalars<false, 3>, U, 0, st);
  else u_launch(apply ? k_u_advect_scalars<true, 1> : k_u_advect_scalars<false, 1>, U, 0, st);
}
// The sweeps of one mip level from its prolongation (or from zero) into p, the
// iterate before the last into p~. Larger levels take the dense passes from
// U.tv[0], where their prolongation goes, with U.tv[0] and U.tv[1], free until
// the next velocity advection, as scratch; below kDenseCells a launch per
// sweep is faster (48^3: 4.1 against 4.7 us per sweep; 64^3: 6.1 and 5.6; 192^3:
// 55 and 13).
constexpr long long kDenseCells = 200000;
static void u_sweeps(const UDev &U, int level, int sweeps, bool zero, int sms, cudaStream_t st) {
  const long long n = ucells(U, level);
  const size_t o = (size_t)U.mip_off[level];
  const bool dense = n > kDenseCells && sweeps > 0;
  if (!zero) u_launch(k_u_prolongate, U, level, st, level, dense ? U.tv[0] : U.p + o);
  if (dense) {
    const int s = 1 << level;
    const float alpha = U.ph.dx * U.ph.dx * (float)s * (float)s;
    const DenseSweep v{U.gx / s,  U.gy / s,  U.gz / s,  U.tv[0], U.div + o, U.tv[0],
                       U.tv[1],   U.p + o,   U.pt + o,  -alpha,  zero,      false};
    launch_dense_sweeps(&v, 1, sweeps, true, sms, st);
    return;
  }
  for (int i = 0; i < sweeps / 2; i++) {
    u_launch(k_u_jacobi, U, level, st, level, (const float *)U.p, U.pt);
    u_launch(k_u_jacobi, U, level, st, level, (const float *)U.pt, U.p);
  }
}
// FluidSimulationUniform::project / projectLocal (fluid_simulation_uniform.cu:96-135)
// apply = false leaves out the pressure application (k_u_advect_scalars<true> follows)
void launch_u_project(const UDev &U, int top_pairs, int pairs, bool local, bool apply, int sms, cudaStream_t st) {
  u_launch(k_u_divergence, U, 0, st);
  if (local) {
    u_sweeps(U, 0, 2 * pairs, true, sms, st);
  } else {
    for (int l = 1; l < U.levels; l++) u_launch(k_u_restrict, U, l, st, l);
    const int top = U.levels - 1;
    int l = top;
    while (l >= 0 && ucells(U, l) <= SB_CELLS) l--;
    if (l < top) {  // the levels that one CTA holds; the shared-memory opt-in is the current device's
      const bool clean = cudaPeekAtLastError() == cudaSuccess;
      if (cudaFuncSetAttribute(k_u_small, cudaFuncAttributeMaxDynamicSharedMemorySize, SB_SMEM) == cudaSuccess) {
        k_u_small<<<1, SB_THREADS, SB_SMEM, st>>>(U, top, l + 1, 2 * top_pairs, 2 * pairs);
      } else {
        if (clean) cudaGetLastError();  // a launch per sweep takes its place
        l = top;
      }
    }
    for (; l >= 0; l--) u_sweeps(U, l, 2 * (l == top ? top_pairs : pairs), l == top, sms, st);
  }
  if (apply) u_launch(k_u_apply_pressure, U, 0, st);
}
void launch_u_add_noise(const UDev &U, unsigned long long seed, float amp, cudaStream_t st) {
  u_launch(k_u_noise, U, 0, st, seed, amp);
}
void launch_u_stats(const UDev &U, cudaStream_t st) {
  cudaMemsetAsync(U.red, 0, sizeof(double) * 32, st);
  k_u_stats<<<ugrid(U.nc), 256, 0, st>>>(U);
}

}  // namespace dcg
