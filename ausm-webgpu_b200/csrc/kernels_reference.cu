// Reference-shaped engine: the reference's five dispatches per RK stage as two CUDA
// kernels (boundary, j- and i-flux; residual and RK stage), fluxes and states going through
// memory, on the reference's buffer layout (main.js:110-125):
//   boundary  ausm.js:23-120   M x (N+3)   ghost rows + pass-through copy
//   j-flux    ausm.js:128-392  M x (N+1)   faces below each interior cell
//   i-flux    ausm.js:128-392  M x N       faces left of each interior cell (the
//                                          reference's extra column i=M is never read,
//                                          ausm.js:420, and is not computed)
//   residual  ausm.js:402-436  M x N
//   RK stage  ausm.js:441-527  M x N       interior rows only
// plus the wave-speed max reduction (ausm.js:617-630, 535-581) and the grid metrics
// (shaders/grid.js:115-147).  This translation unit is compiled with -fmad=false and
// uses the exact (FAST=false) arithmetic, so it matches the float oracle bit for bit.
// It is the plain baseline of the benchmarks.
// Bound by its IEEE divisions and square roots (some 50 a cell and stage) and by latency.  A
// step of 510 x 381 (AUSM+-up) took 100 us with one kernel per dispatch (full copies in the
// boundary pass, the residual through memory, eight conversions to primitives per cell),
// 75 us with those kernels under programmatic dependent launch, and takes 53 us.
#include "ausm_internal.h"
#include "tma.cuh"

namespace ausm {

// State of cell (i, j), j in [-2, N + 1], from interior rows alone: loadState (ausm.js:138-143;
// i wraps, interior row + 1, clamped at the wall ghost) with the ghost rows of the boundary
// pass (ausm.js:23-120) computed where they are read.
__device__ __forceinline__ float4 ref_load(const float4* st, const float2* V, const Consts& c, int M, int N, int i, int j) {
  const int ii = (i + M) % M, jj = max(j + 1, 0);
  if (jj >= 1 && jj <= N) return st[(size_t)jj * M + ii];
  const int r = (ii + 1) % M;
  if (jj == 0) return wall_ghost<false>(st[(size_t)M + ii], V[ii], V[r]);
  float4 g1, g2;
  far_ghosts<false>(st[(size_t)N * M + ii], V[(size_t)N * M + ii], V[(size_t)N * M + r], c, g1, g2);
  return jj == N + 1 ? g1 : g2;
}

__global__ void k_ref_metrics(const float2* __restrict__ V, float* __restrict__ area, float4* __restrict__ flen,
                              int M, int N) {
  int i = blockIdx.x * blockDim.x + threadIdx.x, j = blockIdx.y * blockDim.y + threadIdx.y;
  if (i >= M || j >= N) return;
  int r = (i + 1) % M;
  float2 a = V[(size_t)j * M + i], b = V[(size_t)j * M + r], c = V[(size_t)(j + 1) * M + i],
         d = V[(size_t)(j + 1) * M + r];
  size_t k = (size_t)j * M + i;
  area[k] = quad_area(a, b, c, d);
  float4 l;
  l.x = sqrtf((a.x - c.x) * (a.x - c.x) + (a.y - c.y) * (a.y - c.y));
  l.y = sqrtf((b.x - d.x) * (b.x - d.x) + (b.y - d.y) * (b.y - d.y));
  l.z = sqrtf((c.x - d.x) * (c.x - d.x) + (c.y - d.y) * (c.y - d.y));
  l.w = sqrtf((a.x - b.x) * (a.x - b.x) + (a.y - b.y) * (a.y - b.y));
  flen[k] = l;
}

__global__ void k_ref_boundary(const float4* __restrict__ in, float4* __restrict__ out,
                               const float2* __restrict__ V, const Consts c, int M, int N) {
  int i = blockIdx.x * blockDim.x + threadIdx.x, y = blockIdx.y * blockDim.y + threadIdx.y;
  if (i >= M || y >= N + 3) return;
  int r = (i + 1) % M;
  grid_dep_wait();
  grid_dep_launch();
  if (y == 0) {
    out[i] = wall_ghost<false>(in[(size_t)M + i], V[i], V[r]);
  } else if (y > N) {
    float4 g1, g2;
    far_ghosts<false>(in[(size_t)N * M + i], V[(size_t)N * M + i], V[(size_t)N * M + r], c, g1, g2);
    out[(size_t)y * M + i] = (y == N + 1) ? g1 : g2;
  } else {
    out[(size_t)y * M + i] = in[(size_t)y * M + i];
  }
}

// The j- and i-flux passes: a block converts the cells of its 32 x 8 faces (with the three
// rows and columns beside them) to primitives once, in shared memory, and its threads take
// one face of each direction.  Two kernels that converted the four cells of every face
// spent a quarter of their time on that (8 conversions per cell, two divisions each).
template <int SCHEME>
__global__ void __launch_bounds__(256)
    k_ref_fluxes(const float4* __restrict__ st, const float2* __restrict__ V, float4* __restrict__ fx,
                 float4* __restrict__ fy, const Consts c, int M, int N) {
  __shared__ float4 P[11][35];
  const int tx = threadIdx.x, ty = threadIdx.y, across = (M + 31) / 32;  // blocks row by row
  const int i0 = (int)(blockIdx.x % across) * 32, j0 = (int)(blockIdx.x / across) * 8;
  const int i = i0 + tx, j = j0 + ty;
  const bool jf = i < M && j <= N, jn = i < M && j < N;
  float nx = 0, ny = 0, mx = 0, my = 0, len;
  if (jf) edge_normal<false>(V[(size_t)j * M + i], V[(size_t)j * M + (i + 1) % M], nx, ny, len);
  if (jn) edge_normal<false>(V[(size_t)(j + 1) * M + i], V[(size_t)j * M + i], mx, my, len);
  grid_dep_wait();
  grid_dep_launch();
  for (int k = ty * 32 + tx; k < 11 * 35; k += 256) {
    const int r = k / 35, cc = k % 35;
    if (j0 - 2 + r <= N + 1 && i0 - 2 + cc <= M)
      P[r][cc] = to_prim<false>(ref_load(st, V, c, M, N, i0 - 2 + cc, j0 - 2 + r), c.gm1);
  }
  __syncthreads();
  if (jf)
    fy[(size_t)j * M + i] = face_flux<SCHEME>(P[ty][tx + 2], P[ty + 1][tx + 2], P[ty + 2][tx + 2], P[ty + 3][tx + 2], nx, ny, c);
  if (jn)
    fx[(size_t)j * M + i] = face_flux<SCHEME>(P[ty + 2][tx], P[ty + 2][tx + 1], P[ty + 2][tx + 2], P[ty + 2][tx + 3], mx, my, c);
}

// residual of a cell from its faces (ausm.js:402-436)
__device__ __forceinline__ float4 residual_of(const float4* __restrict__ fx, const float4* __restrict__ fy,
                                              const float4* __restrict__ flen, const float* __restrict__ area, int M,
                                              int i, int j) {
  size_t k = (size_t)j * M + i;
  float4 xl = fx[k], xr = fx[(size_t)j * M + (i + 1) % M], yu = fy[(size_t)(j + 1) * M + i], yd = fy[k];
  float4 l = flen[k];
  float A = area[k];
  float4 R;
  R.x = -(xr.x * l.y - xl.x * l.x + yu.x * l.z - yd.x * l.w) / A;
  R.y = -(xr.y * l.y - xl.y * l.x + yu.y * l.z - yd.y * l.w) / A;
  R.z = -(xr.z * l.y - xl.z * l.x + yu.z * l.z - yd.z * l.w) / A;
  R.w = -(xr.w * l.y - xl.w * l.x + yu.w * l.z - yd.w * l.w) / A;
  return R;
}
__global__ void k_ref_residual(const float4* __restrict__ fx, const float4* __restrict__ fy,
                               const float4* __restrict__ flen, const float* __restrict__ area,
                               float4* __restrict__ res, int M, int N) {
  int i = blockIdx.x * blockDim.x + threadIdx.x, j = blockIdx.y * blockDim.y + threadIdx.y;
  if (i >= M || j >= N) return;
  grid_dep_wait();
  grid_dep_launch();
  res[(size_t)j * M + i] = residual_of(fx, fy, flen, area, M, i, j);
}

// residual and RK stage (ausm.js:402-527) of the interior rows; the residual, which only
// this stage uses, stays in registers
template <int STAGE>
__global__ void k_ref_stage(const float4* __restrict__ fx, const float4* __restrict__ fy,
                            const float4* __restrict__ flen, const float* __restrict__ area, const float4* s0,
                            const float4* __restrict__ s1, float4* out, const float* __restrict__ dtp, int M,
                            int N) {
  int i = blockIdx.x * blockDim.x + threadIdx.x, j = blockIdx.y * blockDim.y + threadIdx.y;
  if (i >= M || j >= N) return;
  grid_dep_wait();
  grid_dep_launch();
  const float dt = *dtp;
  size_t o = (size_t)(j + 1) * M + i;
  const float4 Rr = residual_of(fx, fy, flen, area, M, i, j), Q = s0[o];
  float4 o4;
  if constexpr (STAGE == 1) {
    o4 = make_float4(Q.x + dt * Rr.x, Q.y + dt * Rr.y, Q.z + dt * Rr.z, Q.w + dt * Rr.w);
  } else if constexpr (STAGE == 2) {
    float4 Q1 = s1[o];
    o4 = make_float4(0.75f * Q.x + 0.25f * (Q1.x + dt * Rr.x), 0.75f * Q.y + 0.25f * (Q1.y + dt * Rr.y),
                     0.75f * Q.z + 0.25f * (Q1.z + dt * Rr.z), 0.75f * Q.w + 0.25f * (Q1.w + dt * Rr.w));
  } else {
    float4 Q2 = s1[o];
    o4 = make_float4((Q.x + 2.0f * (Q2.x + dt * Rr.x)) / 3.0f, (Q.y + 2.0f * (Q2.y + dt * Rr.y)) / 3.0f,
                     (Q.z + 2.0f * (Q2.z + dt * Rr.z)) / 3.0f, (Q.w + 2.0f * (Q2.w + dt * Rr.w)) / 3.0f);
  }
  out[o] = o4;
}

__global__ void k_ref_wave(const float4* __restrict__ st, const float4* __restrict__ flen,
                           const float* __restrict__ area, float gamma, int M, int N, uint32_t* wave) {
  grid_dep_wait();
  grid_dep_launch();
  uint32_t wm = 0u;
  size_t total = (size_t)M * N;
  for (size_t k = blockIdx.x * (size_t)blockDim.x + threadIdx.x; k < total; k += (size_t)gridDim.x * blockDim.x) {
    float4 l = flen[k];
    float w = wave_speed<false>(st[k + M], ((l.x + l.y) + l.z) + l.w, area[k], gamma);
    wm = max(wm, __float_as_uint(w));
  }
  block_max_to(wave, wm);
}

// dt = min(maxdt, cfl / maxWaveSpeed) (ausm.js:457)
__global__ void k_dt(const uint32_t* __restrict__ wave, float* __restrict__ dt, float maxdt, float cfl) {
  dt[0] = fminf(maxdt, cfl / __uint_as_float(wave[0]));
}

// ---- launchers ----
static inline dim3 grid16(int w, int h) { return dim3((w + 15) / 16, (h + 15) / 16); }
static const dim3 B16(16, 16);

void launch_ref_metrics(const float2* V, float* area, float4* flen, int M, int N, cudaStream_t s) {
  k_ref_metrics<<<grid16(M, N), B16, 0, s>>>(V, area, flen, M, N);
}
void launch_ref_boundary(const float4* in, float4* out, const float2* V, const Consts& c, int M, int N,
                         cudaStream_t s) {
  launch_pdl(k_ref_boundary, grid16(M, N + 3), B16, 0, s, in, out, V, c, M, N);
}
void launch_ref_fluxes(int scheme, const float4* st, const float2* V, float4* fx, float4* fy, const Consts& c, int M,
                       int N, cudaStream_t s) {
  const dim3 g((M + 31) / 32 * ((N + 8) / 8)), b(32, 8);
  if (scheme == 0) launch_pdl(k_ref_fluxes<0>, g, b, 0, s, st, V, fx, fy, c, M, N);
  else if (scheme == 1) launch_pdl(k_ref_fluxes<1>, g, b, 0, s, st, V, fx, fy, c, M, N);
  else launch_pdl(k_ref_fluxes<2>, g, b, 0, s, st, V, fx, fy, c, M, N);
}
void launch_ref_residual(const float4* fx, const float4* fy, const float4* flen, const float* area, float4* res, int M,
                         int N, cudaStream_t s) {
  launch_pdl(k_ref_residual, grid16(M, N), B16, 0, s, fx, fy, flen, area, res, M, N);
}
void launch_ref_stage(int stage, const float4* fx, const float4* fy, const float4* flen, const float* area,
                      const float4* s0, const float4* s1, float4* out, const float* dt, int M, int N, cudaStream_t s) {
  auto k = stage == 1 ? k_ref_stage<1> : (stage == 2 ? k_ref_stage<2> : k_ref_stage<3>);
  launch_pdl(k, grid16(M, N), B16, 0, s, fx, fy, flen, area, s0, s1, out, dt, M, N);
}
void launch_ref_wave(const float4* st, const float4* flen, const float* area, float gamma, int M, int N,
                     uint32_t* wave, cudaStream_t s) {
  int blocks = (int)std::min<size_t>(((size_t)M * N + 255) / 256, 148 * 8);
  launch_pdl(k_ref_wave, dim3(blocks), dim3(256), 0, s, st, flen, area, gamma, M, N, wave);
}
void launch_dt(const uint32_t* wave, float* dt, float maxdt, float cfl, cudaStream_t s) {
  k_dt<<<1, 1, 0, s>>>(wave, dt, maxdt, cfl);
}

}  // namespace ausm
