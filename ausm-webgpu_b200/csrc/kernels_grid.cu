// O-grid generation: the initial guess and the elliptic sweeps (shaders/grid.js:18-113),
// compiled with -fmad=false like the reference's arithmetic.
//
// Sweeps run several to a launch on tiles in shared memory.  A CTA loads its tile with a
// halo as deep as the sweeps reach, applies them in place (multicolour) or between two
// copies (Jacobi) on a region that shrinks by one vertex per colour or sweep, and writes
// its own vertices to a second buffer; vertices of the halo are computed again by the
// tiles that own them, from the same operands, so the result has the bits of one launch
// per colour or sweep.  One launch per colour left three lanes of four idle, read the
// nine neighbours from L2 with a stride and cost a launch per colour.  Measured on B200,
// FP64 multicolour, us per sweep before / now: 128 x 96 18.4 / 2.9, 512 x 384 25.1 / 5.4,
// 1024 x 768 41.6 / 13.0, 4096 x 3072 563 / 168.  What is left at 1024 x 768: some 5 us of FP64
// arithmetic (72 operations a vertex at half rate, halo and idle lanes included) and the
// tiles' way in and out of L2, which all CTAs of the launch take at the same time; on
// small grids the latency of the colour steps, 0.4 us each.
#include <mutex>
#include <set>

#include "ausm_internal.h"
#include "tma.cuh"

namespace ausm {

// ---- initial guess ----
// Position of row j on the line of a column, as a fraction t: j / N (reference) or a
// geometric progression with first cell height `h1` relative to the body-outer distance.
// The growth ratio q solves h (q^N - 1)/(q - 1) = 1 by bisection; once the midpoint is
// one of its ends it stays there, so the loop ends with the q that 200 iterations give.
// It is found once per column and block, not by every vertex: guess, conversion and face
// records of 1024 x 768 cells took 2.5 ms (boundary rows sent with all others as zeros),
// now 0.09 ms; of 4096 x 3072, 106 ms and 0.7 ms.
__device__ __forceinline__ double growth_ratio(double h, int N) {
  double lo = 1.0 + 1e-12, hi = 2.0;
  if (h * N >= 1.0) { lo = 1e-6; hi = 1.0 - 1e-12; }
  for (int it = 0; it < 200; it++) {
    double q = 0.5 * (lo + hi);
    if (q == lo || q == hi) break;
    double s = h * (pow(q, (double)N) - 1.0) / (q - 1.0);
    if ((s > 1.0) == (h * N < 1.0)) hi = q; else lo = q;
  }
  return 0.5 * (lo + hi);
}

constexpr int kInitRows = 64;  // rows of a block of the initial guess

// Initial guess (shaders/grid.js:18-27): mix(body, outer, t) along each i line.
template <class V2T, class R>
__global__ void __launch_bounds__(256) k_grid_guess(V2T* __restrict__ V, int M, int N, double first_spacing) {
  __shared__ double sh[32], sq[32];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int i = blockIdx.x * 32 + lane;
  V2T a{}, b{};
  if (i < M) {
    a = V[i];
    b = V[(size_t)N * M + i];
  }
  if (first_spacing > 0.0) {
    if (warp == 0 && i < M) {
      // the line's length, with the coordinate differences rounded as R
      const double L = sqrt((double)(b.x - a.x) * (b.x - a.x) + (double)(b.y - a.y) * (b.y - a.y));
      sh[lane] = first_spacing / L;  // first step as a fraction of the line length
      sq[lane] = growth_ratio(sh[lane], N);
    }
    __syncthreads();
  }
  if (i >= M) return;
  const int j1 = min(N, (int)(blockIdx.y + 1) * kInitRows);
  for (int j = max(1, (int)blockIdx.y * kInitRows) + warp; j < j1; j += 8) {
    R t;
    if (first_spacing <= 0.0) {
      t = R(j) / R(N);
    } else {
      const double h = sh[lane], q = sq[lane];
      t = (R)(h * (pow(q, (double)j) - 1.0) / (q - 1.0));
    }
    V2T v;
    v.x = a.x * (R(1) - t) + b.x * t;
    v.y = a.y * (R(1) - t) + b.y * t;
    V[(size_t)j * M + i] = v;
  }
}

// ---- sweeps ----
// TTM/Winslow update with P = Q = 0 of the vertex at `s` from its eight neighbours, applied
// only where the Jacobian is negative (shaders/grid.js:55-108).
template <class V2T, class R>
__device__ __forceinline__ V2T ttm(V2T c, V2T L, V2T Rt, V2T D, V2T U, V2T DL, V2T DR, V2T UL, V2T UR, R omega) {
  R xix = R(0.5) * (Rt.x - L.x), xiy = R(0.5) * (Rt.y - L.y);
  R etx = R(0.5) * (U.x - D.x), ety = R(0.5) * (U.y - D.y);
  R xex = R(0.25) * (UR.x + DL.x - UL.x - DR.x), xey = R(0.25) * (UR.y + DL.y - UL.y - DR.y);
  R alpha = etx * etx + ety * ety, gam = xix * xix + xiy * xiy, beta = xix * etx + xiy * ety;
  R den = R(2) * (alpha + gam);
  R ax = L.x + Rt.x, ay = L.y + Rt.y, gx = D.x + U.x, gy = D.y + U.y;
  if constexpr (sizeof(R) == 4) {  // the reference's zero control functions keep their place in its sums
    const R P = R(0), Q = R(0);
    ax = ax + P * xix; ay = ay + P * xiy;
    gx = gx + Q * etx; gy = gy + Q * ety;
  }
  R npx = (alpha * ax + gam * gx - R(2) * beta * xex) / den;
  R npy = (alpha * ay + gam * gy - R(2) * beta * xey) / den;
  R jac = xix * ety - xiy * etx;
  V2T o;
  o.x = c.x * (R(1) - omega) + npx * omega;
  o.y = c.y * (R(1) - omega) + npy * omega;
  return jac < R(0) ? o : c;
}

// A tile: W vertices of a row of 64 (with the halo H on both sides) and h rows, cut in
// nearly equal parts.  The sweeps change rows 1 .. N - 1; src and dst hold those, rows 0
// and N come from `ends` (a full vertex array).
constexpr int GW = 64;
struct GridTile {
  int i0, w, j0, h;
};
__device__ __forceinline__ GridTile grid_tile(int M, int N) {
  GridTile t;
  t.i0 = (int)((long long)blockIdx.x * M / gridDim.x);
  t.w = (int)((long long)(blockIdx.x + 1) * M / gridDim.x) - t.i0;
  t.j0 = 1 + (int)((long long)blockIdx.y * (N - 1) / gridDim.y);
  t.h = 1 + (int)((long long)(blockIdx.y + 1) * (N - 1) / gridDim.y) - t.j0;
  return t;
}
template <class V2T>
__device__ __forceinline__ const V2T* grid_row(const V2T* src, const V2T* ends, int M, int N, int j) {
  return j == 0 ? ends : (j == N ? ends + (size_t)N * M : src + (size_t)(j - 1) * M);
}

// Fetches the tile's rows (with the halo) that the grid has, two columns gi[] per lane, and
// hands them to put(tile row, grid row, values), eight loads of a lane in flight (against
// row by row: multicolour 1024 x 768 13.4 -> 13.0, 4096 x 3072 184 -> 168 us per sweep).
template <class V2T, int NW, class Put>
__device__ __forceinline__ void load_rows(const GridTile& t, int H, const V2T* src, const V2T* ends, int M, int N,
                                          const int (&gi)[2], int warp, Put put) {
  constexpr int B = 4;
  for (int r = warp; r < t.h + 2 * H; r += B * NW) {
    V2T v[B][2];
#pragma unroll
    for (int q = 0; q < B; q++) {
      const int j = t.j0 - H + r + q * NW;
      if (r + q * NW < t.h + 2 * H && j >= 0 && j <= N) {
        const V2T* row = grid_row(src, ends, M, N, j);
        v[q][0] = row[gi[0]];
        v[q][1] = row[gi[1]];
      }
    }
#pragma unroll
    for (int q = 0; q < B; q++) {
      const int j = t.j0 - H + r + q * NW;
      if (r + q * NW < t.h + 2 * H && j >= 0 && j <= N) put(r + q * NW, j, v[q]);
    }
  }
}

// FP64 multicolour Gauss-Seidel.  Colour (i & 1) * 2 + (j & 1); with odd M the seam column
// i = M - 1 has the colours 4 + (j & 1), so no two vertices of a colour touch (9-point
// stencil, periodic in i).  A row of the tile is one warp: lane k has the columns 2 k and
// 2 k + 1, of which at most one has a given colour; even and odd columns are stored apart,
// so that the lanes of a colour read consecutive 16-byte words.  move: max vertex move of
// the last sweep (float bits), or null.
template <int NC, int S, int NW>
__global__ void __launch_bounds__(32 * NW)
    k_grid_multicolor(const double2* __restrict__ src, double2* __restrict__ dst, const double2* __restrict__ ends,
                      const int M, const int N, const int sweeps, const double omega, uint32_t* move) {
  constexpr int H = NC * S;
  extern __shared__ double2 smem_d[];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const GridTile t = grid_tile(M, N);
  auto at = [&](int r, int c) -> double2& { return smem_d[r * GW + (c & 1) * (GW / 2) + (c >> 1)]; };
  int gi[2], sel[3] = {-1, -1, -1};
#pragma unroll
  for (int k = 0; k < 2; k++) {
    const int x = (t.i0 - H + 2 * lane + k) % M, i = x < 0 ? x + M : x;
    gi[k] = i;
    sel[(M & 1) && i == M - 1 ? 2 : (i & 1)] = 2 * lane + k;
  }
  grid_dep_wait();
  grid_dep_launch();
  load_rows<double2, NW>(t, H, src, ends, M, N, gi, warp, [&](int r, int, const double2* v) {
#pragma unroll
    for (int k = 0; k < 2; k++) at(r, 2 * lane + k) = v[k];
  });
  __syncthreads();
  const int steps = NC * sweeps;
  uint32_t mv = 0u;
  for (int st = 0, col = 0; st < steps; st++, col = col == NC - 1 ? 0 : col + 1) {
    const int e = steps - 1 - st;
    const int c = col < 2 ? sel[0] : (col < 4 ? sel[1] : sel[2]);
    const int lo = max(H - e, H + 1 - t.j0), hi = min(H + t.h + e, H + N - t.j0);
    const int first = lo + ((t.j0 - H + lo + col) & 1);  // first row of the colour's parity
    if (c >= H - e && c < H + t.w + e)
      for (int r = first + 2 * warp; r < hi; r += 2 * NW) {
        const double2 o = at(r, c);
        const double2 p = ttm<double2, double>(o, at(r, c - 1), at(r, c + 1), at(r - 1, c), at(r + 1, c), at(r - 1, c - 1),
                                               at(r - 1, c + 1), at(r + 1, c - 1), at(r + 1, c + 1), omega);
        at(r, c) = p;
        if (move && st >= steps - NC && c >= H && c < H + t.w && r >= H && r < H + t.h)
          mv = max(mv, __float_as_uint((float)fmax(fabs(p.x - o.x), fabs(p.y - o.y))));
      }
    __syncthreads();
  }
  for (int r = H + warp; r < H + t.h; r += NW) {
    double2* row = dst + (size_t)(t.j0 - H + r - 1) * M;
#pragma unroll
    for (int k = 0; k < 2; k++) {
      const int c = 2 * lane + k;
      if (c >= H && c < H + t.w) row[gi[k]] = at(r, c);
    }
  }
  if (move) block_max_to(move, mv);
}

// FP32 Jacobi sweeps (omega = 1), the reference's generator; lane k has the columns k and
// k + 32 of a row.
template <int S, int NW>
__global__ void __launch_bounds__(32 * NW)
    k_grid_jacobi(const float2* __restrict__ src, float2* __restrict__ dst, const float2* __restrict__ ends,
                  const int M, const int N, const int sweeps) {
  constexpr int H = S;
  extern __shared__ float2 smem_f[];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const GridTile t = grid_tile(M, N);
  const int rows = t.h + 2 * H;
  float2 *a = smem_f, *b = smem_f + rows * GW;
  int gi[2];
#pragma unroll
  for (int k = 0; k < 2; k++) {
    const int x = (t.i0 - H + lane + 32 * k) % M;
    gi[k] = x < 0 ? x + M : x;
  }
  grid_dep_wait();
  grid_dep_launch();
  load_rows<float2, NW>(t, H, src, ends, M, N, gi, warp, [&](int r, int j, const float2* v) {
#pragma unroll
    for (int k = 0; k < 2; k++) {
      a[r * GW + lane + 32 * k] = v[k];
      if (j == 0 || j == N) b[r * GW + lane + 32 * k] = v[k];  // fixed rows, in both copies
    }
  });
  __syncthreads();
  for (int st = 0; st < sweeps; st++) {
    const int e = sweeps - 1 - st;
    const int lo = max(H - e, H + 1 - t.j0), hi = min(H + t.h + e, H + N - t.j0);
    for (int r = lo + warp; r < hi; r += NW)
#pragma unroll
      for (int k = 0; k < 2; k++) {
        const int c = lane + 32 * k;
        if (c >= H - e && c < H + t.w + e) {
          const float2 *m = a + r * GW + c, *d = m - GW, *u = m + GW;
          b[r * GW + c] = ttm<float2, float>(m[0], m[-1], m[1], d[0], u[0], d[-1], d[1], u[-1], u[1], 1.0f);
        }
      }
    __syncthreads();
    float2* x = a;
    a = b;
    b = x;
  }
  for (int r = H + warp; r < H + t.h; r += NW) {
    float2* row = dst + (size_t)(t.j0 - H + r - 1) * M;
#pragma unroll
    for (int k = 0; k < 2; k++) {
      const int c = lane + 32 * k;
      if (c >= H && c < H + t.w) row[gi[k]] = a[r * GW + c];
    }
  }
}

// ---- launchers ----
namespace {
constexpr int kSMs = 148;
// Tiles of an M x N grid: as wide as the halo lets them be, and as many rows of tiles as
// fill whole rounds of the SMs, at most `max_h` vertex rows each.
dim3 grid_tiles(int M, int N, int halo, int max_h) {
  const int nx = (M + GW - 2 * halo - 1) / (GW - 2 * halo);
  const int need = (N - 1 + max_h - 1) / max_h;
  const int rounds = (nx * need + kSMs - 1) / kSMs;
  return dim3(nx, std::max(need, std::min(std::max(1, kSMs * rounds / nx), N - 1)));
}
// Lets KERN take `bytes`, what its largest tile needs, on the current device: once per
// device and before its first launch there.  The limit belongs to the kernel and is shared
// by all host threads; set per launch to the launch's own size, it changed under another
// thread's launch, and grids of two sizes generated at once came out wrong.
template <auto KERN> void allow_smem(int bytes) {
  static std::mutex mu;
  static std::set<int> done;
  int dev = 0;
  cudaGetDevice(&dev);
  std::lock_guard<std::mutex> lk(mu);
  if (done.count(dev)) return;
  if (cudaFuncSetAttribute(KERN, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes) == cudaSuccess) done.insert(dev);
}
template <int NC, int S, int NW, int MAX_H>
void sweeps_d(const double2* src, double2* dst, const double2* ends, int M, int N, int sweeps, double omega,
              uint32_t* move, cudaStream_t s) {
  constexpr int ROW = GW * (int)sizeof(double2);
  const dim3 g = grid_tiles(M, N, NC * S, MAX_H);
  const int h = (N - 1 + g.y - 1) / g.y;
  constexpr auto kern = k_grid_multicolor<NC, S, NW>;
  allow_smem<kern>((MAX_H + 2 * NC * S) * ROW);
  launch_pdl(kern, g, dim3(32 * NW), (size_t)(h + 2 * NC * S) * ROW, s, src, dst, ends, M, N, sweeps, omega, move);
}
// One or two sweeps to a launch.  Two halve the launches and the trips through L2, for a
// deeper halo (tiles of 48 columns instead of 56, with odd M 40 instead of 52).
// Even M: two while the tiles of one sweep are cut for two rounds of the SMs at most; three
// rounds are lower tiles that run three to an SM, and one sweep wins (us per sweep, one /
// two: 64 x 33 3.0 / 2.7, 512 x 384 6.6 / 5.3, 640 x 480 8.2 / 7.0, 900 x 600 13.1 / 11.4,
// 4096 x 160 14.1 / 12.6; beyond, 1000 x 650 11.1 / 12.7, 256 x 2400 11.0 / 13.7, 1024 x 768
// 13.0 / 15.4).  Odd M, whose halos are half as deep again: two while their tiles fit the SMs
// one each (129 x 97 4.3 / 4.3, 201 x 151 4.5 / 4.7, 401 x 300 6.9 / 6.5, 513 x 300 7.5 / 7.1;
// beyond, 513 x 385 8.6 / 8.7, 721 x 481 11.7 / 11.3, 801 x 600 15.0 / 16.8).
bool two_sweeps(int M, int N) {
  auto tiles = [&](int cols, int rows) { return (long long)((M + cols - 1) / cols) * ((N - 1 + rows - 1) / rows); };
  return M & 1 ? tiles(40, 32) <= kSMs : tiles(56, 40) <= 2 * kSMs;
}
}  // namespace

void launch_grid_init(float2* V, int M, int N, double first_spacing, cudaStream_t s) {
  k_grid_guess<float2, float><<<dim3((M + 31) / 32, (N + kInitRows - 1) / kInitRows), 256, 0, s>>>(V, M, N, first_spacing);
}
void launch_grid_init_d(double2* V, int M, int N, double first_spacing, cudaStream_t s) {
  k_grid_guess<double2, double><<<dim3((M + 31) / 32, (N + kInitRows - 1) / kInitRows), 256, 0, s>>>(V, M, N, first_spacing);
}

// 6 sweeps (a halo of 6) in tiles of 52 x up to 48: us per sweep, one launch each / now:
// 128 x 96 4.1 / 0.8, 512 x 384 4.1 / 1.8, 1024 x 768 8.2 / 4.4 (8 sweeps 4.8).
constexpr int kJacobiSweeps = 6;
int grid_jacobi_sweeps() { return kJacobiSweeps; }
void launch_grid_jacobi(const float2* src, float2* dst, const float2* ends, int M, int N, int sweeps, cudaStream_t s) {
  constexpr int NW = 16, MAX_H = 48, ROW = 2 * GW * (int)sizeof(float2);
  const dim3 g = grid_tiles(M, N, kJacobiSweeps, MAX_H);
  const int h = (N - 1 + g.y - 1) / g.y;
  constexpr auto kern = k_grid_jacobi<kJacobiSweeps, NW>;
  allow_smem<kern>((MAX_H + 2 * kJacobiSweeps) * ROW);
  launch_pdl(kern, g, dim3(32 * NW), (size_t)(h + 2 * kJacobiSweeps) * ROW, s, src, dst, ends, M, N, sweeps);
}

int grid_multicolor_sweeps(int M, int N) { return two_sweeps(M, N) ? 2 : 1; }
void launch_grid_multicolor_d(const double2* src, double2* dst, const double2* ends, int M, int N, int sweeps,
                              double omega, uint32_t* move, cudaStream_t s) {
  if (two_sweeps(M, N)) {
    if (M & 1) sweeps_d<6, 2, 16, 32>(src, dst, ends, M, N, sweeps, omega, move, s);
    else sweeps_d<4, 2, 16, 32>(src, dst, ends, M, N, sweeps, omega, move, s);
  } else {
    if (M & 1) sweeps_d<6, 1, 8, 40>(src, dst, ends, M, N, sweeps, omega, move, s);
    else sweeps_d<4, 1, 8, 40>(src, dst, ends, M, N, sweeps, omega, move, s);
  }
}

}  // namespace ausm
