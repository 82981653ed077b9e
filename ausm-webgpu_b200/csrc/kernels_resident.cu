// Resident engine: the n RK3 steps of a step(n) call in one cooperative launch, for grids
// whose tiles all fit on the chip at once.
//
// One CTA keeps one tile for the whole launch: conserved state in registers, Qn, the
// face records, the primitives with their 2-cell halo and the face fluxes in shared
// memory.  Between stages only the two outermost rows and columns of each tile travel,
// as primitives, through a small exchange buffer that stays in L2; a tile waits for the
// edges of its four neighbours and for nothing else.  Global memory sees the state once
// per launch in and once out.
//
// Why: on these grids the stage kernels (kernels_fused.cu) are bound by latency, not by
// work.  Each launch drains the chip, fetches records and state again and waits for the
// last CTA of the grid; a stage of 128 x 96 cells takes 4.1 us and one of 512 x 384 7.0 us
// with about 1.6 us of arithmetic in it.
//
// Exchange: every 8-byte word carries one float and a 32-bit tag (the number of the stage
// that wrote it), so data and its arrival are one transaction and no fence or separate
// flag is needed: a reader polls the words themselves until all tags are the stage's.
// 8-byte accesses are single-copy atomic, so a word is never half old.  Two copies of
// the buffer, by the parity of the tag: a tile writes stage s + 2 only after it has read
// its neighbours' stage s + 1, which they wrote after reading this tile's stage s, so a
// word is never overwritten before it has been read.  Tags go on from launch to launch of
// a buffer, counted on the host, and a buffer is cleared before they would wrap (after 2^32
// stages, an hour and a half of the smallest grids): so whoever uses it next finds none of
// its own tags in cells that only larger launches write.
//
// Every wait is bounded (c_wait_polls); a CTA that gives up sets *err, which the host reads,
// marks its solve and writes nothing; the other tiles of the solve see the mark in their own
// waits.  Other solves of a batch, and later launches while *err is set, are not touched.
//
// Tiling: the grid is cut into ceil(M / 32) x ceil(N / TY) tiles of nearly equal size,
// not into full tiles and a remainder: all tiles of a stage take the same time, and no
// tile is narrower than 4 cells or (for N >= 2) lower than 2, so a tile's halo always
// lies in its direct neighbours.
//
// Two tile heights.  4 rows: warps 0..3 own a row each; while the edges travel they
// evaluate the i-faces of their row that need no halo, then every warp has one more face
// (j-face rows 0..4 and, on the sixth warp, the four i-face columns at the halo), so no
// warp has two in a row.  8 rows: warps 0..3 own two rows each and evaluate their faces
// interleaved, the fifth takes the top row and the right column; more work per warp and
// no early faces (they were 5 % slower there: other CTAs of the SM fill the wait).
//
// Measured on B200 (us per stage; stage kernels at their best height / this one), SLAU2,
// MUSCL:
//     64 x 33    4.35 / 1.25 (4 rows)
//    128 x 96    4.12 / 1.25
//    257 x 131   4.38 / 1.57
//    300 x 220   4.81 / 2.01
//    333 x 250   5.09 / 2.46
//    460 x 340   5.56 / 3.86 (8 rows)
//    512 x 384   6.98 / 4.48   (44 G cell-stages/s)
// (8-row tiles where 4 rows fit: 64 x 33 and 128 x 96 2.1, 257 x 131 2.4, 300 x 220 2.5,
// 333 x 250 2.8.)
// Bound by latency: of some 2400 cycles of a 4-row stage on an idle chip more than half pass
// between publishing an edge and having the neighbours' (two L2 trips, with the early
// faces inside), the rest in equal parts in one face evaluation and in the combination.  At
// 512 x 384 the fullest SM holds 6 tiles and issues about 60 % of the time.
#include <map>
#include <mutex>
#include <type_traits>
#include <vector>

#include "ausm_internal.h"
#include "stage_tile.cuh"
#include "tma.cuh"

namespace ausm {
using namespace tile;

namespace {

constexpr int RW = 4;  // warps that own cells
// ... and warps that fetch the halo and share the last faces: two where each owning warp
// has one row, so that none of them has two faces in a row there
constexpr int aux_warps(int TY) { return TY == 4 ? 2 : 1; }
// Each height is built twice: for one CTA per SM fewer than would fit, with registers to
// interleave more of a face's arithmetic, and for all that fit.  A launch takes the first
// while its tiles fit (us per stage, all that fit / fewer: 128 x 96 1.33 / 1.25, 257 x 131
// 1.61 / 1.57, 300 x 220 2.11 / 2.01; 8 rows: 460 x 340 3.99 / 3.86, 400 x 380 AUSM+-up
// 4.21 / 4.08; three CTAs of 4 rows instead of four gain another 1-2 % on the smallest).
constexpr int few_ctas(int TY) { return TY == 4 ? 4 : 5; }
constexpr int more_ctas(int TY) { return TY == 4 ? 5 : 6; }
constexpr int kMaxTiles4 = more_ctas(4) * 148, kMaxTiles8 = more_ctas(8) * 148;  // tiles of a launch
constexpr int threads_of(int TY) { return 32 * (RW + aux_warps(TY)); }

// Exchange cells of one tile and parity: bottom rows 2 x 32, top rows 2 x 32, left
// columns 2 x TY, right columns 2 x TY; a cell is two 16-byte halves, kept apart so
// that the halves of a row are contiguous.
template <int TY> struct Ex {
  static constexpr int NC = 128 + 4 * TY;
  static constexpr int BOTTOM = 0, TOP = 64, LEFT = 128, RIGHT = 128 + 2 * TY;
  static constexpr size_t TILE = 4 * (size_t)NC;  // 16-byte words of a tile (2 parities x 2 halves)
};

__device__ __forceinline__ unsigned long long tagged(float v, uint32_t tag) {
  return ((unsigned long long)tag << 32) | __float_as_uint(v);
}
__device__ __forceinline__ void st_pair(ulonglong2* p, unsigned long long a, unsigned long long b) {
  asm volatile("st.relaxed.gpu.global.v2.b64 [%0], {%1, %2};" ::"l"(p), "l"(a), "l"(b) : "memory");
}
__device__ __forceinline__ ulonglong2 ld_pair(const ulonglong2* p) {
  ulonglong2 v;
  asm volatile("ld.relaxed.gpu.global.v2.b64 {%0, %1}, [%2];" : "=l"(v.x), "=l"(v.y) : "l"(p) : "memory");
  return v;
}
__device__ __forceinline__ uint32_t tag_of(unsigned long long w) { return (uint32_t)(w >> 32); }
__device__ __forceinline__ float value_of(unsigned long long w) { return __uint_as_float((uint32_t)w); }

struct Tile {
  int i0, w, j0, h, nx, ny, tx, ty;
};
template <int TY> __device__ __forceinline__ Tile tile_of(int M, int N, int t) {
  Tile q;
  q.nx = (M + TX - 1) / TX;
  q.ny = (N + TY - 1) / TY;
  q.ty = t / q.nx;
  q.tx = t - q.ty * q.nx;
  q.i0 = (int)((long long)q.tx * M / q.nx);
  q.w = (int)((long long)(q.tx + 1) * M / q.nx) - q.i0;
  q.j0 = (int)((long long)q.ty * N / q.ny);
  q.h = (int)((long long)(q.ty + 1) * N / q.ny) - q.j0;
  return q;
}

template <int TY> struct Smem {
  float4 P[TY + 4][TX + 4];   // primitives with halo (corners unused)
  float4 Ti[TY][TX + 1];      // face records of the tile
  float4 Tj[TY + 1][TX];
  float4 Fi[TY][TX + 1];      // flux x length of each face
  float4 Fj[TY + 1][TX];
  float4 Qn[TY][TX];          // state at the start of the step
};

constexpr uint32_t kGaveUp = 1u << 16;  // above the most tiles of a launch

// What a CTA of the launch works on (one tile of one solve).
struct Job {
  const float4* Qs;
  float4* Qo;
  const float4* Mi;
  const float4* Mj;
  float* dt;
  uint32_t* wave;  // [0] max wave speed bits, [1] a launch's accumulator, [2] its finished tiles, plus kGaveUp
                   // for each that gave up
  float* out;      // (dt, wave speed) for the host, or null
  int* out_err;    // copy of *err for the host, or null
  int M, N, t;     // t: tile of the solve
};

// ex: the solve's tiles in the exchange buffer; tag0: tag of the state before the first stage.
template <int SF, int TY>
__device__ __forceinline__ void resident_tile(Smem<TY>& sm, const Job& b, const Consts& c, ulonglong2* ex, const uint32_t tag0, int nsteps,
                                              bool first, bool last, int* err) {
  using E = Ex<TY>;
  constexpr int CPT = TY / RW;
  constexpr bool EARLY = TY == 4;
  const int tx = threadIdx.x, ty = threadIdx.y, tid = ty * 32 + tx;
  const int M = b.M, N = b.N;
  const Tile q = tile_of<TY>(M, N, b.t);
  const int w = q.w, h = q.h, i0 = q.i0, j0 = q.j0;
  const bool wall = q.ty == 0, far = q.ty == q.ny - 1;
  const bool owner = ty < RW && tx < w;  // of cells (tx, ty + RW * k)

  // the halo entry this thread fetches: its place in P and the neighbour's exchange cell
  constexpr int AUX = aux_warps(TY);
  int pr, pc, cell, nb;
  bool fetch;
  if (ty < RW) {  // rows -2, -1, h, h + 1
    pr = ty < 2 ? ty : h + ty;
    pc = tx + 2;
    fetch = tx < w && (ty < 2 ? !wall : !far);
    nb = ty < 2 ? b.t - q.nx : b.t + q.nx;
    cell = (ty < 2 ? E::TOP + 32 * ty : E::BOTTOM + 32 * (ty - 2)) + tx;
  } else {  // columns -2, -1, w, w + 1
    const int sel = tx / TY, r = tx % TY;
    pr = r + 2;
    pc = sel < 2 ? sel : w + sel;
    fetch = ty == RW && sel < 4 && r < h;
    nb = sel < 2 ? (q.tx == 0 ? b.t + q.nx - 1 : b.t - 1) : (q.tx == q.nx - 1 ? b.t - q.nx + 1 : b.t + 1);
    cell = (sel < 2 ? E::RIGHT + TY * sel : E::LEFT + TY * (sel - 2)) + r;
  }
  const ulonglong2* const from = ex + (fetch ? (size_t)nb * E::TILE + cell : 0);
  float4* const halo = &sm.P[0][0] + (fetch ? pr * (TX + 4) + pc : 0);
  ulonglong2* mine = ex + (size_t)b.t * E::TILE;
  // The first stage's halo comes from the state itself, except when the launch writes its
  // result over that state: then it is exchanged like any other, so that no tile reads
  // cells that another one writes.
  const bool in_place = b.Qs == b.Qo;

  // face records (the column past the last face wraps through the seam)
  for (int r = ty; r < h; r += RW + AUX)
    for (int cc = tx; cc <= w; cc += 32) sm.Ti[r][cc] = __ldg(&b.Mi[(size_t)(j0 + r) * M + wrap_i(i0 + cc, M)]);
  for (int r = ty; r <= h; r += RW + AUX)
    if (tx < w) sm.Tj[r][tx] = __ldg(&b.Mj[(size_t)(j0 + r) * M + i0 + tx]);
  float4 s[CPT];
#pragma unroll
  for (int k = 0; k < CPT; k++)
    s[k] = owner && ty + RW * k < h ? b.Qs[(size_t)(j0 + ty + RW * k) * M + i0 + tx] : make_float4(1.0f, 0.0f, 0.0f, 1.0f);
  if (fetch && !in_place) *halo = to_prim<true>(b.Qs[(size_t)(j0 - 2 + pr) * M + wrap_i(i0 - 2 + pc, M)], c.gm1);
  const float dt = first ? fminf(c.maxdt, c.cfl / __uint_as_float(b.wave[0])) : *b.dt;
  __syncthreads();  // the records: the ghost rows take their normals from them

  // primitives of an own cell into P (and the ghost rows next to it, boundary pass
  // ausm.js:34-120), and its edges into the exchange buffer when the next stage follows
  const int side = tx < 2 ? E::LEFT + TY * tx : E::RIGHT + TY * (tx - (w - 2));
  const bool at_side = tx < 2 || tx >= w - 2;
  auto own = [&](int r, float4 v, bool put, uint32_t tag) {
    const float4 p = to_prim<true>(v, c.gm1);
    if (put) {
      ulonglong2* e = mine + (tag & 1u) * (2 * E::NC);
      const unsigned long long x = tagged(p.x, tag), y = tagged(p.y, tag), z = tagged(p.z, tag), u = tagged(p.w, tag);
      auto to = [&](ulonglong2* g) {
        st_pair(g, x, y);
        st_pair(g + E::NC, z, u);
      };
      if (r < 2 && !wall) to(e + E::BOTTOM + 32 * r + tx);
      if (r >= h - 2 && !far) to(e + E::TOP + 32 * (r - (h - 2)) + tx);
      if (at_side) to(e + side + r);
    }
    sm.P[r + 2][tx + 2] = p;
    if (wall && r == 0) {
      const float4 g = to_prim<true>(wall_ghost_n<true>(v, sm.Tj[0][tx].x, sm.Tj[0][tx].y), c.gm1);
      sm.P[0][tx + 2] = g;
      sm.P[1][tx + 2] = g;
    }
    if (far && r == h - 1) {
      float4 g1, g2;
      far_ghosts_n<true>(v, sm.Tj[h][tx].x, sm.Tj[h][tx].y, c, g1, g2);
      sm.P[h + 2][tx + 2] = to_prim<true>(g1, c.gm1);
      sm.P[h + 3][tx + 2] = to_prim<true>(g2, c.gm1);
    }
  };
  if (owner) {
#pragma unroll
    for (int k = 0; k < CPT; k++)
      if (ty + RW * k < h) {
        sm.Qn[ty + RW * k][tx] = s[k];
        own(ty + RW * k, s[k], in_place, tag0);
      }
  }

  auto iface = [&](int r, int cc) {
    const float4 m = sm.Ti[r][cc];
    const float4* p = &sm.P[r + 2][cc];
    sm.Fi[r][cc] = face_flux_len<SF>(p[0], p[1], p[2], p[3], m.x, m.y, m.z, c);
  };
  auto jface = [&](int r, int cc) {
    constexpr int PW = TX + 4;
    const float4 m = sm.Tj[r][cc];
    const float4* p = &sm.P[r][cc + 2];
    sm.Fj[r][cc] = face_flux_len<SF>(p[0], p[PW], p[2 * PW], p[3 * PW], m.x, m.y, m.z, c);
  };

  const int stages = 3 * nsteps;
  const float2 dt2 = make_float2(dt, dt), m1 = make_float2(-1.0f, -1.0f);
  bool ok = true;
  int rk = 1;
  for (int st = 0; st < stages; st++) {
    const bool wants = fetch && (st > 0 || in_place);  // the neighbours' edges
    const uint32_t tag = tag0 + st;
    const ulonglong2* e = from + (tag & 1u) * (2 * E::NC);
    const unsigned polls = c_wait_polls * 64u;
    auto gave_up = [&] { return *(volatile uint32_t*)&b.wave[2] >= kGaveUp; };  // a tile of this solve
    auto arrived = [&](ulonglong2 x, ulonglong2 y) {
      if (tag_of(x.x) != tag || tag_of(x.y) != tag || tag_of(y.x) != tag || tag_of(y.y) != tag) return false;
      *halo = make_float4(value_of(x.x), value_of(x.y), value_of(y.x), value_of(y.y));
      return true;
    };
    if constexpr (EARLY) {
      // The edges are asked for in the middle of the early face: by the time the words are
      // read in L2 they have mostly arrived, and the answer is back soon after the face is
      // done (asked for after the face: 7 % more a stage).
      ulonglong2 x{}, y{};
      if (ty < RW) {
        __syncwarp();  // the own row of P
        const bool inner = tx >= 2 && tx <= w - 2;
        float4 L, R;
        if (inner) {
          const float4* p = &sm.P[ty + 2][tx];
          face_states<SF>(p[0], p[1], p[2], p[3], c, L, R);
        }
        if (wants) {
          x = ld_pair(e);
          y = ld_pair(e + E::NC);
        }
        if (inner) {
          const float4 m = sm.Ti[ty][tx];
          sm.Fi[ty][tx] = face_flux_states<SF>(L, R, m.x, m.y, m.z, c);
        }
      } else if (wants) {
        x = ld_pair(e);
        y = ld_pair(e + E::NC);
      }
      if (wants) {
        ok = false;
        for (unsigned it = 0; it < polls; it++) {
          if (arrived(x, y)) {
            ok = true;
            break;
          }
          if ((it & 1023u) == 1023u && gave_up()) break;
          x = ld_pair(e);
          y = ld_pair(e + E::NC);
        }
      }
    } else if (wants) {
      ok = false;
      for (unsigned it = 0; it < polls; it++) {
        const ulonglong2 x = ld_pair(e), y = ld_pair(e + E::NC);
        if (arrived(x, y)) {
          ok = true;
          break;
        }
        if ((it & 1023u) == 1023u && gave_up()) break;
      }
    }
    if (__syncthreads_or(!ok)) {  // P is complete, or a wait gave up
      if (tid == 0) {
        atomicExch(err, 1);
        atomicAdd(&b.wave[2], kGaveUp);
      }
      ok = false;
      break;
    }
    if constexpr (EARLY) {
      if (ty <= RW) {
        if (tx < w && ty <= h) jface(ty, tx);
      } else {
        const int sel = tx / TY, r = tx % TY;  // i-face columns 0, 1, w - 1, w
        if (sel < 4 && r < h) iface(r, sel < 2 ? sel : w - 3 + sel);
      }
    } else if (ty < RW) {
      if (tx < w) {
#pragma unroll
        for (int k = 0; k < CPT; k++)
          if (ty + RW * k < h) {
            iface(ty + RW * k, tx);
            jface(ty + RW * k, tx);
          }
      }
    } else {
      if (tx < h) iface(tx, w);
      if (tx < w) jface(h, tx);
    }
    __syncthreads();
    const bool end = st == stages - 1;
    if (owner) {
#pragma unroll
      for (int k = 0; k < CPT; k++) {
        const int r = ty + RW * k;
        if (r < h) {
          const float iA = sm.Ti[r][tx].w;
          const float2 niA = make_float2(-iA, -iA);
          const float4 fl = sm.Fi[r][tx], fr = sm.Fi[r][tx + 1], fd = sm.Fj[r][tx], fu = sm.Fj[r + 1][tx];
          // as combine_phase (stage_tile.cuh)
          const float2 R01 = mul2(fma2(lo2(fd), m1, add2(fma2(lo2(fl), m1, lo2(fr)), lo2(fu))), niA);
          const float2 R23 = mul2(fma2(hi2(fd), m1, add2(fma2(hi2(fl), m1, hi2(fr)), hi2(fu))), niA);
          float2 o01 = fma2(dt2, R01, lo2(s[k])), o23 = fma2(dt2, R23, hi2(s[k]));
          if (rk == 2) {
            const float4 n = sm.Qn[r][tx];
            const float2 c25 = make_float2(0.25f, 0.25f), c75 = make_float2(0.75f, 0.75f);
            o01 = fma2(c75, lo2(n), mul2(c25, o01));
            o23 = fma2(c75, hi2(n), mul2(c25, o23));
          } else if (rk == 3) {
            const float4 n = sm.Qn[r][tx];
            const float2 two = make_float2(2.0f, 2.0f);
            o01 = div3(fma2(two, o01, lo2(n)));
            o23 = div3(fma2(two, o23, hi2(n)));
          }
          s[k] = make_float4(o01.x, o01.y, o23.x, o23.y);
          if (!end) {
            own(r, s[k], true, tag0 + st + 1);
            if (rk == 3) sm.Qn[r][tx] = s[k];
          }
        }
      }
    }
    rk = rk == 3 ? 1 : rk + 1;
  }

  uint32_t wmax = 0u;
  if (ok && owner) {
#pragma unroll
    for (int k = 0; k < CPT; k++) {
      const int r = ty + RW * k;
      if (r < h) {
        b.Qo[(size_t)(j0 + r) * M + i0 + tx] = s[k];
        if (last) wmax = max(wmax, __float_as_uint(wave_speed_w<true>(s[k], sm.Tj[r][tx].w, c.gamma)));
      }
    }
  }
  // Every tile of the solve has read wave[0] by the time the last one gets here; that one
  // publishes the max wave speed of the new state (none if a tile gave up).  Accumulator and
  // count are zero again for the next launch, also when a wait gave up.
  if (last) block_max_to(&b.wave[1], wmax);
  if (tid == 0) {
    __threadfence();
    const uint32_t done = atomicAdd(&b.wave[2], 1u);
    if ((done & (kGaveUp - 1)) == (uint32_t)(q.nx * q.ny) - 1) {
      __threadfence();
      b.wave[2] = 0u;
      *b.dt = dt;
      if (last) {
        const uint32_t bits = atomicExch(&b.wave[1], 0u);
        if (done < kGaveUp) b.wave[0] = bits;
        if (b.out) {
          b.out[0] = dt;
          b.out[1] = __uint_as_float(bits);
        }
      }
      if (b.out_err) *b.out_err = *(volatile int*)err;
    }
  }
}

// OCC: CTAs per SM the registers are sized for (few_ctas and more_ctas above).
template <int SF, int TY, int OCC>
__global__ void __launch_bounds__(threads_of(TY), OCC)
    k_resident(const float4* Qs, float4* Qo, const float4* __restrict__ Mi, const float4* __restrict__ Mj, float* dt,
               uint32_t* wave, ulonglong2* ex, const uint32_t tag0, const int nsteps, const int first, const int last, float* out, int* out_err, int* err, const Consts c,
               const int M, const int N) {
  __shared__ Smem<TY> sm;
  const Job b = {Qs, Qo, Mi, Mj, dt, wave, out, out_err, M, N, (int)blockIdx.x};
  resident_tile<SF, TY>(sm, b, c, ex, tag0, nsteps, first != 0, last != 0, err);
}

// All solves of a batch in one launch: items[blockIdx.x] is a solve and one of its tiles.
// The schemes are separate bodies, chosen once per CTA, so that the registers are those
// of the largest one.
template <int TY, int OCC>
__global__ void __launch_bounds__(threads_of(TY), OCC)
    k_resident_batch(const BatchSolve* __restrict__ solves, const int2* __restrict__ items, ulonglong2* ex,
                     const uint32_t tag0, const int nsteps, const int first, const int last, int* err) {
  __shared__ Smem<TY> sm;
  const int2 it = items[blockIdx.x];
  const BatchSolve& d = solves[it.x];
  const Consts c = d.c;
  const Job b = {d.Q[d.cur], d.Q[(d.cur + nsteps) % 3], d.Mi, d.Mj, d.dt, d.wave, nullptr, nullptr, d.M, d.N, it.y};
  auto go = [&](auto sf) {
    resident_tile<decltype(sf)::value, TY>(sm, b, c, ex + (size_t)d.rtile0 * Ex<TY>::TILE, tag0, nsteps, first != 0,
                                           last != 0, err);
  };
  switch (d.scheme) {
    case 0: go(std::integral_constant<int, 0>()); break;
    case 1: go(std::integral_constant<int, 1>()); break;
    case 2: go(std::integral_constant<int, 2>()); break;
    case 4: go(std::integral_constant<int, 4>()); break;
    case 5: go(std::integral_constant<int, 5>()); break;
    default: go(std::integral_constant<int, 6>());
  }
}

template <int TY> int tiles_of(int M, int N) { return ((M + TX - 1) / TX) * ((N + TY - 1) / TY); }

// CTAs of `kern` the current device holds at once (0 when cooperative launches are not
// available).
int resident_ctas(const void* kern, int threads) {
  int dev = 0, sms = 0, per = 0, coop = 0;
  if (cudaGetDevice(&dev) != cudaSuccess) return 0;
  if (cudaDeviceGetAttribute(&coop, cudaDevAttrCooperativeLaunch, dev) != cudaSuccess || !coop) return 0;
  if (cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess) return 0;
  if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per, kern, threads, 0) != cudaSuccess) return 0;
  return sms * per;
}

using Kern = void (*)(const float4*, float4*, const float4*, const float4*, float*, uint32_t*, ulonglong2*, uint32_t, int,
                      int, int, float*, int*, int*, Consts, int, int);
template <int TY, int OCC> Kern kernel_of(int sf) {
  switch (sf) {
    case 0: return k_resident<0, TY, OCC>;
    case 1: return k_resident<1, TY, OCC>;
    case 2: return k_resident<2, TY, OCC>;
    case 4: return k_resident<4, TY, OCC>;
    case 5: return k_resident<5, TY, OCC>;
    default: return k_resident<6, TY, OCC>;
  }
}
// Tiles of height TY a launch can take, by the kernels built for OCC CTAs per SM (every
// scheme's is built for the same).
template <int TY, int OCC> int capacity() {
  static const int n = std::min(resident_ctas((const void*)k_resident<4, TY, OCC>, threads_of(TY)),
                                resident_ctas((const void*)k_resident_batch<TY, OCC>, threads_of(TY)));
  return n;
}
template <int TY> bool few(int tiles) { return tiles <= capacity<TY, few_ctas(TY)>(); }
template <int TY> Kern kernel_of(int sf, int tiles) {
  return few<TY>(tiles) ? kernel_of<TY, few_ctas(TY)>(sf) : kernel_of<TY, more_ctas(TY)>(sf);
}

}  // namespace

int resident_tiles(int M, int N, int rows) { return rows == 4 ? tiles_of<4>(M, N) : tiles_of<8>(M, N); }

// 4 rows wherever all tiles fit at that height (740 tiles of 128 cells on 148 SMs): the
// lower tiles have the shorter stage at every size that fits (table above).  8 rows up to
// 888 tiles (227 K cells); beyond, a CTA would have to work on several tiles in turn.
int resident_rows(int tiles4, int tiles8) {
  if (tiles4 <= std::min(capacity<4, more_ctas(4)>(), kMaxTiles4)) return 4;
  return tiles8 <= std::min(capacity<8, more_ctas(8)>(), kMaxTiles8) ? 8 : 0;
}

// ---- exchange buffers ----
// A launch needs one for its own duration only, so they are kept for the process and not
// per solve (a solve would hold up to 72 bytes a cell for it): at most kMaxBuffers per
// device, created with a solver or a batch for which none is large enough, so that its steps
// allocate nothing, and as launches overlap; freed with the device's last solver, batch or
// server.  A launch takes, of those that are large enough, the buffer its stream used last,
// or one whose last launch is over, or waits (on the device) for the oldest.  A device without the memory for a first buffer refuses
// the launch, and the caller steps by the stage kernels, which need none.
namespace {
constexpr int kMaxBuffers = 8;
// Up to 9.1 MB, 10 MiB with the rounding.  Sizes up to 1 MiB share mappings with other small arrays (1 us to allocate
// instead of 340), larger ones take whole mappings of 2 MiB.
size_t bytes_of(int tiles, int rows) {
  const size_t need = 16 * tiles * (rows == 4 ? Ex<4>::TILE : Ex<8>::TILE), unit = need <= (1u << 20) ? 1u << 18 : 1u << 21;
  return (need + unit - 1) / unit * unit;
}
struct Buffer {
  ulonglong2* p = nullptr;
  size_t bytes = 0;
  uint32_t tag = 1;  // of the next launch's first exchange; 0 is that of a cleared buffer
  cudaEvent_t done = nullptr;
  cudaStream_t stream = nullptr;
  uint64_t used = 0;
};
struct Pool {
  int users = 0;
  uint64_t clock = 0;
  std::vector<Buffer> buffers;
};
std::mutex g_pool_mu;
std::map<int, Pool> g_pool;  // per device

void free_buffer(Buffer& b) {
  cudaEventSynchronize(b.done);
  cudaFree(b.p);
  cudaEventDestroy(b.done);
}

// One more buffer, cleared on s.  With g_pool_mu held and the device current.
cudaError_t add_buffer(Pool& pool, size_t bytes, cudaStream_t s) {
  Buffer b;
  b.bytes = bytes;
  cudaError_t e = cudaMalloc((void**)&b.p, bytes);
  if (e == cudaSuccess) e = cudaEventCreateWithFlags(&b.done, cudaEventDisableTiming);
  if (e == cudaSuccess) e = cudaMemsetAsync(b.p, 0, bytes, s);
  if (e == cudaSuccess) e = cudaEventRecord(b.done, s);
  if (e != cudaSuccess) {
    if (b.done) cudaEventDestroy(b.done);
    if (b.p) cudaFree(b.p);
    return e;
  }
  b.stream = s;
  pool.buffers.push_back(b);
  return cudaSuccess;
}

// A buffer of at least `bytes` for a launch of `stages` stages on s.  With g_pool_mu held and
// the device current.
cudaError_t take(Pool& pool, cudaStream_t s, size_t bytes, uint32_t stages, Buffer** out) {
  Buffer *best = nullptr, *oldest = nullptr;  // oldest: of those large enough
  for (Buffer& b : pool.buffers)
    if (b.bytes >= bytes) {
      if (b.stream == s) best = &b;
      if (!oldest || b.used < oldest->used) oldest = &b;
    }
  if (!best)
    for (Buffer& b : pool.buffers) {
      if (best) break;
      if (b.bytes < bytes) continue;
      if (cudaEventQuery(b.done) == cudaSuccess) best = &b;
      else cudaGetLastError();  // busy, or not to be asked now: not an error of this thread's calls
    }
  if (!best && ((int)pool.buffers.size() < kMaxBuffers || !oldest)) {
    if ((int)pool.buffers.size() == kMaxBuffers) {  // all too small: the one unused for longest makes room
      auto b = std::min_element(pool.buffers.begin(), pool.buffers.end(),
                                [](const Buffer& x, const Buffer& y) { return x.used < y.used; });
      free_buffer(*b);
      pool.buffers.erase(b);
    }
    const cudaError_t e = add_buffer(pool, bytes, s);
    if (e == cudaSuccess) {
      best = &pool.buffers.back();
    } else {
      if (e != cudaErrorMemoryAllocation || !oldest) return e;
      cudaGetLastError();  // no memory for one more: share those there are
    }
  }
  if (!best) {
    best = oldest;
    const cudaError_t e = cudaStreamWaitEvent(s, best->done, 0);
    if (e != cudaSuccess) return e;
  }
  best->stream = s;
  best->used = ++pool.clock;
  if (best->tag > UINT32_MAX - stages) {  // the tags would wrap: start again on a cleared buffer
    const cudaError_t e = cudaMemsetAsync(best->p, 0, best->bytes, s);
    if (e != cudaSuccess) return e;
    best->tag = 1;
  }
  *out = best;
  return cudaSuccess;
}

template <class... KArgs, class... Args>
cudaError_t launch_coop(void (*kern)(KArgs...), int ctas, int threads, cudaStream_t s, Args&&... args) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(ctas);
  cfg.blockDim = dim3(32, threads / 32);
  cfg.stream = s;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeCooperative;
  attr[0].val.cooperative = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  return cudaLaunchKernelEx(&cfg, kern, static_cast<Args&&>(args)...);
}

// Takes a buffer of the current device for `nsteps` steps of `tiles` tiles on s, calls
// launch(cells, first tag), notes when the buffer is free.  None of it belongs to a stream capture another
// thread may have open.
template <class F> cudaError_t with_buffer(cudaStream_t s, int tiles, int rows, int nsteps, F launch) {
  int dev = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e != cudaSuccess) return e;
  cudaStreamCaptureMode mode = cudaStreamCaptureModeRelaxed;
  cudaThreadExchangeStreamCaptureMode(&mode);
  {
    std::lock_guard<std::mutex> lk(g_pool_mu);
    Buffer* b = nullptr;
    e = take(g_pool[dev], s, bytes_of(tiles, rows), 3u * nsteps, &b);
    if (e == cudaSuccess) {
      e = launch(b->p, b->tag);
      if (e == cudaSuccess) b->tag += 3u * nsteps;
      const cudaError_t e2 = cudaEventRecord(b->done, s);
      if (e == cudaSuccess) e = e2;
    }
  }
  cudaThreadExchangeStreamCaptureMode(&mode);
  return e;
}
}  // namespace

void set_exchange_tag(int dev, uint32_t tag) {
  std::lock_guard<std::mutex> lk(g_pool_mu);
  for (Buffer& b : g_pool[dev].buffers) b.tag = std::max(tag, 1u);
}

void resident_user(int dev, int change) {
  std::lock_guard<std::mutex> lk(g_pool_mu);
  Pool& pool = g_pool[dev];
  pool.users += change;
  if (pool.users > 0) return;
  for (Buffer& b : pool.buffers) free_buffer(b);
  pool.buffers.clear();
}

void resident_reserve(int dev, int tiles, int rows, cudaStream_t s) {
  std::lock_guard<std::mutex> lk(g_pool_mu);
  Pool& pool = g_pool[dev];
  const size_t bytes = bytes_of(tiles, rows);
  if ((int)pool.buffers.size() == kMaxBuffers) return;
  for (const Buffer& b : pool.buffers)
    if (b.bytes >= bytes) return;
  if (add_buffer(pool, bytes, s) != cudaSuccess) cudaGetLastError();  // a step will ask again
}

cudaError_t launch_resident(int scheme, const float4* Qs, float4* Qo, const float4* Mi, const float4* Mj, float* dt,
                            uint32_t* wave, int rows, int nsteps, bool first, bool last, float* out, int* out_err,
                            int* err, const Consts& c, int M, int N, cudaStream_t s) {
  const int sf = scheme + (c.muscl > 0 ? 4 : 0), tiles = resident_tiles(M, N, rows);
  return with_buffer(s, tiles, rows, nsteps, [&](ulonglong2* ex, uint32_t tag0) {
    return launch_coop(rows == 4 ? kernel_of<4>(sf, tiles) : kernel_of<8>(sf, tiles), tiles, threads_of(rows), s, Qs,
                       Qo, Mi, Mj, dt, wave, ex, tag0, nsteps, (int)first, (int)last, out, out_err, err, c, M, N);
  });
}

cudaError_t launch_resident_batch(const BatchSolve* solves, const int2* items, int tiles, int rows, int nsteps,
                                  bool first, bool last, int* err, cudaStream_t s) {
  return with_buffer(s, tiles, rows, nsteps, [&](ulonglong2* ex, uint32_t tag0) {
    auto k = rows == 4 ? (few<4>(tiles) ? k_resident_batch<4, few_ctas(4)> : k_resident_batch<4, more_ctas(4)>)
                       : (few<8>(tiles) ? k_resident_batch<8, few_ctas(8)> : k_resident_batch<8, more_ctas(8)>);
    return launch_coop(k, tiles, threads_of(rows), s, solves, items, ex, tag0, nsteps, (int)first, (int)last, err);
  });
}

bool resident_refused(cudaError_t e) {
  if (e != cudaErrorCooperativeLaunchTooLarge && e != cudaErrorMemoryAllocation) return false;
  cudaGetLastError();
  return true;
}

cudaError_t set_wait_polls_resident(unsigned polls) { return cudaMemcpyToSymbol(c_wait_polls, &polls, sizeof polls); }

}  // namespace ausm
