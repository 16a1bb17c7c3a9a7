// Plain compensated DD matmul on the FP64 pipe (real and complex), plus the
// matrix-vector forms.
//
// Semantics (src/float64x2/matmul.inc:6-239): C(m,n) = A(m,k) * B(k,n),
// column-major, leading dimension = first extent, C overwritten.  For every
// output the reference runs mac_inl(A[i,p], B[p,j]) for p = 0..k-1 in order,
// renormalises after each full chunk of `renorm_interval` steps when more
// steps remain, and renormalises once at the end.  The kernels below keep the
// k-loop of each output sequential and reproduce that cadence, so results are
// bit-identical to matmuldd_mm / _mv / _vm.  The complex kernel reproduces the
// Fortran cdd_matmul_mm (fsrc/multifloats.fypp:2609-2621): four real products
// rr, ii, ri, ir accumulated side by side, then re = rr - ii, im = ri + ir with
// the DD operators.
//
// Tiling: a 256-thread CTA owns a square output tile of edge 64, 32 or 16 (32
// or 16 complex); each thread owns a register tile of (s_hi, s_lo)
// accumulators.  A and B k-slices are staged in shared memory with cp.async
// (16-byte copies, zero-filled past the matrix edge) in a two-stage ring.
// Bound: FP64 pipe, 13 FP64 instructions per MAC plus 6 per renormalisation.
// Which tiles a product is cut into is decided by pick_tiles.
#include "common.cuh"
#include "dd_device.cuh"
#include "gemm_tile.cuh"

namespace mfcuda {

using gtile::load_dd;
using gtile::cp_async_commit;
using gtile::cp_async_wait_all;

// ---------------------------------------------------------------------------
// Cutting a product into tiles.  The k loop of an output cannot be split (the
// MAC order is fixed), so a product fills the chip only by its output tiles,
// and the SM that gets one tile more than the others sets the time.  A tile
// of edge E costs (start + n per_tile) k for the n tiles of the busiest SM,
// measured at k = 1024 on 148 SMs (in units of 0.1 ns per step: real tiles
// of 64 / 32 / 16: 300 + 5000 n, 150 + 1320 n, 110 + 385 n; complex tiles of
// 32 / 16: 300 + 5100 n, 270 + 1335 n): a small tile loses 5-20 % per MAC but
// quantises better.  Candidates: every tile of one edge, or the largest edge
// for the whole rounds over the SMs and the remaining tiles cut into 4 or 16
// (run at the large tile's two CTAs per SM: 1390 / 433, complex 1460).  The
// cheapest one is launched.  256^3: 16 tiles of 64 took 180 us, 256 of 16
// take 25 us; 1531 x 977 x 1203: 456 tiles of 64 took 2.34 ms, 444 of them and
// 192 of 16 take 1.56 ms.
// ---------------------------------------------------------------------------
constexpr int kThreads = gtile::kThreads;

struct TilePick {
  int edge;        // of the uniform tiles, or of the whole ones
  int64_t blocks;  // grid
  int64_t whole;   // mixed: this many whole tiles, then the rest cut into `cut` pieces
  int cut;         // 0: uniform
};
struct TileCost {
  int64_t start, per_tile;
};
// Tiles of the edges 16 TMAX, 8 TMAX, ... 16 with their costs, largest first.
static TilePick pick_tiles(int64_t m, int64_t n, const TileCost *cost, int nedges, const int64_t *cut_cost) {
  const int64_t sms = sm_count();
  auto tiles = [&](int e) { return ((m + e - 1) / e) * ((n + e - 1) / e); };
  const int top = 16 << (nedges - 1);
  TilePick best = {0, 0, 0, 0};
  int64_t best_cost = INT64_MAX;
  for (int i = 0; i < nedges; ++i) {
    const int64_t t = tiles(top >> i), c = cost[i].start + (t + sms - 1) / sms * cost[i].per_tile;
    if (c < best_cost && t <= INT32_MAX) {
      best_cost = c;
      best = {top >> i, t, 0, 0};
    }
  }
  const int64_t t = tiles(top), rounds = t / sms, rest = t % sms;
  for (int i = 1; i < nedges && rounds > 0 && rest > 0; ++i) {
    const int64_t pieces = rest << (2 * i);
    const int64_t c = cost[0].start + rounds * cost[0].per_tile + (pieces + sms - 1) / sms * cut_cost[i - 1];
    if (c < best_cost && t <= INT32_MAX) {
      best_cost = c;
      best = {top, rounds * sms + pieces, rounds * sms, 1 << (2 * i)};
    }
  }
  return best;
}
constexpr TileCost kRealCost[3] = {{300, 5000}, {150, 1320}, {110, 385}};
constexpr int64_t kRealCutCost[2] = {1390, 433};
constexpr TileCost kCplxCost[2] = {{300, 5100}, {270, 1335}};
constexpr int64_t kCplxCutCost[1] = {1460};

// Origin of block b's tile among tiles of edge E, gx of them along M.
__device__ __forceinline__ void tile_origin(int64_t b, int64_t gx, int E, int64_t &m0, int64_t &n0) {
  m0 = b % gx * E;
  n0 = b / gx * E;
}
// Piece q of the tile at (m0, n0) cut into side x side pieces of edge E.
__device__ __forceinline__ void piece_origin(int q, int side, int E, int64_t &m0, int64_t &n0) {
  m0 += q % side * E;
  n0 += q / side * E;
}

// ---------------------------------------------------------------------------
// Real GEMM.  Mixed: blocks 0 .. whole - 1 own a 64 x 64 tile (4 x 4 outputs
// per thread), the others a piece of the tiles after those.
// ---------------------------------------------------------------------------
template <bool ALIGNED, bool SHORT>
__global__ void __launch_bounds__(kThreads, 2)
    gemm_dd_kernel(const double *__restrict__ A, const double *__restrict__ B,
                   double *__restrict__ C, int64_t M, int64_t K, int64_t N, int64_t ri,
                   int64_t whole, int cut) {
  __shared__ gtile::Smem sm;
  const int64_t gx = (M + 63) / 64;
  int64_t b = blockIdx.x, m0, n0;
  if (b < whole) {
    tile_origin(b, gx, 64, m0, n0);
    gtile::gemm_tile<4, 4, ALIGNED, SHORT>(A, B, C, M, K, N, ri, m0, n0, sm);
    return;
  }
  b -= whole;
  const int q = (int)(b % cut);
  tile_origin(whole + b / cut, gx, 64, m0, n0);
  if (cut == 4) {
    piece_origin(q, 2, 32, m0, n0);
    if (m0 < M && n0 < N) gtile::gemm_tile<2, 2, ALIGNED, SHORT>(A, B, C, M, K, N, ri, m0, n0, sm);
  } else {
    piece_origin(q, 4, 16, m0, n0);
    if (m0 < M && n0 < N) gtile::gemm_tile<1, 1, ALIGNED, SHORT>(A, B, C, M, K, N, ri, m0, n0, sm);
  }
}
// Uniform tiles of edge 16 T (three CTAs of edge 32 per SM, four of edge 16).
template <int T, bool ALIGNED, bool SHORT>
__global__ void __launch_bounds__(kThreads, T == 2 ? 3 : 4)
    gemm_dd_small_kernel(const double *__restrict__ A, const double *__restrict__ B,
                         double *__restrict__ C, int64_t M, int64_t K, int64_t N, int64_t ri) {
  __shared__ gtile::Smem sm;
  int64_t m0, n0;
  tile_origin(blockIdx.x, (M + 16 * T - 1) / (16 * T), 16 * T, m0, n0);
  gtile::gemm_tile<T, T, ALIGNED, SHORT>(A, B, C, M, K, N, ri, m0, n0, sm);
}

// ---------------------------------------------------------------------------
// Complex GEMM (gtile::cgemm_tile): the same with tiles of 32 and 16.
// ---------------------------------------------------------------------------
template <bool ALIGNED, bool SHORT>
__global__ void __launch_bounds__(kThreads, 2)
    cgemm_dd_kernel(const double *__restrict__ A, const double *__restrict__ B,
                    double *__restrict__ C, int64_t M, int64_t K, int64_t N, int64_t ri,
                    int64_t whole, int cut) {
  __shared__ gtile::CSmem sm;
  const int64_t gx = (M + 31) / 32;
  int64_t b = blockIdx.x, m0, n0;
  if (b < whole) {
    tile_origin(b, gx, 32, m0, n0);
    gtile::cgemm_tile<2, 2, ALIGNED, SHORT>(A, B, C, M, K, N, ri, m0, n0, sm);
    return;
  }
  b -= whole;
  tile_origin(whole + b / cut, gx, 32, m0, n0);
  piece_origin((int)(b % cut), 2, 16, m0, n0);
  if (m0 < M && n0 < N) gtile::cgemm_tile<1, 1, ALIGNED, SHORT>(A, B, C, M, K, N, ri, m0, n0, sm);
}
template <bool ALIGNED, bool SHORT>
__global__ void __launch_bounds__(kThreads, 4)
    cgemm_dd_small_kernel(const double *__restrict__ A, const double *__restrict__ B,
                          double *__restrict__ C, int64_t M, int64_t K, int64_t N, int64_t ri) {
  __shared__ gtile::CSmem sm;
  int64_t m0, n0;
  tile_origin(blockIdx.x, (M + 15) / 16, 16, m0, n0);
  gtile::cgemm_tile<1, 1, ALIGNED, SHORT>(A, B, C, M, K, N, ri, m0, n0, sm);
}

// ---------------------------------------------------------------------------
// Matrix-vector forms.  Every output keeps the reference's sequential MAC over
// p = 0..k-1, so there is one dependency chain per output and only a few
// thousand of them; a CTA owns 32 outputs and splits each MAC
// (matmul.inc:6-19) in two:
//   * eight producer warps stream the matrix (a stage is 32 outputs x 32 k, four
//     columns of it per warp, P stages ahead in registers) and compute the
//     accumulator-independent part of every MAC, p = ah*bh and
//     q = fma(ah,bh,-p) + fma(ah,bl,al*bh), into a double-buffered array;
//   * one warp runs the accumulator chain (two_sum of s_hi with p, then
//     s_lo += q + (aerr + berr)) and the renorm cadence, lane = output.
// The operations and their order per output are the reference's, so results
// are bit-identical; the warps hand over through one named barrier per stage.
//
// Bound: the chain, 15 dependent additions of 8 cycles per eight steps and 62
// FP64 instructions; as compiled it takes 28-32 cycles a step, where HBM at one
// CTA per SM would take 19.  So the chain warp has a scheduler to itself (the
// producers use the other three; the roles rotate with the wave of CTAs, so
// that the chains of the CTAs of one SM land on different schedulers), no
// test between its steps in the default cadence, and the shared memory nearly
// to itself: with the matrix staged there too, its traffic cost the chain a
// quarter of its time.  The matrix reaches the registers through L2, where each
// producer prefetches its columns eight stages ahead (none: a third slower; 24
// ahead of 16384 rows: likewise).  P = 4 stages (one CTA per SM) when the outputs are one wave, 2 (two
// CTAs) otherwise.
// Inputs not in L2: 4099 x 3001 144 -> 49 us (y = A x), 142 -> 48 (y = x A); 200
// x 6000 278 -> 85; 16384 x 8192 904 -> 353, 866 -> 351 (HBM alone 328).
// ---------------------------------------------------------------------------
constexpr int kGvN = 32, kGvK = 32;
constexpr int kGvWarps = 12, kGvThreads = 32 * kGvWarps;  // chain, eight producers, three without work
constexpr int kGvProd = 8, kGvActive = 32 * (1 + kGvProd);
// Row of the term array, padded for the producers of y = x B, which write it
// transposed (and the same for both: the chain's code is then one).
constexpr int kGvPitch = 33;
constexpr int kGvAhead = 8;   // stages of the matrix ahead in L2
constexpr int kGvXStages = 8;  // stages of the vector in flight

template <int N>
__device__ __forceinline__ void cp_async_wait_n() {
  asm volatile("cp.async.wait_group %0;\n" ::"n"(N));
}

// The accumulator half of mac_inl for one output: p and q from the producers.
__device__ __forceinline__ void mac_chain(double p, double q, double &s_hi, double &s_lo) {
  double t = mfdev::add(s_hi, p);
  double bp = mfdev::sub(t, s_hi);
  double ap = mfdev::sub(t, bp);
  double aerr = mfdev::sub(s_hi, ap);
  double berr = mfdev::sub(p, bp);
  s_lo = mfdev::add(s_lo, mfdev::add(q, mfdev::add(aerr, berr)));
  s_hi = t;
}
// The accumulator-independent half: p = ah bh, q = e + cross (same operations as mac).
__device__ __forceinline__ double2 mac_terms(double ah, double al, double bh, double bl) {
  double p = mfdev::mul(ah, bh);
  double e = mfdev::fma_(ah, bh, -p);
  double cross = mfdev::fma_(ah, bl, mfdev::mul(al, bh));
  return make_double2(p, mfdev::add(e, cross));
}

// Runs the chain over a whole stage with a renormalisation after every group of
// eight steps.
template <int PITCH>
__device__ __forceinline__ void chain_groups(const double2 *__restrict__ v, double &sh, double &sl) {
  constexpr int G = gtile::kGroup;
#pragma unroll
  for (int g = 0; g < kGvK / G; ++g) {
    double2 u[G];
#pragma unroll
    for (int r = 0; r < G; ++r) u[r] = v[(g * G + r) * PITCH];
#pragma unroll
    for (int r = 0; r < G; ++r) mac_chain(u[r].x, u[r].y, sh, sl);
    mfdev::renorm(sh, sl);
  }
}
// Runs the chain over cmax terms of a stage that starts at step p0 (v: this
// lane's column of the term array), renorm cadence as in the reference: after
// each full chunk of ri steps when more remain.
template <int PITCH>
__device__ __forceinline__ void chain_stage(const double2 *__restrict__ v, int cmax, int64_t p0, int64_t K,
                                            gtile::Cadence &cad, double &sh, double &sl) {
  constexpr int G = gtile::kGroup;
  auto group = [&](int c) {
    double2 u[G];
#pragma unroll
    for (int r = 0; r < G; ++r) u[r] = v[(c + r) * PITCH];
#pragma unroll
    for (int r = 0; r < G; ++r) mac_chain(u[r].x, u[r].y, sh, sl);
    if (cad.ends(G) && p0 + c + G < K) mfdev::renorm(sh, sl);
  };
  int c = 0;
  if (cad.grouped) {
#pragma unroll 1
    for (; c + G <= cmax; c += G) group(c);
  }
  while (c < cmax) {  // the steps up to the next chunk's end
    const int run = cad.run(cmax - c);
    const double2 *w = v + c * PITCH;
#pragma unroll 4
    for (int r = 0; r < run; ++r) mac_chain(w[r * PITCH].x, w[r * PITCH].y, sh, sl);
    c += run;
    if (cad.ends(run) && p0 + c < K) mfdev::renorm(sh, sl);
  }
}

// VM false: y(M) = A(M,K) x(K) (gaxpy_mv_panel, matmul.inc:47-88; A is the
// MAC's first operand); a stage is 32 columns of A, 32 rows (512 contiguous
// bytes) each.  VM true: y(M) = x(K) A(K,M) (vm_impl, matmul.inc:213-239; x is
// the MAC's first operand); a stage is 32 columns (outputs), 32 k each.
template <bool VM, int P, bool ALIGNED>
__global__ void __launch_bounds__(kGvThreads, P > 2 ? 1 : 2) gemv_dd_kernel(const double *__restrict__ A,
                                                                            const double *__restrict__ x,
                                                                            double *__restrict__ y, int64_t M,
                                                                            int64_t K, int64_t ri, int sms) {
  constexpr int PITCH = kGvPitch, S = kGvXStages;
  __shared__ __align__(16) double2 xs[S * kGvK];           // [stage][k] of the vector
  __shared__ __align__(16) double2 pq[2 * kGvK * PITCH];   // [2][k][output]
  const int lane = threadIdx.x & 31;
  // role 0: chain; 4 and 8, which share its scheduler, and 11: none; else a producer
  const int rot = (int)(blockIdx.x / (unsigned)sms) & 3;
  const int role = ((int)(threadIdx.x >> 5) + kGvWarps - rot) % kGvWarps;
  if (role == 4 || role == 8 || role == 11) return;
  auto sync = [] { asm volatile("bar.sync 1, %0;" ::"n"(kGvActive) : "memory"); };
  const int64_t i0 = (int64_t)blockIdx.x * kGvN;
  const int64_t nst = (K + kGvK - 1) / kGvK;

  if (role == 0) {  // ---- accumulator chain
    double sh = 0.0, sl = 0.0;
    gtile::Cadence cad(ri);
    sync();  // the vector's first stage landed
    sync();  // the terms of stage 0 are ready
    // stages with more steps after them in the default cadence: no tests at all
    const int64_t plain = cad.ri == gtile::kGroup ? (K - 1) / kGvK : 0;
    const double2 *v = pq + lane;
    int64_t st = 0;
    for (; st < plain; ++st) {
      chain_groups<PITCH>(v + (st & 1) * kGvK * PITCH, sh, sl);
      sync();
    }
    for (; st < nst; ++st) {
      const int64_t p0 = st * kGvK;
      const int cmax = (K - p0) < kGvK ? (int)(K - p0) : kGvK;
      chain_stage<PITCH>(v + (st & 1) * kGvK * PITCH, cmax, p0, K, cad, sh, sl);
      sync();
    }
    const int64_t i = i0 + lane;
    if (i < M) {
      mfdev::renorm(sh, sl);
      y[2 * i] = sh;
      y[2 * i + 1] = sl;
    }
    return;
  }
  // ---- producer w: the columns w, w + 8, w + 16, w + 24 of every stage
  constexpr int COLS = kGvN / kGvProd;
  const int w = role < 4 ? role - 1 : role < 8 ? role - 2 : role - 3;
  // (not evict-first: a column of odd length starts inside a 128-byte line, and
  // the CTA that shares it comes a little later -- 4099 x 3001 64 instead of 49 us)
  auto load = [&](int64_t st, double2 (&a)[COLS]) {
    const int64_t p0 = st * kGvK;
    const double *src = VM ? A + 2 * ((i0 + w) * K + p0 + lane) : A + 2 * ((p0 + w) * M + i0 + lane);
    const int64_t step = 2 * kGvProd * (VM ? K : M);
    const bool ok = VM ? p0 + lane < K : i0 + lane < M;
    const int64_t left = (VM ? M - i0 : K - p0) - w;  // columns from this warp's first one on
#pragma unroll
    for (int u = 0; u < COLS; ++u) {
      a[u] = make_double2(0.0, 0.0);
      if (ok && u * kGvProd < left) {
        const double *q = src + u * step;
        a[u] = ALIGNED ? __ldg(reinterpret_cast<const double2 *>(q)) : make_double2(q[0], q[1]);
      }
    }
  };
  // the same entries into L2, one 128-byte line per eight lanes
  auto prefetch = [&](int64_t st) {
    const int64_t p0 = st * kGvK;
    const double *src = VM ? A + 2 * ((i0 + w) * K + p0 + lane) : A + 2 * ((p0 + w) * M + i0 + lane);
    const int64_t step = 2 * kGvProd * (VM ? K : M);
    const bool ok = (lane & 7) == 0 && (VM ? p0 + lane < K : i0 + lane < M);
    const int64_t left = (VM ? M - i0 : K - p0) - w;
#pragma unroll
    for (int u = 0; u < COLS; ++u)
      if (ok && u * kGvProd < left) asm volatile("prefetch.global.L2 [%0];" ::"l"(src + u * step));
  };
  auto load_x = [&](int64_t st) {  // by the first producer, for all
    if (st < nst) {
      const int64_t p = st * kGvK + lane;
      load_dd<ALIGNED>(xs + (st % S) * kGvK + lane, x + 2 * p, p < K, x);
    }
    cp_async_commit();
  };
  double2 a[P][COLS];
  if (w == 0) {
    for (int st = 0; st < S - 1; ++st) load_x(st);
    cp_async_wait_n<S - 2>();
  }
#pragma unroll
  for (int q = 0; q < P; ++q) load(q, a[q]);
  for (int q = P; q < kGvAhead; ++q) prefetch(q);
  sync();  // the vector's first stage landed
  for (int64_t base = 0; base <= nst; base += P) {
#pragma unroll
    for (int q = 0; q < P; ++q) {
      const int64_t st = base + q;
      if (st > nst) break;
      if (w == 0) {
        load_x(st + S - 1);        // into the slot of stage st - 1, read an iteration ago
        cp_async_wait_n<S - 2>();  // stage st + 1 landed, for everyone after this iteration's barrier
      }
      if (st < nst) {
        const double2 *xp = xs + (st % S) * kGvK;
        double2 *out = pq + (st & 1) * kGvK * PITCH;
        double2 v[VM ? 1 : COLS];
        if (VM) {
          v[0] = xp[lane];
        } else {
#pragma unroll
          for (int u = 0; u < COLS; ++u) v[VM ? 0 : u] = xp[w + u * kGvProd];
        }
#pragma unroll
        for (int u = 0; u < COLS; ++u) {
          const int c = w + u * kGvProd;
          if (VM)
            out[lane * PITCH + c] = mac_terms(v[0].x, v[0].y, a[q][u].x, a[q][u].y);  // pitch 33: conflict-free
          else
            out[c * PITCH + lane] = mac_terms(a[q][u].x, a[q][u].y, v[VM ? 0 : u].x, v[VM ? 0 : u].y);
        }
        load(st + P, a[q]);
        prefetch(st + kGvAhead);
      }
      sync();
    }
  }
  if (w == 0) cp_async_wait_n<0>();
}

static bool aligned16(const void *a, const void *b, const void *c) {
  return ((reinterpret_cast<uintptr_t>(a) | reinterpret_cast<uintptr_t>(b) |
           reinterpret_cast<uintptr_t>(c)) & 15) == 0;
}

static bool shape_ok(int64_t m, int64_t k, int64_t n, size_t elem) {
  return size_ok(m, elem) && size_ok(k, elem) && size_ok(n, elem) && mul_ok(m, k) &&
         mul_ok(k, n) && mul_ok(m, n) && size_ok(m * k, elem) && size_ok(k * n, elem) &&
         size_ok(m * n, elem);
}

// Output with k == 0: the reference finalises zero accumulators -> +0.
__global__ void zero_fill_kernel(double *p, int64_t n) {
  int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  int64_t stride = (int64_t)gridDim.x * blockDim.x;
  for (; i < n; i += stride) p[i] = 0.0;
}
static int zero_fill(double *p, int64_t ndoubles, cudaStream_t s) {
  if (ndoubles == 0) return MFCUDA_OK;
  int64_t blocks = (ndoubles + 255) / 256;
  if (blocks > 4096) blocks = 4096;
  zero_fill_kernel<<<(int)blocks, 256, 0, s>>>(p, ndoubles);
  MF_TRY_CUDA(cudaGetLastError());
  return MFCUDA_OK;
}

template <bool ALIGNED, bool SHORT>
static void launch_gemm(const TilePick &p, const double *A, const double *B, double *C, int64_t m, int64_t k,
                        int64_t n, int64_t ri, cudaStream_t s) {
  const unsigned g = (unsigned)p.blocks;
  if (p.edge == 64)
    gemm_dd_kernel<ALIGNED, SHORT><<<g, kThreads, 0, s>>>(A, B, C, m, k, n, ri, p.cut ? p.whole : p.blocks, p.cut);
  else if (p.edge == 32)
    gemm_dd_small_kernel<2, ALIGNED, SHORT><<<g, kThreads, 0, s>>>(A, B, C, m, k, n, ri);
  else
    gemm_dd_small_kernel<1, ALIGNED, SHORT><<<g, kThreads, 0, s>>>(A, B, C, m, k, n, ri);
}
template <bool ALIGNED, bool SHORT>
static void launch_cgemm(const TilePick &p, const double *A, const double *B, double *C, int64_t m, int64_t k,
                         int64_t n, int64_t ri, cudaStream_t s) {
  const unsigned g = (unsigned)p.blocks;
  if (p.edge == 32)
    cgemm_dd_kernel<ALIGNED, SHORT><<<g, kThreads, 0, s>>>(A, B, C, m, k, n, ri, p.cut ? p.whole : p.blocks, p.cut);
  else
    cgemm_dd_small_kernel<ALIGNED, SHORT><<<g, kThreads, 0, s>>>(A, B, C, m, k, n, ri);
}

int gemm_dev(const float64x2 *a, const float64x2 *b, float64x2 *c, int64_t m, int64_t k,
             int64_t n, int64_t ri, cudaStream_t s) {
  if (!shape_ok(m, k, n, sizeof(float64x2))) return MFCUDA_ERR_INVALID_ARG;
  if (m == 0 || n == 0) return MFCUDA_OK;
  if (!c || (k > 0 && (!a || !b))) return MFCUDA_ERR_INVALID_ARG;
  MF_TRY(require_device());
  double *C = reinterpret_cast<double *>(c);
  if (k == 0) return zero_fill(C, 2 * m * n, s);
  const double *A = reinterpret_cast<const double *>(a);
  const double *B = reinterpret_cast<const double *>(b);
  if ((n + 63) / 64 > 65535) return MFCUDA_ERR_UNSUPPORTED;
  const TilePick p = pick_tiles(m, n, kRealCost, 3, kRealCutCost);
  if (p.blocks <= 0 || p.blocks > INT32_MAX) return MFCUDA_ERR_UNSUPPORTED;
  const bool sh = gtile::short_interval(ri);
  if (aligned16(a, b, c))
    (sh ? launch_gemm<true, true> : launch_gemm<true, false>)(p, A, B, C, m, k, n, ri, s);
  else
    (sh ? launch_gemm<false, true> : launch_gemm<false, false>)(p, A, B, C, m, k, n, ri, s);
  MF_TRY_CUDA(cudaGetLastError());
  return MFCUDA_OK;
}

int cgemm_dev(const complex64x2 *a, const complex64x2 *b, complex64x2 *c, int64_t m, int64_t k,
              int64_t n, int64_t ri, cudaStream_t s) {
  if (!shape_ok(m, k, n, sizeof(complex64x2))) return MFCUDA_ERR_INVALID_ARG;
  if (m == 0 || n == 0) return MFCUDA_OK;
  if (!c || (k > 0 && (!a || !b))) return MFCUDA_ERR_INVALID_ARG;
  MF_TRY(require_device());
  double *C = reinterpret_cast<double *>(c);
  if (k == 0) return zero_fill(C, 4 * m * n, s);
  const double *A = reinterpret_cast<const double *>(a);
  const double *B = reinterpret_cast<const double *>(b);
  if ((n + 31) / 32 > 65535) return MFCUDA_ERR_UNSUPPORTED;
  const TilePick p = pick_tiles(m, n, kCplxCost, 2, kCplxCutCost);
  if (p.blocks <= 0 || p.blocks > INT32_MAX) return MFCUDA_ERR_UNSUPPORTED;
  const bool sh = gtile::short_interval(ri);
  if (aligned16(a, b, c))
    (sh ? launch_cgemm<true, true> : launch_cgemm<true, false>)(p, A, B, C, m, k, n, ri, s);
  else
    (sh ? launch_cgemm<false, true> : launch_cgemm<false, false>)(p, A, B, C, m, k, n, ri, s);
  MF_TRY_CUDA(cudaGetLastError());
  return MFCUDA_OK;
}

// y(m) = A(m,k) x(k), or with VM y(m) = x(k) A(k,m).
template <bool VM, int P, bool ALIGNED>
static int launch_gemv(const double *A, const double *x, double *y, int64_t m, int64_t k, int64_t ri, int sms,
                       cudaStream_t s) {
  gemv_dd_kernel<VM, P, ALIGNED><<<(unsigned)((m + kGvN - 1) / kGvN), kGvThreads, 0, s>>>(A, x, y, m, k, ri, sms);
  MF_TRY_CUDA(cudaGetLastError());
  return MFCUDA_OK;
}
template <bool VM>
static int gemv_any(const float64x2 *a, const float64x2 *x, float64x2 *y, int64_t m, int64_t k, int64_t ri,
                    cudaStream_t s) {
  if (!shape_ok(m, k, 1, sizeof(float64x2))) return MFCUDA_ERR_INVALID_ARG;
  if (m == 0) return MFCUDA_OK;
  if (!y || (k > 0 && (!a || !x))) return MFCUDA_ERR_INVALID_ARG;
  MF_TRY(require_device());
  const int64_t blocks = (m + kGvN - 1) / kGvN;
  if (blocks > INT32_MAX) return MFCUDA_ERR_UNSUPPORTED;
  const double *A = reinterpret_cast<const double *>(a), *X = reinterpret_cast<const double *>(x);
  double *Y = reinterpret_cast<double *>(y);
  const int sms = sm_count();
  const bool one_wave = blocks <= sms;
  if (aligned16(a, x, y))
    return one_wave ? launch_gemv<VM, 4, true>(A, X, Y, m, k, ri, sms, s)
                    : launch_gemv<VM, 2, true>(A, X, Y, m, k, ri, sms, s);
  return one_wave ? launch_gemv<VM, 4, false>(A, X, Y, m, k, ri, sms, s)
                  : launch_gemv<VM, 2, false>(A, X, Y, m, k, ri, sms, s);
}
int gemv_dev(const float64x2 *a, const float64x2 *x, float64x2 *y, int64_t m, int64_t k,
             int64_t ri, cudaStream_t s) {
  return gemv_any<false>(a, x, y, m, k, ri, s);
}
int gevm_dev(const float64x2 *x, const float64x2 *b, float64x2 *y, int64_t k, int64_t n,
             int64_t ri, cudaStream_t s) {
  return gemv_any<true>(b, x, y, n, k, ri, s);
}

// ---- host-pointer (drop-in) forms -----------------------------------------
static int gemm_host(const float64x2 *a, const float64x2 *b, float64x2 *c, int64_t m, int64_t k,
                     int64_t n, int64_t ri) {
  if (!shape_ok(m, k, n, sizeof(float64x2))) return MFCUDA_ERR_INVALID_ARG;
  if (m == 0 || n == 0) return MFCUDA_OK;
  if (!c || (k > 0 && (!a || !b))) return MFCUDA_ERR_INVALID_ARG;
  MF_TRY(require_device());
  size_t ba = (size_t)(m * k) * sizeof(float64x2), bb = (size_t)(k * n) * sizeof(float64x2),
         bc = (size_t)(m * n) * sizeof(float64x2);
  size_t sz[4] = {ba, bb, bc, 0};
  Staging st;
  MF_TRY(staging_acquire(st, sz));
  auto *da = static_cast<float64x2 *>(st.buf[0]);
  auto *db = static_cast<float64x2 *>(st.buf[1]);
  auto *dc = static_cast<float64x2 *>(st.buf[2]);
  if (ba) MF_TRY_CUDA(cudaMemcpyAsync(da, a, ba, cudaMemcpyHostToDevice, st.stream));
  if (bb) MF_TRY_CUDA(cudaMemcpyAsync(db, b, bb, cudaMemcpyHostToDevice, st.stream));
  MF_TRY(gemm_dev(da, db, dc, m, k, n, ri, st.stream));
  MF_TRY_CUDA(cudaMemcpyAsync(c, dc, bc, cudaMemcpyDeviceToHost, st.stream));
  MF_TRY_CUDA(cudaStreamSynchronize(st.stream));
  return MFCUDA_OK;
}

static int cgemm_host(const complex64x2 *a, const complex64x2 *b, complex64x2 *c, int64_t m,
                      int64_t k, int64_t n, int64_t ri) {
  if (!shape_ok(m, k, n, sizeof(complex64x2))) return MFCUDA_ERR_INVALID_ARG;
  if (m == 0 || n == 0) return MFCUDA_OK;
  if (!c || (k > 0 && (!a || !b))) return MFCUDA_ERR_INVALID_ARG;
  MF_TRY(require_device());
  size_t ba = (size_t)(m * k) * sizeof(complex64x2), bb = (size_t)(k * n) * sizeof(complex64x2),
         bc = (size_t)(m * n) * sizeof(complex64x2);
  size_t sz[4] = {ba, bb, bc, 0};
  Staging st;
  MF_TRY(staging_acquire(st, sz));
  auto *da = static_cast<complex64x2 *>(st.buf[0]);
  auto *db = static_cast<complex64x2 *>(st.buf[1]);
  auto *dc = static_cast<complex64x2 *>(st.buf[2]);
  if (ba) MF_TRY_CUDA(cudaMemcpyAsync(da, a, ba, cudaMemcpyHostToDevice, st.stream));
  if (bb) MF_TRY_CUDA(cudaMemcpyAsync(db, b, bb, cudaMemcpyHostToDevice, st.stream));
  MF_TRY(cgemm_dev(da, db, dc, m, k, n, ri, st.stream));
  MF_TRY_CUDA(cudaMemcpyAsync(c, dc, bc, cudaMemcpyDeviceToHost, st.stream));
  MF_TRY_CUDA(cudaStreamSynchronize(st.stream));
  return MFCUDA_OK;
}

static int gemv_host(const float64x2 *a, const float64x2 *x, float64x2 *y, int64_t m, int64_t k,
                     int64_t ri) {
  if (!shape_ok(m, k, 1, sizeof(float64x2))) return MFCUDA_ERR_INVALID_ARG;
  if (m == 0) return MFCUDA_OK;
  if (!y || (k > 0 && (!a || !x))) return MFCUDA_ERR_INVALID_ARG;
  MF_TRY(require_device());
  size_t ba = (size_t)(m * k) * sizeof(float64x2), bx = (size_t)k * sizeof(float64x2),
         by = (size_t)m * sizeof(float64x2);
  size_t sz[4] = {ba, bx, by, 0};
  Staging st;
  MF_TRY(staging_acquire(st, sz));
  auto *da = static_cast<float64x2 *>(st.buf[0]);
  auto *dx = static_cast<float64x2 *>(st.buf[1]);
  auto *dy = static_cast<float64x2 *>(st.buf[2]);
  if (ba) MF_TRY_CUDA(cudaMemcpyAsync(da, a, ba, cudaMemcpyHostToDevice, st.stream));
  if (bx) MF_TRY_CUDA(cudaMemcpyAsync(dx, x, bx, cudaMemcpyHostToDevice, st.stream));
  MF_TRY(gemv_dev(da, dx, dy, m, k, ri, st.stream));
  MF_TRY_CUDA(cudaMemcpyAsync(y, dy, by, cudaMemcpyDeviceToHost, st.stream));
  MF_TRY_CUDA(cudaStreamSynchronize(st.stream));
  return MFCUDA_OK;
}

static int gevm_host(const float64x2 *x, const float64x2 *b, float64x2 *y, int64_t k, int64_t n,
                     int64_t ri) {
  if (!shape_ok(1, k, n, sizeof(float64x2))) return MFCUDA_ERR_INVALID_ARG;
  if (n == 0) return MFCUDA_OK;
  if (!y || (k > 0 && (!b || !x))) return MFCUDA_ERR_INVALID_ARG;
  MF_TRY(require_device());
  size_t bx = (size_t)k * sizeof(float64x2), bb = (size_t)(k * n) * sizeof(float64x2),
         by = (size_t)n * sizeof(float64x2);
  size_t sz[4] = {bx, bb, by, 0};
  Staging st;
  MF_TRY(staging_acquire(st, sz));
  auto *dx = static_cast<float64x2 *>(st.buf[0]);
  auto *db = static_cast<float64x2 *>(st.buf[1]);
  auto *dy = static_cast<float64x2 *>(st.buf[2]);
  if (bx) MF_TRY_CUDA(cudaMemcpyAsync(dx, x, bx, cudaMemcpyHostToDevice, st.stream));
  if (bb) MF_TRY_CUDA(cudaMemcpyAsync(db, b, bb, cudaMemcpyHostToDevice, st.stream));
  MF_TRY(gevm_dev(dx, db, dy, k, n, ri, st.stream));
  MF_TRY_CUDA(cudaMemcpyAsync(y, dy, by, cudaMemcpyDeviceToHost, st.stream));
  MF_TRY_CUDA(cudaStreamSynchronize(st.stream));
  return MFCUDA_OK;
}

}  // namespace mfcuda

extern "C" {

MULTIFLOATS_CUDA_API int mfcuda_matmuldd_mm(const float64x2 *a, const float64x2 *b, float64x2 *c,
                                            int64_t m, int64_t k, int64_t n, int64_t ri,
                                            void *stream) {
  return mfcuda::gemm_dev(a, b, c, m, k, n, ri, mfcuda::as_stream(stream));
}
MULTIFLOATS_CUDA_API int mfcuda_matmuldd_mv(const float64x2 *a, const float64x2 *x, float64x2 *y,
                                            int64_t m, int64_t k, int64_t ri, void *stream) {
  return mfcuda::gemv_dev(a, x, y, m, k, ri, mfcuda::as_stream(stream));
}
MULTIFLOATS_CUDA_API int mfcuda_matmuldd_vm(const float64x2 *x, const float64x2 *b, float64x2 *y,
                                            int64_t k, int64_t n, int64_t ri, void *stream) {
  return mfcuda::gevm_dev(x, b, y, k, n, ri, mfcuda::as_stream(stream));
}
MULTIFLOATS_CUDA_API int mfcuda_cmatmuldd_mm(const complex64x2 *a, const complex64x2 *b,
                                             complex64x2 *c, int64_t m, int64_t k, int64_t n,
                                             int64_t ri, void *stream) {
  return mfcuda::cgemm_dev(a, b, c, m, k, n, ri, mfcuda::as_stream(stream));
}

MULTIFLOATS_CUDA_API void matmuldd_mm(const float64x2 *a, const float64x2 *b, float64x2 *c,
                                      int64_t m, int64_t k, int64_t n, int64_t ri) {
  mfcuda::set_last_error(mfcuda::gemm_host(a, b, c, m, k, n, ri));
}
MULTIFLOATS_CUDA_API void matmuldd_mv(const float64x2 *a, const float64x2 *x, float64x2 *y,
                                      int64_t m, int64_t k, int64_t ri) {
  mfcuda::set_last_error(mfcuda::gemv_host(a, x, y, m, k, ri));
}
MULTIFLOATS_CUDA_API void matmuldd_vm(const float64x2 *x, const float64x2 *b, float64x2 *y,
                                      int64_t k, int64_t n, int64_t ri) {
  mfcuda::set_last_error(mfcuda::gevm_host(x, b, y, k, n, ri));
}
MULTIFLOATS_CUDA_API void matmulf64x2_mm(const float64x2 *a, const float64x2 *b, float64x2 *c,
                                         int64_t m, int64_t k, int64_t n, int64_t ri) {
  matmuldd_mm(a, b, c, m, k, n, ri);
}
MULTIFLOATS_CUDA_API void matmulf64x2_mv(const float64x2 *a, const float64x2 *x, float64x2 *y,
                                         int64_t m, int64_t k, int64_t ri) {
  matmuldd_mv(a, x, y, m, k, ri);
}
MULTIFLOATS_CUDA_API void matmulf64x2_vm(const float64x2 *x, const float64x2 *b, float64x2 *y,
                                         int64_t k, int64_t n, int64_t ri) {
  matmuldd_vm(x, b, y, k, n, ri);
}
MULTIFLOATS_CUDA_API void cmatmuldd_mm(const complex64x2 *a, const complex64x2 *b,
                                       complex64x2 *c, int64_t m, int64_t k, int64_t n,
                                       int64_t ri) {
  mfcuda::set_last_error(mfcuda::cgemm_host(a, b, c, m, k, n, ri));
}

}  // extern "C"
