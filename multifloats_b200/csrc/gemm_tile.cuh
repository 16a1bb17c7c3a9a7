// One output tile of the plain compensated DD matmul (src/float64x2/matmul.inc:6-39
// semantics: per output, the MAC over p = 0..k-1 in order, renormalised after
// each full chunk of `ri` steps when more remain and once at the end), shared
// by the single-problem kernel and the grouped (batched) kernel.
//
// A 256-thread CTA owns a (16 TM) x (16 TN) tile; thread t owns rows
// tx + 16 i (i < TM) and columns ty + 16 j (j < TN), tx = t % 16, ty = t / 16.
// A and B k-slices go through a two-stage cp.async ring in shared memory
// (zero-filled past the edges), deeper for smaller tiles (8, 16 or 32 steps),
// so that a stage always holds about the same bytes and the small tiles do
// not meet a barrier every few MACs.
//
// Bound: FP64 pipe, 13 instructions per MAC plus 6 per renormalisation, two
// issue cycles each.  The steps run in branch-free groups of eight: with the
// chunk counter tested after every step the accumulators had to sit in fixed
// registers at each merge, and the moves that took (8 of 26 issue cycles per
// MAC) were paid on top of the FP64 issue -- 4096^3 66.6 -> 56.8 ms, 16.6 of the
// pipe's 18.6 T instructions/s (64 a cycle and SM at 1.965 GHz; a chain-free loop
// of multiply-adds alone reaches 17.1).  An interval that is not a multiple of eight runs from chunk end
// to chunk end in a counted loop; the shortest ones have kernels of their own.
#pragma once
#include "dd_device.cuh"

namespace mfcuda {
namespace gtile {

__device__ __forceinline__ unsigned smem_u32(const void *p) {
  return static_cast<unsigned>(__cvta_generic_to_shared(p));
}
// 16-byte async copy; src_bytes = 0 zero-fills the destination.
__device__ __forceinline__ void cp_async16(void *dst, const void *src, int src_bytes) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], 16, %2;\n" ::"r"(smem_u32(dst)), "l"(src),
               "r"(src_bytes));
}
__device__ __forceinline__ void cp_async8(void *dst, const void *src, int src_bytes) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], 8, %2;\n" ::"r"(smem_u32(dst)), "l"(src),
               "r"(src_bytes));
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;\n" ::); }
__device__ __forceinline__ void cp_async_wait_all() { asm volatile("cp.async.wait_group 0;\n" ::); }

// Copy one DD (16 bytes) or zero-fill it.  `safe` is an in-bounds address
// (the matrix base) handed to the copy when nothing is read.
template <bool ALIGNED>
__device__ __forceinline__ void load_dd(double2 *dst, const double *src, bool valid,
                                        const double *safe) {
  if constexpr (ALIGNED) {
    cp_async16(dst, valid ? src : safe, valid ? 16 : 0);
  } else {
    double *d = reinterpret_cast<double *>(dst);
    cp_async8(d, valid ? src : safe, valid ? 8 : 0);
    cp_async8(d + 1, valid ? src + 1 : safe, valid ? 8 : 0);
  }
}


constexpr int kThreads = 256;
constexpr int kGroup = 8;  // steps of a branch-free group

// Depth of a stage for a tile of edge e: 8 steps of 64, 16 of 32, 32 of 16.
__host__ __device__ constexpr int depth(int edge) { return 512 / edge; }
// A row of the B stage is one entry longer than the tile: the threads of a
// copy run along k, and without it eight of them meet in the same banks.
__host__ __device__ constexpr int b_pitch(int bn) { return bn + 1; }

// Staging of any tile (edges 16, 32, 64).
struct Smem {
  double2 A[2][512];
  double2 B[2][depth(16) * b_pitch(16)];
};

// The renormalisation cadence: where the chunks of `ri` steps end.
struct Cadence {
  int64_t ri, cnt;   // interval (<= 0: no renormalisation), steps since the last one
  bool grouped;      // the interval is none or a multiple of kGroup
  __device__ __forceinline__ explicit Cadence(int64_t r) : ri(r), cnt(0), grouped(r <= 0 || r % kGroup == 0) {}
  // steps until the chunk's end, at most `left`
  __device__ __forceinline__ int run(int left) const {
    return ri > 0 && ri - cnt < left ? (int)(ri - cnt) : left;
  }
  // `steps` more MACs done (never past a chunk's end): does a chunk end here?
  __device__ __forceinline__ bool ends(int steps) {
    if (ri <= 0 || (cnt += steps) != ri) return false;
    cnt = 0;
    return true;
  }
  // one more MAC done, interval known to be positive: does a chunk end here?
  __device__ __forceinline__ bool step_ends() {
    const bool end = ++cnt == ri;
    if (end) cnt = 0;
    return end;
  }
};
// Intervals of up to three steps have kernels of their own (SHORT): their chunks are
// too short for a counted loop each.  Real tiles of 32 and 16 and complex ones of 16
// test the chunk counter after every step of an unrolled group, complex tiles of 32
// renormalise without a test where the interval is one.  Counted loops -> these, us:
// 777 x 333 x 555 interval 1 376 -> 232, 2 261 -> 220; 256^3 interval 1 64 -> 35, 3
// 39 -> 33; complex batches interval 1 a fifth less.  With four steps
// and more the test costs the tiles of 32 up to 15 %; in the same kernel as the
// longer intervals this code cost those up to 5 %.
constexpr int kShort = 3;
inline bool short_interval(int64_t ri) { return ri > 0 && ri <= kShort; }

template <int TM, int TN, bool ALIGNED, bool SHORT>
__device__ __forceinline__ void gemm_tile(const double *__restrict__ A, const double *__restrict__ B,
                                          double *__restrict__ C, int64_t M, int64_t K, int64_t N,
                                          int64_t ri, int64_t m0, int64_t n0, Smem &sm) {
  constexpr int BM = 16 * TM, BN = 16 * TN, BK = depth(BM > BN ? BM : BN), PB = b_pitch(BN);
  static_assert(BK * BM <= 512 && BK * PB <= depth(16) * b_pitch(16), "stage fits Smem");
  const int t = threadIdx.x;
  const int tx = t % 16, ty = t / 16;

  double s_hi[TM][TN], s_lo[TM][TN];
#pragma unroll
  for (int i = 0; i < TM; ++i)
#pragma unroll
    for (int j = 0; j < TN; ++j) s_hi[i][j] = s_lo[i][j] = 0.0;

  auto issue = [&](int stage, int64_t k0) {
#pragma unroll
    for (int idx = t; idx < BK * BM; idx += kThreads) {
      int row = idx % BM, kk = idx / BM;
      int64_t gi = m0 + row, gk = k0 + kk;
      bool v = gi < M && gk < K;
      load_dd<ALIGNED>(&sm.A[stage][kk * BM + row], A + 2 * (gk * M + gi), v, A);
    }
#pragma unroll
    for (int idx = t; idx < BK * BN; idx += kThreads) {
      int kk = idx % BK, col = idx / BK;
      int64_t gj = n0 + col, gk = k0 + kk;
      bool v = gj < N && gk < K;
      load_dd<ALIGNED>(&sm.B[stage][kk * PB + col], B + 2 * (gj * K + gk), v, B);
    }
    cp_async_commit();
  };
  auto step = [&](const double2 *as, const double2 *bs) {
    double ah[TM], al[TM], bh[TN], bl[TN];
#pragma unroll
    for (int i = 0; i < TM; ++i) {
      double2 v = as[16 * i];
      ah[i] = v.x;
      al[i] = v.y;
    }
#pragma unroll
    for (int j = 0; j < TN; ++j) {
      double2 v = bs[16 * j];
      bh[j] = v.x;
      bl[j] = v.y;
    }
#pragma unroll
    for (int j = 0; j < TN; ++j)
#pragma unroll
      for (int i = 0; i < TM; ++i) mfdev::mac(ah[i], al[i], bh[j], bl[j], s_hi[i][j], s_lo[i][j]);
  };
  auto renorm_all = [&]() {
#pragma unroll
    for (int i = 0; i < TM; ++i)
#pragma unroll
      for (int j = 0; j < TN; ++j) mfdev::renorm(s_hi[i][j], s_lo[i][j]);
  };

  const int64_t ntiles = (K + BK - 1) / BK;
  Cadence cad(ri);
  if (ntiles > 0) issue(0, 0);
  for (int64_t kt = 0; kt < ntiles; ++kt) {
    const int stage = (int)(kt & 1);
    cp_async_wait_all();
    __syncthreads();
    if (kt + 1 < ntiles) issue(stage ^ 1, (kt + 1) * BK);
    const int64_t k0 = kt * BK;
    const int kmax = (K - k0) < BK ? (int)(K - k0) : BK;
    const double2 *as = sm.A[stage] + tx, *bs = sm.B[stage] + ty;
    int kk = 0;
    if constexpr (SHORT && TM * TN < 16) {  // whole groups with more steps after them
#pragma unroll 1
      for (; kk + kGroup <= kmax && k0 + kk + kGroup < K; kk += kGroup) {
#pragma unroll
        for (int u = 0; u < kGroup; ++u) {
          step(as + (kk + u) * BM, bs + (kk + u) * PB);
          if (cad.step_ends()) renorm_all();
        }
      }
    } else if (!SHORT && cad.grouped) {
#pragma unroll 1
      for (; kk + kGroup <= kmax; kk += kGroup) {
#pragma unroll
        for (int u = 0; u < kGroup; ++u) step(as + (kk + u) * BM, bs + (kk + u) * PB);
        if (cad.ends(kGroup) && k0 + kk + kGroup < K) renorm_all();
      }
    }
    while (kk < kmax) {  // the steps up to the next chunk's end
      const int run = cad.run(kmax - kk);
      const double2 *ar = as + kk * BM, *br = bs + kk * PB;
#pragma unroll(TM * TN >= 16 ? 1 : 4)
      for (int u = 0; u < run; ++u) step(ar + u * BM, br + u * PB);
      kk += run;
      if (cad.ends(run) && k0 + kk < K) renorm_all();
    }
    __syncthreads();
  }
#pragma unroll
  for (int j = 0; j < TN; ++j) {
    int64_t gj = n0 + ty + 16 * j;
#pragma unroll
    for (int i = 0; i < TM; ++i) {
      int64_t gi = m0 + tx + 16 * i;
      double h = s_hi[i][j], l = s_lo[i][j];
      mfdev::renorm(h, l);
      if (gi < M && gj < N) {
        double *dst = C + 2 * (gj * M + gi);
        if constexpr (ALIGNED) {
          *reinterpret_cast<double2 *>(dst) = make_double2(h, l);
        } else {
          dst[0] = h;
          dst[1] = l;
        }
      }
    }
  }
}


// ---------------------------------------------------------------------------
// One (16 TM) x (16 TN) output tile of the complex product (the Fortran
// cdd_matmul_mm composition, fsrc/multifloats.fypp:2609-2621): each thread owns
// TM x TN complex outputs with four real accumulators each (rr, ii, ri, ir),
// each run with the real MAC and renorm cadence, then re = rr - ii,
// im = ri + ir with the DD operators.
// ---------------------------------------------------------------------------
// Staging of any complex tile (edges 16, 32): real and imaginary part adjacent.
struct CSmem {
  double2 A[2][512];
  double2 B[2][2 * depth(32) * b_pitch(16)];
};

template <int TM, int TN, bool ALIGNED, bool SHORT>
__device__ __forceinline__ void cgemm_tile(const double *__restrict__ A, const double *__restrict__ B,
                                           double *__restrict__ C, int64_t M, int64_t K, int64_t N,
                                           int64_t ri, int64_t m0, int64_t n0, CSmem &sm) {
  // complex element = 4 doubles = two double2 (re, im)
  constexpr int BM = 16 * TM, BN = 16 * TN, BK = depth(2 * (BM > BN ? BM : BN)), PB = b_pitch(BN);
  static_assert(2 * BK * BM <= 512 && BK * PB <= depth(32) * b_pitch(16), "stage fits CSmem");
  const int t = threadIdx.x;
  const int tx = t % 16, ty = t / 16;

  double s_hi[TM][TN][4], s_lo[TM][TN][4];
#pragma unroll
  for (int i = 0; i < TM; ++i)
#pragma unroll
    for (int j = 0; j < TN; ++j)
#pragma unroll
      for (int q = 0; q < 4; ++q) s_hi[i][j][q] = s_lo[i][j][q] = 0.0;

  auto issue = [&](int stage, int64_t k0) {
#pragma unroll
    for (int idx = t; idx < 2 * BK * BM; idx += kThreads) {
      int part = idx & 1, e = idx >> 1;
      int row = e % BM, kk = e / BM;
      int64_t gi = m0 + row, gk = k0 + kk;
      bool v = gi < M && gk < K;
      load_dd<ALIGNED>(&sm.A[stage][2 * (kk * BM + row) + part], A + 4 * (gk * M + gi) + 2 * part, v, A);
    }
#pragma unroll
    for (int idx = t; idx < 2 * BK * BN; idx += kThreads) {
      int part = idx & 1, e = idx >> 1;
      int kk = e % BK, col = e / BK;
      int64_t gj = n0 + col, gk = k0 + kk;
      bool v = gj < N && gk < K;
      load_dd<ALIGNED>(&sm.B[stage][2 * (kk * PB + col) + part], B + 4 * (gj * K + gk) + 2 * part, v, B);
    }
    cp_async_commit();
  };
  auto step = [&](const double2 *as, const double2 *bs) {
    double2 ar[TM], ai[TM], br[TN], bi[TN];
#pragma unroll
    for (int i = 0; i < TM; ++i) {
      ar[i] = as[32 * i];
      ai[i] = as[32 * i + 1];
    }
#pragma unroll
    for (int j = 0; j < TN; ++j) {
      br[j] = bs[32 * j];
      bi[j] = bs[32 * j + 1];
    }
#pragma unroll
    for (int j = 0; j < TN; ++j)
#pragma unroll
      for (int i = 0; i < TM; ++i) {
        mfdev::mac(ar[i].x, ar[i].y, br[j].x, br[j].y, s_hi[i][j][0], s_lo[i][j][0]);
        mfdev::mac(ai[i].x, ai[i].y, bi[j].x, bi[j].y, s_hi[i][j][1], s_lo[i][j][1]);
        mfdev::mac(ar[i].x, ar[i].y, bi[j].x, bi[j].y, s_hi[i][j][2], s_lo[i][j][2]);
        mfdev::mac(ai[i].x, ai[i].y, br[j].x, br[j].y, s_hi[i][j][3], s_lo[i][j][3]);
      }
  };
  auto renorm_all = [&]() {
#pragma unroll
    for (int i = 0; i < TM; ++i)
#pragma unroll
      for (int j = 0; j < TN; ++j)
#pragma unroll
        for (int q = 0; q < 4; ++q) mfdev::renorm(s_hi[i][j][q], s_lo[i][j][q]);
  };

  const int64_t ntiles = (K + BK - 1) / BK;
  Cadence cad(ri);
  if (ntiles > 0) issue(0, 0);
  for (int64_t kt = 0; kt < ntiles; ++kt) {
    const int stage = (int)(kt & 1);
    cp_async_wait_all();
    __syncthreads();
    if (kt + 1 < ntiles) issue(stage ^ 1, (kt + 1) * BK);
    const int64_t k0 = kt * BK;
    const int kmax = (K - k0) < BK ? (int)(K - k0) : BK;
    const double2 *as = sm.A[stage] + 2 * tx, *bs = sm.B[stage] + 2 * ty;
    int kk = 0;
    if constexpr (SHORT && TM * TN >= 4) {
      if (ri == 1) {
        const int each = K - 1 - k0 < kmax ? (int)(K - 1 - k0) : kmax;  // steps with more after them
#pragma unroll 2
        for (; kk < each; ++kk) {
          step(as + 2 * kk * BM, bs + 2 * kk * PB);
          renorm_all();
        }
      }
    } else if constexpr (SHORT) {  // whole groups with more steps after them
#pragma unroll 1
      for (; kk + kGroup <= kmax && k0 + kk + kGroup < K; kk += kGroup) {
#pragma unroll
        for (int u = 0; u < kGroup; ++u) {
          step(as + 2 * (kk + u) * BM, bs + 2 * (kk + u) * PB);
          if (cad.step_ends()) renorm_all();
        }
      }
    } else if (!SHORT && cad.grouped) {
#pragma unroll 1
      for (; kk + kGroup <= kmax; kk += kGroup) {
#pragma unroll
        for (int u = 0; u < kGroup; ++u) step(as + 2 * (kk + u) * BM, bs + 2 * (kk + u) * PB);
        if (cad.ends(kGroup) && k0 + kk + kGroup < K) renorm_all();
      }
    }
    while (kk < kmax) {  // the steps up to the next chunk's end
      const int run = cad.run(kmax - kk);
      const double2 *ar = as + 2 * kk * BM, *br = bs + 2 * kk * PB;
#pragma unroll(TM * TN >= 4 ? 1 : 4)
      for (int u = 0; u < run; ++u) step(ar + 2 * u * BM, br + 2 * u * PB);
      kk += run;
      if (cad.ends(run) && k0 + kk < K) renorm_all();
    }
    __syncthreads();
  }
#pragma unroll
  for (int j = 0; j < TN; ++j) {
    int64_t gj = n0 + ty + 16 * j;
#pragma unroll
    for (int i = 0; i < TM; ++i) {
      int64_t gi = m0 + tx + 16 * i;
      mfdev::dd p[4];
#pragma unroll
      for (int q = 0; q < 4; ++q) {
        double h = s_hi[i][j][q], l = s_lo[i][j][q];
        mfdev::renorm(h, l);
        p[q] = mfdev::make(h, l);
      }
      mfdev::dd re = mfdev::dd_sub(p[0], p[1]);
      mfdev::dd im = mfdev::dd_add(p[2], p[3]);
      if (gi < M && gj < N) {
        double *dst = C + 4 * (gj * M + gi);
        if constexpr (ALIGNED) {
          reinterpret_cast<double2 *>(dst)[0] = make_double2(re.hi, re.lo);
          reinterpret_cast<double2 *>(dst)[1] = make_double2(im.hi, im.lo);
        } else {
          dst[0] = re.hi;
          dst[1] = re.lo;
          dst[2] = im.hi;
          dst[3] = im.lo;
        }
      }
    }
  }
}

}  // namespace gtile
}  // namespace mfcuda
