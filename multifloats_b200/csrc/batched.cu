// Batched ragged work in grouped launches, captured once in a CUDA graph.
//
// A batch plan binds a list of independent problems (device pointers) and
// captures their execution as a CUDA graph that mfcuda_batch_run replays:
//
//  * plain DD GEMMs: ONE persistent grouped kernel.  Its work list holds every
//    output tile of every problem, longest K first; CTAs take items from an
//    atomic counter.  Each item runs the same tile code as the single-problem
//    kernel (gemm_tile.cuh) with the tile shape the autotuner picked for that
//    problem's shape bucket (64x64, 32x32 or 16x16), so every output is
//    bit-identical to matmuldd_mm.
//  * split-INT8 DD GEMMs: each phase of the split pipeline (exponent scan,
//    plan, slicing, tcgen05 MMA, recombination) is one grouped launch over all
//    problems; the tensor-core phase is one persistent kernel whose work list,
//    written on the device from the plans, holds every problem's items: one or
//    two diagonals (digits) or one modulus (CRT) of a K chunk and tile.  Per
//    problem: slice count from its plan, tile width N (256/128/64) from the
//    autotuner; one K chunk for the whole plan.  Results are bit-identical to
//    mfcuda_matmuldd_mm_split with that K chunk.
//  * ragged elementwise arrays: one grid-stride launch over the concatenated
//    index space.
//
// The autotuner times the candidate configurations of each shape bucket on
// synthetic problems of that bucket the first time the bucket is seen and keeps
// the winners in a small text cache (MFCUDA_AUTOTUNE_CACHE, default
// $HOME/.cache/multifloats_b200/autotune.txt).
#include <cudaTypedefs.h>
#include <sys/stat.h>

#include <algorithm>
#include <cmath>
#include <cstddef>
#include <cstdio>
#include <cstdlib>
#include <map>
#include <mutex>
#include <string>
#include <vector>

#include "common.cuh"
#include "dd_device.cuh"
#include "gemm_tile.cuh"
#include "crt_device.cuh"
#include "log_queue.cuh"
#include "split_device.cuh"
#include "tcgen05.cuh"

struct mfcuda_batch;

namespace mfcuda {
int unary_dev(int op, const float64x2 *x, float64x2 *y, int64_t n, cudaStream_t s);

namespace batch {

// ===========================================================================
// plain grouped GEMM
// ===========================================================================
struct PProb {
  const double *A;
  const double *B;
  double *C;
  int64_t m, k, n;
};
struct PItem {
  int prob, cfg, tm, tn;
};
constexpr int kPlainCfgs = 3;  // 0: 64x64 (4x4 per thread), 1: 32x32 (2x2), 2: 16x16 (1x1)
static int cfg_edge(int cfg) { return cfg == 0 ? 64 : cfg == 1 ? 32 : 16; }

template <bool ALIGNED, bool SHORT>
__global__ void __launch_bounds__(256, 2)
    plain_grouped_kernel(const PProb *__restrict__ probs, const PItem *__restrict__ items, int nitems,
                         int64_t ri, int *counter) {
  __shared__ gtile::Smem sm;
  __shared__ int next;
  for (;;) {
    if (threadIdx.x == 0) next = atomicAdd(counter, 1);
    __syncthreads();
    const int w = next;
    __syncthreads();  // everyone has read `next` before thread 0 overwrites it
    if (w >= nitems) break;
    const PItem it = items[w];
    const PProb p = probs[it.prob];
    switch (it.cfg) {
      case 0:
        gtile::gemm_tile<4, 4, ALIGNED, SHORT>(p.A, p.B, p.C, p.m, p.k, p.n, ri, (int64_t)it.tm * 64,
                                               (int64_t)it.tn * 64, sm);
        break;
      case 1:
        gtile::gemm_tile<2, 2, ALIGNED, SHORT>(p.A, p.B, p.C, p.m, p.k, p.n, ri, (int64_t)it.tm * 32,
                                               (int64_t)it.tn * 32, sm);
        break;
      default:
        gtile::gemm_tile<1, 1, ALIGNED, SHORT>(p.A, p.B, p.C, p.m, p.k, p.n, ri, (int64_t)it.tm * 16,
                                               (int64_t)it.tn * 16, sm);
        break;
    }
  }
}

// Complex problems (complex64x2): every 32 x 32 output tile runs the
// single-problem complex tile code (gtile::cgemm_tile).
template <bool ALIGNED, bool SHORT>
__global__ void __launch_bounds__(256, 2)
    cplain_grouped_kernel(const PProb *__restrict__ probs, const PItem *__restrict__ items, int nitems,
                          int64_t ri, int *counter) {
  __shared__ gtile::CSmem sm;
  __shared__ int next;
  for (;;) {
    if (threadIdx.x == 0) next = atomicAdd(counter, 1);
    __syncthreads();
    const int w = next;
    __syncthreads();
    if (w >= nitems) break;
    const PItem it = items[w];
    const PProb p = probs[it.prob];
    gtile::cgemm_tile<2, 2, ALIGNED, SHORT>(p.A, p.B, p.C, p.m, p.k, p.n, ri, (int64_t)it.tm * 32,
                                            (int64_t)it.tn * 32, sm);
  }
}

// ===========================================================================
// ragged elementwise
// ===========================================================================
struct RArr {
  const double *x;
  double *y;
  int64_t off;  // first index of this array in the concatenated space
};

template <int OP>
__device__ __forceinline__ mfdev::dd apply(mfdev::dd x) {
  if constexpr (OP == MFCUDA_EXP) return mfdev::dd_exp(x);
  if constexpr (OP == MFCUDA_LOG) return mfdev::dd_log(x);
  if constexpr (OP == MFCUDA_SIN) return mfdev::dd_sin(x);
  if constexpr (OP == MFCUDA_COS) return mfdev::dd_cos(x);
  return mfdev::dd_sqrt(x);
}

// last array whose start is <= e (offsets ascending, arrays may be empty)
__device__ __forceinline__ int find_array(const RArr *arrs, int narr, int64_t e) {
  int lo = 0, hi = narr - 1;
  while (lo < hi) {
    int mid = (lo + hi + 1) >> 1;
    if (arrs[mid].off <= e)
      lo = mid;
    else
      hi = mid - 1;
  }
  return lo;
}

template <int OP>
__global__ void __launch_bounds__(256) ragged_unary_kernel(const RArr *__restrict__ arrs, int narr,
                                                           int64_t total) {
  auto ld = [&](int64_t e, mfdev::dd &v, double *&y) {
    const RArr a = arrs[find_array(arrs, narr, e)];
    const int64_t i = e - a.off;
    v = mfdev::make(a.x[2 * i], a.x[2 * i + 1]);
    y = a.y + 2 * i;
  };
  auto st = [](double *y, mfdev::dd r) {
    y[0] = r.hi;
    y[1] = r.lo;
  };
  if constexpr (log_op<OP>) {
    __shared__ LogQueue q;
    log_map(q, total, ld, [](mfdev::dd v) { return apply<OP>(v); }, st);
  } else {
    const int64_t stride = (int64_t)gridDim.x * blockDim.x;
    for (int64_t e = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; e < total; e += stride) {
      mfdev::dd v;
      double *y;
      ld(e, v, y);
      st(y, apply<OP>(v));
    }
  }
}

// ===========================================================================
// split grouped pipeline
// ===========================================================================
using namespace split;

// One real product of the grouped split pipeline: a real problem, or one of
// the four real products of a complex problem (re = ArBr - AiBi,
// im = ArBi + AiBr).  Operands and the output are strided views (DD element e
// at double2 index e * stride); a product may reuse the statistics and slices
// of another product's A or B operand and share its plan (the four products
// of a complex problem use one slice count, planned from all four operands).
struct SProb {
  const double *A, *B;
  double *C;
  int64_t astride, bstride, cstride;
  int mode;  // recombination: 0 store, 1 C - P, 2 C + P
  int own_a, own_b, own_plan;
  int64_t m, k, n, M_pad, N_pad, K_pad;
  int bn, kcb, nkc, kblocks, ntm, ntn;
  int *sigA, *muA, *flagA, *sigB, *muB, *flagB;
  int *sigA2, *muA2, *sigB2, *muB2;  // the plan's second A and B operands (complex), or null
  int8_t *As, *Bs;
  int32_t *D;
  Plan *plan;
  int crt;       // CRT form (crt_device.cuh): slices are residues, items single products
  int nsl;       // slice slots per operand: SMAX digits, or the most moduli the CRT plan can use
  int diags;     // diagonals of an item (CRT: 1, the product of one modulus)
  CrtConst *cc;  // the plan's reconstruction constants (CRT form)
};
// K indices whose digits or residues the tensor cores read: whole steps of 32.
__host__ __device__ constexpr int64_t k_fill(int64_t k) { return k < 1 ? 32 : (k + 31) / 32 * 32; }

// phases with a per-problem block count (and the items, with their prefix sums); the
// recombination runs in two launches: stores first, then the - / + updates
enum { PH_SCAN_A, PH_SCAN_B, PH_SLICE_A, PH_SLICE_B, PH_COMBINE, PH_COMBINE2, PH_ITEMS, PH_COUNT };

// A block's problem and its index among the problem's blocks of the phase, from
// a table made with the plan: a bisection over the problems' block counts
// was eleven dependent loads at the head of every block (2000 products, both
// slicers, the scans and the recombination together 6.1 -> 5.6 ms).
struct Owner {
  int p, local;
};

__global__ void __launch_bounds__(256) g_scan_a(const SProb *probs, const Owner *owner) {
  const Owner own = owner[blockIdx.x];
  const SProb &P = probs[own.p];
  const int64_t l = own.local;
  const int64_t nbx = (P.m + 255) / 256;
  scan_a_body(P.A, P.m, P.k, P.astride, 64, P.sigA, P.muA, P.flagA, l % nbx, l / nbx);
}
// a warp per column, 8 columns per block
__global__ void __launch_bounds__(256) g_scan_b(const SProb *probs, const Owner *owner) {
  const Owner own = owner[blockIdx.x];
  const SProb &P = probs[own.p];
  const int64_t j = (int64_t)own.local * 8 + (threadIdx.x >> 5);
  if (j < P.n) scan_b_warp(P.B, P.k, P.bstride, P.sigB, P.muB, P.flagB, j);
}
__global__ void __launch_bounds__(256) g_plan(const SProb *probs, int slices, double target) {
  const SProb &P = probs[blockIdx.x];
  if (!P.own_plan) return;
  StatSet st;
  st.n = 0;
  auto add = [&](int *sig, const int *mu, int64_t count, int side) {
    st.sig[st.n] = sig;
    st.mu[st.n] = mu;
    st.count[st.n] = count;
    st.side[st.n] = side;
    ++st.n;
  };
  add(P.sigA, P.muA, P.m, 0);
  if (P.sigA2) add(P.sigA2, P.muA2, P.m, 0);
  add(P.sigB, P.muB, P.n, 1);
  if (P.sigB2) add(P.sigB2, P.muB2, P.n, 1);
  if (P.crt)
    crt_plan_body(st, slices, target, P.k, P.plan, P.cc);  // slices: the operand bits W (0 = from target)
  else
    plan_body(st, slices, target, P.plan);
}
__global__ void __launch_bounds__(256) g_slice_a(const SProb *probs, const Owner *owner) {
  const Owner own = owner[blockIdx.x];
  const SProb &P = probs[own.p];
  const int64_t l = own.local;
  const int64_t nbx = (P.m + 31) / 32;
  slice_a_body(P.A, P.m, P.k, P.astride, P.M_pad, P.K_pad, P.sigA, P.flagA, P.plan, P.As, l % nbx, l / nbx);
}
// CRT form: residues instead of digits, in MN-major planes As[t][p][i] (the
// rows of one K index contiguous); flat: thread t of the problem takes K
// index t / ceil(m / 8), rows 8 (t % ceil(m / 8)) .. + 7
__global__ void __launch_bounds__(256) g_crt_slice_a(const SProb *probs, const Owner *owner) {
  const Owner own = owner[blockIdx.x];
  const SProb &P = probs[own.p];
  const int64_t t = (int64_t)own.local * 256 + threadIdx.x;
  const int64_t per_k = (P.m + 7) / 8;
  const int64_t kp = t / per_k;
  CrtSlice c;
  c.a(P.A, P.m, P.k, P.astride, P.M_pad, P.K_pad, P.sigA, P.flagA, P.As, (t % per_k) * 8,
      kp < k_fill(P.k) ? kp : P.K_pad);
  c.run(P.plan);
}
__global__ void __launch_bounds__(256) g_crt_slice_b(const SProb *probs, const Owner *owner) {
  const Owner own = owner[blockIdx.x];
  const SProb &P = probs[own.p];
  const int64_t t = (int64_t)own.local * 256 + threadIdx.x;
  const int64_t per_col = k_fill(P.k) / 8;
  const int64_t j = t / per_col;
  CrtSlice c;
  c.b(P.B, P.k, P.n, P.bstride, P.N_pad, P.K_pad, P.sigB, P.flagB, P.Bs, j, (t % per_col) * 8);
  c.run(P.plan);
}
// flat: thread t of the problem takes column t / (k_fill / 8), entries 8 (t % (k_fill / 8)) .. + 7
__global__ void __launch_bounds__(256) g_slice_b(const SProb *probs, const Owner *owner) {
  const Owner own = owner[blockIdx.x];
  const SProb &P = probs[own.p];
  const int64_t t = (int64_t)own.local * 256 + threadIdx.x;
  const int64_t per_col = k_fill(P.k) / 8;
  const int64_t j = t / per_col;
  if (j < P.n)
    slice_b_one(P.B, P.k, P.n, P.bstride, P.N_pad, P.K_pad, P.sigB, P.flagB, P.plan, P.Bs, j, (t % per_col) * 8);
}
// flat: thread t of the problem owns rows 4 (t % q) .. + 3 of column t / q,
// q = ceil(m / 4) (combine4_body)
constexpr int kCombineThreads = COMBINE_THREADS;
static int64_t combine_blocks(int64_t m, int64_t n) {
  return (((m + 3) / 4) * n + kCombineThreads - 1) / kCombineThreads;
}
__global__ void __launch_bounds__(kCombineThreads, COMBINE_BLOCKS) g_combine(const SProb *probs, const Owner *owner) {
  const Owner own = owner[blockIdx.x];
  const SProb &P = probs[own.p];
  const int64_t t = (int64_t)own.local * kCombineThreads + threadIdx.x;
  const int64_t q = (P.m + 3) / 4;
  combine4_body(P.D, P.plan, P.sigA, P.flagA, P.sigB, P.flagB, P.m, P.n, P.M_pad, P.N_pad, P.nkc, P.C,
                P.cstride, P.mode, t % q, t / q);
}

// CRT form: the tensor-core reconstruction (crt_combine_tc_body), a block
// per 128 rows and CTC_QUADS column quads of a problem.
static int64_t crt_combine_blocks(int64_t m, int64_t n) {
  return ((m + CTC_THREADS - 1) / CTC_THREADS) * (((n + 3) / 4 + CTC_QUADS - 1) / CTC_QUADS);
}
__global__ void __launch_bounds__(CTC_THREADS, 4) g_crt_combine(const SProb *probs, const Owner *owner,
                                                             int *status, uint64_t wait_ns) {
  extern __shared__ uint8_t ctc_raw[];
  uint8_t *smem = reinterpret_cast<uint8_t *>((reinterpret_cast<uintptr_t>(ctc_raw) + 1023) & ~uintptr_t(1023));
  const Owner own = owner[blockIdx.x];
  const SProb &P = probs[own.p];
  const int64_t l = own.local, nbx = (P.m + CTC_THREADS - 1) / CTC_THREADS;
  crt_combine_tc_body(reinterpret_cast<const uint8_t *>(P.D), P.plan, P.cc, P.sigA, P.flagA, P.sigB, P.flagB, P.m,
                      P.n, P.M_pad, P.N_pad, P.nkc, P.k, P.C, P.cstride, P.mode, (l % nbx) * CTC_THREADS,
                      (l / nbx) * CTC_QUADS, smem, status, wait_ns);
}

// Work item of the tensor-core kernels, with all they need to know of its
// problem.  The list is written on the device once the plans are known
// (g_items) and every role reads its next entry while it works on the current
// one: finding an item's problem by bisection and walking to its plan was a
// dozen dependent loads per role and item, about 10 of the 13 us an item took.
struct __align__(16) GItem {
  int p;           // problem (its tensor maps)
  int g, nd;       // digits: diagonals g, g - 1, ... (nd of them); CRT: modulus g, nd = 1; nd = 0: beyond the plan
  int kb0, kb1;    // K blocks
  int a_row, b_row;  // first row of A and column of B
  int bn;          // columns of the tile: those of the output, rounded up to 32
  int M_pad;
  int rows;        // rows of the tile that the output has
  int klast, pad;  // K steps of 32 of block kb1 - 1: those of the operands
  int32_t *dst;    // D of diagonal / modulus g, K chunk and tile
  int64_t gstride;  // INT32 sums between diagonals
};
static_assert(sizeof(GItem) == 64 && offsetof(GItem, M_pad) == 32 && offsetof(GItem, dst) == 48, "read by load_item");
// Field by field: a struct filled through a pointer would live in local memory
// and be read again after every barrier wait.
__device__ __forceinline__ GItem load_item(const GItem *items, int64_t w, int64_t n) {
  GItem it;
  it.nd = 0;
  if (w < n) {
    const int4 *src = reinterpret_cast<const int4 *>(items + w);
    const int4 a = __ldg(src), b = __ldg(src + 1);
    const int4 c = __ldg(src + 2);
    const longlong2 e = __ldg(reinterpret_cast<const longlong2 *>(src + 3));
    it.p = a.x;
    it.g = a.y;
    it.nd = a.z;
    it.kb0 = a.w;
    it.kb1 = b.x;
    it.a_row = b.y;
    it.b_row = b.z;
    it.bn = b.w;
    it.M_pad = c.x;
    it.rows = c.y;
    it.klast = c.z;
    it.dst = reinterpret_cast<int32_t *>(e.x);
    it.gstride = e.y;
  }
  return it;
}
// Tiles come in boxes of 64 rows, only those the output has, and the MMAs, the
// drain and the slicers stop at the same bounds (columns rounded up to 32, K to the
// 32 of a step): the problems of a batch are small, and whole tiles of 128 x 256 x
// 128 were 2.3 times the work.  B200, whole tiles -> these, us: 2000 problems up to
// 1024 digits 10950 -> 10560, CRT 13760 -> 12690; 300 up to 256 330 -> 313, 514 ->
// 448; 1000 up to 64 458 -> 442, 708 -> 553.
constexpr int G_BOX = 64;
// Tensor maps of a problem.  CRT: A (boxes of 128 rows), B (boxes of G_BOX columns).
// Digits: boxes of 128 rows and of G_BOX for A, of G_BOX, 128 and 256 columns for B,
// and a tile is loaded in as few as there are for it: a box costs the copy engine as
// much as its bytes where one CTA's loads are the bound (100 x 500 x 200, 14 items:
// 46 us in boxes of 64, 38 so).  The CRT form's items are short and gain nothing
// (1000 products up to 64: 566 -> 576 us with the choice).
enum { GM_A, GM_B, GM_CRT, GM_A_BOX = GM_CRT, GM_B128, GM_B256, GM_COUNT };
// nb G_BOX columns of B (1 <= nb <= 4) from column b_row on.
__device__ __forceinline__ void load_b(uint8_t *dst, const CUtensorMap *m, uint64_t *bar, int nb, int k, int b_row,
                                       int slice) {
  if (nb == 4) {
    mftc::tma_load_3d(dst, m + GM_B256, bar, k, b_row, slice);
    return;
  }
  if (nb >= 2) mftc::tma_load_3d(dst, m + GM_B128, bar, k, b_row, slice);
  if (nb & 1) mftc::tma_load_3d(dst + (nb - 1) * G_BOX * BK, m + GM_B, bar, k, b_row + (nb - 1) * G_BOX, slice);
}
// Diagonals of an item of the digit-sliced form: two, or one in a batch that has at
// most five single ones per SM (`items` of them).  Two share their loads and take 7/8
// of the time of two single items where a batch is long; but the longest item, which
// by chance starts last, is 1.75 times as long as a single one, and in a short batch
// that counts for more: with the mean item half as long as the longest, up to
// five or six per SM.  260 random batches, one against two by single items per SM: up to 1
// 0.93, 1 to 3 0.96, 3 to 5 0.97, 5 to 7 1.00, 7 to 17 1.05.  B200, two -> one, us: 512^3
// 82 -> 71, 5 of 100 x 500 x 200 (0.5) 82 -> 70, 4 of 465 x 559 x 22 (3) 109 -> 94, 42
// of 200 x 1000 x 300 (16) 651 -> 714.
constexpr int GD_DIAGS = 2;
static int digit_diags(int64_t items) { return items <= 5 * (int64_t)sm_count() ? 1 : GD_DIAGS; }
__host__ __device__ constexpr int g_groups(int nsl, int diags) { return (nsl + diags - 1) / diags; }
// A block per problem: its items, the longest first.
__global__ void __launch_bounds__(128) g_items(const SProb *probs, const int64_t *prefix, GItem *items) {
  const SProb &P = probs[blockIdx.x];
  const int G = P.plan->G, ntiles = P.ntm * P.ntn, per_g = P.nkc * ntiles, groups = g_groups(P.nsl, P.diags);
  for (int64_t l = threadIdx.x; l < (int64_t)groups * per_g; l += blockDim.x) {
    GItem it;
    const int q = (int)(l / per_g), r = (int)(l % per_g), kc = r / ntiles, tile = r % ntiles;
    it.p = (int)blockIdx.x;
    it.g = P.crt ? P.nsl - 1 - q : G - P.diags * q;
    it.nd = P.crt ? (it.g <= G ? 1 : 0) : max(0, min(P.diags, it.g + 1));
    it.kb0 = kc * P.kcb;
    it.kb1 = min(P.kblocks, it.kb0 + P.kcb);
    it.a_row = tile % P.ntm * BM;
    it.b_row = tile / P.ntm * P.bn;
    it.bn = ((int)min((int64_t)P.bn, P.n - it.b_row) + 31) / 32 * 32;
    it.M_pad = (int)P.M_pad;
    it.rows = (int)min((int64_t)BM, P.m - it.a_row);
    it.klast = it.kb1 < P.kblocks ? BK / UMMA_K : (int)(k_fill(P.k) - (int64_t)(P.kblocks - 1) * BK) / UMMA_K;
    it.pad = 0;
    it.gstride = (int64_t)P.nkc * P.N_pad * P.M_pad;
    const int64_t off = (int64_t)max(it.g, 0) * it.gstride + ((int64_t)kc * P.N_pad + it.b_row) * P.M_pad + it.a_row;
    // CRT: one byte per output, four columns per 32-bit word (crt_device.cuh)
    it.dst = P.crt ? P.D + crt_word_index(off, P.M_pad) : P.D + off;
    items[prefix[blockIdx.x] + l] = it;
  }
}

// Persistent tensor-core kernel of the CRT form over every problem's items,
// one product of a modulus, K chunk and tile each (static round-robin).  The
// warp roles and barriers of split_mma_kernel, with eight epilogue warps (two
// per TMEM lane quadrant, each draining half of the accumulator's columns); per
// item it uses the problem's tensor maps (global memory) and tile width.
constexpr int G_EPI_WARPS = 8;
constexpr int G_THREADS = 64 + 32 * G_EPI_WARPS;  // warp 0 TMA, warp 1 MMA, warps 2-9 epilogue
__global__ void __launch_bounds__(G_THREADS, 1)
    g_crt_mma(const GItem *__restrict__ items, int64_t nitems, const CUtensorMap *__restrict__ maps, int *status,
              uint64_t wait_ns) {
  extern __shared__ uint8_t smem_raw[];
  uint8_t *smem = reinterpret_cast<uint8_t *>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  uint8_t *sA = smem;
  uint8_t *sB = smem + NSTAGE * A_STAGE;
  uint64_t *full = reinterpret_cast<uint64_t *>(smem + NSTAGE * STAGE);
  uint64_t *empty = full + NSTAGE;
  uint64_t *tfull = empty + NSTAGE;
  uint64_t *tempty = tfull + 2;
  uint64_t *drain = tempty + 2;
  uint32_t *tmem_slot = reinterpret_cast<uint32_t *>(drain + 1);
  volatile int *abort_flag = reinterpret_cast<volatile int *>(tmem_slot + 1);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;

  if (threadIdx.x == 0) {
    for (int s = 0; s < NSTAGE; ++s) {
      mftc::mbar_init(&full[s], 1);
      mftc::mbar_init(&empty[s], 1);
    }
    for (int a = 0; a < 2; ++a) {
      mftc::mbar_init(&tfull[a], 1);
      mftc::mbar_init(&tempty[a], G_EPI_WARPS);
    }
    mftc::mbar_init(drain, 1);
    *abort_flag = 0;
    mftc::fence_mbar_init();
  }
  if (warp == 1) {
    mftc::tmem_alloc(tmem_slot, TMEM_COLS);
    mftc::tmem_relinquish();
  }
  mftc::tc_fence_before();
  __syncthreads();
  mftc::tc_fence_after();
  const uint32_t tmem_base = *tmem_slot;
  auto fail = [&](int code) {
    *abort_flag = 1;
    record_abort(status, code);
  };
  ArmedStages<NSTAGE> arm;  // the producer's armed stages
  arm.clear();
  if (warp == 0) {
    if (lane == 0) {
      int stage = 0;
      uint32_t phase = 0;
      bool ok = true;
      GItem next = load_item(items, blockIdx.x, nitems);
      for (int64_t w = blockIdx.x; w < nitems && ok; w += gridDim.x) {
        const GItem it = next;
        next = load_item(items, w + gridDim.x, nitems);
        if (!it.nd) continue;
        const int nb = (it.bn + G_BOX - 1) / G_BOX;
        const uint32_t bytes = (uint32_t)(A_STAGE + nb * G_BOX * BK);
        for (int kb = it.kb0; kb < it.kb1; ++kb) {
          if (!wait_bar(&empty[stage], phase ^ 1, abort_flag, wait_ns)) {
            fail(1);
            ok = false;
            break;
          }
          mftc::mbar_arrive_expect_tx(&full[stage], bytes);
          // A: MN-major residue planes (row, K index, modulus)
          mftc::tma_load_3d(sA + stage * A_STAGE, &maps[GM_CRT * it.p + GM_A], &full[stage], it.a_row, kb * BK, it.g);
          for (int b = 0; b < nb; ++b)
            mftc::tma_load_3d(sB + stage * B_STAGE + b * G_BOX * BK, &maps[GM_CRT * it.p + GM_B], &full[stage], kb * BK,
                              it.b_row + b * G_BOX, it.g);
          arm.arm(stage, phase);
          if (++stage == NSTAGE) {
            stage = 0;
            phase ^= 1;
          }
        }
      }
    }
  } else if (warp == 1) {
    if (lane == 0) {
      int stage = 0;
      uint32_t phase = 0;
      int acc = 0;
      uint32_t acc_phase = 0;
      bool ok = true;
      GItem next = load_item(items, blockIdx.x, nitems);
      for (int64_t w = blockIdx.x; w < nitems && ok; w += gridDim.x) {
        const GItem it = next;
        next = load_item(items, w + gridDim.x, nitems);
        if (!it.nd) continue;
        const uint32_t idesc = mftc::idesc_u8(BM, it.bn) | mftc::IDESC_A_MN;
        const uint32_t a_kstep = 32 * 128;  // a K step of 32 rows of the MN-major A tile
        if (!wait_bar(&tempty[acc], acc_phase ^ 1, abort_flag, wait_ns)) {
          fail(2);
          break;
        }
        mftc::tc_fence_after();
        const uint32_t d_tmem = tmem_base + (uint32_t)(acc * BN);
        uint32_t accumulate = 0;
        for (int kb = it.kb0; kb < it.kb1; ++kb) {
          if (!wait_bar(&full[stage], phase, abort_flag, wait_ns)) {
            fail(4);
            ok = false;
            break;
          }
          mftc::tc_fence_after();
          const uint32_t a0 = mftc::smem_u32(sA + stage * A_STAGE);
          const uint32_t b0 = mftc::smem_u32(sB + stage * B_STAGE);
          const int ks = kb == it.kb1 - 1 ? it.klast : BK / UMMA_K;
#pragma unroll
          for (int kk = 0; kk < BK / UMMA_K; ++kk) {
            if (kk >= ks) break;
            mftc::umma_i8(d_tmem, mftc::smem_desc_k_sw128(a0 + kk * a_kstep),
                          mftc::smem_desc_k_sw128(b0 + kk * UMMA_K), idesc, accumulate);
            accumulate = 1;
          }
          mftc::umma_commit(&empty[stage]);
          if (++stage == NSTAGE) {
            stage = 0;
            phase ^= 1;
          }
        }
        if (!ok) break;
        mftc::umma_commit(&tfull[acc]);
        if (++acc == 2) {
          acc = 0;
          acc_phase ^= 1;
        }
      }
      mftc::umma_commit(drain);
      uint64_t t0 = globaltimer();
      while (!mftc::mbar_try_wait(drain, 0) && globaltimer() - t0 < WAIT_NS) {
      }
    }
  } else {
    const int quad = warp & 3;           // TMEM lanes this warp may read
    const int half = (warp - 2) / 4;     // which half of the accumulator's columns
    const int row = quad * 32 + lane;
    int acc = 0;
    uint32_t acc_phase = 0;
    GItem next = load_item(items, blockIdx.x, nitems);
    for (int64_t w = blockIdx.x; w < nitems; w += gridDim.x) {
      const GItem it = next;
      next = load_item(items, w + gridDim.x, nitems);
      if (!it.nd) continue;
      bool got = wait_bar(&tfull[acc], acc_phase, abort_flag, wait_ns);
      if (!__all_sync(0xffffffffu, got)) {
        if (lane == 0) fail(8);
        break;
      }
      mftc::tc_fence_after();
      const int nch = quad * 32 < it.rows ? it.bn / 32 : 0;  // 32-column chunks, every other one this warp's
      for (int chunk = half; chunk < nch; chunk += 2) {
        // residues modulo m_g, four columns per 32-bit word (crt_device.cuh)
        uint32_t *dst = reinterpret_cast<uint32_t *>(it.dst) + row + (int64_t)chunk * 8 * it.M_pad;
        uint32_t r[32];
        mftc::tmem_ld_32x32b_x32(tmem_base + ((uint32_t)(quad * 32) << 16) + (uint32_t)(acc * BN + chunk * 32), r);
        mftc::tmem_wait_ld();
#pragma unroll
        for (int g = 0; g < 8; ++g) {
          __stcs(dst, crt_pack4(r[4 * g], r[4 * g + 1], r[4 * g + 2], r[4 * g + 3], it.g));
          dst += it.M_pad;
        }
      }
      mftc::tc_fence_before();
      __syncwarp();
      if (lane == 0) mftc::mbar_arrive(&tempty[acc]);
      if (++acc == 2) {
        acc = 0;
        acc_phase ^= 1;
      }
    }
  }
  mftc::tc_fence_before();
  __syncthreads();
  mftc::tc_fence_after();
  if (*abort_flag) {  // read after the barrier: the same value in every thread
    // copies in flight that no MMA consumed land before shared memory is released
    if (warp == 0 && lane == 0) arm.drain(full, NSTAGE);
    __syncthreads();
  }
  if (warp == 1) {
    __syncwarp();
    mftc::tmem_dealloc(tmem_base, TMEM_COLS);
  }
}

// Persistent tensor-core kernel of the digit-sliced form.  An item is one diagonal g
// (digit_diags), or two consecutive ones g, g - 1, of one tile (128 rows x bn <= 256 columns) and
// K chunk, accumulated side by side in tensor memory.  Per K block the slices
// come in the order A_0, B_g, B_{g-1}, A_1, B_{g-2}, ...: step s multiplies A_s
// with B_{g-s} and B_{g-s-1}, one product per diagonal, and then lets A_s and
// B_{g-s} go, so each slice is loaded once for both diagonals.  B has more slots
// than A because a step holds two B tiles but one A tile; as every step takes one
// of each and frees one of each, the n-th tiles of both belong together: one
// barrier says that what steps up to n multiply has landed (A_n and the B tiles
// loaded with it, one ahead), one that the n-th tile of both is free, which with
// one slot of B more also frees the one ahead.
//
// CTAs take items from a counter (the producer does, one item ahead, and hands
// each to the other roles through a small ring in shared memory): dealt round
// robin the busiest CTA had 16 % more work than the mean.
//
// Bound: the operands from L2 (45 GB for 2000 products up to 1024: 10 TB/s; the MMAs
// alone would take 2.6 ms of the 4.5), then the drain, hidden only
// behind the next item's loads (the accumulators fill tensor memory; they are
// handed back one by one in the order the next item needs them).  Four
// diagonals on 128 x 128 tiles load less, but a 128-column MMA takes 102 cycles
// instead of its 64 (shared-memory reads).  2000 products of sizes up to 1024:
// 9.0 ms with one diagonal at a time and items found by bisection, 7.8 four by
// 128 columns, 6.0 two by 256.  With barriers and commits of their own for A and B
// a step cost 0.2 us more: 5.65 -> 4.50 ms with one (under ncu, both); 100 x 500 x 200
// alone 52 -> 41 us.
constexpr int GD_BN = BN, GD_NA = 4, GD_NB = 5, GD_NW = 4;
constexpr int GD_TILE_A = A_STAGE, GD_TILE_B = B_STAGE;  // bytes of a slot
constexpr int GD_SMEM = GD_NA * GD_TILE_A + GD_NB * GD_TILE_B + 1024 /*align*/ + 512 /*barriers, items*/;
static_assert(GD_DIAGS * GD_BN == TMEM_COLS, "accumulators fill tensor memory");
static_assert(GD_NB >= GD_NA + GD_DIAGS - 1, "a free step of A means free slots of B");

// Position in a ring of N slots and the parity of its current pass.
template <int N>
struct RingPos {
  int slot = 0;
  uint32_t phase = 0;
  __device__ __forceinline__ void advance() {
    if (++slot == N) {
      slot = 0;
      phase ^= 1;
    }
  }
  __device__ __forceinline__ int at(int d) const { return slot + d < N ? slot + d : slot + d - N; }
};

__global__ void __launch_bounds__(G_THREADS, 1)
    g_digit_mma(const GItem *__restrict__ items, int64_t nitems, int *counter, const CUtensorMap *__restrict__ maps,
                int *status, uint64_t wait_ns) {
  extern __shared__ uint8_t smem_raw[];
  uint8_t *sA = reinterpret_cast<uint8_t *>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  uint8_t *sB = sA + GD_NA * GD_TILE_A;
  uint64_t *full = reinterpret_cast<uint64_t *>(sB + GD_NB * GD_TILE_B);
  uint64_t *empty = full + GD_NA;
  uint64_t *tempty = empty + GD_NA;     // per accumulator
  uint64_t *tfull = tempty + GD_DIAGS;  // the item's accumulators
  uint64_t *wfull = tfull + 1;  // the ring of items
  uint64_t *wempty = wfull + GD_NW;
  uint64_t *drain = wempty + GD_NW;
  GItem *work = reinterpret_cast<GItem *>((reinterpret_cast<uintptr_t>(drain + 2) + 15) & ~uintptr_t(15));
  uint32_t *tmem_slot = reinterpret_cast<uint32_t *>(drain + 1);
  volatile int *abort_flag = reinterpret_cast<volatile int *>(tmem_slot + 1);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;

  if (threadIdx.x == 0) {
    for (int s = 0; s < GD_NA; ++s) {
      mftc::mbar_init(&full[s], 1);
      mftc::mbar_init(&empty[s], 1);
    }
    for (int d = 0; d < GD_DIAGS; ++d) mftc::mbar_init(&tempty[d], G_EPI_WARPS);
    mftc::mbar_init(tfull, 1);
    for (int s = 0; s < GD_NW; ++s) {
      mftc::mbar_init(&wfull[s], 1);
      mftc::mbar_init(&wempty[s], 1 + G_EPI_WARPS);  // the issuer and every epilogue warp
    }
    mftc::mbar_init(drain, 1);
    *abort_flag = 0;
    mftc::fence_mbar_init();
  }
  if (warp == 1) {
    mftc::tmem_alloc(tmem_slot, TMEM_COLS);
    mftc::tmem_relinquish();
  }
  mftc::tc_fence_before();
  __syncthreads();
  mftc::tc_fence_after();
  const uint32_t tmem_base = *tmem_slot;
  auto fail = [&](int code) {
    *abort_flag = 1;
    record_abort(status, code);
  };
  ArmedStages<GD_NA> arm;  // the producer's armed steps
  arm.clear();

  if (warp == 0) {
    if (lane == 0) {  // ---- TMA producer
      RingPos<GD_NA> ra;
      RingPos<GD_NB> rb;
      RingPos<GD_NW> rw;
      bool ok = true;
      int64_t w = (unsigned)atomicAdd(counter, 1);
      GItem next = load_item(items, w, nitems);
      while (ok) {
        const GItem it = next;
        const bool end = w >= nitems;
        if (!end) {
          w = (unsigned)atomicAdd(counter, 1);
          next = load_item(items, w, nitems);
        }
        if (!end && !it.nd) continue;
        if (!wait_bar(&wempty[rw.slot], rw.phase ^ 1, abort_flag, wait_ns)) {
          fail(1);
          break;
        }
        work[rw.slot] = it;  // nd = 0: no more items
        mftc::mbar_arrive(&wfull[rw.slot]);
        rw.advance();
        if (end) break;
        const CUtensorMap *m = &maps[GM_COUNT * it.p];
        const int na = (it.rows + G_BOX - 1) / G_BOX, nb = (it.bn + G_BOX - 1) / G_BOX;
        for (int kb = it.kb0; kb < it.kb1 && ok; ++kb) {
          int t = it.g;  // next slice of B
          for (int s = 0; s <= it.g; ++s) {
            if (!wait_bar(&empty[ra.slot], ra.phase ^ 1, abort_flag, wait_ns)) {
              fail(1);
              ok = false;
              break;
            }
            const int upto = max(it.g - s - it.nd + 1, 0);  // the last slice of B that step s multiplies
            mftc::mbar_arrive_expect_tx(&full[ra.slot], (uint32_t)((na + (t - upto + 1) * nb) * G_BOX * BK));
            mftc::tma_load_3d(sA + ra.slot * GD_TILE_A, m + (na == 1 ? GM_A_BOX : GM_A), &full[ra.slot], kb * BK,
                              it.a_row, s);
            for (; t >= upto; --t) {
              load_b(sB + rb.slot * GD_TILE_B, m, &full[ra.slot], nb, kb * BK, it.b_row, t);
              rb.advance();
            }
            arm.arm(ra.slot, ra.phase);
            ra.advance();
          }
        }
      }
    }
  } else if (warp == 1) {
    if (lane == 0) {  // ---- MMA issuer
      const uint64_t descA = mftc::smem_desc_k_sw128(mftc::smem_u32(sA));
      const uint64_t descB = mftc::smem_desc_k_sw128(mftc::smem_u32(sB));
      RingPos<GD_NA> ra;
      RingPos<GD_NB> rb;
      uint32_t acc_phase = 0;  // bit d: parity of tempty[d]
      bool ok = true;
      RingPos<GD_NW> rw;
      while (ok) {
        if (!wait_bar(&wfull[rw.slot], rw.phase, abort_flag, wait_ns)) {
          fail(4);
          break;
        }
        const int g = work[rw.slot].g, it_nd = work[rw.slot].nd, kb0 = work[rw.slot].kb0, kb1 = work[rw.slot].kb1,
                  bn = work[rw.slot].bn, klast = work[rw.slot].klast;
        mftc::mbar_arrive(&wempty[rw.slot]);
        rw.advance();
        if (!it_nd) break;
        const uint32_t idesc = mftc::idesc_i8(BM, bn);
        uint32_t accumulate = 0;
        for (int kb = kb0; kb < kb1 && ok; ++kb) {
          const int ks = kb == kb1 - 1 ? klast : BK / UMMA_K;
          for (int s = 0; s <= g; ++s) {
            const int nd = min(it_nd, g - s + 1);
            if (!wait_bar(&full[ra.slot], ra.phase, abort_flag, wait_ns)) {
              fail(4);
              ok = false;
              break;
            }
            mftc::tc_fence_after();
            const uint64_t ad = descA + (uint64_t)(ra.slot * (GD_TILE_A / 16));
#pragma unroll
            for (int d = 0; d < GD_DIAGS; ++d) {
              if (d >= nd) break;
              if (!accumulate) {  // first step: the previous item's drain handed this accumulator back
                if (!wait_bar(&tempty[d], ((acc_phase >> d) & 1u) ^ 1u, abort_flag, wait_ns)) {
                  fail(2);
                  ok = false;
                  break;
                }
                acc_phase ^= 1u << d;
                mftc::tc_fence_after();
              }
              const uint64_t bd = descB + (uint64_t)(rb.at(d) * (GD_TILE_B / 16));
              const uint32_t acc = tmem_base + (uint32_t)(d * GD_BN);
#pragma unroll
              for (int kk = 0; kk < BK / UMMA_K; ++kk)
                if (kk < ks) mftc::umma_i8(acc, ad + (uint64_t)(kk * UMMA_K / 16), bd + (uint64_t)(kk * UMMA_K / 16), idesc,
                              kk == 0 ? accumulate : 1u);
            }
            if (!ok) break;
            accumulate = 1;
            mftc::umma_commit(&empty[ra.slot]);
            ra.advance();
            rb.advance();
          }
        }
        if (!ok) break;
        mftc::umma_commit(tfull);
      }
      mftc::umma_commit(drain);
      uint64_t t0 = globaltimer();
      while (!mftc::mbar_try_wait(drain, 0) && globaltimer() - t0 < WAIT_NS) {
      }
    }
  } else {  // ---- epilogue
    const int quad = warp & 3;        // TMEM lanes this warp may read
    const int half = (warp - 2) / 4;  // which half of an accumulator's columns
    const int row = quad * 32 + lane;
    uint32_t item_phase = 0;
    RingPos<GD_NW> rw;
    while (true) {
      bool got = wait_bar(&wfull[rw.slot], rw.phase, abort_flag, wait_ns);
      if (!__all_sync(0xffffffffu, got)) {
        if (lane == 0) fail(8);
        break;
      }
      int32_t *const it_dst = work[rw.slot].dst;
      const int64_t gstride = work[rw.slot].gstride;
      const int nd = work[rw.slot].nd, M_pad = work[rw.slot].M_pad;
      // 32-column chunks, every other one this warp's
      const int nch = quad * 32 < work[rw.slot].rows ? work[rw.slot].bn / 32 : 0;
      __syncwarp();
      if (lane == 0) mftc::mbar_arrive(&wempty[rw.slot]);
      rw.advance();
      if (!nd) break;
      got = wait_bar(tfull, item_phase, abort_flag, wait_ns);
      if (!__all_sync(0xffffffffu, got)) {
        if (lane == 0) fail(8);
        break;
      }
      item_phase ^= 1;
      mftc::tc_fence_after();
      for (int d = 0; d < nd; ++d) {
        for (int chunk = half; chunk < nch; chunk += 2) {
          int32_t *dst = it_dst - d * gstride + (int64_t)chunk * 32 * M_pad + row;
          uint32_t r[32];
          mftc::tmem_ld_32x32b_x32(
              tmem_base + ((uint32_t)(quad * 32) << 16) + (uint32_t)(d * GD_BN + chunk * 32), r);
          mftc::tmem_wait_ld();
#pragma unroll
          for (int q = 0; q < 32; ++q) {
            __stcs(dst, (int32_t)r[q]);  // evict-first: keep L2 for the slices
            dst += M_pad;
          }
        }
        mftc::tc_fence_before();
        __syncwarp();
        if (lane == 0) mftc::mbar_arrive(&tempty[d]);
      }
    }
  }
  mftc::tc_fence_before();
  __syncthreads();
  mftc::tc_fence_after();
  if (*abort_flag) {  // read after the barrier: the same value in every thread
    // copies in flight that no MMA consumed land before shared memory is released
    if (warp == 0 && lane == 0) arm.drain(full, GD_NA);
    __syncthreads();
  }
  if (warp == 1) {
    __syncwarp();
    mftc::tmem_dealloc(tmem_base, TMEM_COLS);
  }
}

__global__ void fill_kernel(int *p, int64_t n, int v) {
  int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n) p[i] = v;
}

// ===========================================================================
// autotuner cache
// ===========================================================================
static std::mutex g_tune_mu;
static std::map<std::string, int> g_tune;
static bool g_tune_loaded = false;

static std::string cache_path() {
  const char *p = std::getenv("MFCUDA_AUTOTUNE_CACHE");
  if (p && *p) return p;
  const char *home = std::getenv("HOME");
  return std::string(home ? home : "/tmp") + "/.cache/multifloats_b200/autotune.txt";
}
static void tune_load() {
  if (g_tune_loaded) return;
  g_tune_loaded = true;
  FILE *f = std::fopen(cache_path().c_str(), "r");
  if (!f) return;
  char key[256];
  int v;
  while (std::fscanf(f, "%255s %d", key, &v) == 2) g_tune[key] = v;
  std::fclose(f);
}
static void tune_save() {
  std::string path = cache_path();
  std::string dir = path.substr(0, path.find_last_of('/'));
  for (size_t i = 1; i <= dir.size(); ++i)  // create the directory chain
    if (i == dir.size() || dir[i] == '/') (void)::mkdir(dir.substr(0, i).c_str(), 0755);
  FILE *f = std::fopen(path.c_str(), "w");
  if (!f) return;
  for (auto &kv : g_tune) std::fprintf(f, "%s %d\n", kv.first.c_str(), kv.second);
  std::fclose(f);
}


// ===========================================================================
// host side
// ===========================================================================
static int clog2(int64_t v) {
  int b = 0;
  while (((int64_t)1 << b) < v) ++b;
  return b;
}
static int64_t ru(int64_t v, int64_t m) { return (v + m - 1) / m * m; }

static bool aligned16(const void *p) { return (reinterpret_cast<uintptr_t>(p) & 15) == 0; }

// Tiles of a plain batch: the tuner's winner, or 32 x 32, or 16 x 16 for problems
// under 24 rows or columns; smaller ones where a tile's k loop outlasts the batch,
// which the tuner, timing a bucket alone at one k, cannot see.  With
// two CTAs per SM a tile of 32 costs its SM 0.139 us per step and takes 0.28 us
// to do one, a tile of 16 0.043 and 0.087 (measured): a problem whose k steps
// of 0.28 us exceed the whole batch's work spread over the SMs would set the
// time alone.  Tiles of 64 do the same work 2 % cheaper but take 1.0 us a step:
// 2000 problems up to 1024 29.1 ms with 64, 29.0 with 32; 30 up to 600 603 us
// against 222 by this rule, 60 up to 300 308 against 96, 20 up to 200 105
// against 23; tuned ones 603 -> 223, 307 -> 102, 105 -> 23.
constexpr double kStep32 = 0.139, kLatency32 = 0.28, kLatency64 = 1.0;
static int plain_heuristic(int64_t m, int64_t n) { return std::min(m, n) >= 24 ? 1 : 2; }
static void plain_small_tiles(const mfcuda_gemm_desc *d, int64_t count, std::vector<int> &cfg) {
  double work = 0.0;
  for (int64_t p = 0; p < count; ++p)
    work += (double)((d[p].m + 31) / 32) * (double)((d[p].n + 31) / 32) * (double)d[p].k * kStep32;
  const double balanced = work / sm_count();
  for (int64_t p = 0; p < count; ++p) {
    if (cfg[p] == 0 && (double)d[p].k * kLatency64 > balanced) cfg[p] = 1;
    if (cfg[p] == 1 && (double)d[p].k * kLatency32 > balanced) cfg[p] = 2;
  }
}

// Plan memory: one device allocation holding the tables and the workspace.
struct Arena {
  size_t off = 0;
  size_t take(size_t bytes, size_t align = 256) {
    off = (off + align - 1) / align * align;
    size_t o = off;
    off += bytes;
    return o;
  }
};

}  // namespace batch
}  // namespace mfcuda

struct mfcuda_batch {
  int kind = 0;  // 0 plain GEMM, 1 split GEMM, 2 ragged unary
  int kchunk = 0;  // split: K chunk in elements
  int device = 0;
  void *mem = nullptr;
  size_t mem_bytes = 0;
  cudaGraph_t graph = nullptr;
  cudaGraphExec_t exec = nullptr;
  int64_t count = 0, work = 0;
  int *status = nullptr;
  std::vector<int> cfg;
};

namespace mfcuda {
namespace batch {

static void destroy(mfcuda_batch *b) {
  if (!b) return;
  if (b->exec) cudaGraphExecDestroy(b->exec);
  if (b->graph) cudaGraphDestroy(b->graph);
  if (b->mem) cudaFree(b->mem);
  delete b;
}

// Captures `enqueue` (a sequence of launches on the given stream) into the
// plan's graph.
template <class F>
static int capture(mfcuda_batch *b, F enqueue) {
  cudaStream_t cs;
  MF_TRY_CUDA(cudaStreamCreateWithFlags(&cs, cudaStreamNonBlocking));
  int rc = MFCUDA_OK;
  if (cudaStreamBeginCapture(cs, cudaStreamCaptureModeThreadLocal) != cudaSuccess) {
    rc = MFCUDA_ERR_CUDA;
  } else {
    enqueue(cs);
    cudaError_t e1 = cudaGetLastError();
    cudaError_t e2 = cudaStreamEndCapture(cs, &b->graph);
    if (e1 != cudaSuccess || e2 != cudaSuccess)
      rc = MFCUDA_ERR_CUDA;
    else if (cudaGraphInstantiate(&b->exec, b->graph, 0) != cudaSuccess)
      rc = MFCUDA_ERR_CUDA;
  }
  (void)cudaGetLastError();
  cudaStreamDestroy(cs);
  return rc;
}

// ---- plain ------------------------------------------------------------------
// complex = true: complex64x2 problems, 32 x 32 tiles (cfg ignored).
static int create_plain(const mfcuda_gemm_desc *d, int64_t count, int64_t ri, const std::vector<int> &cfg,
                        mfcuda_batch **out, bool complex = false) {
  std::vector<int64_t> order;
  bool aligned = true;
  for (int64_t p = 0; p < count; ++p) {
    if (d[p].m > 0 && d[p].n > 0) order.push_back(p);
    aligned = aligned && aligned16(d[p].a) && aligned16(d[p].b) && aligned16(d[p].c);
  }
  std::stable_sort(order.begin(), order.end(), [&](int64_t x, int64_t y) { return d[x].k > d[y].k; });
  std::vector<PProb> probs(count);
  std::vector<PItem> items;
  for (int64_t p = 0; p < count; ++p)
    probs[p] = {static_cast<const double *>(d[p].a), static_cast<const double *>(d[p].b),
                static_cast<double *>(d[p].c), d[p].m, d[p].k, d[p].n};
  for (int64_t p : order) {
    const int e = complex ? 32 : cfg_edge(cfg[p]);
    for (int64_t tn = 0; tn < (d[p].n + e - 1) / e; ++tn)
      for (int64_t tm = 0; tm < (d[p].m + e - 1) / e; ++tm)
        items.push_back({(int)p, complex ? 1 : cfg[p], (int)tm, (int)tn});
  }
  if (items.size() > (size_t)INT32_MAX) return MFCUDA_ERR_UNSUPPORTED;
  auto *b = new mfcuda_batch;
  b->kind = 0;
  b->count = count;
  b->work = (int64_t)items.size();
  b->cfg = cfg;
  cudaGetDevice(&b->device);
  Arena ar;
  size_t o_probs = ar.take(sizeof(PProb) * std::max<int64_t>(count, 1));
  size_t o_items = ar.take(sizeof(PItem) * std::max<size_t>(items.size(), 1));
  size_t o_ctr = ar.take(sizeof(int));
  b->mem_bytes = ar.off;
  if (injected_alloc_failure() || device_malloc(&b->mem, b->mem_bytes) != cudaSuccess) {
    (void)cudaGetLastError();
    destroy(b);
    return MFCUDA_ERR_ALLOC;
  }
  uint8_t *base = static_cast<uint8_t *>(b->mem);
  PProb *dp = reinterpret_cast<PProb *>(base + o_probs);
  PItem *di = reinterpret_cast<PItem *>(base + o_items);
  int *ctr = reinterpret_cast<int *>(base + o_ctr);
  if (cudaMemcpy(dp, probs.data(), sizeof(PProb) * count, cudaMemcpyHostToDevice) != cudaSuccess ||
      (!items.empty() &&
       cudaMemcpy(di, items.data(), sizeof(PItem) * items.size(), cudaMemcpyHostToDevice) != cudaSuccess)) {
    destroy(b);
    return MFCUDA_ERR_CUDA;
  }
  const int nitems = (int)items.size();
  int grid = sm_count() * 2;
  if (grid > nitems) grid = nitems > 0 ? nitems : 1;
  auto pick = [&](auto al, auto sh) {
    return complex ? cplain_grouped_kernel<al, sh> : plain_grouped_kernel<al, sh>;
  };
  const std::true_type yes;
  const std::false_type no;
  const bool sh = gtile::short_interval(ri);
  auto *kernel = aligned ? (sh ? pick(yes, yes) : pick(yes, no)) : sh ? pick(no, yes) : pick(no, no);
  int rc = capture(b, [&](cudaStream_t cs) {
    cudaMemsetAsync(ctr, 0, sizeof(int), cs);
    kernel<<<grid, 256, 0, cs>>>(dp, di, nitems, ri, ctr);
  });
  if (rc != MFCUDA_OK) {
    destroy(b);
    return rc;
  }
  *out = b;
  return MFCUDA_OK;
}

// ---- split ------------------------------------------------------------------
static std::once_flag g_gmma_attr;

static PFN_cuTensorMapEncodeTiled_v12000 encode_fn() {
  static PFN_cuTensorMapEncodeTiled_v12000 fn = [] {
    void *p = nullptr;
    cudaDriverEntryPointQueryResult q;
    if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &p, cudaEnableDefault, &q) != cudaSuccess ||
        q != cudaDriverEntryPointSuccess)
      p = nullptr;
    return reinterpret_cast<PFN_cuTensorMapEncodeTiled_v12000>(p);
  }();
  return fn;
}
static bool make_map(CUtensorMap *map, void *base, int64_t rows, int64_t K_pad, uint32_t box_rows, int nsl) {
  auto fn = encode_fn();
  if (!fn) return false;
  cuuint64_t dims[3] = {(cuuint64_t)K_pad, (cuuint64_t)rows, (cuuint64_t)nsl};
  cuuint64_t strides[2] = {(cuuint64_t)K_pad, (cuuint64_t)(rows * K_pad)};
  cuuint32_t box[3] = {(cuuint32_t)BK, box_rows, 1};
  cuuint32_t estr[3] = {1, 1, 1};
  return fn(map, CU_TENSOR_MAP_DATA_TYPE_UINT8, 3, base, dims, strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE,
            CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
            CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

// MN-major residue planes (row, K index, modulus) of the CRT form's A side:
// boxes of 128 rows x BK K indices, 128-byte swizzle.
static bool make_map_mn(CUtensorMap *map, void *base, int64_t M_pad, int64_t K_pad, int nsl) {
  auto fn = encode_fn();
  if (!fn) return false;
  cuuint64_t dims[3] = {(cuuint64_t)M_pad, (cuuint64_t)K_pad, (cuuint64_t)nsl};
  cuuint64_t strides[2] = {(cuuint64_t)M_pad, (cuuint64_t)(M_pad * K_pad)};
  cuuint32_t box[3] = {128, (cuuint32_t)BK, 1};
  cuuint32_t estr[3] = {1, 1, 1};
  return fn(map, CU_TENSOR_MAP_DATA_TYPE_UINT8, 3, base, dims, strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE,
            CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
            CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

// One real product to plan (host side of SProb): operand / output views, its
// tile width, and where its A operand, B operand and plan come from (-1: its
// own; else the index of the product that provides them).  A plan owner lists
// in plan_a2 / plan_b2 the products whose A / B statistics also enter its plan.
struct Spec {
  const double *A, *B;
  double *C;
  int64_t astride, bstride, cstride;
  int mode;
  int64_t m, k, n;
  int bn;
  int a_src, b_src, plan_src, plan_a2, plan_b2;
};

// kcb: K chunk in blocks of 128 (shared by all products).  crt: the CRT form,
// `slices` then being the operand bits W (0: chosen for `target`).
static int create_split_specs(std::vector<Spec> specs, int64_t count, int slices, double target,
                              const std::vector<int> &cfg, int kcb_all, mfcuda_batch **out, bool crt) {
  // longest K first (stable: the products of one complex problem stay together)
  const int np = (int)specs.size();
  std::vector<int> order(np), pos(np);
  for (int q = 0; q < np; ++q) order[q] = q;
  std::stable_sort(order.begin(), order.end(), [&](int x, int y) { return specs[x].k > specs[y].k; });
  for (int q = 0; q < np; ++q) pos[order[q]] = q;
  std::vector<Spec> sp(np);
  for (int q = 0; q < np; ++q) {
    sp[q] = specs[order[q]];
    for (int *r : {&sp[q].a_src, &sp[q].b_src, &sp[q].plan_src, &sp[q].plan_a2, &sp[q].plan_b2})
      if (*r >= 0) *r = pos[*r];
  }
  std::vector<SProb> probs(np);
  Arena ar;
  size_t o_probs = ar.take(sizeof(SProb) * std::max(np, 1));
  size_t o_prefix = ar.take(sizeof(int64_t) * std::max(np, 1));
  const size_t nmaps = crt ? GM_CRT : GM_COUNT;  // per problem
  size_t o_maps = ar.take(sizeof(CUtensorMap) * nmaps * std::max(np, 1), 128);
  size_t o_status = ar.take(2 * sizeof(int));  // abort codes, the digit kernel's item counter
  std::vector<size_t> o_plan(np, 0), o_cc(np, 0), o_as(np, 0), o_bs(np, 0), o_d(np);
  std::vector<int64_t> rowA(np, -1), rowB(np, -1);  // statistics rows of owned operands
  int64_t rows_total = 0;
  std::vector<int64_t> prefix((size_t)std::max(np, 1), 0);  // of the items
  std::vector<Owner> owner[PH_ITEMS];                         // of the blocks of the other phases
  int64_t total[PH_COUNT] = {0, 0, 0, 0, 0, 0, 0};
  int64_t singles = 0;  // items of one diagonal each, at the most slices a plan may take
  for (const Spec &g : sp) {
    const int64_t kblocks = ru(g.k < 1 ? 1 : g.k, BK) / BK, kcb = std::min(kcb_all, KC_BLOCKS);
    singles += (slices > 0 ? slices : SMAX) * ((kblocks + kcb - 1) / kcb) * (ru(g.m, BM) / BM) * (ru(g.n, g.bn) / g.bn);
  }
  const int diags = crt ? 1 : digit_diags(singles);
  for (int q = 0; q < np; ++q) {
    const Spec &g = sp[q];
    SProb &P = probs[q];
    P.A = g.A;
    P.B = g.B;
    P.C = g.C;
    P.astride = g.astride;
    P.bstride = g.bstride;
    P.cstride = g.cstride;
    P.mode = g.mode;
    P.own_a = g.a_src < 0;
    P.own_b = g.b_src < 0;
    P.own_plan = g.plan_src < 0;
    P.m = g.m;
    P.k = g.k;
    P.n = g.n;
    P.bn = g.bn;
    P.M_pad = ru(g.m, BM);
    P.N_pad = ru(g.n, P.bn);
    P.K_pad = ru(g.k < 1 ? 1 : g.k, BK);
    P.kblocks = (int)(P.K_pad / BK);
    P.kcb = std::min(kcb_all, KC_BLOCKS);
    P.nkc = (P.kblocks + P.kcb - 1) / P.kcb;
    P.ntm = (int)(P.M_pad / BM);
    P.ntn = (int)(P.N_pad / P.bn);
    P.crt = crt ? 1 : 0;
    P.nsl = crt ? crt_slices_max(g.k < 1 ? 1 : g.k, slices) : SMAX;
    P.diags = diags;
    P.cc = nullptr;
    if (P.own_plan) {
      o_plan[q] = ar.take(sizeof(Plan));
      if (crt) o_cc[q] = ar.take(sizeof(CrtConst));
    }
    if (P.own_a) {
      rowA[q] = rows_total;
      rows_total += P.M_pad;
      o_as[q] = ar.take((size_t)P.nsl * P.M_pad * P.K_pad, 1024);
    }
    if (P.own_b) {
      rowB[q] = rows_total;
      rows_total += P.N_pad;
      o_bs[q] = ar.take((size_t)P.nsl * P.N_pad * P.K_pad, 1024);
    }
    // INT32 diagonal sums, or (CRT) byte residues four columns to a word
    o_d[q] = ar.take((size_t)P.nsl * P.nkc * P.N_pad * P.M_pad * (crt ? 1 : sizeof(int32_t)));
    const int64_t comb = crt ? crt_combine_blocks(P.m, P.n) : combine_blocks(P.m, P.n);
    const int64_t blocks[PH_COUNT] = {
        P.own_a ? ((P.m + 255) / 256) * ((P.k + 63) / 64) : 0,
        P.own_b && P.k > 0 ? (P.n + 7) / 8 : 0,
        P.own_a ? (crt ? (k_fill(P.k) * ((P.m + 7) / 8) + 255) / 256 : ((P.m + 31) / 32) * ((k_fill(P.k) + 63) / 64)) : 0,
        P.own_b ? (P.n * (k_fill(P.k) / 8) + 255) / 256 : 0,
        P.mode == 0 ? comb : 0,
        P.mode != 0 ? comb : 0,
        (int64_t)g_groups(P.nsl, P.diags) * P.nkc * P.ntm * P.ntn};
    prefix[q] = total[PH_ITEMS];
    for (int ph = 0; ph < PH_COUNT; ++ph) {
      total[ph] += blocks[ph];
      if (total[ph] > INT32_MAX) return MFCUDA_ERR_UNSUPPORTED;
      if (ph != PH_ITEMS)
        for (int64_t l = 0; l < blocks[ph]; ++l) owner[ph].push_back({q, (int)l});
    }
  }
  size_t o_owner[PH_ITEMS];
  for (int ph = 0; ph < PH_ITEMS; ++ph) o_owner[ph] = ar.take(sizeof(Owner) * std::max<int64_t>(total[ph], 1));
  const size_t o_items = ar.take(sizeof(GItem) * std::max<int64_t>(total[PH_ITEMS], 1));
  // exponent statistics of all owned operands in three contiguous arrays
  const size_t o_sig = ar.take(sizeof(int) * std::max<int64_t>(rows_total, 1));
  const size_t o_mu = ar.take(sizeof(int) * std::max<int64_t>(rows_total, 1));
  const size_t o_flag = ar.take(sizeof(int) * std::max<int64_t>(rows_total, 1));
  auto *b = new mfcuda_batch;
  b->kind = 1;
  b->kchunk = std::min(kcb_all, KC_BLOCKS) * BK;
  b->count = count;
  b->work = total[PH_ITEMS];
  b->cfg = cfg;
  cudaGetDevice(&b->device);
  b->mem_bytes = ar.off;
  if (injected_alloc_failure() || device_malloc(&b->mem, b->mem_bytes) != cudaSuccess) {
    (void)cudaGetLastError();
    destroy(b);
    return MFCUDA_ERR_ALLOC;
  }
  uint8_t *base = static_cast<uint8_t *>(b->mem);
  int *sig0 = reinterpret_cast<int *>(base + o_sig), *mu0 = reinterpret_cast<int *>(base + o_mu),
      *flag0 = reinterpret_cast<int *>(base + o_flag);
  // owned storage first, then the borrowed pointers
  for (int q = 0; q < np; ++q) {
    SProb &P = probs[q];
    if (P.own_plan) {
      P.plan = reinterpret_cast<Plan *>(base + o_plan[q]);
      if (crt) P.cc = reinterpret_cast<CrtConst *>(base + o_cc[q]);
    }
    if (P.own_a) {
      P.sigA = sig0 + rowA[q];
      P.muA = mu0 + rowA[q];
      P.flagA = flag0 + rowA[q];
      P.As = reinterpret_cast<int8_t *>(base + o_as[q]);
    }
    if (P.own_b) {
      P.sigB = sig0 + rowB[q];
      P.muB = mu0 + rowB[q];
      P.flagB = flag0 + rowB[q];
      P.Bs = reinterpret_cast<int8_t *>(base + o_bs[q]);
    }
    P.D = reinterpret_cast<int32_t *>(base + o_d[q]);
  }
  std::vector<CUtensorMap> maps(nmaps * std::max(np, 1));
  for (int q = 0; q < np; ++q) {
    SProb &P = probs[q];
    const Spec &g = sp[q];
    if (!P.own_plan) {
      P.plan = probs[g.plan_src].plan;
      P.cc = probs[g.plan_src].cc;
    }
    if (!P.own_a) {
      const SProb &S = probs[g.a_src];
      P.sigA = S.sigA;
      P.muA = S.muA;
      P.flagA = S.flagA;
      P.As = S.As;
    }
    if (!P.own_b) {
      const SProb &S = probs[g.b_src];
      P.sigB = S.sigB;
      P.muB = S.muB;
      P.flagB = S.flagB;
      P.Bs = S.Bs;
    }
    P.sigA2 = g.plan_a2 >= 0 ? probs[g.plan_a2].sigA : nullptr;
    P.muA2 = g.plan_a2 >= 0 ? probs[g.plan_a2].muA : nullptr;
    P.sigB2 = g.plan_b2 >= 0 ? probs[g.plan_b2].sigB : nullptr;
    P.muB2 = g.plan_b2 >= 0 ? probs[g.plan_b2].muB : nullptr;
    CUtensorMap *m = &maps[nmaps * q];
    bool made = (crt ? make_map_mn(m + GM_A, P.As, P.M_pad, P.K_pad, P.nsl)
                     : make_map(m + GM_A, P.As, P.M_pad, P.K_pad, BM, P.nsl)) &&
                make_map(m + GM_B, P.Bs, P.N_pad, P.K_pad, G_BOX, P.nsl);
    if (!crt)
      made = made && make_map(m + GM_A_BOX, P.As, P.M_pad, P.K_pad, G_BOX, P.nsl) &&
             (P.bn < 128 || make_map(m + GM_B128, P.Bs, P.N_pad, P.K_pad, 128, P.nsl)) &&
             (P.bn < 256 || make_map(m + GM_B256, P.Bs, P.N_pad, P.K_pad, 256, P.nsl));
    if (!made) {
      destroy(b);
      return MFCUDA_ERR_CUDA;
    }
  }
  SProb *dp = reinterpret_cast<SProb *>(base + o_probs);
  int64_t *dprefix = reinterpret_cast<int64_t *>(base + o_prefix);
  Owner *downer[PH_ITEMS];
  bool copied = true;
  for (int ph = 0; ph < PH_ITEMS; ++ph) {
    downer[ph] = reinterpret_cast<Owner *>(base + o_owner[ph]);
    if (!owner[ph].empty() && cudaMemcpy(downer[ph], owner[ph].data(), sizeof(Owner) * owner[ph].size(),
                                         cudaMemcpyHostToDevice) != cudaSuccess)
      copied = false;
  }
  CUtensorMap *dmaps = reinterpret_cast<CUtensorMap *>(base + o_maps);
  GItem *ditems = reinterpret_cast<GItem *>(base + o_items);
  b->status = reinterpret_cast<int *>(base + o_status);
  if (np > 0 && (cudaMemcpy(dp, probs.data(), sizeof(SProb) * np, cudaMemcpyHostToDevice) != cudaSuccess ||
                 cudaMemcpy(dprefix, prefix.data(), sizeof(int64_t) * np, cudaMemcpyHostToDevice) != cudaSuccess ||
                 !copied ||
                 cudaMemcpy(dmaps, maps.data(), sizeof(CUtensorMap) * nmaps * np, cudaMemcpyHostToDevice) !=
                     cudaSuccess)) {
    destroy(b);
    return MFCUDA_ERR_CUDA;
  }
  std::call_once(g_gmma_attr, [] {
    cudaFuncSetAttribute(g_crt_mma, cudaFuncAttributeMaxDynamicSharedMemorySize, MMA_SMEM);
    cudaFuncSetAttribute(g_digit_mma, cudaFuncAttributeMaxDynamicSharedMemorySize, GD_SMEM);
    cudaFuncSetAttribute(g_crt_combine, cudaFuncAttributeMaxDynamicSharedMemorySize,
                         crt_tc_smem((CRT_NMAX + 31) / 32));
  });
  // the reconstruction's shared tiles hold the most moduli of any product
  int nsl_max = 1;
  for (int q = 0; q < np; ++q) nsl_max = std::max(nsl_max, probs[q].nsl);
  int mma_grid = sm_count();
  if (mma_grid > total[PH_ITEMS]) mma_grid = (int)std::max<int64_t>(total[PH_ITEMS], 1);
  const uint64_t wait_ns = wait_limit_ns();  // captured into the graph with the plan
  int rc = capture(b, [&](cudaStream_t cs) {
    cudaMemsetAsync(b->status, 0, 2 * sizeof(int), cs);
    if (np == 0) return;
    const unsigned fb = (unsigned)((rows_total + 255) / 256);
    fill_kernel<<<fb, 256, 0, cs>>>(sig0, rows_total, SENT_LO);
    fill_kernel<<<fb, 256, 0, cs>>>(mu0, rows_total, SENT_HI);
    fill_kernel<<<fb, 256, 0, cs>>>(flag0, rows_total, 0);
    if (total[PH_SCAN_A]) g_scan_a<<<(unsigned)total[PH_SCAN_A], 256, 0, cs>>>(dp, downer[PH_SCAN_A]);
    if (total[PH_SCAN_B]) g_scan_b<<<(unsigned)total[PH_SCAN_B], 256, 0, cs>>>(dp, downer[PH_SCAN_B]);
    g_plan<<<np, 256, 0, cs>>>(dp, slices, target);
    if (total[PH_SLICE_A] && crt)
      g_crt_slice_a<<<(unsigned)total[PH_SLICE_A], 256, 0, cs>>>(dp, downer[PH_SLICE_A]);
    else if (total[PH_SLICE_A])
      g_slice_a<<<(unsigned)total[PH_SLICE_A], 256, 0, cs>>>(dp, downer[PH_SLICE_A]);
    if (total[PH_SLICE_B] && crt)
      g_crt_slice_b<<<(unsigned)total[PH_SLICE_B], 256, 0, cs>>>(dp, downer[PH_SLICE_B]);
    else if (total[PH_SLICE_B])
      g_slice_b<<<(unsigned)total[PH_SLICE_B], 256, 0, cs>>>(dp, downer[PH_SLICE_B]);
    g_items<<<np, 128, 0, cs>>>(dp, dprefix, ditems);
    if (crt)
      g_crt_mma<<<mma_grid, G_THREADS, MMA_SMEM, cs>>>(ditems, total[PH_ITEMS], dmaps, b->status, wait_ns);
    else
      g_digit_mma<<<mma_grid, G_THREADS, GD_SMEM, cs>>>(ditems, total[PH_ITEMS], b->status + 1, dmaps, b->status,
                                                        wait_ns);
    for (int ph : {PH_COMBINE, PH_COMBINE2}) {
      if (!total[ph]) continue;
      if (crt)
        g_crt_combine<<<(unsigned)total[ph], CTC_THREADS, crt_tc_smem((nsl_max + 31) / 32), cs>>>(
            dp, downer[ph], b->status, wait_ns);
      else
        g_combine<<<(unsigned)total[ph], kCombineThreads, 0, cs>>>(dp, downer[ph]);
    }
  });
  if (rc != MFCUDA_OK) {
    destroy(b);
    return rc;
  }
  *out = b;
  return MFCUDA_OK;
}

// Given-up waits of the grouped tensor-core kernels (this file's record).
int wait_sticky_batched(bool clear) { return take_wait_sticky(clear); }

static bool split_args_ok(const mfcuda_gemm_desc &g) {
  return aligned16(g.a) && aligned16(g.b) && aligned16(g.c) && g.n <= 65535;
}

// Real problems: one product each.  cfg[p] = tile width N (256, 128 or 64).
static int create_split(const mfcuda_gemm_desc *d, int64_t count, int slices, double target,
                        const std::vector<int> &cfg, int kcb_all, mfcuda_batch **out, bool crt) {
  std::vector<Spec> specs;
  for (int64_t p = 0; p < count; ++p) {
    if (!split_args_ok(d[p])) return MFCUDA_ERR_UNSUPPORTED;
    if (d[p].m <= 0 || d[p].n <= 0) continue;
    specs.push_back({static_cast<const double *>(d[p].a), static_cast<const double *>(d[p].b),
                     static_cast<double *>(d[p].c), 1, 1, 1, 0, d[p].m, d[p].k, d[p].n, cfg[p], -1, -1, -1, -1,
                     -1});
  }
  return create_split_specs(std::move(specs), count, slices, target, cfg, kcb_all, out, crt);
}

// Complex problems (complex64x2 operands): four real products each, in the
// order and with the combination of mfcuda_cmatmuldd_mm_split (re = ArBr, then
// re - AiBi; im = ArBi, then im + AiBr), one plan from all four operands, each
// operand sliced once.
static int create_csplit(const mfcuda_gemm_desc *d, int64_t count, int slices, double target,
                         const std::vector<int> &cfg, int kcb_all, mfcuda_batch **out, bool crt) {
  std::vector<Spec> specs;
  for (int64_t p = 0; p < count; ++p) {
    if (!split_args_ok(d[p])) return MFCUDA_ERR_UNSUPPORTED;
    if (d[p].m <= 0 || d[p].n <= 0) continue;
    const double *A = static_cast<const double *>(d[p].a), *B = static_cast<const double *>(d[p].b);
    double *Cm = static_cast<double *>(d[p].c);
    const int64_t m = d[p].m, k = d[p].k, n = d[p].n;
    const int q = (int)specs.size();
    //           A      B      C       strides  mode  shape    bn      a_src  b_src  plan_src plan_a2 plan_b2
    specs.push_back({A, B, Cm, 2, 2, 2, 0, m, k, n, cfg[p], -1, -1, -1, q + 1, q + 1});          // re  = Ar Br
    specs.push_back({A + 2, B + 2, Cm, 2, 2, 2, 1, m, k, n, cfg[p], -1, -1, q, -1, -1});          // re -= Ai Bi
    specs.push_back({A, B + 2, Cm + 2, 2, 2, 2, 0, m, k, n, cfg[p], q, q + 1, q, -1, -1});        // im  = Ar Bi
    specs.push_back({A + 2, B, Cm + 2, 2, 2, 2, 2, m, k, n, cfg[p], q + 1, q, q, -1, -1});        // im += Ai Br
  }
  return create_split_specs(std::move(specs), count, slices, target, cfg, kcb_all, out, crt);
}

// ---- ragged elementwise -------------------------------------------------------
static int ragged_table(const float64x2 *const *xs, float64x2 *const *ys, const int64_t *ns, int64_t count,
                        std::vector<RArr> &tab, int64_t &total) {
  total = 0;
  tab.resize(count);
  for (int64_t a = 0; a < count; ++a) {
    if (ns[a] < 0 || !size_ok(ns[a], sizeof(float64x2))) return MFCUDA_ERR_INVALID_ARG;
    if (ns[a] > 0 && (!xs[a] || !ys[a])) return MFCUDA_ERR_INVALID_ARG;
    tab[a] = {reinterpret_cast<const double *>(xs[a]), reinterpret_cast<double *>(ys[a]), total};
    total += ns[a];
  }
  return MFCUDA_OK;
}
static void launch_ragged(int op, const RArr *tab, int narr, int64_t total, cudaStream_t s) {
  int64_t want = (total + 255) / 256, cap = (int64_t)sm_count() * 16;
  unsigned grid = (unsigned)std::max<int64_t>(1, std::min(want, cap));
  switch (op) {
    case MFCUDA_EXP: ragged_unary_kernel<MFCUDA_EXP><<<grid, 256, 0, s>>>(tab, narr, total); break;
    case MFCUDA_LOG: ragged_unary_kernel<MFCUDA_LOG><<<grid, 256, 0, s>>>(tab, narr, total); break;
    case MFCUDA_SIN: ragged_unary_kernel<MFCUDA_SIN><<<grid, 256, 0, s>>>(tab, narr, total); break;
    case MFCUDA_COS: ragged_unary_kernel<MFCUDA_COS><<<grid, 256, 0, s>>>(tab, narr, total); break;
    default: ragged_unary_kernel<MFCUDA_SQRT><<<grid, 256, 0, s>>>(tab, narr, total); break;
  }
}
static int create_unary(int op, const float64x2 *const *xs, float64x2 *const *ys, const int64_t *ns,
                        int64_t count, mfcuda_batch **out) {
  std::vector<RArr> tab;
  int64_t total;
  MF_TRY(ragged_table(xs, ys, ns, count, tab, total));
  auto *b = new mfcuda_batch;
  b->kind = 2;
  b->count = count;
  b->work = total;
  cudaGetDevice(&b->device);
  b->mem_bytes = sizeof(RArr) * std::max<int64_t>(count, 1);
  if (injected_alloc_failure() || device_malloc(&b->mem, b->mem_bytes) != cudaSuccess) {
    (void)cudaGetLastError();
    destroy(b);
    return MFCUDA_ERR_ALLOC;
  }
  RArr *dt = static_cast<RArr *>(b->mem);
  if (count > 0 && cudaMemcpy(dt, tab.data(), sizeof(RArr) * count, cudaMemcpyHostToDevice) != cudaSuccess) {
    destroy(b);
    return MFCUDA_ERR_CUDA;
  }
  int rc = capture(b, [&](cudaStream_t cs) {
    if (total > 0) launch_ragged(op, dt, (int)count, total, cs);
  });
  if (rc != MFCUDA_OK) {
    destroy(b);
    return rc;
  }
  *out = b;
  return MFCUDA_OK;
}

// ---- autotuner ------------------------------------------------------------------
// Candidates are timed on synthetic problems of the bucket's representative
// shape, in a batch as large as the bucket's population (at least enough
// tiles to fill the GPU), once per bucket; winners are cached on disk.
__global__ void synth_fill_kernel(double *p, int64_t n_dd, uint64_t seed) {
  int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n_dd) return;
  uint64_t z = seed + (uint64_t)i * 0x9E3779B97F4A7C15ull;  // splitmix64
  z = (z ^ (z >> 30)) * 0xBF58476D1CE4E5B9ull;
  z = (z ^ (z >> 27)) * 0x94D049BB133111EBull;
  z ^= z >> 31;
  double u = (double)(z >> 11) * 0x1p-53 * 2.0 - 1.0;
  p[2 * i] = u;
  p[2 * i + 1] = u * 0x1p-60;
}

static double time_plan(mfcuda_batch *b, int reps) {
  cudaStream_t s;
  cudaStreamCreateWithFlags(&s, cudaStreamNonBlocking);
  cudaEvent_t e0, e1;
  cudaEventCreate(&e0);
  cudaEventCreate(&e1);
  cudaGraphLaunch(b->exec, s);  // warm-up
  cudaEventRecord(e0, s);
  for (int r = 0; r < reps; ++r) cudaGraphLaunch(b->exec, s);
  cudaEventRecord(e1, s);
  cudaEventSynchronize(e1);
  float ms = 0.f;
  cudaEventElapsedTime(&ms, e0, e1);
  cudaEventDestroy(e0);
  cudaEventDestroy(e1);
  cudaStreamDestroy(s);
  return cudaGetLastError() == cudaSuccess ? ms / reps : 1e30;
}

struct Bucket {
  int bm, bn, bk;
  int64_t population;
};

// form 0: candidate = plain tile config; form 1: candidate = split tile width N.
static int tune_bucket(int form, const Bucket &bk, int64_t ri) {
  const int64_t m = (int64_t)1 << bk.bm, n = (int64_t)1 << bk.bn, k = (int64_t)1 << bk.bk;
  std::vector<int> cands = form == 0 ? std::vector<int>{0, 1, 2} : std::vector<int>{256, 128, 64};
  const int64_t tiles16 = ((m + 15) / 16) * ((n + 15) / 16);
  int64_t copies = std::max<int64_t>(bk.population, 1);
  if (form == 0) {
    copies = std::max<int64_t>(copies, (int64_t)sm_count() * 4 * 16 / std::max<int64_t>(tiles16, 1));
    copies = std::min<int64_t>(copies, 256);
  } else {
    copies = std::min<int64_t>(copies, 16);
  }
  void *buf = nullptr;
  const int64_t per = 2 * (m * k + k * n + m * n);
  if (device_malloc(&buf, sizeof(double) * per * copies) != cudaSuccess) {
    (void)cudaGetLastError();
    return form == 0 ? plain_heuristic(m, n) : 256;
  }
  double *p = static_cast<double *>(buf);
  synth_fill_kernel<<<(unsigned)((per * copies / 2 + 255) / 256), 256>>>(p, per * copies / 2, 12345);
  std::vector<mfcuda_gemm_desc> descs(copies);
  for (int64_t c = 0; c < copies; ++c) {
    double *base = p + c * per;
    descs[c] = {base, base + 2 * m * k, base + 2 * (m * k + k * n), m, k, n};
  }
  int best = cands[0];
  double best_ms = 1e30;
  for (int cand : cands) {
    if (form != 0 && cand > 64 && cand >= 2 * n) continue;  // wider than twice the problem: pure padding
    mfcuda_batch *b = nullptr;
    std::vector<int> cfg(copies, cand);
    int rc = form == 0 ? create_plain(descs.data(), copies, ri, cfg, &b)
                       : create_split(descs.data(), copies, 0, 8.0, cfg, KC_BLOCKS, &b, form == 2);
    if (rc != MFCUDA_OK) continue;
    double ms = time_plan(b, 2);
    destroy(b);
    if (ms < best_ms) {
      best_ms = ms;
      best = cand;
    }
  }
  cudaDeviceSynchronize();
  cudaFree(buf);
  return best;
}

// Part of a winner's key, raised with every change of the tiles' kernels: a winner
// timed on other kernels says nothing about these (cache files outlive the library
// that wrote them; entries without this number are from before it was there).
constexpr int kTuneGeneration = 2;
static std::string bucket_key(int form, const Bucket &b) {
  char dev[256] = "gpu";
  cudaDeviceProp prop;
  int d = 0;
  if (cudaGetDevice(&d) == cudaSuccess && cudaGetDeviceProperties(&prop, d) == cudaSuccess)
    std::snprintf(dev, sizeof dev, "%s", prop.name);
  for (char *c = dev; *c; ++c)
    if (*c == ' ') *c = '_';
  char key[512];
  std::snprintf(key, sizeof key, "%s:%s:%d:%d:%d:g%d", dev, form == 0 ? "plain" : form == 1 ? "split" : "crt", b.bm,
                b.bn, b.bk, kTuneGeneration);
  return key;
}

// Chooses per-problem configurations: the cached or freshly tuned winner of
// each shape bucket when tune != 0, else the built-in heuristic.
static std::vector<int> choose(int form, const mfcuda_gemm_desc *d, int64_t count, int tune, int64_t ri) {
  std::vector<int> cfg(count);
  std::map<std::tuple<int, int, int>, Bucket> buckets;
  // plain: the tile edge depends on m and n; split: the tile width N on n and
  // a coarse K class (m only changes the number of 128-row tiles)
  auto bucket_of = [&](const mfcuda_gemm_desc &g) {
    int bn = std::min(std::max(clog2(g.n), 4), 10);
    if (form == 0) return std::make_tuple(std::min(std::max(clog2(g.m), 4), 10), bn, 8);
    return std::make_tuple(bn, bn, std::min(std::max(clog2(g.k), 7), 10));
  };
  for (int64_t p = 0; p < count; ++p) {
    auto t = bucket_of(d[p]);
    auto &b = buckets[t];
    b.bm = std::get<0>(t);
    b.bn = std::get<1>(t);
    b.bk = std::get<2>(t);
    b.population++;
  }
  std::map<std::tuple<int, int, int>, int> win;
  {
    std::lock_guard<std::mutex> lk(g_tune_mu);
    tune_load();
    bool dirty = false;
    for (auto &kv : buckets) {
      const std::string key = bucket_key(form, kv.second);
      auto it = g_tune.find(key);
      if (it != g_tune.end()) {
        win[kv.first] = it->second;
      } else if (tune) {
        int best = tune_bucket(form, kv.second, ri);
        g_tune[key] = best;
        win[kv.first] = best;
        dirty = true;
      }
    }
    if (dirty) tune_save();
  }
  for (int64_t p = 0; p < count; ++p) {
    auto it = win.find(bucket_of(d[p]));
    if (it != win.end()) {
      cfg[p] = it->second;
    } else if (form == 0) {
      cfg[p] = plain_heuristic(d[p].m, d[p].n);
    } else {
      cfg[p] = d[p].n <= 64 ? 64 : d[p].n <= 128 ? 128 : 256;
    }
  }
  if (form == 0) plain_small_tiles(d, count, cfg);
  return cfg;
}

// Split-K rule: K chunks of at most KC_BLOCKS blocks (the INT32 bound); when
// the whole batch has fewer than four products of one diagonal or modulus per SM,
// shorter chunks raise their number (the chunks' INT32 partials are summed exactly
// in the combine).  The results depend on the chunk (the combine rounds once per
// chunk), so it follows from shapes alone and not from how many diagonals an item has.
// nsl(k): slice slots (and so products per tile) of a product with inner size k.
template <class SlotFn>
static int choose_kcb(const mfcuda_gemm_desc *d, int64_t count, const std::vector<int> &cfg, int prods, SlotFn nsl) {
  int64_t items = 0, kmax = 1;
  for (int64_t p = 0; p < count; ++p) {
    if (d[p].m <= 0 || d[p].n <= 0) continue;
    int64_t kb = (ru(std::max<int64_t>(d[p].k, 1), BK)) / BK;
    kmax = std::max(kmax, kb);
    items += (int64_t)prods * nsl(d[p].k) * ((kb + KC_BLOCKS - 1) / KC_BLOCKS) * (ru(d[p].m, BM) / BM) *
             (ru(d[p].n, cfg[p]) / cfg[p]);
  }
  const int64_t want = (int64_t)sm_count() * 4;
  if (items >= want || items == 0) return KC_BLOCKS;
  int64_t split = (want + items - 1) / items;
  int64_t kcb = (std::min<int64_t>(kmax, KC_BLOCKS) + split - 1) / split;
  return (int)std::max<int64_t>(4, std::min<int64_t>(kcb, KC_BLOCKS));
}

}  // namespace batch
}  // namespace mfcuda

extern "C" {

static int batch_create(const mfcuda_gemm_desc *descs, int64_t count, int form, int64_t renorm_interval,
                        int slices, double target, int tune, mfcuda_batch **plan, bool complex) {
  using namespace mfcuda;
  if (!plan || count < 0 || (count > 0 && !descs)) return MFCUDA_ERR_INVALID_ARG;
  *plan = nullptr;
  if (form != MFCUDA_FORM_PLAIN && form != MFCUDA_FORM_SPLIT && form != MFCUDA_FORM_CRT)
    return MFCUDA_ERR_INVALID_ARG;
  if (form == MFCUDA_FORM_SPLIT && (slices < 0 || slices > split::SMAX || slices == 1 || !(target > 0.0)))
    return MFCUDA_ERR_INVALID_ARG;
  if (form == MFCUDA_FORM_CRT &&
      (slices < 0 || (slices > 0 && slices < 8) || slices > split::CRT_WMAX || !(target > 0.0)))
    return MFCUDA_ERR_INVALID_ARG;
  for (int64_t p = 0; p < count; ++p) {
    const mfcuda_gemm_desc &g = descs[p];
    if (g.m < 0 || g.k < 0 || g.n < 0 || !mul_ok(g.m, g.k) || !mul_ok(g.k, g.n) || !mul_ok(g.m, g.n))
      return MFCUDA_ERR_INVALID_ARG;
    if (g.m > 0 && g.n > 0 && (!g.c || (g.k > 0 && (!g.a || !g.b)))) return MFCUDA_ERR_INVALID_ARG;
  }
  MF_TRY(require_device());
  if (complex && form == MFCUDA_FORM_PLAIN)
    return batch::create_plain(descs, count, renorm_interval, std::vector<int>(count, 1), plan, true);
  std::vector<int> cfg = batch::choose(form, descs, count, tune, renorm_interval);
  if (form == MFCUDA_FORM_PLAIN) return batch::create_plain(descs, count, renorm_interval, cfg, plan);
  const bool crt = form == MFCUDA_FORM_CRT;
  int kcb = batch::choose_kcb(descs, count, cfg, complex ? 4 : 1, [&](int64_t k) {
    return crt ? split::crt_slices_max(k < 1 ? 1 : k, slices) : split::SMAX;
  });
  if (complex) return batch::create_csplit(descs, count, slices, target, cfg, kcb, plan, crt);
  return batch::create_split(descs, count, slices, target, cfg, kcb, plan, crt);
}

MULTIFLOATS_CUDA_API int mfcuda_batch_create_gemm(const mfcuda_gemm_desc *descs, int64_t count, int form,
                                                  int64_t renorm_interval, int slices, double target, int tune,
                                                  mfcuda_batch **plan) {
  return batch_create(descs, count, form, renorm_interval, slices, target, tune, plan, false);
}

MULTIFLOATS_CUDA_API int mfcuda_batch_create_cgemm(const mfcuda_gemm_desc *descs, int64_t count, int form,
                                                   int64_t renorm_interval, int slices, double target, int tune,
                                                   mfcuda_batch **plan) {
  return batch_create(descs, count, form, renorm_interval, slices, target, tune, plan, true);
}

MULTIFLOATS_CUDA_API int mfcuda_batch_create_unary(int op, const float64x2 *const *xs,
                                                   float64x2 *const *ys, const int64_t *ns, int64_t count,
                                                   mfcuda_batch **plan) {
  using namespace mfcuda;
  if (!plan || count < 0 || (count > 0 && (!xs || !ys || !ns))) return MFCUDA_ERR_INVALID_ARG;
  *plan = nullptr;
  if (op < MFCUDA_EXP || op > MFCUDA_SQRT || count > INT32_MAX) return MFCUDA_ERR_INVALID_ARG;
  MF_TRY(require_device());
  return batch::create_unary(op, xs, ys, ns, count, plan);
}

MULTIFLOATS_CUDA_API int mfcuda_batch_run(mfcuda_batch *plan, void *stream) {
  if (!plan || !plan->exec) return MFCUDA_ERR_INVALID_ARG;
  if (cudaGraphLaunch(plan->exec, mfcuda::as_stream(stream)) != cudaSuccess) {
    (void)cudaGetLastError();
    return MFCUDA_ERR_CUDA;
  }
  return MFCUDA_OK;
}

MULTIFLOATS_CUDA_API int mfcuda_batch_status(mfcuda_batch *plan) {
  if (!plan) return MFCUDA_ERR_INVALID_ARG;
  if (cudaDeviceSynchronize() != cudaSuccess) {
    (void)cudaGetLastError();
    return MFCUDA_ERR_CUDA;
  }
  if (plan->status) {
    int st = 0;
    if (cudaMemcpy(&st, plan->status, sizeof(int), cudaMemcpyDeviceToHost) != cudaSuccess)
      return MFCUDA_ERR_CUDA;
    if (st) return MFCUDA_ERR_TIMEOUT;
  }
  return MFCUDA_OK;
}

MULTIFLOATS_CUDA_API int64_t mfcuda_batch_config(const mfcuda_batch *plan, int64_t i) {
  if (!plan || i < 0 || i >= (int64_t)plan->cfg.size()) return -1;
  if (plan->kind == 0) return mfcuda::batch::cfg_edge(plan->cfg[i]);
  return plan->cfg[i];
}

MULTIFLOATS_CUDA_API int64_t mfcuda_batch_work_items(const mfcuda_batch *plan) {
  return plan ? plan->work : -1;
}

MULTIFLOATS_CUDA_API int64_t mfcuda_batch_kchunk(const mfcuda_batch *plan) {
  return plan && plan->kind == 1 ? plan->kchunk : -1;
}

MULTIFLOATS_CUDA_API void mfcuda_batch_destroy(mfcuda_batch *plan) {
  if (plan) {
    cudaDeviceSynchronize();
    mfcuda::batch::destroy(plan);
  }
}

MULTIFLOATS_CUDA_API int mfcuda_unary_dd_ragged(int op, const float64x2 *const *xs, float64x2 *const *ys,
                                                const int64_t *ns, int64_t count, void *stream) {
  using namespace mfcuda;
  if (count < 0 || (count > 0 && (!xs || !ys || !ns))) return MFCUDA_ERR_INVALID_ARG;
  if (op < MFCUDA_EXP || op > MFCUDA_SQRT || count > INT32_MAX) return MFCUDA_ERR_INVALID_ARG;
  if (count == 0) return MFCUDA_OK;
  MF_TRY(require_device());
  std::vector<batch::RArr> tab;
  int64_t total;
  MF_TRY(batch::ragged_table(xs, ys, ns, count, tab, total));
  if (total == 0) return MFCUDA_OK;
  cudaStream_t s = as_stream(stream);
  void *dt = nullptr;
  MF_TRY(ws_alloc(&dt, sizeof(batch::RArr) * count, s));
  MF_TRY_CUDA(cudaMemcpyAsync(dt, tab.data(), sizeof(batch::RArr) * count, cudaMemcpyHostToDevice, s));
  // the host table must outlive the asynchronous copy
  cudaError_t e = cudaStreamSynchronize(s);
  if (e == cudaSuccess) {
    batch::launch_ragged(op, static_cast<batch::RArr *>(dt), (int)count, total, s);
    e = cudaGetLastError();
  }
  ws_free(dt, s);
  return e == cudaSuccess ? MFCUDA_OK : MFCUDA_ERR_CUDA;
}

}  // extern "C"
