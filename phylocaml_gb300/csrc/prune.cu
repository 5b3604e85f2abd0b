// Felsenstein pruning: the tree log-likelihood of weighted site patterns.
//
// The reference's likelihood character is a stub (Likelihood_c.median_2 is
// `failwith "TODO"`, lib/likelihood_c.ml:15); this is the computation that
// slot exists for, over the transition matrices MlModel.compose builds
// (lib/mlModel.ml:585-587, lib/mlmodel.c:325-342, P[i][j] = Pr(j | i, t)):
//
//   CLV_v[r][i] = (sum_j P_{a,r}[i][j] CLV_a[r][j]) * (sum_j P_{b,r}[i][j] CLV_b[r][j])
//   L_s         = sum_r probs[r] sum_i pi[i] CLV_root[r][i]
//   lnL         = sum_s w_s (log L_s + e_s ln 2)
//
// A subtree of two or three tips has few distinct columns however many
// patterns there are: n_codes^2 or n_codes^3 combinations of codes.  Where
// that is less than half the patterns, every such subtree (the largest ones
// of at most three tips) becomes one leaf of a reduced tree, and
// prune_prep_kernel fills its rows P(t) CLV for every combination with the
// same arithmetic as a node of the walk.  In a Yule tree half the internal
// nodes lie in such subtrees.
//
// One kernel then scores the whole tree (prune_tree_kernel):
//   warp 0, lane 0   producer: streams the transition matrices of each
//                    step's internal children into a shared ring with 1-D
//                    bulk copies on mbarriers;
//   consumer warps   one (pattern, rate class) per thread; the conditional
//                    likelihood vectors of internal nodes live on a
//                    per-thread stack in shared memory (top entry in
//                    registers), so no CLV ever goes to HBM.  A leaf's row is
//                    gathered by the thread itself, three leaves ahead, with
//                    cp.async into its own shared slots, by an index that
//                    prune_prep_kernel formed from the tips' codes.  After
//                    every node the vector is rescaled by an exact power of
//                    two when its largest entry drops below 2^-32 (FP32) or
//                    2^-256 (FP64) and the exponent is added to the
//                    pattern's integer scaler e_s.
// The root log-likelihoods are weighted and summed in FP64 with error-free
// TwoSum steps (a compensated reduction), one (sum, compensation) pair per
// CTA; the last CTA adds the pairs in contiguous chunks, so the result does
// not depend on scheduling.
//
// T = float is the FP32 form, T = double the FP64 comparison form; both use
// P matrices built in FP64 on the GPU (pmatrix.cu), the FP32 form rounding
// them once.
#include <algorithm>
#include <cmath>
#include <cstring>
#include <type_traits>

#include "pgpu_internal.cuh"
#include "forms.cuh"
#include "pmatrix.cuh"

namespace {
using namespace pgpu_forms;

struct PruneArgs {
  const uint16_t *index;      // [n_leaf + PR_PAD][ld_index]: each pattern's row of the leaf
  const void *P;              // per branch: 16-byte unit k of rate class r at k RT + r
  const void *rows;           // leaf rows, [n_codes^k][R] per leaf (form's values)
  const int *row_exp;         // power of two taken out of each collapsed leaf's row
  const int *row_flag;        // per model: some exponent is not zero
  const double *pi;           // [S]
  const double *probs;        // [R]
  const double *weights;      // [n_pat] or null
  double *site_lnl;           // [n_pat] or null
  double2 *partials;          // [n_models][n_tiles_total], by tile
  unsigned *done;             // [n_models] CTAs finished, zeroed by the setup kernel
  double *lnl;                // [n_models]
  const int4 *ops;            // {internal children, branch of the first, of the second, -}
  const uint32_t *leaf_unit;  // 16-byte unit of each leaf's first row, in the order the steps read them
  int *flag;
  // several models over the same tree and patterns: CTA row blockIdx.y
  // scores model blockIdx.y, whose P blocks and leaf rows lie P_stride and
  // rows_stride bytes after the previous model's, pi and probs 4 and R
  // doubles after, its exponents exp_stride ints after, and whose partial
  // sums follow the previous model's
  size_t P_stride, rows_stride, exp_stride;
  // a launch may cover tiles tile_base .. tile_base + gridDim.x - 1 of
  // n_tiles_total (the host-buffer entry point launches one per copied chunk)
  size_t tile_base, n_tiles_total;
  size_t index_col;           // pattern of index's first column
  size_t ld_index, n_pat;
  uint32_t exp_unit;          // unit of row_exp's first row
  int n_ops, n_leaf, R, NP, depth;
};

__host__ __device__ inline size_t align16(size_t x) { return (x + 15) & ~size_t(15); }

constexpr int PR_THREADS = 256;   // consumer threads per CTA
constexpr int PR_LEAVES = 3;      // leaf rows in flight per thread
constexpr int PR_PAD = PR_LEAVES + 1;   // row-0 leaves after the last, so that the pipeline runs on unchecked

// CTAs each SM should hold, and growth: how much larger each column chunk of
// host tip codes is than the one before; a chunk's copy must end while the
// previous chunk is scored.
template <typename Pol> struct PruneTune {
  static constexpr int min_ctas = 1, growth = 8;
};
template <> struct PruneTune<pgpu_forms::Ff32> {
  static constexpr int min_ctas = 3, growth = 2;
};
template <> struct PruneTune<pgpu_forms::Fp32> {
  static constexpr int min_ctas = 4, growth = 2;
};
// Ring of the coefficient blocks, in postorder steps (a power of two).  The
// producer stages PR_GROUP consecutive steps under one mbarrier phase, so
// the consumers wait and release once per group.
constexpr int PR_STAGES = 8, PR_GROUP = 4;

// Shared memory of one CTA: the ring of step slots (the coefficient blocks
// RT x 16 of the internal children), the threads'
// leaf slots, then the CLV stack (the results set aside: one less than the
// schedule's depth, the top being in registers).
template <typename Pol>
struct PruneLayout {
  using V = typename Pol::V;
  using Coef = typename Pol::Coef;
  __host__ __device__ static constexpr uint32_t coef_bytes(int RT) { return (uint32_t)(RT * 16 * sizeof(Coef)); }
  __host__ __device__ static constexpr uint32_t ring_off() { return 128; }
  __host__ __device__ static constexpr uint32_t leaf_off(int RT) {
    return ring_off() + PR_STAGES * 2 * coef_bytes(RT);
  }
  __host__ __device__ static constexpr uint32_t stk_off(int RT) {
    return leaf_off(RT) + (uint32_t)(PR_LEAVES * 4 * PR_THREADS * sizeof(V));
  }
  __host__ __device__ static size_t bytes(int RT, int depth) {
    return stk_off(RT) + (size_t)(depth > 1 ? depth - 1 : 0) * 4 * PR_THREADS * sizeof(V);
  }
};

// Exact power-of-two rescaling of one rate class's vector (each rate class
// keeps its own scaler; the root aligns them).  An all-zero vector (a site
// the tree cannot produce) rescales to zeros again and ends as log 0 = -inf.
template <typename Pol, typename M>
__device__ __forceinline__ void rescale_vec(typename Pol::V *acc, M mx, int &escale) {
  const int ex = frexp_exp(mx);
  escale += ex;
  // two steps when the largest entry is subnormal, so each factor stays a
  // normal power of two
  const int k1 = min(-ex, 120), k2 = -ex - k1;
#pragma unroll
  for (int e = 0; e < 4; ++e) acc[e] = Pol::scale(acc[e], k1);
  if (k2 > 0) {
#pragma unroll
    for (int e = 0; e < 4; ++e) acc[e] = Pol::scale(acc[e], k2);
  }
}
template <typename Pol>
__device__ __forceinline__ auto largest(const typename Pol::V *acc) {
  return fmax(fmax(Pol::mag(acc[0]), Pol::mag(acc[1])), fmax(Pol::mag(acc[2]), Pol::mag(acc[3])));
}

// Rows of the collapsed leaves: P(t_v) CLV_v for every combination of the
// leaf's codes, (c0 n + c1) for tips 0 and 1, ((c0 n + c1) n + c2) with tip 2
// beside the cherry of tips 0 and 1.  A thread per (c0, c1), which forms the
// cherry once for every c2.
struct TableArgs {
  void *rows;            // tips' rows first: [n_tips][n_codes][R]
  const void *P;
  const int4 *leaves;
  const int4 *made;      // {leaf, branch of the leaf, branch of its cherry or -1, -}
  int *row_exp, *row_flag;
  size_t P_stride, rows_stride, exp_stride;
  size_t exp_base;       // row of row_exp's first entry
  int R, RT, n_codes, n_made, blocks;   // blocks: CTAs per (leaf, rate class)
  const int *status;     // model m at m
};

// Row of every leaf for every pattern, in the leaves' reading order, so that
// the walk reads one 16-bit index where it would read up to three codes in
// each of a pattern's rate classes.  A code outside the table raises the
// error word and reads as the last.
struct IndexArgs {
  const uint8_t *tip_codes;   // [n_tips][ld_pat]
  const int4 *leaves;         // {tip, tip or -1, tip or -1, first row}
  uint16_t *index;            // [n_leaf][ld_index], column 0 = pattern col0
  size_t ld_pat, ld_index, col0, cols, n_pat;
  int n_codes, blocks;        // blocks: CTAs per leaf, 256 x IX_PATTERNS patterns each
  int *flag;
};

// 16 patterns per thread: one 16-byte load per tip and two 16-byte stores
// (128 against 220 us for 256 leaves of 446,427 patterns with 4).
constexpr int IX_PATTERNS = 16;

__device__ __forceinline__ void leaf_index(const IndexArgs &p, int block) {
  const int4 lf = __ldg(p.leaves + block / p.blocks);
  const size_t col = ((size_t)(block % p.blocks) * 256 + threadIdx.x) * IX_PATTERNS;
  if (col >= p.cols) return;
  const size_t pat = p.col0 + col;   // a multiple of 16, as are the rows' lengths
  const uint32_t top = (uint32_t)p.n_codes - 1u;
  const int tips[3] = {lf.x, lf.y, lf.z};
  uint4 w[3];
#pragma unroll
  for (int h = 0; h < 3; ++h)
    if (tips[h] >= 0) w[h] = __ldg(reinterpret_cast<const uint4 *>(p.tip_codes + (size_t)tips[h] * p.ld_pat + pat));
  uint32_t row[IX_PATTERNS];
#pragma unroll
  for (int q = 0; q < IX_PATTERNS; ++q) row[q] = 0u;
  bool bad = false;
#pragma unroll
  for (int h = 0; h < 3; ++h) {
    if (tips[h] < 0) break;
    const uint32_t v[4] = {w[h].x, w[h].y, w[h].z, w[h].w};
#pragma unroll
    for (int q = 0; q < IX_PATTERNS; ++q) {
      const uint32_t c = (v[q / 4] >> (8 * (q % 4))) & 255u;
      bad |= c > top && pat + q < p.n_pat;
      row[q] = row[q] * (uint32_t)p.n_codes + min(c, top);
    }
  }
  if (bad) atomicOr(p.flag, PGPU_FLAG_BADCODE);
  uint4 *out = reinterpret_cast<uint4 *>(p.index + (size_t)(block / p.blocks) * p.ld_index + col);
#pragma unroll
  for (int q = 0; q < IX_PATTERNS; q += 8)
    out[q / 8] = make_uint4(row[q] | row[q + 1] << 16, row[q + 2] | row[q + 3] << 16,
                            row[q + 4] | row[q + 5] << 16, row[q + 6] | row[q + 7] << 16);
}

// CTAs 0 .. n_table - 1: the collapsed leaves' rows (model by model); the
// rest: leaf indexes.
template <typename Pol>
__global__ void __launch_bounds__(256) prune_prep_kernel(const TableArgs p, const IndexArgs ix, int n_table) {
  using V = typename Pol::V;
  using Coef = typename Pol::Coef;
  if ((int)blockIdx.x >= n_table) {
    leaf_index(ix, (int)blockIdx.x - n_table);
    return;
  }
  const int per_model = p.n_made * p.R * p.blocks;
  const int m = blockIdx.x / per_model, at_block = blockIdx.x % per_model, lr = at_block / p.blocks;
  const int4 mk = __ldg(p.made + lr / p.R);
  const int r = lr % p.R, NC = p.n_codes;
  const int4 lf = __ldg(p.leaves + mk.x);
  const int q = (at_block % p.blocks) * 256 + threadIdx.x;   // codes of tips 0 and 1
  if (q >= NC * NC || p.status[m]) return;
  char *rows = static_cast<char *>(p.rows) + m * p.rows_stride;
  const char *P = static_cast<const char *>(p.P) + m * p.P_stride;
  auto coef = [&](int branch) {
    return reinterpret_cast<const Coef *>(P + (size_t)branch * p.RT * 16 * sizeof(Coef) + 16 * r);
  };
  auto tip = [&](int t, int c, V *y) { Pol::load_tip(rows, ((size_t)t * NC + c) * p.R + r, y); };
  auto node = [&](const V *x, const V *y, V *acc, int ex) {
    Pol::mul4(x, y, acc);
    const auto mx = largest<Pol>(acc);
    if (mx < Pol::thresh) rescale_vec<Pol>(acc, mx, ex);
    return ex;
  };
  auto put = [&](const V *x, int combination, int ex) {
    const size_t at = (size_t)(uint32_t)lf.w + (size_t)combination * p.R + r;
    Pol::store4(rows, at, x);
    p.row_exp[m * p.exp_stride + (at - p.exp_base)] = ex;
    if (ex) p.row_flag[m] = 1;   // every writer writes 1
  };
  V x[4], y[4], acc[4];
  tip(lf.x, q / NC, x);
  tip(lf.y, q % NC, y);
  const int ex = node(x, y, acc, 0);
  if (lf.z < 0) {
    Pol::rows(coef(mk.y), acc, x, p.RT);
    put(x, q, ex);
    return;
  }
  V cherry[4];
  Pol::rows(coef(mk.z), acc, cherry, p.RT);
  for (int c = 0; c < NC; ++c) {
    tip(lf.z, c, y);
    const int e2 = node(cherry, y, acc, ex);
    Pol::rows(coef(mk.y), acc, x, p.RT);
    put(x, q * NC + c, e2);
  }
}

__device__ __forceinline__ void cp_async_16(uint32_t dst, const void *src) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], 16;" ::"r"(dst), "l"(src) : "memory");
}

// One CTA: 32 producer threads + PR_THREADS consumers.  Consumer c works on
// rate class c % RT (R <= RT of them active) of pattern c / RT of the tile;
// it holds the 4 state values and its own power-of-two scaler.  The classes
// of a pattern sit in neighbouring lanes and interleaved in memory, so a
// pattern's leaf row is one 128-byte line for all of them (four classes of
// the pair form): a warp's gather touches 8 lines.  With a warp per class it
// touched up to 32, and the line lookups bounded the kernel.
//
// 512 taxa x 446,427 patterns, 4 rate classes, pair form: 3.83 ms with
// the collapsed subtrees (about half the steps), 7.12 ms walking every node
// with the tip rows staged per step by the producer.  Issue slots 57 % busy,
// FMA pipe 50 %; the first stall is the wait for gathered leaf rows (2.8 of
// 10 an instruction), then the pair arithmetic's own chains.
template <typename Pol, int RT>
__global__ void __launch_bounds__(32 + PR_THREADS, PruneTune<Pol>::min_ctas)
    prune_tree_kernel(const PruneArgs p) {
  using V = typename Pol::V;
  using Coef = typename Pol::Coef;
  using L = PruneLayout<Pol>;
  constexpr int ST = PR_STAGES, NT = PR_THREADS, G = PR_GROUP, NB = ST / G;
  constexpr int VU = 4 * sizeof(V) / 16;   // 16-byte units of a row
  static_assert(ST % G == 0 && (NB & (NB - 1)) == 0, "ring depth must be a power-of-two number of groups");
  extern __shared__ __align__(128) unsigned char smem[];
  __shared__ double2 red[NT / 32];
  __shared__ double2 xch[RT][NT / RT];   // per pattern and rate class: (part, scaler)
  __shared__ int step_kind[ST];          // per step slot: internal children
  __shared__ int last_cta;
  constexpr int NP = NT / RT;
  const int R = p.R;
  uint64_t *full = reinterpret_cast<uint64_t *>(smem);     // [NB]
  uint64_t *empty = full + NB;                              // [NB]
  constexpr uint32_t CB = L::coef_bytes(RT), SB = 2 * CB;
  unsigned char *ring = smem + L::ring_off();               // [ST][SB]
  V *stk = reinterpret_cast<V *>(smem + L::stk_off(RT));    // [depth - 1][4][NT]
  const size_t tile = p.tile_base + blockIdx.x;
  const size_t tile0 = tile * NP;
  const int tid = threadIdx.x;

  if (tid == 0) {
    for (int s = 0; s < NB; ++s) {
      mbar_init(&full[s], 1);
      mbar_init(&empty[s], NT / 32);
    }
    fence_mbarrier_init();
  }
  __syncthreads();

  if (tid < 32) {
    // producer: the coefficient blocks step i reads go into slot i % ST
    if (tid == 0) {
      const unsigned char *Pg = static_cast<const unsigned char *>(p.P) + blockIdx.y * p.P_stride;
      // group q (steps qG .. qG + G - 1) completes barrier q % NB once per
      // pass over the ring
      int groups = 0;
      for (int g0 = 0; g0 < p.n_ops; g0 += G) {
        const int q = g0 / G, b = q & (NB - 1), round = q / NB;
        if (round > 0 && !mbar_wait_bounded(&empty[b], (round - 1) & 1, p.flag)) break;
        const int gn = min(G, p.n_ops - g0);
        int4 ops[G];
        uint32_t tx = 0;
        for (int k = 0; k < gn; ++k) {
          ops[k] = __ldg(p.ops + g0 + k);
          tx += (uint32_t)ops[k].x * CB;
          // the arrive below releases this store to the consumers' wait
          step_kind[(g0 + k) & (ST - 1)] = ops[k].x;
        }
        mbar_arrive_expect_tx(&full[b], tx);
        for (int k = 0; k < gn; ++k) {
          unsigned char *sl = ring + (size_t)((g0 + k) & (ST - 1)) * SB;
          if (ops[k].x > 0) bulk_g2s(sl, Pg + (size_t)ops[k].y * CB, CB, &full[b]);
          if (ops[k].x > 1) bulk_g2s(sl + CB, Pg + (size_t)ops[k].z * CB, CB, &full[b]);
        }
        groups = q + 1;
      }
      // do not leave while copies into this CTA's shared memory are in flight
      for (int q = max(0, groups - NB); q < groups; ++q)
        (void)mbar_wait_bounded(&full[q & (NB - 1)], (q / NB) & 1, p.flag);
    }
    return;
  }

  const int c = tid - 32, lane = tid & 31;
  const int r = c % RT, pl = c / RT;
  const size_t pat = tile0 + pl;
  // lanes of a rate class beyond R (R < RT) repeat class R - 1 and are
  // dropped at the root, so the step loop has no branch on the rate
  const int rr = min(r, R - 1);

  // leaf pipeline: the slots hold the rows of the next PR_LEAVES leaves, get
  // the first of them; a slot is refilled with the row PR_LEAVES on as soon
  // as its values are in use, by an index read a leaf before that
  const uint16_t *index = p.index + (min(pat, p.n_pat - 1) - p.index_col);   // idle lanes repeat the last pattern
  const char *rows = static_cast<const char *>(p.rows) + blockIdx.y * p.rows_stride + (size_t)rr * (4 * sizeof(V));
  const uint32_t *unit = p.leaf_unit;
  const uint32_t RU = (uint32_t)R * VU;
  constexpr uint32_t SLOT = VU * NT * 16u;
  const uint32_t slot0 = smem_u32(smem + L::leaf_off(RT)) + 16u * c;   // [slot][VU][NT] of 16 bytes
  const bool scaled_rows = p.row_flag[blockIdx.y] != 0;
  int escale = 0;
  uint32_t next_row = __ldg(index), next_unit = __ldg(unit);
  auto after = [&](uint32_t slot) { return slot == slot0 + (PR_LEAVES - 1) * SLOT ? slot0 : slot + SLOT; };
  auto refill = [&](uint32_t slot) {
    const uint32_t u = next_unit + next_row * RU;
    const char *src = rows + (size_t)u * 16;
#pragma unroll
    for (int k = 0; k < VU; ++k) cp_async_16(slot + k * NT * 16u, src + 16 * k);
    asm volatile("cp.async.commit_group;" ::: "memory");
    if (scaled_rows && u >= p.exp_unit)
      escale += __ldg(p.row_exp + blockIdx.y * p.exp_stride + (u - p.exp_unit) / VU + rr);
    index += p.ld_index;
    next_row = __ldg(index);
    next_unit = __ldg(++unit);
  };
  uint32_t get = slot0;
#pragma unroll
  for (int j = 0; j < PR_LEAVES; ++j) refill(slot0 + j * SLOT);

  // The stack discipline is fixed by the schedule: in postorder the result
  // of step i - 1 is always a child of step i when any child of it is
  // internal; a step with two leaves sets the previous result aside (push),
  // and a step with two internal children takes its first child from the
  // stack (pop).  So the top of the stack lives in registers and each step is
  // one of three straight-line cases, chosen by a warp-uniform branch.
  V top[4];
  V *my = stk + c;   // this thread's column of the stack: entry (k, e) at my[(4 k + e) NT]
  int sp = -1;       // entries set aside, -1 before the first step
  bool ok = true;
  const unsigned char *coefs = ring + rr * 16;

#pragma unroll 1
  for (int g0 = 0; g0 < p.n_ops; g0 += G) {
    const int q = g0 / G, b = q & (NB - 1);
    if (!__all_sync(0xffffffffu, mbar_wait_bounded(&full[b], (q / NB) & 1, p.flag))) {
      ok = false;
      break;
    }
    const int g1 = min(g0 + G, p.n_ops);
#pragma unroll 1
    for (int i = g0; i < g1; ++i) {
      const int slot = i & (ST - 1), kind = step_kind[slot];
      const Coef *coef = reinterpret_cast<const Coef *>(coefs + slot * SB);
      V acc[4], y0[4], y1[4];
      if (kind == 1) {          // the previous result and a leaf
        asm volatile("cp.async.wait_group %0;" ::"n"(PR_LEAVES - 1) : "memory");
        Pol::load_row_s(get, get + NT * 16u, y1);
        Pol::rows(coef, top, y0, RT);
        Pol::mul4(y0, y1, acc);
        refill(get);
        get = after(get);
      } else if (kind == 0) {   // two leaves; the previous result waits on the stack
        if (sp >= 0) {
#pragma unroll
          for (int e = 0; e < 4; ++e) my[(4 * sp + e) * NT] = top[e];
        }
        ++sp;
        asm volatile("cp.async.wait_group %0;" ::"n"(PR_LEAVES - 2) : "memory");
        const uint32_t second = after(get);
        Pol::load_row_s(get, get + NT * 16u, y0);
        Pol::load_row_s(second, second + NT * 16u, y1);
        Pol::mul4(y0, y1, acc);
        refill(get);
        refill(second);
        get = after(second);
      } else {                  // both internal: the first from the stack
        --sp;
        V xa[4];
#pragma unroll
        for (int e = 0; e < 4; ++e) xa[e] = my[(4 * sp + e) * NT];
        Pol::rows(coef, xa, y0, RT);
        Pol::rows(reinterpret_cast<const Coef *>(coefs + slot * SB + CB), top, y1, RT);
        Pol::mul4(y0, y1, acc);
      }
      // rare, so the warp only enters when some lane needs it
      const auto mx = largest<Pol>(acc);
      if (__any_sync(0xffffffffu, mx < Pol::thresh)) {
        if (mx < Pol::thresh) rescale_vec<Pol>(acc, mx, escale);
      }
#pragma unroll
      for (int e = 0; e < 4; ++e) top[e] = acc[e];
    }
    // this warp is done with the group's step slots
    __syncwarp();
    if (lane == 0) mbar_arrive(&empty[b]);
  }
  asm volatile("cp.async.wait_all;" ::: "memory");

  // root: sum over rate classes of probs[r] 2^e_r sum_i pi_i x_i, in FP64;
  // the rate classes of a pattern meet in shared memory
  double part = 0.0;
  if (ok && r < R) {
    const double *pi = p.pi + (size_t)blockIdx.y * 4, *probs = p.probs + (size_t)blockIdx.y * R;
    double lr = 0.0;
#pragma unroll
    for (int e = 0; e < 4; ++e) lr += pi[e] * Pol::to_d(top[e]);
    part = probs[r] * lr;
  }
  xch[r][pl] = make_double2(part, (double)escale);
  asm volatile("bar.sync 1, %0;" ::"r"(NT) : "memory");
  double s = 0.0, comp = 0.0;
  // the first NP threads take a pattern each: FP64 costs a warp the same
  // however few of its lanes work
  if (c < NP) {
    int emax = -0x7fffffff;
    for (int q = 0; q < R; ++q) emax = max(emax, (int)xch[q][c].y);
    double site = 0.0;
    for (int q = 0; q < R; ++q) {
      const double2 v = xch[q][c];
      site += ldexp(v.x, (int)v.y - emax);
    }
    const size_t mine = tile0 + c;
    if (ok && mine < p.n_pat) {
      const double lnl = log(site) + (double)emax * 0.69314718055994530942;
      if (p.site_lnl) p.site_lnl[mine] = lnl;
      s = p.weights ? p.weights[mine] * lnl : lnl;
    }
  }
  warp_csum(s, comp);
  const int cw = c >> 5;
  if (lane == 0) red[cw] = make_double2(s, comp);
  asm volatile("bar.sync 1, %0;" ::"r"(NT) : "memory");
  const double2 *parts = p.partials + (size_t)blockIdx.y * p.n_tiles_total;
  if (cw == 0) {
    double2 v = lane < NT / 32 ? red[lane] : make_double2(0.0, 0.0);
    double ss = v.x, cc = v.y;
    warp_csum(ss, cc);
    if (lane == 0) {
      p.partials[(size_t)blockIdx.y * p.n_tiles_total + tile] = make_double2(ss, cc);
      __threadfence();
      last_cta = atomicAdd(p.done + blockIdx.y, 1u) == (unsigned)p.n_tiles_total - 1u;
    }
  }
  asm volatile("bar.sync 1, %0;" ::"r"(NT) : "memory");
  if (!last_cta) return;
  // the model's last CTA: every partial, in contiguous chunks of the tiles
  // and a fixed butterfly, so the total does not depend on which CTA it is
  __threadfence();
  const size_t per = (p.n_tiles_total + NT - 1) / NT;
  const size_t lo = min((size_t)c * per, p.n_tiles_total), hi = min(lo + per, p.n_tiles_total);
  s = comp = 0.0;
  for (size_t i = lo; i < hi; ++i) {
    const double2 v = __ldcg(parts + i);
    double u, e;
    two_sum(s, v.x, u, e);
    s = u;
    comp += e + v.y;
  }
  warp_csum(s, comp);
  if (lane == 0) red[cw] = make_double2(s, comp);
  asm volatile("bar.sync 1, %0;" ::"r"(NT) : "memory");
  if (cw == 0) {
    double2 v = lane < NT / 32 ? red[lane] : make_double2(0.0, 0.0);
    double ss = v.x, cc = v.y;
    warp_csum(ss, cc);
    if (lane == 0) p.lnl[blockIdx.y] = ss + cc;
  }
}

template <typename Pol, int RT>
pgpu_status launch_prune_rt(pgpu_ctx *ctx, PruneArgs &a, size_t n_tiles, size_t smem, int n_models,
                            cudaStream_t stream) {
  PGPU_CUDA(ctx, cudaFuncSetAttribute(prune_tree_kernel<Pol, RT>,
                                      cudaFuncAttributeMaxDynamicSharedMemorySize,
                                      (int)std::max<size_t>(smem, 48 * 1024)));
  prune_tree_kernel<Pol, RT><<<dim3((unsigned)n_tiles, (unsigned)n_models), 32 + PR_THREADS, smem,
                               stream>>>(a);
  return pgpu_after_launch(ctx, "prune_tree_kernel");
}

// Tip codes still in host memory: copied column chunk by column chunk on
// the context's copy stream, each chunk's launch waiting only for its own
// columns, so the copy of chunk k + 1 overlaps the scoring of chunk k.
struct HostTips {
  const uint8_t *host;   // [n_tips][n_pat]
  uint8_t *dev;          // [n_tips][ld_pat]
  size_t n_tips, ld_pat;
};

// The launches of one scoring: tile ranges [bounds[k], bounds[k + 1]).
struct ChunkPlan {
  size_t bounds[PGPU_COPY_CHUNKS + 1];
  int K;
  size_t smem;
};

// Column chunks for tip codes in host memory: the first chunk is one wave
// of CTAs (the one copy the scoring cannot hide), each next one
// PruneTune::growth times the last, so a chunk's copy ends while the chunk
// before it is scored and few launch boundaries drain the GPU; whole waves
// keep every launch but the last free of a part-filled wave.  Tip codes
// already on the device: one launch.
template <typename Pol, int RT>
pgpu_status plan_chunks_rt(pgpu_ctx *ctx, size_t n_tiles, int n_models, bool host, ChunkPlan &pl) {
  pl.K = 0;
  pl.bounds[0] = 0;
  if (host) {
    PGPU_CUDA(ctx, cudaFuncSetAttribute(prune_tree_kernel<Pol, RT>,
                                        cudaFuncAttributeMaxDynamicSharedMemorySize,
                                        (int)std::max<size_t>(pl.smem, 48 * 1024)));
    int per_sm = 0;
    PGPU_CUDA(ctx, cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, prune_tree_kernel<Pol, RT>,
                                                                 32 + PR_THREADS, pl.smem));
    const size_t wave =
        std::max<size_t>((size_t)std::max(per_sm, 1) * (size_t)ctx->num_sms / (size_t)std::max(n_models, 1), 1);
    size_t t = 0, c = wave;
    while (pl.K < PGPU_COPY_CHUNKS - 1 && n_tiles - t >= c + wave) {
      t += c;
      pl.bounds[++pl.K] = t;
      c *= PruneTune<Pol>::growth;
    }
  }
  pl.bounds[++pl.K] = n_tiles;
  return PGPU_OK;
}

// Sets a's tiling and plans its launches.  With the tip codes in host
// memory it also queues every chunk's copy on the copy stream, chunk k's
// end marked by copy_ev[k], so that the first copy runs beside the model
// setup kernels queued after it.
template <typename Pol>
pgpu_status plan_prune(pgpu_ctx *ctx, PruneArgs &a, int RT, int n_models, const HostTips *ht, ChunkPlan &pl) {
  a.NP = PR_THREADS / RT;
  const size_t n_tiles = (a.n_pat + a.NP - 1) / a.NP;
  a.n_tiles_total = n_tiles;
  a.tile_base = 0;
  pl.smem = PruneLayout<Pol>::bytes(RT, a.depth);
  if (pl.smem > ctx->smem_optin)
    return pgpu_set_err(ctx, PGPU_ERR_LIMIT, "prune: %zu bytes of shared memory needed (tree too deep)",
                        pl.smem);
  const bool host = ht != nullptr;
  switch (RT) {
    case 1: PGPU_TRY((plan_chunks_rt<Pol, 1>(ctx, n_tiles, n_models, host, pl))); break;
    case 2: PGPU_TRY((plan_chunks_rt<Pol, 2>(ctx, n_tiles, n_models, host, pl))); break;
    case 4: PGPU_TRY((plan_chunks_rt<Pol, 4>(ctx, n_tiles, n_models, host, pl))); break;
    default: PGPU_TRY((plan_chunks_rt<Pol, 8>(ctx, n_tiles, n_models, host, pl))); break;
  }
  if (host)
    for (int k = 0; k < pl.K; ++k) {
      const size_t c0 = pl.bounds[k] * a.NP, c1 = std::min(pl.bounds[k + 1] * a.NP, a.n_pat);
      if (c1 > c0)
        PGPU_CUDA(ctx, cudaMemcpy2DAsync(ht->dev + c0, ht->ld_pat, ht->host + c0, a.n_pat, c1 - c0, ht->n_tips,
                                         cudaMemcpyHostToDevice, ctx->copy_stream));
      PGPU_CUDA(ctx, cudaEventRecord(ctx->copy_ev[k], ctx->copy_stream));
    }
  return PGPU_OK;
}

// Tables and leaf indexes of the patterns of tiles [t0, t1), or either alone.
template <typename Pol>
pgpu_status launch_prep(pgpu_ctx *ctx, const TableArgs &t, int n_models, IndexArgs &x, int n_leaf, size_t pat0,
                        size_t pat1, bool tables, cudaStream_t stream) {
  const size_t n_table = tables ? (size_t)t.n_made * t.R * t.blocks * n_models : 0;
  x.col0 = pat0;
  x.cols = pat1 - pat0;
  x.blocks = (int)((x.cols + 256 * IX_PATTERNS - 1) / (256 * IX_PATTERNS));
  const size_t grid = n_table + (size_t)n_leaf * x.blocks;
  if (grid == 0) return PGPU_OK;
  if (grid > 0x7fffffff) return pgpu_set_err(ctx, PGPU_ERR_LIMIT, "prune: too many patterns and leaves");
  prune_prep_kernel<Pol><<<(unsigned)grid, 256, 0, stream>>>(t, x, (int)n_table);
  return pgpu_after_launch(ctx, "prune_prep_kernel");
}

// Launches every tile.  With the codes in host memory in several chunks,
// consecutive launches alternate between the context stream and the
// auxiliary one, so a chunk's CTAs take the SMs the previous chunk's CTAs
// leave instead of waiting for the whole launch to drain (the tiles are
// disjoint; each launch waits only for its own columns).  Where the leaf
// indexes of all patterns would take more than index_cols columns, pieces of
// that many take turns in one buffer, on the context stream alone.
template <typename Pol, int RT>
pgpu_status launch_prune_chunks(pgpu_ctx *ctx, PruneArgs &a, const ChunkPlan &pl, int n_models, bool host,
                                const TableArgs &t, IndexArgs &x, size_t index_cols) {
  const bool whole = index_cols >= a.n_tiles_total * a.NP;
  const bool fork = host && pl.K > 1 && whole;
  const size_t piece = whole ? a.n_tiles_total : index_cols / a.NP;
  bool tables = t.n_made > 0;
  if (fork) {
    if (tables) PGPU_TRY(launch_prep<Pol>(ctx, t, n_models, x, 0, 0, 0, true, ctx->stream));
    tables = false;
    PGPU_CUDA(ctx, cudaEventRecord(ctx->aux_ev[0], ctx->stream));
    PGPU_CUDA(ctx, cudaStreamWaitEvent(ctx->aux_stream, ctx->aux_ev[0], 0));
  }
  uint16_t *index = x.index;
  for (int k = 0; k < pl.K; ++k) {
    const cudaStream_t ks = fork && (k & 1) ? ctx->aux_stream : ctx->stream;
    if (host) PGPU_CUDA(ctx, cudaStreamWaitEvent(ks, ctx->copy_ev[k], 0));
    for (size_t t0 = pl.bounds[k]; t0 < pl.bounds[k + 1]; t0 += piece) {
      const size_t t1 = std::min(t0 + piece, pl.bounds[k + 1]);
      const size_t p0 = t0 * a.NP, p1 = std::min(t1 * a.NP, a.n_pat);
      x.index = whole ? index + p0 : index;
      PGPU_TRY(launch_prep<Pol>(ctx, t, n_models, x, a.n_leaf, p0, p1, tables, ks));
      tables = false;
      a.index = x.index;
      a.index_col = p0;
      a.tile_base = t0;
      PGPU_TRY((launch_prune_rt<Pol, RT>(ctx, a, t1 - t0, pl.smem, n_models, ks)));
    }
  }
  if (fork) {
    PGPU_CUDA(ctx, cudaEventRecord(ctx->aux_ev[1], ctx->aux_stream));
    PGPU_CUDA(ctx, cudaStreamWaitEvent(ctx->stream, ctx->aux_ev[1], 0));
  }
  a.tile_base = 0;
  return PGPU_OK;
}

template <typename Pol>
pgpu_status launch_prune(pgpu_ctx *ctx, PruneArgs &a, int RT, int n_models, const ChunkPlan &pl, bool host,
                         const TableArgs &t, IndexArgs &x, size_t index_cols) {
  switch (RT) {
    case 1: return launch_prune_chunks<Pol, 1>(ctx, a, pl, n_models, host, t, x, index_cols);
    case 2: return launch_prune_chunks<Pol, 2>(ctx, a, pl, n_models, host, t, x, index_cols);
    case 4: return launch_prune_chunks<Pol, 4>(ctx, a, pl, n_models, host, t, x, index_cols);
    default: return launch_prune_chunks<Pol, 8>(ctx, a, pl, n_models, host, t, x, index_cols);
  }
}

}  // namespace

namespace {
using namespace pgpu_forms;

pgpu_status check_model(pgpu_ctx *ctx, const pgpu_model *m, const pgpu_tip_codes *codes) {
  if (!m || !m->Q || !m->pi || !m->rates || !m->probs)
    return pgpu_set_err(ctx, PGPU_ERR_ARG, "prune: null model field");
  if (!codes || !codes->table || codes->n_codes < 1 || codes->n_codes > 256)
    return pgpu_set_err(ctx, PGPU_ERR_ARG, "prune: tip code table must have 1..256 rows");
  if (m->n_rates < 1 || m->n_rates > 8)
    return pgpu_set_err(ctx, PGPU_ERR_LIMIT, "prune: 1..8 rate classes are supported");
  if (m->n_states != 4)
    return pgpu_set_err(ctx, PGPU_ERR_UNSUPPORTED,
                        "prune: the SIMT pruning kernel is built for 4 states (DNA); use "
                        "pgpu_batch_lnl for 20- and 61-state models");
  return PGPU_OK;
}

// all small per-call parameters in one staged block
struct Staged {
  double *Q, *pi, *rates, *probs, *tab, *brlen, *U, *lam, *Ui;
  int *status;
  size_t bytes;
};

Staged stage_layout(int S, int R, int n_codes, int n_br, int V) {
  Staged s{};
  size_t off = 0;
  auto take = [&](size_t n) {
    const size_t o = off;
    off += align16(n * sizeof(double));
    return o;
  };
  s.Q = (double *)take((size_t)V * S * S);
  s.pi = (double *)take((size_t)V * S);
  s.rates = (double *)take((size_t)V * R);
  s.probs = (double *)take((size_t)V * R);
  s.tab = (double *)take((size_t)n_codes * S);
  s.brlen = (double *)take(n_br);
  // the eigen systems, where the host solves them
  s.U = (double *)take((size_t)V * S * S);
  s.lam = (double *)take((size_t)V * S);
  s.Ui = (double *)take((size_t)V * S * S);
  s.status = (int *)take(V);
  s.bytes = off;
  return s;
}

template <typename Ptr>
Ptr *rebase(void *base, Ptr *off) {
  return reinterpret_cast<Ptr *>(static_cast<char *>(base) + reinterpret_cast<size_t>(off));
}

// The reduced tree a call walks, kept on the context (with its device copy)
// for further calls on the same tree.
//
// level: tips of the largest subtree that becomes a leaf (1: none).  A
// collapsed leaf costs n_codes^k table rows where the walk would compute its
// k - 1 nodes for every pattern, so it is worth it while the table is the
// smaller side: at most half the patterns (16 codes: from 8,192 patterns on
// three tips, from 512 on two).  call_bytes is what one row takes over all
// models; the tables of a call stay below 1 GB.  most: the highest level to
// try, lowered when the device has no room for the tables (the plan made then
// serves this tree's later calls too).
pgpu_status prune_plan(pgpu_ctx *ctx, const pgpu_tree *tree, int R, int n_codes, size_t n_pat,
                       size_t row_bytes, size_t call_bytes, int most, const PrunePlan **out) {
  const int32_t n = tree->n_tips, n_int = n - 1;
  const size_t NC = (size_t)n_codes;
  const int asked = 2 * NC * NC * NC <= n_pat && NC * NC * NC <= 65536 ? 3 : 2 * NC * NC <= n_pat ? 2 : 1;
  int level = std::min(asked, most);
  PrunePlan &pl = ctx->prune_plan;
  const bool same_tree = pl.valid && (int32_t)pl.left.size() == n_int &&
                         std::memcmp(pl.left.data(), tree->left, n_int * 4) == 0 &&
                         std::memcmp(pl.right.data(), tree->right, n_int * 4) == 0;
  if (same_tree && pl.R == R && pl.n_codes == n_codes && pl.row_bytes == row_bytes && pl.asked == asked &&
      pl.level <= level && pl.made_rows * call_bytes <= (size_t)1 << 30) {
    *out = &pl;
    return PGPU_OK;
  }
  TreeSchedule sch;
  PGPU_TRY(pgpu_not_capturing(ctx, "a tree or a form that is new to the context"));
  PGPU_TRY(pgpu_check_tree(ctx, tree));
  pl.valid = false;
  pl.asked = asked;
  pl.R = R;
  pl.n_codes = n_codes;
  pl.row_bytes = row_bytes;
  std::vector<int32_t> tips(n_int), id(2 * n - 1), branch, left, right;
  for (int32_t k = 0; k < n_int; ++k) {
    const int32_t a = tree->left[k], b = tree->right[k];
    tips[k] = (a < n ? 1 : tips[a - n]) + (b < n ? 1 : tips[b - n]);
  }
  for (;; --level) {
    // leaves: tips and maximal subtrees of at most `level` tips below the
    // root; {leaf, branch, cherry's branch} of the latter
    std::vector<int4> leaf;
    pl.made.clear();
    pl.made_rows = 0;
    std::vector<uint8_t> inside(2 * n - 1, 0);   // below a collapsed node, or one
    auto small = [&](int32_t v) { return v < n || (v != 2 * n - 2 && tips[v - n] <= level); };
    for (int32_t v = 2 * n - 2; v >= n; --v)
      for (const int32_t c : {tree->left[v - n], tree->right[v - n]})
        if (inside[v] || small(v)) inside[c] = 1;
    branch.clear();
    left.clear();
    right.clear();
    for (int32_t v = 0; v < 2 * n - 2; ++v) {
      if (inside[v] || !small(v)) continue;
      id[v] = (int32_t)leaf.size();
      branch.push_back(v);
      if (v < n) {
        leaf.push_back(make_int4(v, -1, -1, (int)(uint32_t)((size_t)v * R * NC)));
        continue;
      }
      int32_t a = tree->left[v - n], b = tree->right[v - n], cherry = -1;
      if (a < n && b >= n) std::swap(a, b);
      int4 lf = make_int4(a, b, -1, (int)(uint32_t)((size_t)n * R * NC + pl.made_rows));
      if (a >= n) {
        cherry = a;
        lf = make_int4(tree->left[a - n], tree->right[a - n], b, lf.w);
      }
      pl.made.push_back(make_int4((int)leaf.size(), v, cherry, 0));
      pl.made_rows += (size_t)R * NC * NC * (cherry >= 0 ? NC : 1);
      leaf.push_back(lf);
    }
    const size_t n_rows = (size_t)n * R * NC + pl.made_rows;
    if (level > 1 && (n_rows > 0x7fffffffull || pl.made_rows * call_bytes > (size_t)1 << 30 ||
                      pl.made.size() * R * ((NC * NC + 255) / 256) > 0x7fffffff))
      continue;
    if (n_rows > 0x7fffffffull) return pgpu_set_err(ctx, PGPU_ERR_LIMIT, "prune: 2^31 leaf rows or more");
    pl.level = level;
    const int32_t nl = (int32_t)leaf.size();
    int32_t next = nl;
    for (int32_t v = n; v <= 2 * n - 2; ++v) {
      if (inside[v] || small(v)) continue;
      id[v] = next++;
      if (v < 2 * n - 2) branch.push_back(v);
      left.push_back(id[tree->left[v - n]]);
      right.push_back(id[tree->right[v - n]]);
    }
    pgpu_tree red{nl, left.data(), right.data(), nullptr};
    PGPU_TRY(pgpu_build_schedule(ctx, &red, &sch));
    // steps, and the leaves in the order the steps read them, then row 0
    // of the first tip PR_PAD times
    std::vector<int32_t> place(nl);
    for (int32_t j = 0; j < nl; ++j) place[sch.tip_seq[j]] = j;
    pl.ops.clear();
    for (const SchedOp &op : sch.ops) {
      const int br[2] = {op.a >= nl ? branch[op.a] : -1, op.b >= nl ? branch[op.b] : -1};
      const int k = (br[0] >= 0) + (br[1] >= 0);
      pl.ops.push_back(make_int4(k, br[0] >= 0 ? br[0] : br[1], br[1], 0));
    }
    pl.leaves.assign(nl + PR_PAD, make_int4(-1, -1, -1, 0));
    for (int32_t j = 0; j < nl; ++j) pl.leaves[j] = leaf[sch.tip_seq[j]];
    for (int4 &m : pl.made) m.x = place[m.x];
    pl.depth = std::max(sch.max_depth, 1);
    break;
  }
  // resident on the device: {ops, leaves, made, units}
  const size_t n_all = pl.ops.size() + pl.leaves.size() + pl.made.size();
  const size_t bytes = 16 * n_all + 4 * pl.leaves.size();
  void *h, *dst;
  PGPU_TRY(pgpu_buf(ctx, BUF_OPS2, bytes, &dst));
  PGPU_TRY(pgpu_stage(ctx, bytes, &h, nullptr));
  int4 *q = static_cast<int4 *>(h);
  q = std::copy(pl.ops.begin(), pl.ops.end(), q);
  q = std::copy(pl.leaves.begin(), pl.leaves.end(), q);
  q = std::copy(pl.made.begin(), pl.made.end(), q);
  uint32_t *unit = reinterpret_cast<uint32_t *>(q);
  for (const int4 &lf : pl.leaves) *unit++ = (uint32_t)lf.w * (uint32_t)(row_bytes / 16);
  PGPU_TRY(pgpu_stage_copy(ctx, dst, bytes));
  pl.d_ops = static_cast<const int4 *>(dst);
  pl.d_leaves = pl.d_ops + pl.ops.size();
  pl.d_made = pl.d_leaves + pl.leaves.size();
  pl.d_unit = reinterpret_cast<const uint32_t *>(pl.d_made + pl.made.size());
  pl.left.assign(tree->left, tree->left + n_int);
  pl.right.assign(tree->right, tree->right + n_int);
  pl.valid = true;
  *out = &pl;
  return PGPU_OK;
}

// Scores n_models models (same state and rate-class counts) over one tree
// and one set of patterns: lnl_dev[v] for model v.  One launch each for all
// models' eigen systems, P matrices, tip rows and collapsed leaves, then one
// pruning launch whose CTA rows are the models.
// host_tips: the codes are still in host memory (n_pat bytes per row) and
// tips is the device buffer they go to; they are copied in chunks that
// overlap the scoring.
pgpu_status prune_dev(pgpu_ctx *ctx, const pgpu_tree *tree, const pgpu_model *models, int n_models,
                      const pgpu_tip_codes *codes, const uint8_t *tips, size_t ld_pat,
                      const double *weights, size_t n_pat, int precision, double *lnl_dev,
                      double *site_lnl_dev, const uint8_t *host_tips = nullptr) {
  if (!models || n_models < 1) return pgpu_set_err(ctx, PGPU_ERR_ARG, "prune: no model");
  if (n_models > 65535) return pgpu_set_err(ctx, PGPU_ERR_LIMIT, "prune: at most 65,535 models per call");
  for (int v = 0; v < n_models; ++v) {
    PGPU_TRY(check_model(ctx, &models[v], codes));
    if (models[v].n_rates != models[0].n_rates)
      return pgpu_set_err(ctx, PGPU_ERR_ARG, "prune: every model needs the same number of rate classes");
  }
  if (n_models > 1 && site_lnl_dev)
    return pgpu_set_err(ctx, PGPU_ERR_ARG, "prune: site log-likelihoods are for one model at a time");
  if (precision != 32 && precision != 48 && precision != 64)
    return pgpu_set_err(ctx, PGPU_ERR_ARG, "prune: precision must be 32, 48 or 64");
  if (!tree || !tree->brlen) return pgpu_set_err(ctx, PGPU_ERR_ARG, "prune: tree->brlen is required");
  if (!tips || !lnl_dev) return pgpu_set_err(ctx, PGPU_ERR_ARG, "prune: null buffer");
  if (ld_pat % 16 != 0 || ld_pat < n_pat || ((uintptr_t)tips & 15))
    return pgpu_set_err(ctx, PGPU_ERR_ARG,
                        "prune: ld_pat (%zu) must be a multiple of 16 and >= n_pat, rows 16-byte aligned",
                        ld_pat);
  const int V = n_models;
  const int S = models[0].n_states, R = models[0].n_rates, n = tree->n_tips, n_br = 2 * n - 2;
  if (!tree->left || !tree->right || n < 2)
    return pgpu_set_err(ctx, PGPU_ERR_ARG, "tree: null tree or fewer than 2 tips");
  for (int i = 0; i < n_br; ++i)
    if (!(tree->brlen[i] >= 0.0) || !std::isfinite(tree->brlen[i]))
      return pgpu_set_err(ctx, PGPU_ERR_ARG, "prune: branch length %d is negative or not finite", i);
  const size_t row_bytes = precision == 32 ? 16 : 32;
  const int RT = R <= 1 ? 1 : R <= 2 ? 2 : R <= 4 ? 4 : 8;
  const size_t tile = PR_THREADS / RT, n_tiles = (n_pat + tile - 1) / tile;
  const size_t SS = (size_t)S * S;
  const size_t coef = precision == 32 ? 4 : 8;   // float, double, or float pair
  const size_t p_bytes = align16((size_t)n_br * RT * SS * coef);
  const size_t tip_rows = (size_t)n * R * codes->n_codes;
  const size_t clear = align16((size_t)V * 2 * sizeof(int));

  // Device scratch: P matrices, per-CTA partial sums, leaf rows (every tip's,
  // then the collapsed leaves'), CTA counters and exponent flags (cleared by
  // the setup kernel) and the rows' exponents, and the leaf indexes, of all
  // patterns or in pieces of at most 1 GB.  Where the device has no room,
  // smaller pieces, then less collapsed: what a call cannot do without is what
  // the walk over every node takes, and indexes of one tile.
  const PrunePlan *pp;
  void *dP, *dpart, *drows, *dexp, *dix = nullptr;
  size_t cols = 0, rows_bytes = 0;
  PGPU_TRY(pgpu_buf(ctx, BUF_I, (size_t)V * p_bytes, &dP));
  PGPU_TRY(pgpu_buf(ctx, BUF_G, std::max<size_t>(n_tiles, 1) * V * sizeof(double2), &dpart));
  for (int most = 3;; most = pp->level - 1) {
    PGPU_TRY(prune_plan(ctx, tree, R, codes->n_codes, n_pat, row_bytes, row_bytes * V, most, &pp));
    rows_bytes = align16((tip_rows + pp->made_rows) * row_bytes);
    pgpu_status st = pgpu_buf(ctx, BUF_J, (size_t)V * rows_bytes, &drows);
    if (st == PGPU_OK) st = pgpu_buf(ctx, BUF_E, clear + (size_t)V * pp->made_rows * sizeof(int), &dexp);
    const size_t n_leaf = pp->leaves.size();   // the padding included
    size_t piece = std::min(n_tiles, std::max<size_t>(((size_t)1 << 29) / n_leaf / tile, 1));
    for (; st == PGPU_OK && n_tiles > 0; piece = (piece + 1) / 2) {
      cols = piece * tile;
      st = pgpu_buf(ctx, BUF_D, n_leaf * cols * sizeof(uint16_t), &dix);
      if (st != PGPU_ERR_OOM || piece == 1) break;
      st = PGPU_OK;
    }
    if (st == PGPU_OK) break;
    if (st != PGPU_ERR_OOM || pp->level == 1) return st;
    PGPU_TRY(pgpu_buf_release(ctx, BUF_J));   // the larger tables' room
    PGPU_TRY(pgpu_buf_release(ctx, BUF_E));
  }
  const size_t made_rows = pp->made_rows;
  const int n_leaf = (int)pp->leaves.size();

  // stage every model's Q, pi, rates, probs, then the code table and the
  // branch lengths
  Staged lay = stage_layout(S, R, codes->n_codes, n_br, V);
  void *h, *d;
  PGPU_TRY(pgpu_stage(ctx, lay.bytes, &h, &d));
  for (int v = 0; v < V; ++v) {
    const pgpu_model *m = &models[v];
    std::copy(m->Q, m->Q + S * S, rebase(h, lay.Q) + (size_t)v * S * S);
    std::copy(m->pi, m->pi + S, rebase(h, lay.pi) + (size_t)v * S);
    std::copy(m->rates, m->rates + R, rebase(h, lay.rates) + (size_t)v * R);
    std::copy(m->probs, m->probs + R, rebase(h, lay.probs) + (size_t)v * R);
  }
  std::copy(codes->table, codes->table + (size_t)codes->n_codes * S, rebase(h, lay.tab));
  std::copy(tree->brlen, tree->brlen + n_br, rebase(h, lay.brlen));
  // A handful of 4 x 4 eigen systems is quicker on the host (about 1 us
  // each) than in a launch of its own (36 us, however many).
  const bool host_eig = V <= 24;
  if (host_eig)
    for (int v = 0; v < V; ++v)
      rebase(h, lay.status)[v] =
          pgpu_host_eig4(models[v].Q, models[v].pi, rebase(h, lay.U) + (size_t)v * 16,
                         rebase(h, lay.lam) + (size_t)v * 4, rebase(h, lay.Ui) + (size_t)v * 16);
  PGPU_TRY(pgpu_stage_commit(ctx, lay.bytes));

  const double *dU = rebase(d, lay.U), *dUi = rebase(d, lay.Ui), *dlam = rebase(d, lay.lam);
  const int *dst = rebase(d, lay.status);
  if (!host_eig) {
    void *deig;
    PGPU_TRY(pgpu_buf(ctx, BUF_H, (size_t)V * ((2 * SS + S) * 8 + sizeof(int)) + 64, &deig));
    double *u = static_cast<double *>(deig);
    int *st = reinterpret_cast<int *>(u + V * (2 * SS + S));
    PGPU_TRY(pgpu_launch_eig(ctx, rebase(d, lay.Q), rebase(d, lay.pi), S, V, u, u + 2 * V * SS, u + V * SS, st));
    dU = u;
    dUi = u + V * SS;
    dlam = u + 2 * V * SS;
    dst = st;
  }
  PruneArgs a;
  a.P = dP;
  a.rows = drows;
  a.done = static_cast<unsigned *>(dexp);
  a.row_flag = static_cast<const int *>(dexp) + V;
  a.row_exp = reinterpret_cast<const int *>(static_cast<const char *>(dexp) + clear);
  a.pi = rebase(d, lay.pi);
  a.probs = rebase(d, lay.probs);
  a.weights = weights;
  a.site_lnl = site_lnl_dev;
  a.partials = (double2 *)dpart;
  a.lnl = lnl_dev;
  a.ops = pp->d_ops;
  a.leaf_unit = pp->d_unit;
  a.flag = ctx->d_flag;
  a.P_stride = p_bytes;
  a.rows_stride = rows_bytes;
  a.exp_stride = made_rows;
  a.exp_unit = (uint32_t)(tip_rows * (row_bytes / 16));
  a.n_pat = n_pat;
  a.n_ops = (int)pp->ops.size();
  a.n_leaf = n_leaf;
  a.R = R;
  a.NP = 0;
  a.depth = pp->depth;
  HostTips ht{host_tips, const_cast<uint8_t *>(tips), (size_t)n, ld_pat};
  const HostTips *htp = host_tips ? &ht : nullptr;
  ChunkPlan pl;
  if (n_pat > 0) {
    if (precision == 32) PGPU_TRY(plan_prune<Fp32>(ctx, a, RT, V, htp, pl));
    else if (precision == 48) PGPU_TRY(plan_prune<Ff32>(ctx, a, RT, V, htp, pl));
    else PGPU_TRY(plan_prune<Fp64>(ctx, a, RT, V, htp, pl));
  }
  // every model's P matrices and tip rows, formed in FP64 and stored in the
  // form's value type
  PGPU_TRY(pgpu_launch_dna_setup(ctx, dU, dlam, dUi, V, rebase(d, lay.brlen), n, rebase(d, lay.rates), R, RT,
                                 rebase(d, lay.tab), codes->n_codes, precision, dP, p_bytes, drows,
                                 rows_bytes, dst, a.done, const_cast<int *>(a.row_flag), 1));
  if (n_pat == 0) {
    PGPU_CUDA(ctx, cudaMemsetAsync(lnl_dev, 0, (size_t)V * sizeof(double), ctx->stream));
    return PGPU_OK;
  }
  TableArgs t{};
  t.rows = drows;
  t.P = dP;
  t.leaves = pp->d_leaves;
  t.made = pp->d_made;
  t.row_exp = const_cast<int *>(a.row_exp);
  t.row_flag = const_cast<int *>(a.row_flag);
  t.P_stride = p_bytes;
  t.rows_stride = rows_bytes;
  t.exp_stride = made_rows;
  t.exp_base = tip_rows;
  t.R = R;
  t.RT = RT;
  t.n_codes = codes->n_codes;
  t.n_made = (int)pp->made.size();
  t.status = dst;
  t.blocks = (codes->n_codes * codes->n_codes + 255) / 256;
  IndexArgs x{};
  x.tip_codes = tips;
  x.leaves = pp->d_leaves;
  x.ld_pat = ld_pat;
  x.ld_index = a.ld_index = cols;
  x.n_pat = n_pat;
  x.n_codes = codes->n_codes;
  x.flag = ctx->d_flag;
  x.index = static_cast<uint16_t *>(dix);
  if (precision == 32) return launch_prune<Fp32>(ctx, a, RT, V, pl, htp != nullptr, t, x, cols);
  if (precision == 48) return launch_prune<Ff32>(ctx, a, RT, V, pl, htp != nullptr, t, x, cols);
  return launch_prune<Fp64>(ctx, a, RT, V, pl, htp != nullptr, t, x, cols);
}

// Codes and weights of a small call (up to PGPU_STAGE_MOST bytes) through one
// pinned staging block and one copy, rows ld apart: what copies from pageable
// memory cost such a call is waiting (32 taxa x 1,000 patterns: 94 us a
// call against 125 with them).
pgpu_status stage_data(pgpu_ctx *ctx, const uint8_t *tip_codes, size_t n, size_t n_pat, size_t ld,
                       const double *weights, void **dt, void **dw, bool *staged) {
  const size_t cb = n * ld, wb = weights ? n_pat * 8 : 0;
  *staged = n_pat > 0 && cb + wb <= PGPU_STAGE_MOST;
  if (!*staged) return PGPU_OK;
  void *hv;
  PGPU_TRY(pgpu_buf(ctx, BUF_TIPS, cb + wb, dt));
  PGPU_TRY(pgpu_stage(ctx, cb + wb, &hv, nullptr));
  char *h = static_cast<char *>(hv);
  for (size_t i = 0; i < n; ++i) std::memcpy(h + i * ld, tip_codes + i * n_pat, n_pat);
  if (weights) std::memcpy(h + cb, weights, wb);
  *dw = weights ? static_cast<char *>(*dt) + cb : nullptr;
  return pgpu_stage_copy(ctx, *dt, cb + wb);
}

// Results of a host call, with the error word: `bytes` from the device to
// dst (and the double after them to *last), through a staging block when
// they are few.
pgpu_status read_back(pgpu_ctx *ctx, const void *src, void *dst, size_t bytes, double *last = nullptr) {
  const size_t all = bytes + (last ? 8 : 0);
  void *h = nullptr;
  if (all <= PGPU_STAGE_MOST) {
    PGPU_TRY(pgpu_stage(ctx, all, &h, nullptr));
    PGPU_CUDA(ctx, cudaMemcpyAsync(h, src, all, cudaMemcpyDeviceToHost, ctx->stream));
  } else {
    h = ctx->h_pinned;
    PGPU_CUDA(ctx, cudaMemcpyAsync(dst, src, bytes, cudaMemcpyDeviceToHost, ctx->stream));
    if (last)
      PGPU_CUDA(ctx, cudaMemcpyAsync(h, static_cast<const char *>(src) + bytes, 8, cudaMemcpyDeviceToHost,
                                     ctx->stream));
  }
  PGPU_TRY(pgpu_check_flag(ctx, "prune"));
  if (all <= PGPU_STAGE_MOST) {
    std::memcpy(dst, h, bytes);
    if (last) std::memcpy(last, static_cast<char *>(h) + bytes, 8);
  } else if (last) {
    std::memcpy(last, h, 8);
  }
  return PGPU_OK;
}

}  // namespace

extern "C" {

pgpu_status pgpu_prune_lnl_dev(pgpu_ctx *ctx, const pgpu_tree *tree, const pgpu_model *model,
                               const pgpu_tip_codes *codes, const uint8_t *tip_codes_dev,
                               size_t ld_pat, const double *weights_dev, size_t n_pat,
                               int precision, double *lnl_dev, double *site_lnl_dev) {
  if (!ctx) return PGPU_ERR_ARG;
  PGPU_CUDA(ctx, cudaSetDevice(ctx->device));
  return prune_dev(ctx, tree, model, 1, codes, tip_codes_dev, ld_pat, weights_dev, n_pat, precision,
                   lnl_dev, site_lnl_dev);
}

pgpu_status pgpu_prune_lnl_models_dev(pgpu_ctx *ctx, const pgpu_tree *tree,
                                      const pgpu_model *models, int n_models,
                                      const pgpu_tip_codes *codes, const uint8_t *tip_codes_dev,
                                      size_t ld_pat, const double *weights_dev, size_t n_pat,
                                      int precision, double *lnl_dev) {
  if (!ctx) return PGPU_ERR_ARG;
  PGPU_CUDA(ctx, cudaSetDevice(ctx->device));
  return prune_dev(ctx, tree, models, n_models, codes, tip_codes_dev, ld_pat, weights_dev, n_pat,
                   precision, lnl_dev, nullptr);
}

pgpu_status pgpu_prune_lnl_models(pgpu_ctx *ctx, const pgpu_tree *tree, const pgpu_model *models,
                                  int n_models, const pgpu_tip_codes *codes,
                                  const uint8_t *tip_codes, const double *weights, size_t n_pat,
                                  int precision, double *lnl) {
  if (!ctx) return PGPU_ERR_ARG;
  if (!tree || tree->n_tips < 2 || !tip_codes || !lnl || n_models < 1)
    return pgpu_set_err(ctx, PGPU_ERR_ARG, "prune: null argument, no model or fewer than 2 tips");
  PGPU_CUDA(ctx, cudaSetDevice(ctx->device));
  const size_t n = (size_t)tree->n_tips;
  const size_t ld = (n_pat + 15) / 16 * 16;
  void *dt, *dw = nullptr, *dl;
  PGPU_TRY(pgpu_buf(ctx, BUF_SCALAR, std::max<size_t>((size_t)n_models * 8, 64), &dl));
  cudaStream_t s = ctx->stream;
  bool staged;
  PGPU_TRY(stage_data(ctx, tip_codes, n, n_pat, ld, weights, &dt, &dw, &staged));
  if (!staged) {
    PGPU_TRY(pgpu_buf(ctx, BUF_TIPS, std::max<size_t>(n * ld, 16), &dt));
    if (weights) PGPU_TRY(pgpu_buf(ctx, BUF_WEIGHTS, n_pat * 8, &dw));
    if (n_pat) {
      PGPU_CUDA(ctx, cudaMemcpy2DAsync(dt, ld, tip_codes, n_pat, n_pat, n, cudaMemcpyHostToDevice, s));
      if (weights) PGPU_CUDA(ctx, cudaMemcpyAsync(dw, weights, n_pat * 8, cudaMemcpyHostToDevice, s));
    }
  }
  PGPU_TRY(prune_dev(ctx, tree, models, n_models, codes, (const uint8_t *)dt, ld,
                     (const double *)dw, n_pat, precision, (double *)dl, nullptr));
  return read_back(ctx, dl, lnl, (size_t)n_models * 8);
}

pgpu_status pgpu_prune_lnl(pgpu_ctx *ctx, const pgpu_tree *tree, const pgpu_model *model,
                           const pgpu_tip_codes *codes, const uint8_t *tip_codes,
                           const double *weights, size_t n_pat, int precision, double *lnl,
                           double *site_lnl) {
  if (!ctx) return PGPU_ERR_ARG;
  if (!tree || tree->n_tips < 2 || !tip_codes || !lnl)
    return pgpu_set_err(ctx, PGPU_ERR_ARG, "prune: null argument or fewer than 2 tips");
  PGPU_CUDA(ctx, cudaSetDevice(ctx->device));
  const size_t n = (size_t)tree->n_tips;
  const size_t ld = (n_pat + 15) / 16 * 16;
  void *dt, *dw = nullptr, *dl, *dsl = nullptr;
  // the sum follows the patterns' values: one copy back
  PGPU_TRY(pgpu_buf(ctx, BUF_SITECOST, (site_lnl ? n_pat + 1 : 1) * 8, &dsl));
  dl = static_cast<double *>(dsl) + (site_lnl ? n_pat : 0);
  cudaStream_t s = ctx->stream;
  bool staged;
  PGPU_TRY(stage_data(ctx, tip_codes, n, n_pat, ld, weights, &dt, &dw, &staged));
  if (staged) {
    PGPU_TRY(prune_dev(ctx, tree, model, 1, codes, (const uint8_t *)dt, ld, (const double *)dw, n_pat,
                       precision, (double *)dl, site_lnl ? (double *)dsl : nullptr));
    if (!site_lnl) return read_back(ctx, dl, lnl, 8);
    return read_back(ctx, dsl, site_lnl, n_pat * 8, lnl);
  }
  PGPU_TRY(pgpu_buf(ctx, BUF_TIPS, std::max<size_t>(n * ld, 16), &dt));
  if (weights) PGPU_TRY(pgpu_buf(ctx, BUF_WEIGHTS, n_pat * 8, &dw));
  // the tip codes go over in column chunks on the copy stream, after
  // everything already queued on the context's stream (which may still read
  // the device buffer), each chunk's scoring waiting for its own columns
  PGPU_TRY(pgpu_copy_stream(ctx));
  PGPU_CUDA(ctx, cudaEventRecord(ctx->copy_ev[PGPU_COPY_CHUNKS], s));
  PGPU_CUDA(ctx, cudaStreamWaitEvent(ctx->copy_stream, ctx->copy_ev[PGPU_COPY_CHUNKS], 0));
  // the weights go first on the copy stream: the first chunk's event covers them
  if (n_pat && weights)
    PGPU_CUDA(ctx, cudaMemcpyAsync(dw, weights, n_pat * 8, cudaMemcpyHostToDevice, ctx->copy_stream));
  PGPU_TRY(pgpu_settle_copies(ctx, prune_dev(ctx, tree, model, 1, codes, (const uint8_t *)dt, ld,
                                              (const double *)dw, n_pat, precision, (double *)dl,
                                              site_lnl ? (double *)dsl : nullptr, tip_codes)));
  double *hl = reinterpret_cast<double *>(ctx->h_pinned);
  PGPU_CUDA(ctx, cudaMemcpyAsync(hl, dl, 8, cudaMemcpyDeviceToHost, s));
  if (site_lnl && n_pat)
    PGPU_CUDA(ctx, cudaMemcpyAsync(site_lnl, dsl, n_pat * 8, cudaMemcpyDeviceToHost, s));
  PGPU_TRY(pgpu_check_flag(ctx, "prune"));
  *lnl = *hl;
  return PGPU_OK;
}

}  // extern "C"
