// Cost-matrix (TCM) medians of state sets over a tree.
//
// Reference: CostMatrix.Make (lib/costMatrix.ml:124-196) tabulates, for a
// bit-flag alphabet and a transformation cost matrix of its atomic states,
// the median cost and median code of every pair of state-set codes
// (fill_cm, :141-166) with one of three median rules chosen by the matrix's
// declared properties (:145-149): find_median_general (:68-86),
// find_median_metric (:104-122) or find_median_equal (:89-101).  A tree's
// cost under such a character is the postorder of Node.Make1D.median_2
// (lib/node.ml:183-198): each internal node takes the table's median of its
// children's codes and adds the table's cost.  With the unit matrix the
// table is Fitch's rule (test/costMatrixTest.ml:83-108).
//
// GPU layout: DNA-sized alphabets (at most 4 states) as 4-bit lanes, eight
// sites per 32-bit word, like the Fitch kernels.  One thread owns one word
// column and walks the whole postorder; the table is packed
// (cost << 4 | median code, bit 31 = "pair has no median", i.e. an empty or
// out-of-alphabet code) and replicated once per lane in shared memory
// (entry e of lane l at [e][l]), so a warp's 32 lookups never share a bank.
// The top of the node stack stays in a register; pushes and pops follow the
// schedule's fixed discipline (a step with two tip children sets the last
// result aside, one with two internal children takes its first child back).
#include <algorithm>
#include <cstring>

#include "pgpu_internal.cuh"

// The packed pair table (256 words) of a call, staged to the device.
pgpu_status pgpu_tcm_table(pgpu_ctx *ctx, const uint32_t *table, const uint32_t **dev) {
  void *h, *d;
  PGPU_TRY(pgpu_stage(ctx, 256 * sizeof(uint32_t), &h, &d));
  std::memcpy(h, table, 256 * sizeof(uint32_t));
  *dev = static_cast<const uint32_t *>(d);
  return pgpu_stage_commit(ctx, 256 * sizeof(uint32_t));
}

namespace {

constexpr int TC_THREADS = 256;
constexpr uint32_t TC_NONE = 0x80000000u;      // pair without a median
constexpr uint32_t TC_COST_MASK = 0x07ffffffu;  // cost field (bits 4..30)
constexpr int32_t TC_ENTRY_MAX = 1 << 25;       // per TCM entry, so a pair sum fits the field

struct TcmArgs {
  const uint32_t *tips;      // [n_tips][ld]
  const uint32_t *weights;   // [n_sites] or null
  const uint32_t *table;     // [256] packed entries, index (a << 4) | b
  const int4 *ops;           // schedule (k, first, second, -)
  uint32_t *node_sets;       // [n_tips - 1][ld]
  uint32_t *site_cost;       // [n_sites] or null
  unsigned long long *total;
  int *flag;
  size_t ld, n_words, n_sites;
  int n_tips, n_ops, depth;
};

__device__ __forceinline__ uint32_t valid4(size_t w, size_t n_sites) {
  const size_t first = w * 8;
  if (first + 8 <= n_sites) return 0xffffffffu;
  if (first >= n_sites) return 0u;
  return (1u << (4 * int(n_sites - first))) - 1u;
}

__global__ void __launch_bounds__(TC_THREADS) tcm_tree_kernel(const TcmArgs a) {
  __shared__ uint32_t tab[256 * 32];
  __shared__ unsigned long long red[TC_THREADS / 32];
  extern __shared__ uint32_t stk[];   // [depth][TC_THREADS]
  const int t = threadIdx.x, lane = t & 31;
  for (int i = t; i < 256 * 32; i += TC_THREADS) tab[i] = __ldg(a.table + (i >> 5));
  __syncthreads();
  const size_t w = (size_t)blockIdx.x * TC_THREADS + t;
  const bool on = w < a.n_words;
  const uint32_t valid = on ? valid4(w, a.n_sites) : 0u;
  const uint32_t fill = 0x11111111u & ~valid;   // lanes past the last site read as state 1
  const uint32_t *tb = tab + lane;
  auto tip = [&](int ch) -> uint32_t {
    const uint32_t x = on ? __ldg(a.tips + (size_t)ch * a.ld + w) : 0u;
    return (x & valid) | fill;
  };
  uint32_t cnt[8] = {0, 0, 0, 0, 0, 0, 0, 0};
  uint32_t top = 0, none = 0;
  int sp = 0;
  bool ok = true;
  for (int i = 0; i < a.n_ops && ok; ++i) {
    const int4 op = __ldg(a.ops + i);
    const int kind = (op.y >= a.n_tips ? 1 : 0) | (op.z >= a.n_tips ? 2 : 0);
    uint32_t xa, xb;
    if (kind == 0) {   // two tips: the previous result waits on the stack
      if (i > 0) {
        if (sp < a.depth) stk[sp++ * TC_THREADS + t] = top;
        else ok = false;
      }
      xa = tip(op.y);
      xb = tip(op.z);
    } else if (kind == 1) {   // the first child is the previous result
      xa = top;
      xb = tip(op.z);
    } else if (kind == 2) {   // the second child is the previous result
      xa = tip(op.y);
      xb = top;
    } else {                  // both internal: the first from the stack
      if (sp > 0) {
        xa = stk[--sp * TC_THREADS + t];
      } else {
        ok = false;
        xa = 0x11111111u;
      }
      xb = top;
    }
    uint32_t out = 0;
#pragma unroll
    for (int l = 0; l < 8; ++l) {
      const uint32_t ia = (xa >> (4 * l)) & 15u, ib = (xb >> (4 * l)) & 15u;
      const uint32_t e = tb[((ia << 4) | ib) << 5];
      out |= (e & 15u) << (4 * l);
      cnt[l] += e >> 4;   // a no-median entry fails the call, so its bit 31 never matters
      none |= e;
    }
    if (on) a.node_sets[(size_t)op.x * a.ld + w] = out & valid;
    top = out;
  }
  unsigned long long tot = 0;
  if (on && ok) {
#pragma unroll
    for (int l = 0; l < 8; ++l) {
      const size_t s = w * 8 + l;
      if (s < a.n_sites) {
        if (a.site_cost) a.site_cost[s] = cnt[l];
        tot += (unsigned long long)(a.weights ? __ldg(a.weights + s) : 1u) * cnt[l];
      }
    }
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) tot += __shfl_xor_sync(0xffffffffu, tot, o);
  if (lane == 0) red[t >> 5] = tot;
  if (__any_sync(0xffffffffu, (none & TC_NONE) != 0) && lane == 0) atomicOr(a.flag, PGPU_FLAG_BADCODE);
  __syncthreads();
  if (t == 0) {
    unsigned long long s = 0;
    for (int k = 0; k < TC_THREADS / 32; ++k) s += red[k];
    if (s) atomicAdd(a.total, s);
  }
}

// ---- wide alphabets: medians formed on the fly ----------------------------
// For alphabets of up to 32 atomic states (codes of 8, 16 or 32 bits, one
// site per lane) a table over every pair of codes no longer fits, so each
// node forms its medians from the TCM itself, one row per atomic state in
// shared memory.  find_median_general / _metric (lib/costMatrix.ml:68-86,
// 104-122) take, over every atomic pair (a, b) of the two codes, the
// candidates k minimising tcm[a][k] + tcm[b][k], and keep the pairs reaching
// the overall minimum.  That is the same as
//   best = min_k (C_i[k] + C_j[k]),  C_i[k] = min_{a in i} tcm[a][k],
//   code = OR of the k reaching it,
// over all k (general) or the states of i | j (metric): a pair's minimum is
// never below best, and reaches it exactly where some k does.
// find_median_equal (:89-101) intersects at tcm[0][0] or unites at
// tcm[0][1].  All three are symmetric in i and j, so a TCM declared
// symmetric (its table filled for i <= j and mirrored, :150-156) needs no
// ordering of the codes.
//
// tcm_wide_kernel walks the segmented schedule of the Fitch kernel (four
// warps per CTA, each its own subtrees of the same 32 sites, a site per
// lane), so a warp's chain is a quarter of the postorder and 20,000 sites
// give 2,500 warps instead of 625.  C_i is built a whole row at a time: one
// 16-byte shared load and packed minima per 4 words for every state of the
// code, instead of a scalar search per candidate k.  With every cost at most
// 16,383 a word holds two states as 16-bit halves (j and j + W), so a sum of
// two costs stays below the padding's 2 x 0x7fff; larger costs take a word
// per state.  A row for the code "every state" (missing data) makes that
// code as short as a single state.  The row stride is an odd multiple of 16
// bytes, so the rows of 8 lanes' 16-byte loads fall in distinct banks.
// Bound by instruction issue (the per-state minima and sums), not by memory.
// 128 taxa x 20,003 sites of 20 states, metric rule: 59 us a call against
// 1,252 us with one thread per word searching the candidates one by one.
struct TcmWideArgs {
  const uint32_t *tips;      // [n_tips][ld] lanes of LB bits
  const uint32_t *weights;   // [n_sites] or null
  const uint32_t *rows;      // [S + 1][row stride] packed costs, the last row "every state"
  const int4 *ops, *seg, *top, *wseg;
  uint32_t *node_sets;
  uint32_t *site_cost;
  unsigned long long *total;
  int *flag;
  size_t ld, n_words, n_sites;
  int n_tips, n_top, depth, S, mode;
  uint32_t equal, unequal;   // the equal rule's costs tcm[0][0], tcm[0][1]
};

// words from one packed row to the next: an odd number of 16-byte units
__host__ __device__ constexpr int wide_stride(int W) { return W % 8 == 0 ? W + 4 : W; }

constexpr uint32_t TW_PAD16 = 0x7fffu;       // a state that does not exist, 16-bit costs
constexpr uint32_t TW_PAD32 = 0x3fffffffu;   // ... and 32-bit costs
constexpr int32_t TW_MAX16 = 0x3fff;         // largest cost of the 16-bit form

// C[k] = min over the states s of `code` of row s, in W packed words
template <int W, bool U16>
__device__ __forceinline__ void wide_min_rows(const uint32_t *rows, int S, uint32_t all, uint32_t code,
                                              uint32_t (&c)[W]) {
  auto load = [&](int s, uint32_t (&r)[W]) {
    const uint4 *q = reinterpret_cast<const uint4 *>(rows + s * wide_stride(W));
#pragma unroll
    for (int j = 0; j < W / 4; ++j) {
      const uint4 v = q[j];
      r[4 * j] = v.x, r[4 * j + 1] = v.y, r[4 * j + 2] = v.z, r[4 * j + 3] = v.w;
    }
  };
  const bool every = code == all;
  load(every ? S : __ffs(code) - 1, c);
  for (uint32_t m = every ? 0u : code & (code - 1u); m; m &= m - 1u) {
    uint32_t r[W];
    load(__ffs(m) - 1, r);
#pragma unroll
    for (int j = 0; j < W; ++j) c[j] = U16 ? __vminu2(c[j], r[j]) : min(c[j], r[j]);
  }
}

// the median of codes a and b; none is set (and the code is 0) where the
// pair has no median
template <int W, bool U16>
__device__ __forceinline__ uint32_t wide_median(const TcmWideArgs &p, const uint32_t *rows, uint32_t all,
                                                uint32_t a, uint32_t b, uint32_t &cost, bool &none) {
  const bool bad = a == 0u || b == 0u || ((a | b) & ~all);
  none |= bad;
  if (p.mode == PGPU_TCM_EQUAL) {
    const uint32_t inter = a & b;
    cost = bad ? 0u : inter ? p.equal : p.unequal;
    return bad ? 0u : inter ? inter : (a | b);
  }
  if (bad) a = b = 1u;
  const uint32_t cand = p.mode == PGPU_TCM_METRIC ? (a | b) : all;
  uint32_t s[W], t[W];
  wide_min_rows<W, U16>(rows, p.S, all, a, s);
  wide_min_rows<W, U16>(rows, p.S, all, b, t);
  uint32_t best, code;
  if (U16) {
    // sums of states outside the candidates become 0xffff in their half
    const uint32_t out = ~cand;
    const uint32_t out2 = (out & ((1u << W) - 1u)) | ((out >> W) << 16);
    best = 0xffffffffu;
#pragma unroll
    for (int j = 0; j < W; ++j) {
      s[j] = (s[j] + t[j]) | (((out2 >> j) & 0x00010001u) * 0xffffu);
      best = __vminu2(best, s[j]);
    }
    best = min(best & 0xffffu, best >> 16);
    const uint32_t best2 = best * 0x00010001u;
    // 0 in a half that reaches best, else 1 (no half is below best)
    uint32_t off = 0u;
#pragma unroll
    for (int j = 0; j < W; ++j) off |= __vminu2(s[j] - best2, 0x00010001u) << j;
    code = (~off & ((1u << W) - 1u)) | ((~off >> 16) << W);
  } else {
    best = 0xffffffffu;
#pragma unroll
    for (int j = 0; j < W; ++j) {
      s[j] += t[j];
      if (!((cand >> j) & 1u)) s[j] = 0xffffffffu;
      best = min(best, s[j]);
    }
    code = 0u;
#pragma unroll
    for (int j = 0; j < W; ++j) code |= s[j] == best ? 1u << j : 0u;
  }
  cost = bad ? 0u : best;
  return bad ? 0u : code & cand;
}

template <int LB> struct WideLane;
template <> struct WideLane<8> { using T = uint8_t; };
template <> struct WideLane<16> { using T = uint16_t; };
template <> struct WideLane<32> { using T = uint32_t; };

template <int LB, int W, bool U16>
__global__ void __launch_bounds__(PGPU_SPLIT_WARPS * 32) tcm_wide_kernel(const TcmWideArgs p) {
  using T = typename WideLane<LB>::T;
  constexpr int PER = 32 / LB;
  extern __shared__ __align__(16) uint32_t wsm[];
  const int tid = threadIdx.x, w = tid >> 5, lane = tid & 31;
  const int n_row = (p.S + 1) * wide_stride(W);
  uint32_t *rows = wsm;
  uint32_t *stk0 = wsm + n_row + (size_t)w * p.depth * 32 + lane;   // this lane's column
  uint32_t *join = wsm + n_row + (size_t)PGPU_SPLIT_WARPS * p.depth * 32 + lane;
  uint32_t *sitecnt = wsm + n_row + (size_t)(PGPU_SPLIT_WARPS * p.depth + PGPU_SPLIT_JOINS) * 32;
  for (int i = tid; i < n_row; i += PGPU_SPLIT_WARPS * 32) rows[i] = __ldg(p.rows + i);
  if (tid < 32) sitecnt[tid] = 0u;
  __syncthreads();
  const uint32_t all = p.S == 32 ? 0xffffffffu : (1u << p.S) - 1u;
  const size_t site = (size_t)blockIdx.x * 32 + lane;
  const bool in = site < p.n_words * PER;   // the lane's place exists in the rows
  const bool valid = site < p.n_sites;
  // lanes past the last site read as atomic state 0, which always has a
  // median, and are written as zero
  const T *col = reinterpret_cast<const T *>(p.tips) + site;
  T *out = reinterpret_cast<T *>(p.node_sets) + site;
  const size_t ldt = p.ld * PER;
  auto tip = [&](int ch) -> uint32_t { return valid ? (uint32_t)__ldg(col + (size_t)ch * ldt) : 1u; };
  auto put = [&](int k, uint32_t m) {
    if (in) out[(size_t)k * ldt] = (T)(valid ? m : 0u);
  };
  uint32_t acc = 0;
  bool none = false;

  // ---- each warp walks its segments ----
  const int4 ws = p.wseg[w];
  for (int q = 0; q < ws.y; ++q) {
    const int4 sg = p.seg[ws.x + q];   // {op_off, n_ops, tip_off, n_tips}
    uint32_t *stk = stk0 + (q + 1) * 32;   // rows below hold earlier results
    const int4 *ops = p.ops + sg.x;
    int4 op = __ldg(ops);
    // a step's tips are loaded one step ahead, so their latency passes
    // while the step before is computed
    uint32_t ta = op.y < p.n_tips ? tip(op.y) : 0u, tb = op.z < p.n_tips ? tip(op.z) : 0u;
    uint32_t top = 0;
    int sp = 0;
    for (int i = 0; i < sg.y; ++i) {
      const int4 next = i + 1 < sg.y ? __ldg(ops + i + 1) : op;
      uint32_t na = 0u, nb = 0u;
      if (next.y < p.n_tips) na = tip(next.y);
      if (next.z < p.n_tips) nb = tip(next.z);
      const bool a_tip = op.y < p.n_tips, b_tip = op.z < p.n_tips;
      uint32_t x = ta, y = tb;
      if (a_tip && b_tip) {   // the previous result waits on the stack
        if (i > 0) stk[32 * sp++] = top;
      } else if (a_tip) {
        y = top;
      } else {
        x = b_tip ? top : stk[32 * --sp];
        if (!b_tip) y = top;
      }
      uint32_t c;
      top = wide_median<W, U16>(p, rows, all, x, y, c, none);
      acc += c;
      put(op.x, top);
      op = next, ta = na, tb = nb;
    }
    stk0[q * 32] = top;
  }
  __syncthreads();
  // ---- warp 0 joins the segments ----
  if (w == 0)
    for (int i = 0; i < p.n_top; ++i) {
      const int4 op = __ldg(p.top + i);
      uint32_t ch[2];
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        const int ref = h == 0 ? op.y : op.z;
        if (ref >= 0) ch[h] = tip(ref);
        else if (ref > -1000)
          ch[h] = wsm[n_row + ((size_t)((-1 - ref) >> 5) * p.depth + ((-1 - ref) & 31)) * 32 + lane];
        else ch[h] = join[32 * (-1000 - ref)];
      }
      uint32_t c;
      const uint32_t m = wide_median<W, U16>(p, rows, all, ch[0], ch[1], c, none);
      acc += c;
      put(op.x, m);
      join[32 * i] = m;
    }
  atomicAdd(sitecnt + lane, acc);
  if (__any_sync(0xffffffffu, none) && lane == 0) atomicOr(p.flag, PGPU_FLAG_BADCODE);
  __syncthreads();
  if (w == 0) {
    const uint32_t v = sitecnt[lane];
    unsigned long long tot = 0;
    if (valid) {
      if (p.site_cost) p.site_cost[site] = v;
      tot = (unsigned long long)(p.weights ? __ldg(p.weights + site) : 1u) * v;
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) tot += __shfl_xor_sync(0xffffffffu, tot, o);
    if (lane == 0 && tot) atomicAdd(p.total, tot);
  }
}

template <int LB, int W, bool U16>
cudaError_t launch_wide(const TcmWideArgs &a, size_t smem, cudaStream_t s) {
  cudaError_t e = cudaFuncSetAttribute(tcm_wide_kernel<LB, W, U16>,
                                       cudaFuncAttributeMaxDynamicSharedMemorySize,
                                       (int)std::max<size_t>(smem, 48 * 1024));
  if (e != cudaSuccess) return e;
  const size_t grid = (a.n_words * (32 / LB) + 31) / 32;
  tcm_wide_kernel<LB, W, U16><<<(unsigned)grid, PGPU_SPLIT_WARPS * 32, smem, s>>>(a);
  return cudaGetLastError();
}

// W: packed words per row, the smallest multiple of 4 (16-bit halves) or of
// 8 (32-bit) that holds the states
template <bool U16>
cudaError_t launch_wide_lb(int lb, int W, const TcmWideArgs &a, size_t smem, cudaStream_t s) {
  constexpr int U = U16 ? 4 : 8;
  if (lb == 8) return launch_wide<8, U, U16>(a, smem, s);
  if (lb == 16)
    return W == U ? launch_wide<16, U, U16>(a, smem, s) : launch_wide<16, 2 * U, U16>(a, smem, s);
  switch (W / U) {
    case 1: return launch_wide<32, U, U16>(a, smem, s);
    case 2: return launch_wide<32, 2 * U, U16>(a, smem, s);
    case 3: return launch_wide<32, 3 * U, U16>(a, smem, s);
    default: return launch_wide<32, 4 * U, U16>(a, smem, s);
  }
}

// ---- the table (host): restates fill_cm and the three median rules ----

int64_t tcm_cost(const int32_t *tcm, int S, uint32_t x, uint32_t y) {   // x, y atomic codes
  return tcm[(31 - __builtin_clz(x)) * S + (31 - __builtin_clz(y))];
}

// find_median_pair (lib/costMatrix.ml:57-66)
void median_pair(const int32_t *tcm, int S, uint32_t i, uint32_t j, uint32_t candidates,
                 int64_t *cost, uint32_t *code) {
  int64_t best = INT64_MAX;
  uint32_t assign = 0;
  for (int b = 0; b < S; ++b) {
    const uint32_t k = 1u << b;
    if (!(candidates & k)) continue;
    const int64_t c = tcm_cost(tcm, S, i, k) + tcm_cost(tcm, S, j, k);
    if (c == best) assign |= k;
    else if (c < best) best = c, assign = k;
  }
  *cost = best;
  *code = assign;
}

// find_median_general / _metric / _equal (lib/costMatrix.ml:68-122), codes
// of up to 32 atomic states
void median(const int32_t *tcm, int S, int mode, uint32_t i, uint32_t j, int64_t *cost,
            uint32_t *code) {
  const uint32_t all = S == 32 ? 0xffffffffu : (1u << S) - 1u;
  if (mode == PGPU_TCM_EQUAL) {
    const int64_t unequal = tcm_cost(tcm, S, 1, 2), equal = tcm_cost(tcm, S, 1, 1);
    if (i & j) *cost = equal, *code = i & j;
    else *cost = unequal, *code = i | j;
    return;
  }
  const uint32_t cand = mode == PGPU_TCM_METRIC ? (i | j) : all;
  int64_t best = INT64_MAX;
  uint32_t assign = 0;
  for (int bi = 0; bi < S; ++bi) {
    if (!(i >> bi & 1u)) continue;
    for (int bj = 0; bj < S; ++bj) {
      if (!(j >> bj & 1u)) continue;
      int64_t c;
      uint32_t k;
      median_pair(tcm, S, 1u << bi, 1u << bj, cand, &c, &k);
      if (c == best) assign |= k;
      else if (c < best) best = c, assign = k;
    }
  }
  *cost = best;
  *code = assign;
}

// io: the rows are still in host memory (see HostRows); the segmented
// kernel copies them in chunks, the single-walk kernel whole.
pgpu_status tree_dev(pgpu_ctx *ctx, const pgpu_tree *tree, const uint32_t *tips, size_t ld,
                     const uint32_t *weights, size_t n_sites, const uint32_t *table,
                     uint32_t *node_sets, uint32_t *site_cost, unsigned long long *total,
                     const HostRows *io = nullptr) {
  if (!tree || tree->n_tips < 2) return pgpu_set_err(ctx, PGPU_ERR_ARG, "tcm_tree: need at least 2 tips");
  if (!tips || !node_sets || !total || !table) return pgpu_set_err(ctx, PGPU_ERR_ARG, "tcm_tree: null buffer");
  const size_t n_words = (n_sites + 7) / 8;
  if (ld < n_words) return pgpu_set_err(ctx, PGPU_ERR_ARG, "tcm_tree: ld_words (%zu) < %zu", ld, n_words);
  // every site's cost sum must fit uint32
  uint64_t emax = 0;
  for (int e = 0; e < 256; ++e)
    if (!(table[e] & TC_NONE)) emax = std::max<uint64_t>(emax, (table[e] >> 4) & TC_COST_MASK);
  if (emax * (uint64_t)(tree->n_tips - 1) > 0xffffffffull)
    return pgpu_set_err(ctx, PGPU_ERR_OVERFLOW,
                        "tcm_tree: a site's cost can reach %llu x %d, above 2^32 - 1",
                        (unsigned long long)emax, tree->n_tips - 1);
  if (n_words == 0) {
    PGPU_TRY(pgpu_check_tree(ctx, tree));
    PGPU_CUDA(ctx, cudaMemsetAsync(total, 0, sizeof(unsigned long long), ctx->stream));
    return PGPU_OK;
  }
  // the segmented schedule: subtrees walked by four warps per 128-word slice.
  // It sums costs in the low 28 bits of a register under the codes' top 4,
  // flushing every p steps so that a site's sum, at most p * emax, stays
  // below 2^28; below 16 steps between flushes it keeps one sum per register.
  const uint64_t per = ((1ull << 28) - 1) / std::max<uint64_t>(emax, 1);
  const int period = per >= 16 ? (int)std::min<uint64_t>(per, 1u << 30) : 0;
  bool launched = false;
  PGPU_TRY(pgpu_tcm_tree_split(ctx, tree, tips, ld, weights, n_sites,
                               table, period, node_sets, site_cost, total, &launched, io));
  if (launched) return PGPU_OK;
  const TreeSchedule *sch;
  const int4 *d_ops;
  const int32_t *d_seq;
  PGPU_TRY(pgpu_schedule_device(ctx, tree, &sch, &d_ops, &d_seq));
  const size_t n = (size_t)tree->n_tips;
  TcmArgs a;
  PGPU_TRY(pgpu_tcm_table(ctx, table, &a.table));
  PGPU_CUDA(ctx, cudaMemsetAsync(total, 0, sizeof(unsigned long long), ctx->stream));
  if (io)
    PGPU_CUDA(ctx, cudaMemcpy2DAsync(const_cast<uint32_t *>(tips), ld * 4, io->tips, n_words * 4, n_words * 4,
                                     n, cudaMemcpyHostToDevice, ctx->stream));
  a.tips = tips;
  a.weights = weights;
  a.ops = d_ops;
  a.node_sets = node_sets;
  a.site_cost = site_cost;
  a.total = total;
  a.flag = ctx->d_flag;
  a.ld = ld;
  a.n_words = n_words;
  a.n_sites = n_sites;
  a.n_tips = tree->n_tips;
  a.n_ops = (int)sch->ops.size();
  a.depth = std::max(sch->max_depth, 1);
  const size_t smem = (size_t)a.depth * TC_THREADS * sizeof(uint32_t);
  if (smem + sizeof(uint32_t) * 256 * 32 > (size_t)ctx->smem_optin)
    return pgpu_set_err(ctx, PGPU_ERR_LIMIT, "tcm_tree: tree too deep (%d stack entries)", a.depth);
  PGPU_CUDA(ctx, cudaFuncSetAttribute(tcm_tree_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                      (int)smem));
  const unsigned grid = (unsigned)((n_words + TC_THREADS - 1) / TC_THREADS);
  tcm_tree_kernel<<<grid, TC_THREADS, smem, ctx->stream>>>(a);
  PGPU_TRY(pgpu_after_launch(ctx, "tcm_tree_kernel"));
  if (io)
    PGPU_CUDA(ctx, cudaMemcpy2DAsync(io->node_sets, n_words * 4, node_sets, ld * 4, n_words * 4, n - 1,
                                     cudaMemcpyDeviceToHost, ctx->stream));
  return PGPU_OK;
}

pgpu_status tree_wide_dev(pgpu_ctx *ctx, const pgpu_tree *tree, const uint32_t *tips, size_t ld,
                          const uint32_t *weights, size_t n_sites, int lb, const int32_t *tcm,
                          int S, int mode, uint32_t *node_sets, uint32_t *site_cost,
                          unsigned long long *total) {
  if (!tree || tree->n_tips < 2)
    return pgpu_set_err(ctx, PGPU_ERR_ARG, "tcm_tree_wide: need at least 2 tips");
  if (!tips || !node_sets || !total || !tcm)
    return pgpu_set_err(ctx, PGPU_ERR_ARG, "tcm_tree_wide: null buffer");
  if (lb != 8 && lb != 16 && lb != 32)
    return pgpu_set_err(ctx, PGPU_ERR_ARG, "tcm_tree_wide: lane_bits must be 8, 16 or 32");
  if (S < 1 || S > lb)
    return pgpu_set_err(ctx, PGPU_ERR_LIMIT, "tcm_tree_wide: 1..%d states fit %d-bit lanes (got %d)",
                        lb, lb, S);
  if (mode != PGPU_TCM_GENERAL && mode != PGPU_TCM_METRIC && mode != PGPU_TCM_EQUAL)
    return pgpu_set_err(ctx, PGPU_ERR_ARG, "tcm_tree_wide: unknown median rule %d", mode);
  if (mode == PGPU_TCM_EQUAL && S < 2)
    return pgpu_set_err(ctx, PGPU_ERR_ARG, "tcm_tree_wide: the equal-cost rule needs two states");
  int64_t emax = 0;
  for (int e = 0; e < S * S; ++e) {
    if (tcm[e] < 0 || tcm[e] > TC_ENTRY_MAX)
      return pgpu_set_err(ctx, PGPU_ERR_LIMIT,
                          "tcm_tree_wide: costs must lie in [0, 2^25] (entry %d is %d)", e, tcm[e]);
    emax = std::max<int64_t>(emax, tcm[e]);
  }
  // a node adds at most two entries (one for the equal rule)
  if ((uint64_t)(2 * emax) * (uint64_t)(tree->n_tips - 1) > 0xffffffffull)
    return pgpu_set_err(ctx, PGPU_ERR_OVERFLOW,
                        "tcm_tree_wide: a site's cost can reach 2 x %lld x %d, above 2^32 - 1",
                        (long long)emax, tree->n_tips - 1);
  const int per = 32 / lb;
  const size_t n_words = (n_sites + per - 1) / per;
  if (ld < n_words)
    return pgpu_set_err(ctx, PGPU_ERR_ARG, "tcm_tree_wide: ld_words (%zu) < %zu", ld, n_words);
  TcmWideArgs a{};
  const int32_t *d_seq;
  const SplitSchedule *sp;
  PGPU_TRY(pgpu_split_device(ctx, tree, &sp, &a.ops, &a.seg, &a.top, &a.wseg, &d_seq));
  // the packed rows: row x holds tcm[x][k] for every k, row S their minima
  const bool u16 = emax <= TW_MAX16;
  const int unit = u16 ? 4 : 8;
  const int W = ((u16 ? (S + 1) / 2 : S) + unit - 1) / unit * unit, stride = wide_stride(W);
  const size_t n_row = (size_t)(S + 1) * stride;
  void *h, *d;
  PGPU_TRY(pgpu_stage(ctx, n_row * sizeof(uint32_t), &h, &d));
  uint32_t *rows = static_cast<uint32_t *>(h);
  for (int x = 0; x <= S; ++x)
    for (int j = 0; j < stride; ++j) {
      auto cost = [&](int k) -> uint32_t {
        if (j >= W || k >= S) return u16 ? TW_PAD16 : TW_PAD32;
        if (x < S) return (uint32_t)tcm[x * S + k];
        int32_t c = tcm[k];
        for (int y = 1; y < S; ++y) c = std::min(c, tcm[y * S + k]);
        return (uint32_t)c;
      };
      rows[(size_t)x * stride + j] = u16 ? cost(j) | cost(j + W) << 16 : cost(j);
    }
  PGPU_TRY(pgpu_stage_commit(ctx, n_row * sizeof(uint32_t)));
  PGPU_CUDA(ctx, cudaMemsetAsync(total, 0, sizeof(unsigned long long), ctx->stream));
  if (n_words == 0) return PGPU_OK;
  a.tips = tips;
  a.weights = weights;
  a.rows = static_cast<const uint32_t *>(d);
  a.node_sets = node_sets;
  a.site_cost = site_cost;
  a.total = total;
  a.flag = ctx->d_flag;
  a.ld = ld;
  a.n_words = n_words;
  a.n_sites = n_sites;
  a.n_tips = tree->n_tips;
  a.n_top = (int)sp->top.size();
  a.depth = sp->rows - PGPU_SPLIT_RING;   // the kernel keeps no copy ring
  a.S = S;
  a.mode = mode;
  a.equal = (uint32_t)tcm[0];
  a.unequal = S > 1 ? (uint32_t)tcm[1] : 0u;
  const size_t smem =
      (n_row + ((size_t)PGPU_SPLIT_WARPS * a.depth + PGPU_SPLIT_JOINS + 1) * 32) * sizeof(uint32_t);
  if (smem > (size_t)ctx->smem_optin)
    return pgpu_set_err(ctx, PGPU_ERR_LIMIT, "tcm_tree_wide: tree too deep (%d stack entries)",
                        a.depth);
  if ((n_words * per + 31) / 32 > 0x7fffffffu)
    return pgpu_set_err(ctx, PGPU_ERR_LIMIT, "tcm_tree_wide: too many sites");
  const cudaError_t e = u16 ? launch_wide_lb<true>(lb, W, a, smem, ctx->stream)
                            : launch_wide_lb<false>(lb, W, a, smem, ctx->stream);
  PGPU_CUDA(ctx, e);
  return pgpu_after_launch(ctx, "tcm_wide_kernel");
}

}  // namespace

extern "C" {

pgpu_status pgpu_tcm_median(const int32_t *tcm, int n_states, int mode, int symmetric, uint32_t i,
                            uint32_t j, int64_t *cost, uint32_t *code) {
  if (!tcm || !cost || !code) return PGPU_ERR_ARG;
  const int S = n_states;
  if (S < 1 || S > 32) return PGPU_ERR_LIMIT;
  if (mode != PGPU_TCM_GENERAL && mode != PGPU_TCM_METRIC && mode != PGPU_TCM_EQUAL) return PGPU_ERR_ARG;
  if (mode == PGPU_TCM_EQUAL && S < 2) return PGPU_ERR_ARG;
  const uint64_t all = (S == 32 ? 0xffffffffull : (1ull << S) - 1ull);
  if (i == 0 || j == 0 || (i & ~all) || (j & ~all)) {   // the reference's (inf, 0)
    *cost = INT64_MAX;
    *code = 0;
    return PGPU_OK;
  }
  if (symmetric && i > j) std::swap(i, j);
  int64_t c;
  uint32_t k;
  median(tcm, S, mode, i, j, &c, &k);
  *cost = c;
  *code = k;
  return PGPU_OK;
}

pgpu_status pgpu_tcm_tree_wide_dev(pgpu_ctx *ctx, const pgpu_tree *tree, const uint32_t *tips_dev,
                                   size_t ld_words, const uint32_t *weights_dev, size_t n_sites,
                                   int lane_bits, const int32_t *tcm, int n_states, int mode,
                                   int /*symmetric*/, uint32_t *node_sets_dev, uint32_t *site_cost_dev,
                                   uint64_t *total_dev) {
  if (!ctx) return PGPU_ERR_ARG;
  PGPU_CUDA(ctx, cudaSetDevice(ctx->device));
  return tree_wide_dev(ctx, tree, tips_dev, ld_words, weights_dev, n_sites, lane_bits, tcm, n_states,
                       mode, node_sets_dev, site_cost_dev,
                       reinterpret_cast<unsigned long long *>(total_dev));
}

pgpu_status pgpu_tcm_tree_wide(pgpu_ctx *ctx, const pgpu_tree *tree, const uint32_t *tips,
                               const uint32_t *weights, size_t n_sites, int lane_bits,
                               const int32_t *tcm, int n_states, int mode, int /*symmetric*/,
                               uint32_t *node_sets, uint32_t *site_cost, uint64_t *total) {
  if (!ctx) return PGPU_ERR_ARG;
  if (!tree || !tips || !node_sets || !total || !tcm)
    return pgpu_set_err(ctx, PGPU_ERR_ARG, "tcm_tree_wide: null argument");
  if (tree->n_tips < 2) return pgpu_set_err(ctx, PGPU_ERR_ARG, "tree: need at least 2 tips");
  if (lane_bits != 8 && lane_bits != 16 && lane_bits != 32)
    return pgpu_set_err(ctx, PGPU_ERR_ARG, "tcm_tree_wide: lane_bits must be 8, 16 or 32");
  PGPU_CUDA(ctx, cudaSetDevice(ctx->device));
  const int per = 32 / lane_bits;
  const size_t n_words = (n_sites + per - 1) / per;
  const size_t ld = (n_words + 3) / 4 * 4;
  const size_t n = (size_t)tree->n_tips, n_int = n - 1;
  void *dt, *dn, *dw = nullptr, *dsc = nullptr, *dtot;
  PGPU_TRY(pgpu_buf(ctx, BUF_TIPS, std::max<size_t>(n * ld * 4, 16), &dt));
  PGPU_TRY(pgpu_buf(ctx, BUF_OUT, std::max<size_t>(n_int * ld * 4, 16), &dn));
  PGPU_TRY(pgpu_buf(ctx, BUF_SCALAR, 64, &dtot));
  if (weights) PGPU_TRY(pgpu_buf(ctx, BUF_WEIGHTS, std::max<size_t>(n_sites * 4, 16), &dw));
  if (site_cost) PGPU_TRY(pgpu_buf(ctx, BUF_SITECOST, std::max<size_t>(n_sites * 4, 16), &dsc));
  cudaStream_t s = ctx->stream;
  if (n_words) {
    PGPU_CUDA(ctx, cudaMemcpy2DAsync(dt, ld * 4, tips, n_words * 4, n_words * 4, n,
                                     cudaMemcpyHostToDevice, s));
    if (weights) PGPU_CUDA(ctx, cudaMemcpyAsync(dw, weights, n_sites * 4, cudaMemcpyHostToDevice, s));
  }
  PGPU_TRY(tree_wide_dev(ctx, tree, (const uint32_t *)dt, ld, (const uint32_t *)dw, n_sites,
                         lane_bits, tcm, n_states, mode, (uint32_t *)dn, (uint32_t *)dsc,
                         (unsigned long long *)dtot));
  if (n_words) {
    PGPU_CUDA(ctx, cudaMemcpy2DAsync(node_sets, n_words * 4, dn, ld * 4, n_words * 4, n_int,
                                     cudaMemcpyDeviceToHost, s));
    if (site_cost) PGPU_CUDA(ctx, cudaMemcpyAsync(site_cost, dsc, n_sites * 4, cudaMemcpyDeviceToHost, s));
  }
  uint64_t *ht = reinterpret_cast<uint64_t *>(ctx->h_pinned);
  PGPU_CUDA(ctx, cudaMemcpyAsync(ht, dtot, 8, cudaMemcpyDeviceToHost, s));
  PGPU_TRY(pgpu_check_flag(ctx, "tcm_tree_wide"));
  *total = *ht;
  return PGPU_OK;
}


pgpu_status pgpu_tcm_tables(pgpu_ctx *ctx, const int32_t *tcm, int n_states, int mode, int symmetric,
                            uint32_t *table, int64_t *cost, int32_t *assign) {
  if (!tcm || !table) return pgpu_set_err(ctx, PGPU_ERR_ARG, "tcm_tables: null argument");
  const int S = n_states;
  if (S < 1 || S > 4)
    return pgpu_set_err(ctx, PGPU_ERR_LIMIT, "tcm_tables: 1..4 states fit the 4-bit lanes (got %d)", S);
  if (mode != PGPU_TCM_GENERAL && mode != PGPU_TCM_METRIC && mode != PGPU_TCM_EQUAL)
    return pgpu_set_err(ctx, PGPU_ERR_ARG, "tcm_tables: unknown median rule %d", mode);
  if (mode == PGPU_TCM_EQUAL && S < 2)
    return pgpu_set_err(ctx, PGPU_ERR_ARG, "tcm_tables: the equal-cost rule needs two states");
  for (int e = 0; e < S * S; ++e)
    if (tcm[e] < 0 || tcm[e] > TC_ENTRY_MAX)
      return pgpu_set_err(ctx, PGPU_ERR_LIMIT, "tcm_tables: costs must lie in [0, 2^25] (entry %d is %d)",
                          e, tcm[e]);
  for (int i = 0; i < 16; ++i)
    for (int j = 0; j < 16; ++j) {
      table[i * 16 + j] = TC_NONE;
      if (cost) cost[i * 16 + j] = INT64_MAX;
      if (assign) assign[i * 16 + j] = 0;
    }
  const int size = 1 << S;
  for (int i = 1; i < size; ++i)
    for (int j = symmetric ? i : 1; j < size; ++j) {
      int64_t c;
      uint32_t k;
      median(tcm, S, mode, (uint32_t)i, (uint32_t)j, &c, &k);
      const uint32_t packed = ((uint32_t)c << 4) | k;
      table[i * 16 + j] = packed;
      if (cost) cost[i * 16 + j] = c;
      if (assign) assign[i * 16 + j] = k;
      if (symmetric) {
        table[j * 16 + i] = packed;
        if (cost) cost[j * 16 + i] = c;
        if (assign) assign[j * 16 + i] = k;
      }
    }
  return PGPU_OK;
}

pgpu_status pgpu_tcm_tree_dev(pgpu_ctx *ctx, const pgpu_tree *tree, const uint32_t *tips_dev,
                              size_t ld_words, const uint32_t *weights_dev, size_t n_sites,
                              const uint32_t *table, uint32_t *node_sets_dev, uint32_t *site_cost_dev,
                              uint64_t *total_dev) {
  if (!ctx) return PGPU_ERR_ARG;
  PGPU_CUDA(ctx, cudaSetDevice(ctx->device));
  return tree_dev(ctx, tree, tips_dev, ld_words, weights_dev, n_sites, table, node_sets_dev,
                  site_cost_dev, reinterpret_cast<unsigned long long *>(total_dev));
}

pgpu_status pgpu_tcm_tree(pgpu_ctx *ctx, const pgpu_tree *tree, const uint32_t *tips,
                          const uint32_t *weights, size_t n_sites, const uint32_t *table,
                          uint32_t *node_sets, uint32_t *site_cost, uint64_t *total) {
  if (!ctx) return PGPU_ERR_ARG;
  if (!tree || !tips || !node_sets || !total || !table)
    return pgpu_set_err(ctx, PGPU_ERR_ARG, "tcm_tree: null argument");
  if (tree->n_tips < 2) return pgpu_set_err(ctx, PGPU_ERR_ARG, "tree: need at least 2 tips");
  PGPU_CUDA(ctx, cudaSetDevice(ctx->device));
  const size_t n_words = (n_sites + 7) / 8;
  const size_t ld = (n_words + 3) / 4 * 4;
  const size_t n = (size_t)tree->n_tips, n_int = n - 1;
  void *dw = nullptr, *dsc = nullptr, *dtot;
  PGPU_TRY(pgpu_buf(ctx, BUF_SCALAR, 64, &dtot));
  if (weights) PGPU_TRY(pgpu_buf(ctx, BUF_WEIGHTS, n_sites * 4, &dw));
  if (site_cost) PGPU_TRY(pgpu_buf(ctx, BUF_SITECOST, n_sites * 4, &dsc));
  cudaStream_t s = ctx->stream;
  // rows in page-locked host memory the device can address, 16-byte aligned
  // and a multiple of 4 words long: read and written by the kernel over the
  // CPU-GPU link, with no staging buffers
  const uint32_t *tv = nullptr;
  uint32_t *nv = nullptr;
  if (n_words > 0 && n_words % 4 == 0) {
    tv = static_cast<const uint32_t *>(pgpu_host_view(tips));
    nv = static_cast<uint32_t *>(pgpu_host_view(node_sets));
    if (((uintptr_t)tv | (uintptr_t)nv) & 15) tv = nullptr;
  }
  if (tv && nv) {
    if (weights) PGPU_CUDA(ctx, cudaMemcpyAsync(dw, weights, n_sites * 4, cudaMemcpyHostToDevice, s));
    PGPU_TRY(pgpu_settle_copies(ctx, tree_dev(ctx, tree, tv, n_words, (const uint32_t *)dw, n_sites, table,
                                               nv, (uint32_t *)dsc, (unsigned long long *)dtot)));
    if (site_cost)
      PGPU_CUDA(ctx, cudaMemcpyAsync(site_cost, dsc, n_sites * 4, cudaMemcpyDeviceToHost, s));
    uint64_t *ht = reinterpret_cast<uint64_t *>(ctx->h_pinned);
    PGPU_CUDA(ctx, cudaMemcpyAsync(ht, dtot, 8, cudaMemcpyDeviceToHost, s));
    PGPU_TRY(pgpu_check_flag(ctx, "tcm_tree"));
    *total = *ht;
    return PGPU_OK;
  }
  void *dt, *dn;
  PGPU_TRY(pgpu_buf(ctx, BUF_TIPS, n * ld * 4, &dt));
  PGPU_TRY(pgpu_buf(ctx, BUF_OUT, n_int * ld * 4, &dn));
  // the rows go over in column chunks on the copy streams (or whole, where
  // the single-walk kernel runs), after everything already queued on the
  // context's stream
  PGPU_TRY(pgpu_copy_stream(ctx));
  PGPU_CUDA(ctx, cudaEventRecord(ctx->copy_ev[PGPU_COPY_CHUNKS], s));
  PGPU_CUDA(ctx, cudaStreamWaitEvent(ctx->copy_stream, ctx->copy_ev[PGPU_COPY_CHUNKS], 0));
  PGPU_CUDA(ctx, cudaStreamWaitEvent(ctx->d2h_stream, ctx->copy_ev[PGPU_COPY_CHUNKS], 0));
  if (n_words && weights)
    PGPU_CUDA(ctx, cudaMemcpyAsync(dw, weights, n_sites * 4, cudaMemcpyHostToDevice, s));
  const HostRows io{tips, node_sets};
  PGPU_TRY(pgpu_settle_copies(ctx, tree_dev(ctx, tree, (const uint32_t *)dt, ld, (const uint32_t *)dw,
                                             n_sites, table, (uint32_t *)dn, (uint32_t *)dsc,
                                             (unsigned long long *)dtot, n_words ? &io : nullptr)));
  if (n_words && site_cost)
    PGPU_CUDA(ctx, cudaMemcpyAsync(site_cost, dsc, n_sites * 4, cudaMemcpyDeviceToHost, s));
  uint64_t *ht = reinterpret_cast<uint64_t *>(ctx->h_pinned);
  PGPU_CUDA(ctx, cudaMemcpyAsync(ht, dtot, 8, cudaMemcpyDeviceToHost, s));
  PGPU_CUDA(ctx, cudaStreamSynchronize(ctx->d2h_stream));
  PGPU_TRY(pgpu_check_flag(ctx, "tcm_tree"));
  *total = *ht;
  return PGPU_OK;
}

}  // extern "C"
