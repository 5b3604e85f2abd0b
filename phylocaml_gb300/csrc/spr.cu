// SPR rearrangement scoring on the GPU.
//
// phylocaml's tree search stops at the interface: Tree.break / Tree.join
// rearrange a topology (lib/tree.ml:299-494), the neighbourhood enumerators
// are TODOs (lib/treeNeighborhoods.ml:27-75) and the likelihood character is
// a stub (lib/likelihood_c.ml).  This file scores every SPR neighbour of a
// tree in one pass, exactly in the chosen arithmetic form, with the branch
// lengths of the move rule in spr_topo.cpp.
//
// Directed-edge pool (spr_pool_kernel, one pass per tree): for every
// directed edge d the conditional likelihood vector L[d] of the subtree on
// its side, M[d] = P(t) L[d] and H[d] = P(t/2) L[d], with per-pattern
// power-of-two scalers, for all patterns and rate classes, in HBM.  A
// thread owns one (pattern, rate class) and walks the pass order, so no
// thread reads a vector another thread wrote.  H is only read where moves
// are scored, so the pass writes it when that is what it was asked for, and
// spr_half_kernel adds it to a pool made without it (the branch-length
// rounds make several that nothing scores from).
//
// Scan (spr_scan_kernel, one CTA per prune x pattern-block group): removing
// the subtree on p's side of (p,u) changes only the vectors that look
// toward u.  The CTA walks the remaining tree outward from the joined edge
// (s,g), rebuilding each changed vector from its parent's message and the
// sibling's unchanged M, and at every edge (y,c) it scores the regraft:
//   site = sum_r probs_r sum_i pi_i [P(t_yc/2) L'[y|c]]_i H[c->y]_i M[p->u]_i
// The walk descends into the smaller side first and keeps the other
// message on a stack in shared memory, so the stack holds at most
// log2(n) + 1 entries.  Site log-likelihoods are weighted and summed as
// float pairs per warp, per CTA in warp order, then per move over the CTA
// groups in three floats (spr_reduce_kernel), which fixes the summation order.
//
// The Fitch part (spr_fitch_*_kernel) runs the same programs on state sets
// (32 patterns to a word, a word per state): the parsimony length of every neighbour, exactly.
//
// TBR moves that reroot both sides of a cut edge (a,b): the scan program of
// the prune carrying b's side away walks a's side, and in emit mode stores
// its vector at the middle of every edge it would regraft onto (a's side
// rerooted there); the reverse prune does the same for b's side.
// tbr_pair_kernel then scores every pair of attach edges of the cut as one
// dot product per pattern.
#include <algorithm>
#include <type_traits>
#include <cmath>
#include <cstring>

#include "forms.cuh"
#include "pmatrix.cuh"
#include "spr.cuh"

using namespace pgpu_forms;

namespace {

// Threads of a pool or scan CTA: the kernels hold 64 to 128 registers a thread,
// so that small CTAs fill an SM better and wait less for one another (256
// taxa x 45,675 patterns: pool 2.61 ms against 2.91 with 256 threads; the scan
// of 128 taxa x 16,852: 72.2 against 74.2 when it was chosen).
constexpr int SPR_NT = 128;
// What an engine accepts is reckoned in blocks of this many threads.
constexpr int SPR_LIMIT_NT = 256;
constexpr int SPR_NW = SPR_NT / 32;
constexpr int SPR_FEATURES = 64;

__host__ __device__ inline size_t a16(size_t x) { return (x + 15) & ~size_t(15); }

// ---------------------------------------------------------------------------
// rescaling shared by the pool and scan kernels: exact power of two, agreed
// by the RT lanes (rate classes) of one pattern; all lanes of the warp call
// ---------------------------------------------------------------------------
template <typename Pol>
__device__ __forceinline__ auto largest(const typename Pol::V *x) {
  return fmax(fmax(Pol::mag(x[0]), Pol::mag(x[1])), fmax(Pol::mag(x[2]), Pol::mag(x[3])));
}
template <typename Pol, int RT, typename T>
__device__ __forceinline__ void scale_up(typename Pol::V *acc, int &sc, T mx) {
#pragma unroll
  for (int o = 1; o < RT; o <<= 1) mx = fmax(mx, __shfl_xor_sync(0xffffffffu, mx, o));
  if (mx < Pol::thresh && mx > 0) {
    const int ex = frexp_exp(mx);
    sc += ex;
    const int k1 = min(-ex, 120), k2 = -ex - k1;
#pragma unroll
    for (int e = 0; e < 4; ++e) acc[e] = Pol::scale(acc[e], k1);
    if (k2 > 0) {
#pragma unroll
      for (int e = 0; e < 4; ++e) acc[e] = Pol::scale(acc[e], k2);
    }
  }
}
template <typename Pol, int RT>
__device__ __forceinline__ void rescale(typename Pol::V *acc, int &sc) {
  const auto mx = largest<Pol>(acc);
  if (__any_sync(0xffffffffu, mx < Pol::thresh && mx > 0)) scale_up<Pol, RT>(acc, sc, mx);
}
// two vectors, one vote
template <typename Pol, int RT>
__device__ __forceinline__ void rescale2(typename Pol::V *x, int &sx, typename Pol::V *y, int &sy) {
  const auto mx = largest<Pol>(x), my = largest<Pol>(y);
  if (__any_sync(0xffffffffu, (mx < Pol::thresh && mx > 0) || (my < Pol::thresh && my > 0))) {
    scale_up<Pol, RT>(x, sx, mx);
    scale_up<Pol, RT>(y, sy, my);
  }
}

__device__ __forceinline__ void copy16(void *dst, const void *src) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], 16;" ::"r"((uint32_t)__cvta_generic_to_shared(dst)), "l"(src)
               : "memory");
}

// A sum of floats and of products of floats to about 70 bits: three words, each
// the rounding errors of the one before.
struct Sum3 {
  float a = 0.0f, b = 0.0f, c = 0.0f;
  __device__ __forceinline__ void add_low(float x) {
    const ff t = two_sum(b, x);
    b = t.h;
    c = __fadd_rn(c, t.l);
  }
  __device__ __forceinline__ void add(float x) {
    const ff t = two_sum(a, x);
    a = t.h;
    add_low(t.l);
  }
  __device__ __forceinline__ void add_product(float x, float y) {
    const float p = __fmul_rn(x, y);
    add(p);
    add_low(__fmaf_rn(x, y, -p));
  }
  __device__ __forceinline__ double value() const { return (double)a + ((double)b + (double)c); }
};

struct PoolArgs {
  void *L, *M, *H;
  int32_t *sc;
  const void *Dfull, *Dhalf;   // [n_edges][R][16] coefficients
  const int4 *ops;
  const double *pi, *probs, *weights;
  double *site_lnl;
  double2 *partials;
  size_t np;                   // padded patterns
  size_t n_pat;
  int n_ops, R, NP;
};

// HBM-bound: two or three vectors written and up to two read per step.  The
// next step's vectors are read while this step is computed, unless this step
// makes them (then they pass in registers); depth-first order keeps what a
// step reads recent.  256 taxa x 45,675 patterns, pair form: 2.61 ms without
// H; level by level and with nothing read ahead it was 7.2 ms with H.
template <typename Pol, int RT, bool HALF>
__global__ void __launch_bounds__(SPR_NT) spr_pool_kernel(const PoolArgs a) {
  using V = typename Pol::V;
  using Coef = typename Pol::Coef;
  __shared__ double2 red[SPR_NW];
  const int c = threadIdx.x, pl = c / RT, r = c % RT, lane = c & 31;
  const size_t pat = (size_t)blockIdx.x * a.NP + pl;
  const bool on = r < a.R;
  const int R = a.R;
  auto vi = [&](int d) { return ((size_t)d * a.np + pat) * R + r; };
  V x[4], y[4], m[4];
  int sx = 0, sy = 0;
#pragma unroll
  for (int e = 0; e < 4; ++e) x[e] = y[e] = m[e] = Pol::zero();
  auto read = [&](int d, V *v, int &sv) {
    sv = a.sc[(size_t)d * a.np + pat];
    if (on) Pol::load_g(a.M, vi(d), v);
  };
  // a step's transition blocks come one step ahead into the warp's own shared
  // buffer, the 16-byte units of its classes interleaved
  constexpr int U = 16 * sizeof(Coef) / 16, UNITS = U * RT;
  __shared__ uint4 dsh[SPR_NW][2][HALF ? 2 : 1][UNITS];
  auto blocks = [&](int buf, int ed) {
#pragma unroll
    for (int k = 0; k < (UNITS + 31) / 32; ++k) {
      const int q = k * 32 + lane, cls = q / U;
      if (cls < R) {
        const uint4 *src = static_cast<const uint4 *>(a.Dfull) + (size_t)ed * R * U + q;
        copy16(&dsh[c >> 5][buf][0][(q % U) * RT + cls], src);
        if (HALF) copy16(&dsh[c >> 5][buf][HALF ? 1 : 0][(q % U) * RT + cls],
                         static_cast<const uint4 *>(a.Dhalf) + (size_t)ed * R * U + q);
      }
    }
    asm volatile("cp.async.commit_group;");
  };
  int4 op = a.n_ops > 0 ? __ldg(a.ops) : make_int4(0, 0, 0, 0);
  if (a.n_ops > 0) {
    blocks(0, op.x >> 1);
    read(op.y, x, sx);
    read(op.z, y, sy);
  }
  for (int i = 0; i < a.n_ops; ++i) {
    const int4 next = i + 1 < a.n_ops ? __ldg(a.ops + i + 1) : op;
    const bool more = i + 1 < a.n_ops;
    V acc[4];
    int s = sx + sy;
#pragma unroll
    for (int e = 0; e < 4; ++e) acc[e] = Pol::mul(x[e], y[e]);
    const bool from_x = next.y == op.x, from_y = next.z == op.x;
    if (more && !from_x) read(next.y, x, sx);
    if (more && !from_y) read(next.z, y, sy);
    rescale<Pol, RT>(acc, s);
    asm volatile("cp.async.wait_group 0;" ::: "memory");
    __syncwarp();   // this step's blocks are here, and all lanes are done with the step before's
    if (more) blocks((i + 1) & 1, next.x >> 1);
    const uint4(*dw)[UNITS] = dsh[c >> 5][i & 1];
    if (on) {
      Pol::rows(reinterpret_cast<const Coef *>(&dw[0][r]), acc, m, RT);
      Pol::store_g(a.L, vi(op.x), acc);
      Pol::store_g(a.M, vi(op.x), m);
      if (HALF) {
        V h[4];
        Pol::rows(reinterpret_cast<const Coef *>(&dw[HALF ? 1 : 0][r]), acc, h, RT);
        Pol::store_g(a.H, vi(op.x), h);
      }
    }
    if (r == 0) a.sc[(size_t)op.x * a.np + pat] = s;
    if (from_x) {
#pragma unroll
      for (int e = 0; e < 4; ++e) x[e] = m[e];
      sx = s;
    }
    if (from_y) {
#pragma unroll
      for (int e = 0; e < 4; ++e) y[e] = m[e];
      sy = s;
    }
    op = next;
    __syncwarp();   // the scalers of a pattern are written by its first lane
  }
  // log-likelihood across edge 0: L[side a] . P(t) L[side b]
  double part = 0.0;
  if (on) {
    V x[4], y[4];
    Pol::load_g(a.L, vi(0), x);
    Pol::load_g(a.M, vi(1), y);
    double lr = 0.0;
#pragma unroll
    for (int e = 0; e < 4; ++e) lr += a.pi[e] * Pol::to_d(Pol::mul(x[e], y[e]));
    part = a.probs[r] * lr;
  }
#pragma unroll
  for (int o = 1; o < RT; o <<= 1) part += __shfl_xor_sync(0xffffffffu, part, o);
  double sum = 0.0, comp = 0.0;
  if (r == 0 && pat < a.n_pat) {
    const int e2 = a.sc[pat] + a.sc[a.np + pat];
    const double lnl = log(part) + (double)e2 * 0.69314718055994530942;
    if (a.site_lnl) a.site_lnl[pat] = lnl;
    sum = a.weights[pat] * lnl;
  }
  warp_csum(sum, comp);
  if (lane == 0) red[c >> 5] = make_double2(sum, comp);
  __syncthreads();
  if (c < 32) {
    double2 v = lane < SPR_NW ? red[lane] : make_double2(0.0, 0.0);
    double ss = v.x, cc = v.y;
    warp_csum(ss, cc);
    if (lane == 0) a.partials[blockIdx.x] = make_double2(ss, cc);
  }
}

struct TipArgs {
  void *L, *M, *H;
  int32_t *sc;
  const void *tipfull, *tiphalf;   // [n_tips][R][n_codes][4] values of the form
  const void *code_rows;           // [n_codes] vectors of the form
  const uint8_t *codes;            // [n_tips][ld]
  const int4 *tips;                // {dedge, tip, edge, 0}
  int *flag;
  size_t np, n_pat, ld;
  int R, n_codes;
};

// A thread per (pattern, rate class), so that a warp's vectors are one run of
// memory.  LM: L, M and the scalers; HALF: H.  256 taxa x 45,675 patterns, L
// and M: 0.45 ms (6.7 TB/s) with the codes' vectors ready in the form, 1.32
// with their FP64 values converted in every thread.
template <typename Pol, bool LM, bool HALF>
__global__ void __launch_bounds__(256) spr_tip_kernel(const TipArgs a) {
  using V = typename Pol::V;
  const unsigned i = blockIdx.x * 256 + threadIdx.x;   // np R < 2^32: three such arrays per edge fit in memory
  if (i >= a.np * a.R) return;
  const unsigned pat = i / (unsigned)a.R;
  const int r = (int)(i - pat * (unsigned)a.R);
  const int4 t = a.tips[blockIdx.y];
  int code = pat < a.n_pat ? a.codes[(size_t)t.y * a.ld + pat] : 0;
  if (code >= a.n_codes) {
    atomicOr(a.flag, PGPU_FLAG_BADCODE);
    code = 0;
  }
  const size_t at = (size_t)t.x * a.np * a.R + i;
  const size_t tt = ((size_t)t.y * a.R + r) * a.n_codes + code;
  V v[4];
  if (LM) {
    Pol::load_g(a.code_rows, code, v);
    Pol::store_g(a.L, at, v);
    Pol::load_g(a.tipfull, tt, v);
    Pol::store_g(a.M, at, v);
    if (r == 0) a.sc[(size_t)t.x * a.np + pat] = 0;
  }
  if (HALF) {
    Pol::load_g(a.tiphalf, tt, v);
    Pol::store_g(a.H, at, v);
  }
}

// H of every internal directed edge of a pool made without it.
template <typename Pol>
__global__ void __launch_bounds__(256) spr_half_kernel(const void *L, void *H, const void *Dhalf, const int4 *ops,
                                                       size_t np, unsigned R) {
  using V = typename Pol::V;
  using Coef = typename Pol::Coef;
  const unsigned i = blockIdx.x * 256 + threadIdx.x;
  if (i >= np * R) return;
  const int d = __ldg(ops + blockIdx.y).x;
  const int r = (int)(i % R);
  V x[4], h[4];
  Pol::load_g(L, (size_t)d * np * R + i, x);
  Pol::rows(static_cast<const Coef *>(Dhalf) + ((size_t)(d >> 1) * R + r) * 16, x, h);
  Pol::store_g(H, (size_t)d * np * R + i, h);
}

__global__ void __launch_bounds__(1024) spr_pool_finalize_kernel(const double2 *partials, int n,
                                                                double *out) {
  const double v = csum_block<1024>(partials, n);
  if (threadIdx.x == 0) out[0] = v;
}

// ---------------------------------------------------------------------------
// scan
// ---------------------------------------------------------------------------
struct ScanArgs {
  const void *L, *M, *H;
  const int32_t *sc;
  const void *Dhalf, *Dmer;   // [n_edges][R][16], [n_prunes][R][16]
  const SprStep *steps;
  const SprPrune *prunes;
  const double *pi, *probs;
  const float2 *pairs;        // pi [4] and probs [8] as float pairs
  const float2 *wts;          // [np] float pairs, zero beyond n_pat
  const float4 *logtab;       // 64 entries
  float2 *partials;           // [n_groups][n_moves] float pairs
  int *flag;
  size_t np, n_moves;
  int R, NP, G, n_blocks, depth;
  // emit mode (TBR): the attach vector of every wanted edge instead of a score
  const void *Dfull;          // [n_edges][R][16]: P(t) of the cut edge (b's side)
  void *xout;                 // [slot][np][R] x 4
  int32_t *xsc;               // [slot][np]
  long long slot_base;        // move index of slot 0
  int prune_base;             // first prune of the launch
};

// Shared memory of a scan CTA: the logarithm table, a window of SCAN_WIN moves'
// values per warp, the two steps' transition blocks per warp and the stack.
constexpr int SCAN_WIN = 64;
template <typename Pol>
__host__ __device__ constexpr size_t scan_blocks(int RT) {   // of one step, bytes
  return 2 * (size_t)RT * 16 * sizeof(typename Pol::Coef);
}
template <typename Pol>
__host__ __device__ size_t scan_smem(int depth, int RT) {
  return 1024 + (size_t)SPR_NW * SCAN_WIN * sizeof(ff) + 2 * SPR_NW * scan_blocks<Pol>(RT) +
         (size_t)depth * 4 * SPR_NT * sizeof(typename Pol::V) + (size_t)depth * SPR_NT * sizeof(int);
}
// What a scan may ask for: room for every move of a prune at once beside the
// stack, and for the kernel's own memory.
template <typename Pol>
size_t scan_limit(int depth, int max_moves, int RT) {
  const size_t moves = a16((size_t)(SPR_LIMIT_NT / 32) * max_moves * sizeof(ff));
  return std::max(scan_smem<Pol>(depth, RT),
                  1024 + moves + (size_t)depth * SPR_LIMIT_NT * (4 * sizeof(typename Pol::V) + sizeof(int)));
}

// One lane's part of a regraft's site likelihood: sum_e h_e hh_e v_e, v the
// pruned side's vector with the frequencies and (pair form) the class's
// probability in it.
template <typename Pol>
__device__ __forceinline__ typename Pol::V site_part(const typename Pol::V *h, const typename Pol::V *hh,
                                                     const typename Pol::V *v, typename Pol::V prob) {
  using V = typename Pol::V;
  if constexpr (std::is_same<Pol, Ff32>::value) {
    // exact products two to an instruction, then exact sums of the terms
    // (none is negative), the low words left unnormalised until the end
    ff t[4], u[4];
    Pol::mul4(h, hh, t);
    Pol::mul4(t, v, u);
    const float2 a = make_float2(fmaxf(u[0].h, u[2].h), fmaxf(u[1].h, u[3].h));
    const float2 b = make_float2(fminf(u[0].h, u[2].h), fminf(u[1].h, u[3].h));
    const float2 s = __fadd2_rn(a, b);
    const float2 e = __fadd2_rn(b, neg2(__fadd2_rn(s, neg2(a))));
    const float2 lo = __fadd2_rn(__fadd2_rn(make_float2(u[0].l, u[1].l), make_float2(u[2].l, u[3].l)), e);
    const ff w = fast_two_sum(fmaxf(s.x, s.y), fminf(s.x, s.y));
    return fast_two_sum(w.h, __fadd_rn(w.l, __fadd_rn(lo.x, lo.y)));
  } else {
    V p = Pol::zero();
#pragma unroll
    for (int e = 0; e < 4; ++e) p = Pol::add(p, Pol::mul(Pol::mul(h[e], hh[e]), v[e]));
    return Pol::mul(p, prob);
  }
}

// EMIT: instead of scoring a regraft, store the walked side's vector at the
// middle of the edge, [P(t_yc/2) L'[y|c]] (.) H[c->y], with its scaler: the
// side rerooted there, for TBR.  Emit prunes come in pairs per cut edge
// (a,b): the even one walks a's side and stores X weighted by probs_r pi_i,
// the odd one walks b's side and stores P(t_ab) Y, carried across the cut,
// so that a TBR site likelihood is the plain dot product of the two.
//
// Bound by issuing pair arithmetic; with 128 registers a thread 16 warps run
// on an SM, too few to wait for memory, so a step's M vectors (to
// registers) and transition blocks (to shared memory, classes interleaved) are
// read one step ahead and its H vectors at its start.  The lanes of a pattern
// split the two moves of a step: one exchange leaves the even lanes with the
// first move's sum and the odd ones with the second's, and one logarithm and
// one sum over the patterns serve both.  The warps' values meet every
// SCAN_WIN moves.  128 taxa x 16,852 patterns, pair form, 63,000 moves:
// 72.3 ms against 141.8 with none of this.
template <typename Pol, int RT, bool EMIT = false>
__global__ void __launch_bounds__(SPR_NT, 4) spr_scan_kernel(const ScanArgs a) {
  using V = typename Pol::V;
  using Coef = typename Pol::Coef;
  constexpr int NT = SPR_NT, U = sizeof(Coef), UNITS = U * RT;   // 16-byte units of a class's block, of an edge's
  extern __shared__ __align__(16) unsigned char smem[];
  const SprPrune pr = a.prunes[a.prune_base + blockIdx.x];
  const int c = threadIdx.x, lane = c & 31, warp = c >> 5, pl = c / RT, r = c % RT;
  float4 *ltab = reinterpret_cast<float4 *>(smem);
  ff *red = reinterpret_cast<ff *>(smem + 1024);   // [warp][SCAN_WIN]
  uint4 *dsh = reinterpret_cast<uint4 *>(red + SPR_NW * SCAN_WIN) + (size_t)warp * 4 * UNITS;   // [2][2 edges][UNITS]
  V *stk = reinterpret_cast<V *>(smem + 1024 + SPR_NW * SCAN_WIN * sizeof(ff) + 2 * SPR_NW * scan_blocks<Pol>(RT));
  int *stk_sc = reinterpret_cast<int *>(stk + (size_t)a.depth * 4 * NT);
  const bool on = r < a.R;
  const int R = a.R;
  for (int i = c; i < 64; i += NT) ltab[i] = a.logtab[i];
  __syncthreads();
  // the pair form takes these ready: converting them from FP64 in every thread
  // cost 0.4 ms of the 63,000 moves' 72
  auto constant = [&](int k, const double *d) {
    if constexpr (std::is_same<Pol, Ff32>::value) {
      const float2 v = __ldg(a.pairs + k);
      return ff{v.x, v.y};
    } else {
      return Pol::from_d(*d);
    }
  };
  const V prob = on ? constant(4 + r, a.probs + r) : Pol::zero();
  const Coef *Dm = static_cast<const Coef *>(a.Dmer) + ((size_t)(a.prune_base + blockIdx.x) * R + (on ? r : 0)) * 16;
  // blocks of a step's two edges into buffer buf
  auto blocks = [&](int buf, const SprStep &st) {
#pragma unroll
    for (int k = 0; k < (UNITS + 31) / 32; ++k) {
      const int q = k * 32 + lane, cls = q / U;
      if (cls < R) {
        const uint4 *D = static_cast<const uint4 *>(a.Dhalf) + q;
        uint4 *dst = dsh + (size_t)buf * 2 * UNITS + (q % U) * RT + cls;
        copy16(dst, D + (size_t)(st.d1 >> 1) * R * U);
        copy16(dst + UNITS, D + (size_t)(st.d2 >> 1) * R * U);
      }
    }
    asm volatile("cp.async.commit_group;");
  };
  int base = 0;   // first move of the window
  auto flush = [&](int to, bool first) {
    __syncthreads();
    if (c < to - base) {
      auto warp_sum = [&](int w) {
        const ff v = red[w * SCAN_WIN + c];
        return fast_two_sum(v.h, v.l);
      };
      ff s = warp_sum(0);
      for (int w = 1; w < SPR_NW; ++w) s = ff_add(s, warp_sum(w));
      float2 *dst = a.partials + (size_t)blockIdx.y * a.n_moves + pr.move_off + base + c;
      if (!first) s = ff_add(ff{dst->x, dst->y}, s);
      *dst = make_float2(s.h, s.l);
    }
    __syncthreads();
    base = to;
  };
  bool ok = true;

  for (int g = 0; g < a.G && ok; ++g) {
    const int blk = blockIdx.y * a.G + g;
    if (blk >= a.n_blocks) break;
    const size_t pat = (size_t)blk * a.NP + pl;
    // vector of directed edge d, its scaler: one widening product each (the
    // strides fit in 32 bits, as three arrays of 6 edges or more fit in memory)
    const size_t own_vec = pat * R + r;
    const unsigned vec_step = (unsigned)(a.np * R), sc_step = (unsigned)a.np;
    auto vi = [&](int d) { return (unsigned long long)(unsigned)d * vec_step + own_vec; };
    auto scv = [&](int d) { return a.sc[(unsigned long long)(unsigned)d * sc_step + pat]; };
    const float2 wpat = a.wts[pat];
    const ff w{wpat.x, wpat.y};
    V vp[4];
#pragma unroll
    for (int e = 0; e < 4; ++e) vp[e] = Pol::zero();
    const int scp = EMIT ? 0 : scv(pr.dp);
    if (on && !EMIT) {
      Pol::load_g(a.M, vi(pr.dp), vp);
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        vp[e] = Pol::mul(vp[e], constant(e, a.pi + e));
        if constexpr (std::is_same<Pol, Ff32>::value) {
          // normalised after each product: a site's value is then off by 0.88
          // and 1.13 x 2^-48 (rms, values spread evenly and over decades),
          // against 0.96 and 1.18 with the probability multiplied in last and
          // 1.14 and 1.47 with the low words left as they come
          vp[e] = Pol::mul(fast_two_sum(vp[e].h, vp[e].l), prob);
          vp[e] = fast_two_sum(vp[e].h, vp[e].l);
        }
      }
    }
    V in[4];
    int in_sc = 0, sp = 0;
    bool have = false;
    auto push = [&](const V *x, int s) {
      if (sp >= a.depth) {
        ok = false;
        return;
      }
#pragma unroll
      for (int e = 0; e < 4; ++e) stk[((size_t)sp * 4 + e) * NT + c] = x[e];
      stk_sc[sp * NT + c] = s;
      ++sp;
    };
    const SprStep *prog = a.steps + pr.step_off;
    SprStep st = prog[0];
    {
      V ms[4], mg[4];
      if (on) {
        V ls[4], lg[4];
        Pol::load_g(a.L, vi(st.d1), ls);
        Pol::load_g(a.L, vi(st.d2), lg);
        Pol::rows(Dm, lg, ms);   // into s, from g's side across the joined edge
        Pol::rows(Dm, ls, mg);
      } else {
#pragma unroll
        for (int e = 0; e < 4; ++e) ms[e] = mg[e] = Pol::zero();
      }
      const int scs = scv(st.d2), scg = scv(st.d1);
      const bool ds = st.flags & SPR_DOWN1, dg = st.flags & SPR_DOWN2;
      const bool g_first = ds && dg && (st.flags & SPR_FIRST2);
      if (ds && dg) push(g_first ? ms : mg, g_first ? scs : scg);
      const bool take_g = g_first || !ds;
#pragma unroll
      for (int e = 0; e < 4; ++e) in[e] = take_g ? mg[e] : ms[e];
      in_sc = take_g ? scg : scs;
      have = true;
    }
    if (!(st.flags & SPR_START)) ok = false;
    V m1[4], m2[4];
    int s1 = 0, s2 = 0;
#pragma unroll
    for (int e = 0; e < 4; ++e) m1[e] = m2[e] = Pol::zero();
    auto fetch = [&](const SprStep &x) {
      s1 = scv(x.d1);
      s2 = scv(x.d2);
      if (on) {
        Pol::load_g(a.M, vi(x.d1), m1);
        Pol::load_g(a.M, vi(x.d2), m2);
      }
    };
    if (pr.n_steps > 1) {
      st = prog[1];
      __syncwarp();
      blocks(1, st);
      fetch(st);
    }
    for (int si = 1; si < pr.n_steps && ok; ++si) {
      const bool more = si + 1 < pr.n_steps, scored = st.out1 >= 0 || st.out2 >= 0;
      const SprStep nx = more ? prog[si + 1] : st;
      V hh1[4], hh2[4];
      if (!EMIT && on && st.out1 >= 0) Pol::load_g(a.H, vi(st.d1), hh1);
      if (!EMIT && on && st.out2 >= 0) Pol::load_g(a.H, vi(st.d2), hh2);
      if (!have) {
        if (sp == 0) {
          ok = false;
          break;
        }
        --sp;
#pragma unroll
        for (int e = 0; e < 4; ++e) in[e] = stk[((size_t)sp * 4 + e) * NT + c];
        in_sc = stk_sc[sp * NT + c];
      }
      V l1[4], l2[4];
      int sc1 = in_sc + s2, sc2 = in_sc + s1;
      const int at1 = s1, at2 = s2;
      Pol::mul4(in, m2, l1);
      Pol::mul4(in, m1, l2);
      if (more) fetch(nx);
      rescale2<Pol, RT>(l1, sc1, l2, sc2);
      asm volatile("cp.async.wait_group 0;" ::: "memory");
      __syncwarp();   // this step's blocks are here, and all lanes are done with the step before's
      if (more) blocks((si + 1) & 1, nx);
      const Coef *D1 = reinterpret_cast<const Coef *>(dsh + (size_t)(si & 1) * 2 * UNITS + (on ? r : 0));
      const Coef *D2 = reinterpret_cast<const Coef *>(dsh + (size_t)(si & 1) * 2 * UNITS + UNITS + (on ? r : 0));
      V h1[4], h2[4];
      Pol::rows(D1, l1, h1, RT);
      Pol::rows(D2, l2, h2, RT);
      if (EMIT && scored) {
        if (on) {
          const bool side_b = ((a.prune_base + blockIdx.x) & 1) != 0;
          V x[4], y[4];
#pragma unroll
          for (int h = 0; h < 2; ++h) {
            const int out = h == 0 ? st.out1 : st.out2;
            if (out < 0) continue;
            Pol::load_g(a.H, vi(h == 0 ? st.d1 : st.d2), hh1);
#pragma unroll
            for (int e = 0; e < 4; ++e) x[e] = Pol::mul(h == 0 ? h1[e] : h2[e], hh1[e]);
            if (side_b) {
              Pol::rows(static_cast<const Coef *>(a.Dfull) + ((size_t)(pr.dp >> 1) * R + r) * 16, x, y);
            } else {
#pragma unroll
              for (int e = 0; e < 4; ++e) y[e] = Pol::mul(x[e], Pol::from_d(a.probs[r] * a.pi[e]));
            }
            const size_t slot = (size_t)(out - a.slot_base);
            Pol::store_g(a.xout, (slot * a.np + pat) * R + r, y);
            if (r == 0) a.xsc[slot * a.np + pat] = h == 0 ? sc1 + at1 : sc2 + at2;
          }
        }
      } else if (scored) {
        V p1 = Pol::zero(), p2 = Pol::zero();
        if (on && st.out1 >= 0) p1 = site_part<Pol>(h1, hh1, vp, prob);
        if (on && st.out2 >= 0) p2 = site_part<Pol>(h2, hh2, vp, prob);
        const int o1 = st.out1 - pr.move_off, o2 = st.out2 - pr.move_off;
        const int last = st.out2 >= 0 ? o2 : o1;
        if (last - base >= SCAN_WIN) flush(st.out1 >= 0 ? o1 : o2, g == 0);
        ff *own = red + warp * SCAN_WIN - base;
        auto weighed = [&](V p, int e2, bool wanted) {
          ff v{0.0f, 0.0f};
          if (wanted && w.h != 0.0f) {
            if (Pol::positive(p)) v = ff_mul(Pol::site_log(p, e2, ltab), w);
            else atomicOr(a.flag, PGPU_FLAG_NAN);
          }
          return v;
        };
        // pair additions, the last one normalised where it is read (flush)
        auto over_patterns = [&](ff v) {
#pragma unroll
          for (int o = RT; o < 32; o <<= 1) {
            const ff x = ff_shfl_xor(v, o), t = two_sum(v.h, x.h);
            v = {t.h, __fadd_rn(t.l, __fadd_rn(v.l, x.l))};
            if (o < 16) v = fast_two_sum(v.h, v.l);
          }
          return v;
        };
        if constexpr (RT == 1) {
          const ff v1 = over_patterns(weighed(p1, sc1 + at1 + scp, st.out1 >= 0));
          const ff v2 = over_patterns(weighed(p2, sc2 + at2 + scp, st.out2 >= 0));
          if (lane == 0 && st.out1 >= 0) own[o1] = v1;
          if (lane == 0 && st.out2 >= 0) own[o2] = v2;
        } else {
          const bool odd = r & 1;
          V p = Pol::add(odd ? p2 : p1, Pol::shfl_xor(odd ? p1 : p2, 1));
#pragma unroll
          for (int o = 2; o < RT; o <<= 1) p = Pol::add(p, Pol::shfl_xor(p, o));
          const bool wanted = odd ? st.out2 >= 0 : st.out1 >= 0;
          const ff v = over_patterns(weighed(p, (odd ? sc2 + at2 : sc1 + at1) + scp, wanted));
          if (lane < 2 && wanted) own[odd ? o2 : o1] = v;
        }
      }
      const bool dn1 = st.flags & SPR_DOWN1, dn2 = st.flags & SPR_DOWN2;
      if (dn1 || dn2) {
        V n1[4], n2[4];
        if (dn1) Pol::rows(D1, h1, n1, RT);   // P(t/2) P(t/2) L = P(t) L
        if (dn2) Pol::rows(D2, h2, n2, RT);
        const bool second_first = dn1 && dn2 && (st.flags & SPR_FIRST2);
        if (dn1 && dn2) push(second_first ? n1 : n2, second_first ? sc1 : sc2);
        const bool take2 = second_first || !dn1;
#pragma unroll
        for (int e = 0; e < 4; ++e) in[e] = take2 ? n2[e] : n1[e];
        in_sc = take2 ? sc2 : sc1;
        have = true;
      } else {
        have = false;
      }
      st = nx;
    }
    if (!EMIT) {
      flush(pr.n_moves, g == 0);
      base = 0;
    }
  }
  if (!ok && c == 0) atomicOr(a.flag, PGPU_FLAG_EIGEN);   // program and stack disagree
}

// lnl[m] = sum over CTA groups of the partial sums: slice y of a move's groups
// by thread (move, y), the slices in order.  A chain over all the groups kept
// a few moves of 714 groups waiting 210 us; 56 us in 32 slices.  Sums in three
// floats: in FP64 the 33 million partials of 63,000 moves took 0.48 ms, 0.055
// now.
constexpr int RED_Y = 32;
__global__ void __launch_bounds__(32 * RED_Y) spr_reduce_kernel(const float2 *partials, int n_groups, size_t n_moves,
                                                                double *lnl) {
  __shared__ float part[3][RED_Y][33];
  const int x = threadIdx.x, y = threadIdx.y;
  const size_t m = (size_t)blockIdx.x * 32 + x;
  const int per = (n_groups + RED_Y - 1) / RED_Y, g0 = y * per, g1 = min(g0 + per, n_groups);
  Sum3 s;
  if (m < n_moves)
    for (int g = g0; g < g1; ++g) {
      const float2 v = partials[(size_t)g * n_moves + m];
      s.add(v.x);
      s.add_low(v.y);
    }
  part[0][y][x] = s.a;
  part[1][y][x] = s.b;
  part[2][y][x] = s.c;
  __syncthreads();
  if (y != 0 || m >= n_moves) return;
  for (int k = 1; k < RED_Y; ++k) {
    s.add(part[0][k][x]);
    s.add_low(part[1][k][x]);
    s.c = __fadd_rn(s.c, part[2][k][x]);
  }
  lnl[m] = s.value();
}

// ---------------------------------------------------------------------------
// TBR pairs.  For a cut edge (a,b) with the attach vectors of both sides
// from the emit walks (a's side weighted, b's side carried across the cut),
//   site(j, k) = sum_r sum_i X_j[r][i] Z_k[r][i]
//              = sum_r probs_r sum_i pi_i X_j[r][i] [P(t_ab) Y_k][r][i],
// with the two scalers added.  A CTA takes 16 x 16 (j, k) pairs, one per
// thread, over a group of pattern blocks; per block of TB_PB patterns the
// X_j and Z_k are staged in shared memory, rows padded by one element so
// that the 16 Z rows a warp reads fall in distinct banks.
// ---------------------------------------------------------------------------
constexpr int TB_T = 16;
constexpr int TB_PB = 16;

struct TbrCutDev {
  int edge, nA, nB, pad;
  long long slotA, slotB;   // first emit slot of each side
  long long move_off;       // first move of the cut within the launch's range
};

struct PairArgs {
  const void *X;            // [slot][np][R] x 4
  const int32_t *xsc;       // [slot][np]
  const int4 *tiles;        // {cut, j0, k0, 0}
  const TbrCutDev *cuts;
  const float2 *wts;        // [np] float pairs, zero beyond n_pat
  const float4 *logtab;
  float2 *partials;         // [n_groups][n_moves] float pairs
  int *flag;
  size_t np;
  long long n_moves;
  int R, G, n_pblocks;
};

__host__ __device__ inline int tbr_row(int R) { return TB_PB * R * 4 + 1; }

template <typename Pol>
__host__ __device__ size_t pair_smem(int R) {
  return 1024 + 2 * (size_t)TB_T * tbr_row(R) * sizeof(typename Pol::V) + 2 * TB_T * TB_PB * sizeof(int);
}

// sum_q x_q z_q of one site.  In the float-pair form the terms are
// non-negative, so they are summed as the pruning rows sum: exact products
// (TwoProduct and the two cross terms), the high parts added exactly by a
// Fast2Sum of the larger and the smaller, everything else gathered in one
// float; the pair is normalised once at the end.  About 11 instructions a
// term against 15 for a pair add per term.
template <typename Pol>
__device__ __forceinline__ typename Pol::V pair_dot(const typename Pol::V *x, const typename Pol::V *z, int n) {
  if constexpr (std::is_same<Pol, Ff32>::value) {
    float sh = __fmul_rn(x[0].h, z[0].h);
    float lo = __fmaf_rn(x[0].h, z[0].h, -sh);
    lo = __fmaf_rn(x[0].h, z[0].l, lo);
    lo = __fmaf_rn(x[0].l, z[0].h, lo);
    for (int q = 1; q < n; ++q) {
      const float p = __fmul_rn(x[q].h, z[q].h);
      float e = __fmaf_rn(x[q].h, z[q].h, -p);
      e = __fmaf_rn(x[q].h, z[q].l, e);
      e = __fmaf_rn(x[q].l, z[q].h, e);
      const ff t = fast_two_sum(fmaxf(sh, p), fminf(sh, p));
      sh = t.h;
      lo = __fadd_rn(lo, __fadd_rn(t.l, e));
    }
    return fast_two_sum(sh, lo);
  } else {
    typename Pol::V acc = Pol::zero();
    for (int q = 0; q < n; ++q) acc = Pol::add(acc, Pol::mul(x[q], z[q]));
    return acc;
  }
}

template <typename Pol>
__global__ void __launch_bounds__(256) tbr_pair_kernel(const PairArgs a) {
  using V = typename Pol::V;
  extern __shared__ __align__(16) unsigned char smem[];
  const int R = a.R, RS = tbr_row(R);
  float4 *ltab = reinterpret_cast<float4 *>(smem);
  V *Xs = reinterpret_cast<V *>(smem + 1024);
  V *Zs = Xs + (size_t)TB_T * RS;
  int *xs = reinterpret_cast<int *>(Zs + (size_t)TB_T * RS);
  int *ys = xs + TB_T * TB_PB;
  const int t = threadIdx.x;
  for (int i = t; i < 64; i += 256) ltab[i] = a.logtab[i];
  const int4 tl = a.tiles[blockIdx.x];
  const TbrCutDev cut = a.cuts[tl.x];
  const int jj = t / TB_T, kk = t % TB_T;
  const int j = tl.y + jj, k = tl.z + kk;
  const bool mine = j < cut.nA && k < cut.nB;
  const int per_side = TB_T * TB_PB * R;
  ff sum{0.0f, 0.0f};
  for (int g = 0; g < a.G; ++g) {
    const int blk = blockIdx.y * a.G + g;
    if (blk >= a.n_pblocks) break;
    const size_t pat0 = (size_t)blk * TB_PB;
    __syncthreads();   // the previous block's tiles are consumed
    for (int it = t; it < 2 * per_side; it += 256) {
      const int side = it / per_side, rem = it % per_side;
      const int row = rem / (TB_PB * R), p = (rem / R) % TB_PB, r = rem % R;
      const int idx = (side == 0 ? tl.y : tl.z) + row;
      const size_t pat = pat0 + p;
      V v[4];
      int sc = 0;
      if (idx < (side == 0 ? cut.nA : cut.nB)) {
        const size_t slot = (size_t)((side == 0 ? cut.slotA : cut.slotB) + idx);
        Pol::load_g(a.X, (slot * a.np + pat) * R + r, v);
        sc = a.xsc[slot * a.np + pat];
      } else {
#pragma unroll
        for (int e = 0; e < 4; ++e) v[e] = Pol::zero();
      }
      V *dst = (side == 0 ? Xs : Zs) + (size_t)row * RS + ((size_t)p * R + r) * 4;
#pragma unroll
      for (int e = 0; e < 4; ++e) dst[e] = v[e];
      if (r == 0) (side == 0 ? xs : ys)[row * TB_PB + p] = sc;
    }
    __syncthreads();
    if (!mine) continue;
    for (int p = 0; p < TB_PB; ++p) {
      const float2 w = a.wts[pat0 + p];
      if (w.x == 0.0f) continue;
      const V *xr = Xs + (size_t)jj * RS + (size_t)p * R * 4;
      const V *zr = Zs + (size_t)kk * RS + (size_t)p * R * 4;
      const V acc = pair_dot<Pol>(xr, zr, R * 4);
      if (Pol::positive(acc))
        sum = ff_add(sum, ff_mul(Pol::site_log(acc, xs[jj * TB_PB + p] + ys[kk * TB_PB + p], ltab),
                                 ff{w.x, w.y}));
      else
        atomicOr(a.flag, PGPU_FLAG_NAN);
    }
  }
  if (mine)
    a.partials[(size_t)blockIdx.y * a.n_moves + cut.move_off + (long long)j * cut.nB + k] =
        make_float2(sum.h, sum.l);
}

// ---------------------------------------------------------------------------
// Fitch sets on the directed edges and the parsimony length of every move
// ---------------------------------------------------------------------------
// The state sets of 32 patterns are four words, one per state (bit j: pattern
// 32 q + j holds the state), so that a Fitch step is eight three-input logic
// operations on 32 patterns and the empty joins are one word: 28 operations
// with the four states of a pattern side by side in nibbles.
//   empty = no state in both; set = (a & b) or, where empty, a | b
__device__ __forceinline__ uint32_t meet(uint4 a, uint4 b) {
  return (a.x & b.x) | (a.y & b.y) | (a.z & b.z) | (a.w & b.w);
}
__device__ __forceinline__ uint4 fitch4(uint4 a, uint4 b, uint32_t *empty) {
  const uint32_t none = ~meet(a, b);
  *empty = none;
  return make_uint4((a.x & b.x) | ((a.x | b.x) & none), (a.y & b.y) | ((a.y | b.y) & none),
                    (a.z & b.z) | ((a.z | b.z) & none), (a.w & b.w) | ((a.w | b.w) & none));
}
// weighted count of the patterns flagged in a word, the weights as bit planes;
// a thread reads the low planes of its patterns once
constexpr int WPLANES = 8;
struct WeightPlanes {
  const uint32_t *p;
  size_t stride;
  int n;
  uint32_t low[WPLANES];
  __device__ void load(const uint32_t *planes, size_t w4, int n_planes, size_t at, bool in) {
    p = planes + at;
    stride = w4;
    n = in ? n_planes : 0;
#pragma unroll
    for (int b = 0; b < WPLANES; ++b) low[b] = b < n ? p[b * stride] : 0u;
  }
  __device__ uint32_t count(uint32_t f) const {
    uint32_t s = 0;
#pragma unroll
    for (int b = 0; b < WPLANES; ++b)
      if (b < n) s += (uint32_t)__popc(f & low[b]) << b;
    for (int b = WPLANES; b < n; ++b) s += (uint32_t)__popc(f & p[b * stride]) << b;
    return s;
  }
};

struct FitchTipArgs {
  uint4 *F;
  const uint8_t *codes;
  const uint8_t *code_mask;   // [n_codes] state-set bits
  const int4 *tips;
  size_t W4, n_pat, ld;
  int n_codes;
};

__global__ void __launch_bounds__(256) spr_fitch_tip_kernel(const FitchTipArgs a) {
  const size_t pat = (size_t)blockIdx.x * 256 + threadIdx.x;
  const int4 t = a.tips[blockIdx.y];
  uint32_t m = 0;
  if (pat < a.n_pat) {
    const int code = a.codes[(size_t)t.y * a.ld + pat];
    m = code < a.n_codes ? a.code_mask[code] : 0xFu;
  }
  uint4 w;
  w.x = __ballot_sync(0xffffffffu, m & 1u);
  w.y = __ballot_sync(0xffffffffu, m & 2u);
  w.z = __ballot_sync(0xffffffffu, m & 4u);
  w.w = __ballot_sync(0xffffffffu, m & 8u);
  if ((threadIdx.x & 31) == 0 && (pat >> 5) < a.W4) a.F[(size_t)t.x * a.W4 + (pat >> 5)] = w;
}

struct FitchPoolArgs {
  uint4 *F;
  const int4 *ops;
  const uint32_t *planes;   // [n_planes][W4]
  unsigned long long *cnt;   // [n_ops + 1]: local cost of each op, then edge 0's join
  size_t W4;
  int n_ops, n_planes;
};

// Bound by the chain of steps: a thread owns 32 patterns of every directed
// edge, so a small alignment has few warps.  The next step's sets are read
// while this one is computed and each warp adds its own count, with no barrier
// in the chain; CTAs of two warps spread over the SMs.  762 steps x 45,675
// patterns: 0.29 ms against 0.85 with 256-thread CTAs adding up each step.
constexpr int FPOOL_NT = 64;
__global__ void __launch_bounds__(FPOOL_NT) spr_fitch_pool_kernel(const FitchPoolArgs a) {
  const size_t q = (size_t)blockIdx.x * FPOOL_NT + threadIdx.x;
  const bool in = q < a.W4;
  WeightPlanes wp;
  wp.load(a.planes, a.W4, a.n_planes, in ? q : 0, in);
  auto get = [&](int d) { return in ? a.F[(size_t)d * a.W4 + q] : make_uint4(0, 0, 0, 0); };
  auto add = [&](uint32_t e, unsigned long long *dst) {
    const uint32_t v = __reduce_add_sync(0xffffffffu, wp.count(e));
    if ((threadIdx.x & 31) == 0 && v) atomicAdd(dst, (unsigned long long)v);
  };
  uint4 x = make_uint4(0, 0, 0, 0), y = x;
  int4 op = a.n_ops > 0 ? __ldg(a.ops) : make_int4(0, 0, 0, 0);
  if (a.n_ops > 0) {
    x = get(op.y);
    y = get(op.z);
  }
  for (int i = 0; i < a.n_ops; ++i) {
    const bool more = i + 1 < a.n_ops;
    const int4 next = more ? __ldg(a.ops + i + 1) : op;
    uint32_t e;
    const uint4 o = fitch4(x, y, &e);
    if (in) a.F[(size_t)op.x * a.W4 + q] = o;
    if (more) {
      x = next.y == op.x ? o : get(next.y);
      y = next.z == op.x ? o : get(next.z);
    }
    add(e, a.cnt + i);
    op = next;
  }
  uint32_t e;
  (void)fitch4(get(0), get(1), &e);
  add(e, a.cnt + a.n_ops);
}

// lenF[d]: parsimony length of the subtree on d's side; lenF[nd] = tree
// length.  One thread adds along the steps; the others bring the steps and
// hold the lengths in shared memory while the tree has room there (a step
// took 160 ns from global memory).
constexpr int FLEN_NT = 256;
__global__ void __launch_bounds__(FLEN_NT) spr_fitch_len_kernel(const int4 *ops, int n_ops,
                                                                const unsigned long long *cnt,
                                                                unsigned long long *lenF, int nd, int in_shared) {
  extern __shared__ unsigned long long len_sh[];
  __shared__ int4 op_sh[FLEN_NT];
  __shared__ unsigned long long cnt_sh[FLEN_NT];
  unsigned long long *len = in_shared ? len_sh : lenF;
  // tips (and everything) start at 0; ops fill in dependency order
  for (int d = threadIdx.x; d < nd; d += FLEN_NT) len[d] = 0;
  for (int i0 = 0; i0 < n_ops; i0 += FLEN_NT) {
    const int k = min(FLEN_NT, n_ops - i0);
    __syncthreads();
    if ((int)threadIdx.x < k) {
      op_sh[threadIdx.x] = ops[i0 + threadIdx.x];
      cnt_sh[threadIdx.x] = cnt[i0 + threadIdx.x];
    }
    __syncthreads();
    if (threadIdx.x == 0)
      for (int i = 0; i < k; ++i) {
        const int4 op = op_sh[i];
        len[op.x] = len[op.y] + len[op.z] + cnt_sh[i];
      }
  }
  __syncthreads();
  if (in_shared)
    for (int d = threadIdx.x; d < nd; d += FLEN_NT) lenF[d] = len_sh[d];
  if (threadIdx.x == 0) lenF[nd] = len[0] + len[1] + cnt[n_ops];
}

struct FitchScanArgs {
  const uint4 *F;
  const uint32_t *planes;   // [n_planes][W4]
  const SprStep *steps;
  const SprPrune *prunes;
  unsigned long long *ins;     // [n_moves] weighted empty joins with the pruned set
  unsigned long long *join;    // [n_prunes] weighted empty joins of s and g
  size_t W4;
  int n_planes, depth, max_moves, *flag;
};

__global__ void __launch_bounds__(256) spr_fitch_scan_kernel(const FitchScanArgs a) {
  extern __shared__ __align__(16) unsigned char smem[];
  const SprPrune pr = a.prunes[blockIdx.x];
  unsigned int *red = reinterpret_cast<unsigned int *>(smem);   // [max_moves]
  uint4 *stk = reinterpret_cast<uint4 *>(smem + a16((size_t)a.max_moves * 4));
  __shared__ unsigned int join_acc;
  const int c = threadIdx.x;
  for (int i = c; i < a.max_moves; i += 256) red[i] = 0;
  if (c == 0) join_acc = 0;
  __syncthreads();
  const size_t q = (size_t)blockIdx.y * 256 + c;
  const bool in = q < a.W4;
  const size_t qq = in ? q : 0;
  auto Fd = [&](int d) { return in ? a.F[(size_t)d * a.W4 + qq] : make_uint4(0, 0, 0, 0); };
  const uint4 fp = Fd(pr.dp);
  uint4 cur = make_uint4(0, 0, 0, 0);
  int sp = 0;
  bool have = false, ok = true;
  WeightPlanes wp;
  wp.load(a.planes, a.W4, a.n_planes, qq, in);
  auto add = [&](unsigned int *dst, uint32_t v) {
    v = __reduce_add_sync(0xffffffffu, v);
    if ((c & 31) == 0 && v) atomicAdd(dst, v);
  };
  for (int si = 0; si < pr.n_steps && ok; ++si) {
    const SprStep st = a.steps[pr.step_off + si];
    if (st.flags & SPR_START) {
      const uint4 fs = Fd(st.d1), fg = Fd(st.d2);
      add(&join_acc, wp.count(~meet(fs, fg)));
      const bool ds = st.flags & SPR_DOWN1, dg = st.flags & SPR_DOWN2;
      const bool g_first = ds && dg && (st.flags & SPR_FIRST2);
      if (ds && dg) {
        if (sp >= a.depth) { ok = false; break; }
        stk[(size_t)sp * 256 + c] = g_first ? fg : fs;   // set entering s is g's side
        ++sp;
      }
      cur = (g_first || !ds) ? fs : fg;
      have = true;
      continue;
    }
    if (!have) {
      if (sp == 0) { ok = false; break; }
      --sp;
      cur = stk[(size_t)sp * 256 + c];
    }
    const uint4 f1 = Fd(st.d1), f2 = Fd(st.d2);
    uint32_t e;
    const uint4 r1 = fitch4(cur, f2, &e);   // y's side seen from c1
    const uint4 r2 = fitch4(cur, f1, &e);
    if (st.out1 >= 0) {
      add(&red[st.out1 - pr.move_off], wp.count(~meet(fp, fitch4(r1, f1, &e))));
    }
    if (st.out2 >= 0) {
      add(&red[st.out2 - pr.move_off], wp.count(~meet(fp, fitch4(r2, f2, &e))));
    }
    const bool dn1 = st.flags & SPR_DOWN1, dn2 = st.flags & SPR_DOWN2;
    if (dn1 || dn2) {
      const bool second_first = dn1 && dn2 && (st.flags & SPR_FIRST2);
      if (dn1 && dn2) {
        if (sp >= a.depth) { ok = false; break; }
        stk[(size_t)sp * 256 + c] = second_first ? r1 : r2;
        ++sp;
      }
      cur = (second_first || !dn1) ? r2 : r1;
      have = true;
    } else {
      have = false;
    }
  }
  if (!ok && c == 0) atomicOr(a.flag, PGPU_FLAG_EIGEN);
  __syncthreads();
  for (int j = c; j < pr.n_moves; j += 256)
    if (red[j]) atomicAdd(a.ins + pr.move_off + j, (unsigned long long)red[j]);
  if (c == 0 && join_acc) atomicAdd(a.join + blockIdx.x, (unsigned long long)join_acc);
}

// ---------------------------------------------------------------------------
// per-directed-edge summaries and per-move features
// ---------------------------------------------------------------------------
struct SummaryArgs {
  const void *L;
  const double *probs;
  const float2 *weights;   // [np] float pairs
  const double *wd;        // [np] the same in FP64
  float *out;   // [nd][4]
  size_t np, n_pat;
  int R, RT, rt_shift;
  double inv_w;   // 1 / total weight
};

// weighted mean over patterns of the state profile L_i / sum_j L_j.  The FP32
// values of a vector are summed as float pairs (a reciprocal with its
// remainder, exact products, exact sums): 48 bits on the FP32 units, where
// FP64 divisions and sums made the kernel six times as long as reading L.
// 1,018 directed edges x 45,675 patterns x 4 classes: 0.84 ms against 6.3.
// The FP64 form keeps the FP64 sums.
template <typename Pol>
__global__ void __launch_bounds__(256) spr_summary_kernel(const SummaryArgs a) {
  using V = typename Pol::V;
  __shared__ double red[4][8];
  const int d = blockIdx.x, r = threadIdx.x & (a.RT - 1), np_cta = 256 >> a.rt_shift;
  ff acc[4] = {{0.0f, 0.0f}, {0.0f, 0.0f}, {0.0f, 0.0f}, {0.0f, 0.0f}};
  double acc_d[4] = {0.0, 0.0, 0.0, 0.0};
  if (r < a.R)
    for (size_t pat = threadIdx.x >> a.rt_shift; pat < a.n_pat; pat += np_cta) {
      V x[4];
      Pol::load_g(a.L, ((size_t)d * a.np + pat) * a.R + r, x);
      float f[4], s = 0.0f;
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        f[e] = Pol::to_f(x[e]);
        s += f[e];
      }
      if (!(s > 0.0f)) continue;
      if constexpr (std::is_same<Pol, Fp64>::value) {
        const double k = a.wd[pat] / (double)s;
#pragma unroll
        for (int e = 0; e < 4; ++e) acc_d[e] += k * (double)f[e];
        continue;
      }
      if (s < 0x1p-100f) {   // a class far below the others: 1 / s has to be finite
        s *= 0x1p64f;
#pragma unroll
        for (int e = 0; e < 4; ++e) f[e] *= 0x1p64f;
      }
      // q = w / s as a pair
      const float2 w = a.weights[pat];
      const float c = __frcp_rn(s);
      const ff inv{c, __fmul_rn(__fmaf_rn(-c, s, 1.0f), c)};
      const ff q = ff_mul(inv, ff{w.x, w.y});
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        const float p = __fmul_rn(q.h, f[e]);
        float lo = __fmaf_rn(q.h, f[e], -p);
        lo = __fmaf_rn(q.l, f[e], lo);
        const ff t = fast_two_sum(fmaxf(acc[e].h, p), fminf(acc[e].h, p));   // no term is negative
        acc[e] = {t.h, __fadd_rn(acc[e].l, __fadd_rn(t.l, lo))};
      }
    }
  const double prob = r < a.R ? a.probs[r] : 0.0;
  for (int e = 0; e < 4; ++e) {
    double v = prob * (acc_d[e] + ((double)acc[e].h + (double)acc[e].l));
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    if ((threadIdx.x & 31) == 0) red[e][threadIdx.x >> 5] = v;
  }
  __syncthreads();
  if (threadIdx.x < 4) {
    double v = 0.0;
    for (int w = 0; w < 8; ++w) v += red[threadIdx.x][w];
    a.out[(size_t)d * 4 + threadIdx.x] = (float)(v * a.inv_w);
  }
}

struct FeatArgs {
  const SprMove *moves;
  const SprPrune *prunes;
  const int32_t *tipcnt;
  const double *len;               // [n_edges]
  const float *summ;               // [nd][4], already divided by the total weight
  const unsigned long long *lenF;  // [nd + 1]
  const unsigned long long *ins, *join;
  float *X;                        // [n_moves][64]
  size_t n_moves;
  int n_tips, nd;
  double wtot;
};

__global__ void __launch_bounds__(256) spr_feature_kernel(const FeatArgs a) {
  const size_t m = (size_t)blockIdx.x * 256 + threadIdx.x;
  if (m >= a.n_moves) return;
  const SprMove mv = a.moves[m];
  const SprPrune pr = a.prunes[mv.prune];
  const float ln_n = logf((float)a.n_tips);
  const int dp = pr.dp, dc = mv.dc, dy = dc ^ 1;
  float f[SPR_FEATURES];
#pragma unroll
  for (int i = 0; i < SPR_FEATURES; ++i) f[i] = 0.0f;
  const float P = (float)a.tipcnt[dp];
  f[0] = logf(P) / ln_n;
  f[1] = logf((float)a.n_tips - P) / ln_n;
  f[2] = log1pf((float)mv.depth);
  const double t_pu = a.len[dp >> 1], t_s = a.len[pr.ds >> 1], t_g = a.len[pr.dg >> 1],
               t_c = a.len[dc >> 1];
  f[3] = logf((float)t_pu + 1e-4f);
  f[4] = logf((float)(t_s + t_g) + 1e-4f);
  f[5] = logf((float)t_c + 1e-4f);
  // u's other two neighbours are unordered: only symmetric functions of them
  f[6] = logf((float)fmin(t_s, t_g) + 1e-4f);
  f[7] = logf((float)fmax(t_s, t_g) + 1e-4f);
  // parsimony: length of the rearranged tree minus the current length
  const double lenT = (double)a.lenF[a.nd];
  // remaining tree joined at (s,g) plus the pruned subtree, then the new join
  const double lenR = (double)a.lenF[pr.ds] + (double)a.lenF[pr.dg] + (double)a.join[mv.prune] +
                      (double)a.lenF[dp];
  const double dF = lenR + (double)a.ins[m] - lenT;
  const double sc = 100.0 / a.wtot;
  f[8] = (float)(dF * sc);
  f[9] = dF < 0 ? 1.0f : 0.0f;
  f[10] = dF == 0 ? 1.0f : 0.0f;
  f[11] = dF > 0 ? 1.0f : 0.0f;
  f[12] = asinhf((float)dF);
  f[13] = (float)((lenR - lenT) * sc);
  f[14] = (float)((double)a.ins[m] * sc);
  f[15] = logf((float)a.tipcnt[dc]) / ln_n;
  const float *sp = a.summ + (size_t)dp * 4, *sc_ = a.summ + (size_t)dc * 4,
              *sy = a.summ + (size_t)dy * 4, *ss = a.summ + (size_t)pr.ds * 4,
              *sg = a.summ + (size_t)pr.dg * 4;
  float dot_c = 0.0f, dot_s = 0.0f;
#pragma unroll
  for (int e = 0; e < 4; ++e) {
    const float mean_sg = 0.5f * (ss[e] + sg[e]), diff_sg = fabsf(ss[e] - sg[e]);
    f[16 + e] = sp[e];
    f[20 + e] = sc_[e];
    f[24 + e] = sy[e];
    f[28 + e] = mean_sg;
    f[32 + e] = diff_sg;
    f[36 + e] = sp[e] * sc_[e];
    f[40 + e] = sp[e] * sy[e];
    f[44 + e] = sp[e] * mean_sg;
    f[48 + e] = sp[e] * diff_sg;
    dot_c += sp[e] * sc_[e];
    dot_s += sp[e] * mean_sg;
  }
  f[52] = dot_c;
  f[53] = dot_s;
  f[54] = mv.depth == 1 ? 1.0f : 0.0f;
  float *o = a.X + m * SPR_FEATURES;
#pragma unroll
  for (int i = 0; i < SPR_FEATURES; ++i) o[i] = f[i];
}

}  // namespace

// ---------------------------------------------------------------------------
// branch lengths: Newton steps on every edge at once, from the pool
// ---------------------------------------------------------------------------
namespace {

struct BlArgs {
  const void *L;
  const double *U, *Ui, *lam, *pi, *rates, *probs;
  const float2 *w2;         // [np] weights as float pairs
  const float *w3;          // [np] what the pairs leave of the weights, or null: nothing
  float *S;                 // [n_edges][np][R][4]: eigen-basis products
  const double *len_in;
  double *len_out;
  size_t np, n_pat;
  int R, n_edges, iters;
  double tol, tmin, tmax;
};

// S[e][pat][r][k] = (sum_i pi_i L[a|b]_i U_ik) (sum_j Ui_kj L[b|a]_j), so that
// the site likelihood across edge e is sum_r probs_r sum_k S_k exp(lam_k rate_r t)
template <typename Pol>
__device__ __forceinline__ void eigen_values(const BlArgs &a, const typename Pol::V *x, const typename Pol::V *y,
                                             double *xd, double *yd) {
#pragma unroll
  for (int j = 0; j < 4; ++j) {
    xd[j] = a.pi[j] * Pol::to_d(x[j]);
    yd[j] = Pol::to_d(y[j]);
  }
}
__device__ __forceinline__ float eigen_product(const BlArgs &a, const double *x, const double *y, int k) {
  double A = 0.0, B = 0.0;
#pragma unroll
  for (int j = 0; j < 4; ++j) {
    A = fma(x[j], a.U[j * 4 + k], A);
    B = fma(a.Ui[k * 4 + j], y[j], B);
  }
  return (float)(A * B);
}

__global__ void __launch_bounds__(256) bl_sumtab_kernel(const BlArgs a) {
  using Pol = Fp64;
  using V = Pol::V;
  const size_t i = (size_t)blockIdx.x * 256 + threadIdx.x;
  if (i >= a.np * a.R) return;
  const int e = blockIdx.y;
  V x[4], y[4];
  Pol::load_g(a.L, (size_t)(2 * e) * a.np * a.R + i, x);
  Pol::load_g(a.L, (size_t)(2 * e + 1) * a.np * a.R + i, y);
  double xd[4], yd[4];
  eigen_values<Pol>(a, x, y, xd, yd);
  float s[4];
#pragma unroll
  for (int k = 0; k < 4; ++k) s[k] = eigen_product(a, xd, yd, k);
  reinterpret_cast<float4 *>(a.S)[(size_t)e * a.np * a.R + i] = make_float4(s[0], s[1], s[2], s[3]);
}

// The same from FP32 values and float pairs, on the FP32 units: each eigen
// product is a sum of four signed terms, exact products and exact sums
// (TwoSum) in pairs, two eigenvectors to a packed float2 instruction.  S is
// the float that FP64 gives: where the pairs' error leaves two candidates
// (Ziv's rounding test with EIGEN_ERR) the value is formed again in FP64: the
// Newton steps' float exponentials turn a last bit here into 3e-7 of a length,
// and where a whole edge is flat the rounding of sums that cancel is all there
// is to step on.  Nearly all such sums are a missing tip's (1, 1, 1, 1), for
// which FP64's own are formed once per CTA (2.25 ms with each of them formed
// again).
//
// The error of a sum, with u = 2^-24 and T the sum of the terms' sizes: each
// product leaves out its low parts' product and the coefficient's own rest
// (u^2 each) and rounds its low word twice (2 u^2 and 3 u^2): 7 u^2 T in all.
// An addition's low word is its TwoSum rest, at most u T, plus the product's,
// 3 u of its term: forming the three rounds 6 u^2 T, gathering them 15 u^2 T
// (they grow by u T a term).  28 u^2 T.  The product of two such sums A, B
// adds three roundings of its low word, 3 u^2 (T_A |B| + |A| T_B), and the test
// itself and FP64's own error under 2 u^2.  33 u^2 in all; 14 u^2 T is the
// largest error of a sum that a search has found.
// 509 edges x 45,675 patterns x 4 classes, pair form: 1.74 ms against 11.4
// in FP64, which this GPU runs at 1/64 of the FP32 rate.
constexpr float EIGEN_ERR = 0x1p-42f;   // 64 u^2
__device__ __forceinline__ float2 sub2(float2 a, float2 b) { return __fadd2_rn(a, neg2(b)); }
__device__ __forceinline__ void two_sum2(float2 a, float2 b, float2 &s, float2 &e) {
  s = __fadd2_rn(a, b);
  const float2 bb = sub2(s, a);
  e = __fadd2_rn(sub2(a, sub2(s, bb)), sub2(b, bb));
}

// sum_j c_j x_j for two eigenvectors, normalised, and the sum of the terms'
// sizes; c as {hi, hi', lo, lo'}
__device__ __forceinline__ void eigen_pair(const float4 (*c)[2], int kp, const ff *x, float2 &sum, float2 &err,
                                           float2 &mag) {
  float2 s = make_float2(0.0f, 0.0f), lo = s;
#pragma unroll
  for (int j = 0; j < 4; ++j) {
    const float4 q = c[j][kp];
    const float2 ch = make_float2(q.x, q.y), cl = make_float2(q.z, q.w);
    const float2 xh = make_float2(x[j].h, x[j].h), xl = make_float2(x[j].l, x[j].l);
    const float2 p = __fmul2_rn(ch, xh);
    float2 e = __ffma2_rn(ch, xh, neg2(p));
    e = __ffma2_rn(ch, xl, e);
    e = __ffma2_rn(cl, xh, e);
    mag = j == 0 ? make_float2(fabsf(p.x), fabsf(p.y)) : make_float2(mag.x + fabsf(p.x), mag.y + fabsf(p.y));
    if (j == 0) {
      s = p;
      lo = e;
    } else {
      float2 t, te;
      two_sum2(s, p, t, te);
      s = t;
      lo = __fadd2_rn(lo, __fadd2_rn(te, e));
    }
  }
  two_sum2(s, lo, sum, err);
}

__device__ __forceinline__ void take_sum(float4 q, float2 &sum, float2 &err, float2 &mag) {
  sum = make_float2(q.x, q.y);
  err = make_float2(q.z, q.w);
  mag = make_float2(fabsf(q.x), fabsf(q.y));
}

template <typename Pol>
__global__ void __launch_bounds__(256) bl_sumtab_pair_kernel(const BlArgs a) {
  using V = typename Pol::V;
  __shared__ float4 cA[4][2], cB[4][2];   // [j][eigenvector pair]
  __shared__ float4 ones[2][2];           // FP64's sums of a missing tip's vector, as pairs: [side][eigenvector pair]
  if (threadIdx.x < 32) {
    const int side = threadIdx.x >> 4, j = (threadIdx.x >> 2) & 3, k = threadIdx.x & 3;
    const double v = side == 0 ? a.pi[j] * a.U[j * 4 + k] : a.Ui[k * 4 + j];
    float *dst = reinterpret_cast<float *>(side == 0 ? &cA[j][k >> 1] : &cB[j][k >> 1]) + (k & 1);
    const float h = (float)v;
    dst[0] = h;
    dst[2] = (float)(v - (double)h);
  } else if (threadIdx.x < 40) {
    const int side = (threadIdx.x >> 2) & 1, k = threadIdx.x & 3;
    double v = 0.0;   // as eigen_product sums the vector 1, 1, 1, 1
    for (int j = 0; j < 4; ++j) v = side == 0 ? fma(a.pi[j], a.U[j * 4 + k], v) : fma(a.Ui[k * 4 + j], 1.0, v);
    float *dst = reinterpret_cast<float *>(&ones[side][k >> 1]) + (k & 1);
    const float h = (float)v;
    dst[0] = h;
    dst[2] = (float)(v - (double)h);
  }
  __syncthreads();
  const size_t i = (size_t)blockIdx.x * 256 + threadIdx.x;
  if (i >= a.np * a.R) return;
  const int e = blockIdx.y;
  V xv[4], yv[4];
  Pol::load_g(a.L, (size_t)(2 * e) * a.np * a.R + i, xv);
  Pol::load_g(a.L, (size_t)(2 * e + 1) * a.np * a.R + i, yv);
  ff x[4], y[4];
#pragma unroll
  for (int j = 0; j < 4; ++j) {   // normalised: the stored low words may be a few ulps
    x[j] = Pol::to_ff(xv[j]);
    y[j] = Pol::to_ff(yv[j]);
    x[j] = fast_two_sum(x[j].h, x[j].l);
    y[j] = fast_two_sum(y[j].h, y[j].l);
  }
  bool x_ones = true, y_ones = true;
#pragma unroll
  for (int j = 0; j < 4; ++j) {
    x_ones = x_ones && x[j].h == 1.0f && x[j].l == 0.0f;
    y_ones = y_ones && y[j].h == 1.0f && y[j].l == 0.0f;
  }
  float s[4];
  int unsure = 0;
#pragma unroll
  for (int kp = 0; kp < 2; ++kp) {
    float2 ah, al, am, bh, bl, bm;
    eigen_pair(cA, kp, x, ah, al, am);
    eigen_pair(cB, kp, y, bh, bl, bm);
    if (x_ones) take_sum(ones[0][kp], ah, al, am);
    if (y_ones) take_sum(ones[1][kp], bh, bl, bm);
    const float2 p = __fmul2_rn(ah, bh);
    float2 er = __ffma2_rn(ah, bh, neg2(p));
    er = __ffma2_rn(ah, bl, er);
    er = __ffma2_rn(al, bh, er);
    const float2 v = __fadd2_rn(p, er), rest = sub2(er, sub2(v, p));
    const float2 d = __fmul2_rn(make_float2(EIGEN_ERR, EIGEN_ERR),
                                make_float2(fmaf(fabsf(ah.x), bm.x, fabsf(bh.x) * am.x),
                                            fmaf(fabsf(ah.y), bm.y, fabsf(bh.y) * am.y)));
    const float2 up = __fadd2_rn(v, __fadd2_rn(rest, d)), down = __fadd2_rn(v, sub2(rest, d));
    s[2 * kp] = v.x;
    s[2 * kp + 1] = v.y;
    if (!(up.x == down.x)) unsure |= 1 << (2 * kp);
    if (!(up.y == down.y)) unsure |= 2 << (2 * kp);
  }
  if (unsure) {
    double xd[4], yd[4];
    eigen_values<Pol>(a, xv, yv, xd, yd);
#pragma unroll
    for (int k = 0; k < 4; ++k)
      if (unsure >> k & 1) s[k] = eigen_product(a, xd, yd, k);
  }
  reinterpret_cast<float4 *>(a.S)[(size_t)e * a.np * a.R + i] = make_float4(s[0], s[1], s[2], s[3]);
}

// One CTA per edge: Newton iterations on t with the derivatives of
// sum_s w_s log f_s(t) summed over all patterns.  An iteration reads the
// edge's S once and should take no longer than that; FP64 runs at 1/64 of the
// FP32 rate, so the exponentials are formed once per CTA and the sums of an
// iteration kept in three floats, closer than FP64.  509 edges x 45,675
// patterns x 4 classes: 2.0 ms against 2.71 with both in FP64 in every thread.
// A weight is taken with all the bits of its FP64 value.
__global__ void __launch_bounds__(256) bl_newton_kernel(const BlArgs a) {
  __shared__ double red[2][8];
  __shared__ double t_sh;
  __shared__ float cf[8][4], ex[8][4];
  __shared__ int done;
  const int e = blockIdx.x, tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  if (tid == 0) {
    t_sh = a.len_in[e];
    done = 0;
  }
  __syncthreads();
  for (int it = 0; it < a.iters; ++it) {
    const double t = t_sh;
    if (tid < 4 * a.R) {
      const int r = tid >> 2, k = tid & 3;
      cf[r][k] = (float)(a.lam[k] * a.rates[r]);
      ex[r][k] = (float)(exp(a.lam[k] * a.rates[r] * t) * a.probs[r]);
    }
    __syncthreads();
    Sum3 gs, hs;
    const float4 *S = reinterpret_cast<const float4 *>(a.S) + (size_t)e * a.np * a.R;
    for (size_t pat = tid; pat < a.n_pat; pat += 256) {
      float f = 0.0f, f1 = 0.0f, f2 = 0.0f;
      for (int r = 0; r < a.R; ++r) {
        const float4 s = S[pat * a.R + r];
        const float sv[4] = {s.x, s.y, s.z, s.w};
#pragma unroll
        for (int k = 0; k < 4; ++k) {
          const float v = sv[k] * ex[r][k];
          f += v;
          f1 = fmaf(v, cf[r][k], f1);
          f2 = fmaf(v * cf[r][k], cf[r][k], f2);
        }
      }
      if (f > 0.0f) {
        // w d1 and w (f2 / f - d1^2), w in two floats, or three: all of its bits
        const float d1 = f1 / f, d2 = f2 / f, q = __fmul_rn(d1, d1), qe = __fmaf_rn(d1, d1, -q);
        const float2 w = a.w2[pat];
        gs.add_product(w.x, d1);
        hs.add_product(w.x, d2);
        hs.add_product(w.x, -q);
        hs.add_low(__fmul_rn(w.x, -qe));
        if (w.y != 0.0f) {
          gs.add_product(w.y, d1);
          hs.add_product(w.y, d2);
          hs.add_product(w.y, -q);
          hs.add_low(__fmul_rn(w.y, -qe));
          if (a.w3) {
            const float v = a.w3[pat];
            gs.add_low(__fmul_rn(v, d1));
            hs.add_low(__fmul_rn(v, __fadd_rn(d2, -q)));
          }
        }
      }
    }
    double g = gs.value(), h = hs.value();
    for (int o = 16; o > 0; o >>= 1) {
      g += __shfl_xor_sync(0xffffffffu, g, o);
      h += __shfl_xor_sync(0xffffffffu, h, o);
    }
    if (lane == 0) {
      red[0][warp] = g;
      red[1][warp] = h;
    }
    __syncthreads();
    if (tid == 0) {
      double G = 0.0, Hs = 0.0;
      for (int w = 0; w < 8; ++w) {
        G += red[0][w];
        Hs += red[1][w];
      }
      double tn;
      if (Hs < 0.0) tn = t - G / Hs;
      else tn = G > 0.0 ? t * 2.0 : t * 0.5;
      // keep each step inside a factor of ten of the current length
      tn = fmin(fmax(tn, fmax(a.tmin, 0.1 * t)), fmin(a.tmax, 10.0 * fmax(t, a.tmin)));
      if (fabs(tn - t) <= a.tol * fmax(t, 1e-3)) done = 1;
      t_sh = tn;
    }
    __syncthreads();
    if (done) break;
  }
  if (tid == 0) a.len_out[e] = t_sh;
}

__global__ void spr_fitch_moves_kernel(const SprMove *moves, const SprPrune *prunes, size_t n_moves,
                                       const unsigned long long *lenF, const unsigned long long *ins,
                                       const unsigned long long *join, unsigned long long *out) {
  const size_t m = (size_t)blockIdx.x * 256 + threadIdx.x;
  if (m >= n_moves) return;
  const SprMove mv = moves[m];
  const SprPrune pr = prunes[mv.prune];
  // the rest joined at (s,g), the pruned subtree itself, and its new join
  out[m] = lenF[pr.ds] + lenF[pr.dg] + join[mv.prune] + lenF[pr.dp] + ins[m];
}

}  // namespace

// ---------------------------------------------------------------------------
// the engine object
// ---------------------------------------------------------------------------
struct SprPlanDev {
  SprStep *steps = nullptr;
  SprPrune *prunes = nullptr;
  SprMove *moves = nullptr;
  double *mlen = nullptr;   // merged lengths
  void *Dmer = nullptr;
  size_t cap_steps = 0, cap_prunes = 0, cap_moves = 0;
};

struct pgpu_spr {
  pgpu_ctx *ctx = nullptr;
  int precision = 48, R = 1, n = 0, n_codes = 0, RT = 1, NP = 256, n_planes = 0;
  size_t n_pat = 0, np = 0, ld = 0, W4 = 0, vbytes = 0, cbytes = 0;
  double wtot = 0.0;
  const uint8_t *codes = nullptr;
  // model
  double *Q = nullptr, *pi = nullptr, *rates = nullptr, *probs = nullptr, *ctab = nullptr,
         *U = nullptr, *Ui = nullptr, *lam = nullptr;
  void *crows = nullptr;   // the code table as vectors of the form
  int *status = nullptr;
  uint8_t *cmask = nullptr;
  double *w = nullptr;
  float2 *w2 = nullptr;      // weights as float pairs
  float *w3 = nullptr;       // what the pairs leave of them (null: nothing)
  float2 *pairs = nullptr;   // pi [4] and probs [8] as float pairs
  float4 *logtab = nullptr;
  // pool
  void *L = nullptr, *M = nullptr, *H = nullptr;
  int32_t *sc = nullptr;
  void *Dfull = nullptr, *tipfull = nullptr, *tiphalf = nullptr;
  double *elen = nullptr, *tiplen = nullptr, *newlen = nullptr;
  int4 *ops = nullptr, *tips = nullptr, *half_list = nullptr;
  double2 *pool_part = nullptr;
  double *tree_lnl = nullptr, *site_lnl = nullptr;
  // fitch
  uint4 *F = nullptr;
  uint32_t *planes = nullptr;
  unsigned long long *cntF = nullptr, *lenF = nullptr, *ins = nullptr, *join = nullptr;
  float *summ = nullptr;
  // scratch
  float2 *partials = nullptr;
  size_t part_cap = 0;
  float *S = nullptr;
  // host state
  SprTopo T;
  PoolPlan pp;
  SprPlan all, sel;
  SprPlanDev all_d, sel_d;
  bool pp_valid = false, pool_valid = false, half_valid = false, plan_valid = false, fitch_valid = false, summ_valid = false;
  int join_distance = 0;   // 0: every SPR move; d: regraft edges at most d nodes from the break
  // TBR: plan, emit walks on the device, attach vectors of a batch of cuts
  TbrPlan tbr;
  SprPlanDev tbr_d;
  bool tbr_valid = false;
  int tbr_join = 0, tbr_reroot = 0;   // attach-edge limits in nodes from the cut (0: none)
  size_t tbr_budget = size_t(2) << 30;   // attach-vector bytes per batch of cuts
  char *tbr_x = nullptr;
  int32_t *tbr_xsc = nullptr;
  TbrCutDev *tbr_cuts = nullptr;
  int4 *tbr_tiles = nullptr;
  size_t tbr_x_cap = 0, tbr_xsc_cap = 0, tbr_cuts_cap = 0, tbr_tiles_cap = 0;
  // with two different limits: every pair's lnL, and the listed pairs' grid indices
  double *tbr_grid = nullptr;
  int64_t *tbr_keep = nullptr;
  size_t tbr_grid_cap = 0, tbr_keep_cap = 0;
  // host copies of a TBR batch's cut and tile lists, owned by the engine so
  // that they outlive the asynchronous copies to the device
  std::vector<TbrCutDev> h_tbr_cuts;
  std::vector<int4> h_tbr_tiles;
  std::vector<void *> owned;
};

namespace {

pgpu_status dalloc(pgpu_spr *s, size_t bytes, void **p) {
  PGPU_CUDA(s->ctx, cudaMalloc(p, std::max<size_t>(bytes, 16)));
  s->owned.push_back(*p);
  return PGPU_OK;
}
template <typename T>
pgpu_status dalloc_t(pgpu_spr *s, size_t n, T **p) {
  void *v;
  PGPU_TRY(dalloc(s, n * sizeof(T), &v));
  *p = static_cast<T *>(v);
  return PGPU_OK;
}
template <typename T>
pgpu_status grow(pgpu_spr *s, T **p, size_t *cap, size_t n) {
  if (*cap >= n) return PGPU_OK;
  if (*p) {
    cudaFree(*p);
    s->owned.erase(std::find(s->owned.begin(), s->owned.end(), (void *)*p));
  }
  *p = nullptr;
  const size_t want = std::max<size_t>(n + n / 4, 64);
  PGPU_TRY(dalloc_t(s, want, p));
  *cap = want;
  return PGPU_OK;
}
template <typename T>
pgpu_status upload(pgpu_spr *s, T *dst, const T *src, size_t n) {
  if (n) PGPU_CUDA(s->ctx, cudaMemcpyAsync(dst, src, n * sizeof(T), cudaMemcpyHostToDevice, s->ctx->stream));
  return PGPU_OK;
}

int p32_mode(int prec) { return prec == 32 ? P32_MINUS_I : prec == 64 ? P32_PLAIN : P32_PAIRS_ROWS4; }
int tip_form(int prec) { return prec == 32 ? 0 : prec == 64 ? 2 : 3; }

pgpu_status compose(pgpu_spr *s, const double *t_dev, int n_br, void *out) {
  return pgpu_launch_compose(s->ctx, s->U, s->lam, s->Ui, 4, t_dev, n_br, s->rates, s->R,
                             s->precision == 64 ? (double *)out : nullptr,
                             s->precision == 64 ? nullptr : (float *)out, false, s->status,
                             p32_mode(s->precision));
}

template <typename Pol, int RT>
pgpu_status launch_pool_rt(pgpu_spr *s, bool half) {
  PoolArgs a;
  a.L = s->L;
  a.M = s->M;
  a.H = s->H;
  a.sc = s->sc;
  a.Dfull = s->Dfull;
  a.Dhalf = static_cast<char *>(s->Dfull) + (size_t)s->T.n_edges() * s->cbytes;
  a.ops = s->ops;
  a.pi = s->pi;
  a.probs = s->probs;
  a.weights = s->w;
  a.site_lnl = s->site_lnl;
  a.partials = s->pool_part;
  a.np = s->np;
  a.n_pat = s->n_pat;
  a.n_ops = (int)s->pp.ops.size();
  a.R = s->R;
  a.NP = s->NP;
  if (half) spr_pool_kernel<Pol, RT, true><<<(unsigned)(s->np / s->NP), SPR_NT, 0, s->ctx->stream>>>(a);
  else spr_pool_kernel<Pol, RT, false><<<(unsigned)(s->np / s->NP), SPR_NT, 0, s->ctx->stream>>>(a);
  return pgpu_after_launch(s->ctx, "spr_pool_kernel");
}

TipArgs tip_args(pgpu_spr *s) {
  TipArgs t;
  t.L = s->L;
  t.M = s->M;
  t.H = s->H;
  t.sc = s->sc;
  t.tipfull = s->tipfull;
  t.tiphalf = s->tiphalf;
  t.code_rows = s->crows;
  t.codes = s->codes;
  t.tips = s->tips;
  t.flag = s->ctx->d_flag;
  t.np = s->np;
  t.n_pat = s->n_pat;
  t.ld = s->ld;
  t.R = s->R;
  t.n_codes = s->n_codes;
  return t;
}

unsigned item_ctas(const pgpu_spr *s) { return (unsigned)((s->np * s->R + 255) / 256); }

template <typename Pol>
pgpu_status launch_pool(pgpu_spr *s, bool half) {
  const TipArgs t = tip_args(s);
  const dim3 g(item_ctas(s), (unsigned)s->n);
  if (half) spr_tip_kernel<Pol, true, true><<<g, 256, 0, s->ctx->stream>>>(t);
  else spr_tip_kernel<Pol, true, false><<<g, 256, 0, s->ctx->stream>>>(t);
  PGPU_TRY(pgpu_after_launch(s->ctx, "spr_tip_kernel"));
  switch (s->RT) {
    case 1: return launch_pool_rt<Pol, 1>(s, half);
    case 2: return launch_pool_rt<Pol, 2>(s, half);
    case 4: return launch_pool_rt<Pol, 4>(s, half);
    default: return launch_pool_rt<Pol, 8>(s, half);
  }
}

// H of the listed directed edges of a pool made without it: tips {dedge, tip,
// edge, 0} and internal ones {dedge, ...}
template <typename Pol>
pgpu_status launch_half(pgpu_spr *s, const int4 *tips, size_t n_tips, const int4 *ops, size_t n_ops) {
  if (n_tips) {
    TipArgs t = tip_args(s);
    t.tips = tips;
    spr_tip_kernel<Pol, false, true><<<dim3(item_ctas(s), (unsigned)n_tips), 256, 0, s->ctx->stream>>>(t);
    PGPU_TRY(pgpu_after_launch(s->ctx, "spr_tip_kernel"));
  }
  const void *Dhalf = static_cast<char *>(s->Dfull) + (size_t)s->T.n_edges() * s->cbytes;
  for (size_t i = 0; i < n_ops; i += 65535) {
    const unsigned k = (unsigned)std::min<size_t>(n_ops - i, 65535);
    spr_half_kernel<Pol><<<dim3(item_ctas(s), k), 256, 0, s->ctx->stream>>>(s->L, s->H, Dhalf, ops + i, s->np,
                                                                           (unsigned)s->R);
    PGPU_TRY(pgpu_after_launch(s->ctx, "spr_half_kernel"));
  }
  return PGPU_OK;
}

pgpu_status tip_rows(pgpu_spr *s, bool half) {
  return pgpu_launch_tip_table(s->ctx, s->U, s->lam, s->Ui, 4, s->elen + 2 * s->T.n_edges() + (half ? s->n : 0),
                               s->n, s->rates, s->R, s->ctab, s->n_codes, half ? s->tiphalf : s->tipfull,
                               tip_form(s->precision), s->status);
}

pgpu_status add_half(pgpu_spr *s, const int4 *tips, size_t n_tips, const int4 *ops, size_t n_ops) {
  if (n_tips) PGPU_TRY(tip_rows(s, true));
  if (s->precision == 32) return launch_half<Fp32>(s, tips, n_tips, ops, n_ops);
  if (s->precision == 48) return launch_half<Ff32>(s, tips, n_tips, ops, n_ops);
  return launch_half<Fp64>(s, tips, n_tips, ops, n_ops);
}

void ensure_pool_plan(pgpu_spr *s) {
  if (s->pp_valid) return;
  spr_pool_plan(s->T, &s->pp);
  s->pp_valid = true;
}

// Rebuilds everything that depends on the topology and branch lengths; half:
// with the vectors at the edges' middles, which scoring moves reads.
pgpu_status ensure_pool(pgpu_spr *s, bool half = false) {
  if (s->pool_valid) {
    if (!half || s->half_valid) return PGPU_OK;
    PGPU_TRY(add_half(s, s->tips, (size_t)s->n, s->ops, s->pp.ops.size()));
    s->half_valid = true;
    return PGPU_OK;
  }
  SprTopo &T = s->T;
  ensure_pool_plan(s);
  const int ne = T.n_edges();
  std::vector<double> h(2 * ne + 2 * s->n);
  for (int e = 0; e < ne; ++e) {
    h[e] = T.len[e];
    h[ne + e] = 0.5 * T.len[e];
  }
  for (int x = 0; x < s->n; ++x) {
    h[2 * ne + x] = T.len[T.inc[x][0]];
    h[2 * ne + s->n + x] = 0.5 * T.len[T.inc[x][0]];
  }
  PGPU_TRY(upload(s, s->elen, h.data(), h.size()));
  PGPU_TRY(upload(s, s->ops, s->pp.ops.data(), s->pp.ops.size()));
  PGPU_TRY(upload(s, s->tips, s->pp.tips.data(), s->pp.tips.size()));
  PGPU_TRY(compose(s, s->elen, 2 * ne, s->Dfull));
  PGPU_TRY(tip_rows(s, false));
  if (half) PGPU_TRY(tip_rows(s, true));
  if (s->precision == 32) PGPU_TRY(launch_pool<Fp32>(s, half));
  else if (s->precision == 48) PGPU_TRY(launch_pool<Ff32>(s, half));
  else PGPU_TRY(launch_pool<Fp64>(s, half));
  spr_pool_finalize_kernel<<<1, 1024, 0, s->ctx->stream>>>(s->pool_part, (int)(s->np / s->NP), s->tree_lnl);
  PGPU_TRY(pgpu_after_launch(s->ctx, "spr_pool_finalize_kernel"));
  s->pool_valid = true;
  s->half_valid = half;
  return PGPU_OK;
}

pgpu_status upload_plan(pgpu_spr *s, const SprPlan &p, SprPlanDev *d) {
  PGPU_TRY(grow(s, &d->steps, &d->cap_steps, p.steps.size()));
  size_t cp = d->cap_prunes;
  PGPU_TRY(grow(s, &d->prunes, &d->cap_prunes, p.prunes.size()));
  if (d->cap_prunes != cp || !d->mlen) {
    size_t c2 = 0;
    d->mlen = nullptr;
    PGPU_TRY(grow(s, &d->mlen, &c2, d->cap_prunes));
    void *dm;
    PGPU_TRY(dalloc(s, d->cap_prunes * s->cbytes, &dm));
    d->Dmer = dm;
  }
  PGPU_TRY(grow(s, &d->moves, &d->cap_moves, p.moves.size()));
  PGPU_TRY(upload(s, d->steps, p.steps.data(), p.steps.size()));
  PGPU_TRY(upload(s, d->prunes, p.prunes.data(), p.prunes.size()));
  PGPU_TRY(upload(s, d->moves, p.moves.data(), p.moves.size()));
  PGPU_TRY(upload(s, d->mlen, p.merged_len.data(), p.merged_len.size()));
  if (!p.prunes.empty()) PGPU_TRY(compose(s, d->mlen, (int)p.prunes.size(), d->Dmer));
  return PGPU_OK;
}

pgpu_status ensure_plan(pgpu_spr *s) {
  if (s->plan_valid) return PGPU_OK;
  ensure_pool_plan(s);
  spr_plan_all(s->T, s->pp, &s->all, s->join_distance);
  PGPU_TRY(upload_plan(s, s->all, &s->all_d));
  s->plan_valid = true;
  return PGPU_OK;
}

template <typename Pol, int RT>
pgpu_status launch_scan_rt(pgpu_spr *s, const SprPlan &p, const SprPlanDev &d, int G, int n_groups,
                           int n_blocks) {
  ScanArgs a;
  a.L = s->L;
  a.M = s->M;
  a.H = s->H;
  a.sc = s->sc;
  a.Dhalf = static_cast<char *>(s->Dfull) + (size_t)s->T.n_edges() * s->cbytes;
  a.Dmer = d.Dmer;
  a.steps = d.steps;
  a.prunes = d.prunes;
  a.pi = s->pi;
  a.probs = s->probs;
  a.pairs = s->pairs;
  a.wts = s->w2;
  a.logtab = s->logtab;
  a.partials = s->partials;
  a.flag = s->ctx->d_flag;
  a.np = s->np;
  a.n_moves = p.moves.size();
  a.R = s->R;
  a.NP = s->NP;
  a.G = G;
  a.n_blocks = n_blocks;
  a.depth = std::max(p.max_depth, 1);
  a.Dfull = nullptr;
  a.xout = nullptr;
  a.xsc = nullptr;
  a.slot_base = 0;
  a.prune_base = 0;
  const size_t smem = scan_smem<Pol>(a.depth, RT);
  const size_t need = scan_limit<Pol>(a.depth, std::max(p.max_moves_per_prune, 1), RT);
  if (need > s->ctx->smem_optin)
    return pgpu_set_err(s->ctx, PGPU_ERR_LIMIT, "spr: scan needs %zu bytes of shared memory", need);
  PGPU_CUDA(s->ctx, cudaFuncSetAttribute(spr_scan_kernel<Pol, RT>,
                                         cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
  spr_scan_kernel<Pol, RT><<<dim3((unsigned)p.prunes.size(), (unsigned)n_groups), SPR_NT, smem,
                             s->ctx->stream>>>(a);
  return pgpu_after_launch(s->ctx, "spr_scan_kernel");
}

template <typename Pol>
pgpu_status launch_scan(pgpu_spr *s, const SprPlan &p, const SprPlanDev &d, int G, int n_groups,
                        int n_blocks) {
  switch (s->RT) {
    case 1: return launch_scan_rt<Pol, 1>(s, p, d, G, n_groups, n_blocks);
    case 2: return launch_scan_rt<Pol, 2>(s, p, d, G, n_groups, n_blocks);
    case 4: return launch_scan_rt<Pol, 4>(s, p, d, G, n_groups, n_blocks);
    default: return launch_scan_rt<Pol, 8>(s, p, d, G, n_groups, n_blocks);
  }
}

// H of the edges that the moves of plan p regraft onto.  Fewer moves than the
// tree has directed edges read the H of a few of them only, and a pool made
// without H gets just those: 32 moves on 256 taxa x 45,675 patterns took
// 2.52 ms for all 1,018 and 0.06 ms for their own.
pgpu_status ensure_half(pgpu_spr *s, const SprPlan &p) {
  const size_t nd = (size_t)s->T.n_dedges();
  if (p.moves.size() >= nd) return ensure_pool(s, true);
  PGPU_TRY(ensure_pool(s));
  if (s->half_valid) return PGPU_OK;
  std::vector<int4> list[2];   // tips, internal
  std::vector<uint8_t> seen(nd, 0);
  for (const SprMove &m : p.moves) {
    if (seen[m.dc]) continue;
    seen[m.dc] = 1;
    const int src = s->T.dsrc(m.dc);
    list[src < s->n ? 0 : 1].push_back(make_int4(m.dc, src, m.dc >> 1, 0));
  }
  int4 *at = s->half_list;
  PGPU_TRY(upload(s, at, list[0].data(), list[0].size()));
  PGPU_TRY(upload(s, at + list[0].size(), list[1].data(), list[1].size()));
  return add_half(s, at, list[0].size(), at + list[0].size(), list[1].size());
}

// lazy log-likelihood of every move of plan p into lnl_dev
pgpu_status run_scan(pgpu_spr *s, const SprPlan &p, const SprPlanDev &d, double *lnl_dev) {
  const size_t nm = p.moves.size();
  if (nm == 0) return PGPU_OK;
  PGPU_TRY(ensure_half(s, p));
  // CTA groups of G pattern blocks; partial sums at most 256 MB
  const size_t budget = size_t(256) << 20;
  auto groups = [&](int blocks, int *g) {
    *g = (int)std::max<size_t>(1, ((size_t)blocks * nm * 8 + budget - 1) / budget);
    *g = std::min(*g, blocks);
    return (blocks + *g - 1) / *g;
  };
  int G;
  const int lim_np = SPR_LIMIT_NT / s->RT;
  if (groups((int)((s->np + lim_np - 1) / lim_np), &G) > 65535)
    return pgpu_set_err(s->ctx, PGPU_ERR_LIMIT, "spr: too many pattern blocks");
  const int n_blocks = (int)(s->np / s->NP);
  int n_groups = groups(n_blocks, &G);
  if (n_groups > 65535) {   // a grid's second dimension
    G = (n_blocks + 65534) / 65535;
    n_groups = (n_blocks + G - 1) / G;
  }
  PGPU_TRY(grow(s, &s->partials, &s->part_cap, (size_t)n_groups * nm));
  if (s->precision == 32) PGPU_TRY(launch_scan<Fp32>(s, p, d, G, n_groups, n_blocks));
  else if (s->precision == 48) PGPU_TRY(launch_scan<Ff32>(s, p, d, G, n_groups, n_blocks));
  else PGPU_TRY(launch_scan<Fp64>(s, p, d, G, n_groups, n_blocks));
  spr_reduce_kernel<<<(unsigned)((nm + 31) / 32), dim3(32, RED_Y), 0, s->ctx->stream>>>(s->partials, n_groups, nm,
                                                                                       lnl_dev);
  return pgpu_after_launch(s->ctx, "spr_reduce_kernel");
}

// ---------------------------------------------------------------------------
// TBR: per batch of cuts, the emit walks store every attach vector, then the
// pair kernel scores every (j, k) of each cut
// ---------------------------------------------------------------------------
pgpu_status ensure_tbr(pgpu_spr *s) {
  if (s->tbr_valid) return PGPU_OK;
  ensure_pool_plan(s);
  tbr_plan(s->T, s->pp, s->tbr_join, s->tbr_reroot, &s->tbr);
  PGPU_TRY(upload_plan(s, s->tbr.emit, &s->tbr_d));
  if (!s->tbr.keep.empty()) {
    PGPU_TRY(grow(s, &s->tbr_keep, &s->tbr_keep_cap, s->tbr.keep.size()));
    PGPU_TRY(upload(s, s->tbr_keep, s->tbr.keep.data(), s->tbr.keep.size()));
  }
  s->tbr_valid = true;
  return PGPU_OK;
}

template <typename Pol, int RT>
pgpu_status launch_emit_rt(pgpu_spr *s, int prune_base, int n_prunes, long long slot_base) {
  const SprPlan &p = s->tbr.emit;
  ScanArgs a;
  a.L = s->L;
  a.M = s->M;
  a.H = s->H;
  a.sc = s->sc;
  a.Dhalf = static_cast<char *>(s->Dfull) + (size_t)s->T.n_edges() * s->cbytes;
  a.Dmer = s->tbr_d.Dmer;
  a.steps = s->tbr_d.steps;
  a.prunes = s->tbr_d.prunes;
  a.pi = s->pi;
  a.probs = s->probs;
  a.pairs = s->pairs;
  a.wts = s->w2;
  a.logtab = s->logtab;
  a.partials = nullptr;
  a.flag = s->ctx->d_flag;
  a.np = s->np;
  a.n_moves = p.moves.size();
  a.R = s->R;
  a.NP = s->NP;
  a.n_blocks = (int)(s->np / s->NP);
  a.G = (a.n_blocks + 65534) / 65535;   // a grid's second dimension
  a.depth = std::max(p.max_depth, 1);
  a.Dfull = s->Dfull;
  a.xout = s->tbr_x;
  a.xsc = s->tbr_xsc;
  a.slot_base = slot_base;
  a.prune_base = prune_base;
  const int lim_np = SPR_LIMIT_NT / s->RT;
  if ((s->np + lim_np - 1) / lim_np > 65535)
    return pgpu_set_err(s->ctx, PGPU_ERR_LIMIT, "tbr: too many pattern blocks");
  const size_t smem = scan_smem<Pol>(a.depth, RT);
  const size_t need = scan_limit<Pol>(a.depth, std::max(p.max_moves_per_prune, 1), RT);
  if (need > s->ctx->smem_optin)
    return pgpu_set_err(s->ctx, PGPU_ERR_LIMIT, "tbr: walk needs %zu bytes of shared memory", need);
  PGPU_CUDA(s->ctx, cudaFuncSetAttribute(spr_scan_kernel<Pol, RT, true>,
                                         cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
  spr_scan_kernel<Pol, RT, true><<<dim3((unsigned)n_prunes, (unsigned)((a.n_blocks + a.G - 1) / a.G)), SPR_NT, smem,
                                   s->ctx->stream>>>(a);
  return pgpu_after_launch(s->ctx, "spr_scan_kernel (emit)");
}

template <typename Pol>
pgpu_status launch_tbr_batch(pgpu_spr *s, size_t c0, size_t c1, double *lnl_dev) {
  const TbrPlan &tp = s->tbr;
  const SprPlan &P = tp.emit;
  const int pb0 = tp.cuts[c0].pa, n_prunes = tp.cuts[c1 - 1].pb + 1 - pb0;
  const long long slot_base = P.prunes[pb0].move_off;
  switch (s->RT) {
    case 1: PGPU_TRY((launch_emit_rt<Pol, 1>(s, pb0, n_prunes, slot_base))); break;
    case 2: PGPU_TRY((launch_emit_rt<Pol, 2>(s, pb0, n_prunes, slot_base))); break;
    case 4: PGPU_TRY((launch_emit_rt<Pol, 4>(s, pb0, n_prunes, slot_base))); break;
    default: PGPU_TRY((launch_emit_rt<Pol, 8>(s, pb0, n_prunes, slot_base))); break;
  }
  // the batch's cuts and tiles, numbered by their pairs in the grid
  const long long move0 = tp.cuts[c0].grid_off;
  const long long nm = tp.cuts[c1 - 1].grid_off + (long long)tp.cuts[c1 - 1].nA * tp.cuts[c1 - 1].nB - move0;
  // the lists live in the engine; a copy from pageable memory returns once
  // its source has been staged, so the next batch may rewrite them
  std::vector<TbrCutDev> &cuts = s->h_tbr_cuts;
  std::vector<int4> &tiles = s->h_tbr_tiles;
  cuts.clear();
  tiles.clear();
  for (size_t c = c0; c < c1; ++c) {
    const TbrCut &x = tp.cuts[c];
    TbrCutDev d{};
    d.edge = x.edge;
    d.nA = x.nA;
    d.nB = x.nB;
    d.slotA = P.prunes[x.pa].move_off - slot_base;
    d.slotB = P.prunes[x.pb].move_off - slot_base;
    d.move_off = x.grid_off - move0;
    cuts.push_back(d);
    for (int j0 = 0; j0 < x.nA; j0 += TB_T)
      for (int k0 = 0; k0 < x.nB; k0 += TB_T) tiles.push_back(make_int4((int)(c - c0), j0, k0, 0));
  }
  if (tiles.size() > 0x7fffffffu) return pgpu_set_err(s->ctx, PGPU_ERR_LIMIT, "tbr: too many tiles");
  PGPU_TRY(grow(s, &s->tbr_cuts, &s->tbr_cuts_cap, cuts.size()));
  PGPU_TRY(grow(s, &s->tbr_tiles, &s->tbr_tiles_cap, tiles.size()));
  PGPU_CUDA(s->ctx, cudaMemcpyAsync(s->tbr_cuts, cuts.data(), cuts.size() * sizeof(TbrCutDev),
                                    cudaMemcpyHostToDevice, s->ctx->stream));
  PGPU_CUDA(s->ctx, cudaMemcpyAsync(s->tbr_tiles, tiles.data(), tiles.size() * sizeof(int4),
                                    cudaMemcpyHostToDevice, s->ctx->stream));
  // pattern groups: partial sums at most 256 MB
  const int n_pblocks = (int)(s->np / TB_PB);
  const size_t budget = size_t(256) << 20;
  int G = (int)std::max<size_t>(1, ((size_t)n_pblocks * (size_t)nm * 8 + budget - 1) / budget);
  G = std::min(G, n_pblocks);
  const int n_groups = (n_pblocks + G - 1) / G;
  if (n_groups > 65535) return pgpu_set_err(s->ctx, PGPU_ERR_LIMIT, "tbr: too many pattern groups");
  PGPU_TRY(grow(s, &s->partials, &s->part_cap, (size_t)n_groups * nm));
  PairArgs a;
  a.X = s->tbr_x;
  a.xsc = s->tbr_xsc;
  a.tiles = s->tbr_tiles;
  a.cuts = s->tbr_cuts;
  a.wts = s->w2;
  a.logtab = s->logtab;
  a.partials = s->partials;
  a.flag = s->ctx->d_flag;
  a.np = s->np;
  a.n_moves = nm;
  a.R = s->R;
  a.G = G;
  a.n_pblocks = n_pblocks;
  const size_t smem = pair_smem<Pol>(s->R);
  if (smem > s->ctx->smem_optin)
    return pgpu_set_err(s->ctx, PGPU_ERR_LIMIT, "tbr: pairs need %zu bytes of shared memory", smem);
  PGPU_CUDA(s->ctx, cudaFuncSetAttribute(tbr_pair_kernel<Pol>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                         (int)std::max<size_t>(smem, 48 * 1024)));
  tbr_pair_kernel<Pol><<<dim3((unsigned)tiles.size(), (unsigned)n_groups), 256, smem, s->ctx->stream>>>(a);
  PGPU_TRY(pgpu_after_launch(s->ctx, "tbr_pair_kernel"));
  spr_reduce_kernel<<<(unsigned)((nm + 31) / 32), dim3(32, RED_Y), 0, s->ctx->stream>>>(
      s->partials, n_groups, (size_t)nm, lnl_dev + move0);
  return pgpu_after_launch(s->ctx, "spr_reduce_kernel");
}

// out[m] = grid[keep[m]]: the listed moves' lnL out of every pair's
__global__ void __launch_bounds__(256) tbr_gather_kernel(const double *grid, const int64_t *keep,
                                                        size_t n, double *out) {
  for (size_t m = blockIdx.x * (size_t)blockDim.x + threadIdx.x; m < n;
       m += (size_t)gridDim.x * blockDim.x)
    out[m] = grid[keep[m]];
}

// lnL of every TBR move into lnl_dev, in batches of cuts whose attach
// vectors fit in the budget (at least one cut per batch); with two
// different limits every pair goes into the grid buffer first and the
// listed moves are gathered from it
pgpu_status run_tbr_scan(pgpu_spr *s, double *lnl_dev) {
  PGPU_TRY(ensure_pool(s, true));
  PGPU_TRY(ensure_tbr(s));
  const TbrPlan &tp = s->tbr;
  if (tp.n_moves == 0) return PGPU_OK;
  const bool filter = !tp.keep.empty();
  if (filter) PGPU_TRY(grow(s, &s->tbr_grid, &s->tbr_grid_cap, (size_t)tp.n_grid));
  double *out = filter ? s->tbr_grid : lnl_dev;
  const size_t slot_bytes = s->np * s->R * 4 * s->vbytes;
  const size_t max_slots = std::max<size_t>(1, s->tbr_budget / slot_bytes);
  for (size_t c0 = 0; c0 < tp.cuts.size();) {
    size_t c1 = c0, slots = 0;
    while (c1 < tp.cuts.size()) {
      const size_t add = (size_t)tp.cuts[c1].nA + tp.cuts[c1].nB;
      if (c1 > c0 && slots + add > max_slots) break;
      slots += add;
      ++c1;
    }
    PGPU_TRY(grow(s, &s->tbr_x, &s->tbr_x_cap, slots * slot_bytes));
    PGPU_TRY(grow(s, &s->tbr_xsc, &s->tbr_xsc_cap, slots * s->np));
    if (s->precision == 32) PGPU_TRY(launch_tbr_batch<Fp32>(s, c0, c1, out));
    else if (s->precision == 48) PGPU_TRY(launch_tbr_batch<Ff32>(s, c0, c1, out));
    else PGPU_TRY(launch_tbr_batch<Fp64>(s, c0, c1, out));
    c0 = c1;
  }
  if (filter) {
    const size_t n = (size_t)tp.n_moves;
    tbr_gather_kernel<<<(unsigned)std::min<size_t>((n + 255) / 256, 65535), 256, 0, s->ctx->stream>>>(
        s->tbr_grid, s->tbr_keep, n, lnl_dev);
    PGPU_TRY(pgpu_after_launch(s->ctx, "tbr_gather_kernel"));
  }
  return PGPU_OK;
}

pgpu_status ensure_fitch(pgpu_spr *s) {
  if (s->fitch_valid) return PGPU_OK;
  PGPU_TRY(ensure_pool(s));   // pool plan (ops, tips) must match the topology
  FitchTipArgs t;
  t.F = s->F;
  t.codes = s->codes;
  t.code_mask = s->cmask;
  t.tips = s->tips;
  t.W4 = s->W4;
  t.n_pat = s->n_pat;
  t.ld = s->ld;
  t.n_codes = s->n_codes;
  spr_fitch_tip_kernel<<<dim3((unsigned)((s->W4 + 7) / 8), (unsigned)s->n), 256, 0, s->ctx->stream>>>(t);
  PGPU_TRY(pgpu_after_launch(s->ctx, "spr_fitch_tip_kernel"));
  const int n_ops = (int)s->pp.ops.size();
  PGPU_CUDA(s->ctx, cudaMemsetAsync(s->cntF, 0, sizeof(unsigned long long) * (n_ops + 1), s->ctx->stream));
  FitchPoolArgs a;
  a.F = s->F;
  a.ops = s->ops;
  a.planes = s->planes;
  a.cnt = s->cntF;
  a.W4 = s->W4;
  a.n_ops = n_ops;
  a.n_planes = s->n_planes;
  spr_fitch_pool_kernel<<<(unsigned)((s->W4 + FPOOL_NT - 1) / FPOOL_NT), FPOOL_NT, 0, s->ctx->stream>>>(a);
  PGPU_TRY(pgpu_after_launch(s->ctx, "spr_fitch_pool_kernel"));
  const int nd = s->T.n_dedges();
  const size_t len_bytes = (size_t)nd * sizeof(unsigned long long);
  const bool in_shared = len_bytes <= 40 * 1024;   // within 48 KB beside the staged steps
  spr_fitch_len_kernel<<<1, FLEN_NT, in_shared ? len_bytes : 0, s->ctx->stream>>>(s->ops, n_ops, s->cntF, s->lenF, nd,
                                                                                 in_shared);
  PGPU_TRY(pgpu_after_launch(s->ctx, "spr_fitch_len_kernel"));
  s->fitch_valid = true;
  return PGPU_OK;
}

pgpu_status run_fitch_scan(pgpu_spr *s) {
  PGPU_TRY(ensure_fitch(s));
  PGPU_TRY(ensure_plan(s));
  const SprPlan &p = s->all;
  const size_t nm = p.moves.size();
  PGPU_CUDA(s->ctx, cudaMemsetAsync(s->ins, 0, sizeof(unsigned long long) * std::max<size_t>(nm, 1),
                                    s->ctx->stream));
  PGPU_CUDA(s->ctx, cudaMemsetAsync(s->join, 0,
                                    sizeof(unsigned long long) * std::max<size_t>(p.prunes.size(), 1),
                                    s->ctx->stream));
  if (nm == 0) return PGPU_OK;
  FitchScanArgs a;
  a.F = s->F;
  a.planes = s->planes;
  a.steps = s->all_d.steps;
  a.prunes = s->all_d.prunes;
  a.ins = s->ins;
  a.join = s->join;
  a.W4 = s->W4;
  a.n_planes = s->n_planes;
  a.depth = std::max(p.max_depth, 1);
  a.max_moves = std::max(p.max_moves_per_prune, 1);
  a.flag = s->ctx->d_flag;
  const size_t smem = a16((size_t)a.max_moves * 4) + (size_t)a.depth * 256 * sizeof(uint4);
  PGPU_CUDA(s->ctx, cudaFuncSetAttribute(spr_fitch_scan_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                         (int)std::max<size_t>(smem, 48 * 1024)));
  spr_fitch_scan_kernel<<<dim3((unsigned)p.prunes.size(), (unsigned)((s->W4 + 255) / 256)), 256, smem,
                          s->ctx->stream>>>(a);
  return pgpu_after_launch(s->ctx, "spr_fitch_scan_kernel");
}

pgpu_status sync_check(pgpu_spr *s, const char *what) {
  return pgpu_check_flag(s->ctx, what);
}

void invalidate(pgpu_spr *s) {
  s->pp_valid = s->pool_valid = s->half_valid = s->plan_valid = s->fitch_valid = s->summ_valid = s->tbr_valid = false;
}

}  // namespace

extern "C" {

pgpu_status pgpu_spr_create(pgpu_ctx *ctx, const pgpu_model *m, const pgpu_tip_codes *codes,
                            int32_t n_tips, const uint8_t *tip_codes_dev, size_t ld_pat,
                            const double *weights_dev, size_t n_pat, int precision, pgpu_spr **out) {
  if (!ctx || !out) return PGPU_ERR_ARG;
  *out = nullptr;
  if (!m || !m->Q || !m->pi || !m->rates || !m->probs || !codes || !codes->table || !tip_codes_dev)
    return pgpu_set_err(ctx, PGPU_ERR_ARG, "spr: null model, code table or tip codes");
  if (m->n_states != 4)
    return pgpu_set_err(ctx, PGPU_ERR_UNSUPPORTED, "spr: the SPR engine is built for 4 states (DNA)");
  if (m->n_rates < 1 || m->n_rates > 8)
    return pgpu_set_err(ctx, PGPU_ERR_LIMIT, "spr: 1..8 rate classes are supported");
  if (codes->n_codes < 1 || codes->n_codes > 256)
    return pgpu_set_err(ctx, PGPU_ERR_ARG, "spr: the code table needs 1..256 rows");
  if (precision != 32 && precision != 48 && precision != 64)
    return pgpu_set_err(ctx, PGPU_ERR_ARG, "spr: precision must be 32, 48 or 64");
  if (n_tips < 4) return pgpu_set_err(ctx, PGPU_ERR_ARG, "spr: need at least 4 tips");
  if (n_pat < 1 || ld_pat < n_pat) return pgpu_set_err(ctx, PGPU_ERR_ARG, "spr: need n_pat >= 1 and ld_pat >= n_pat");
  PGPU_CUDA(ctx, cudaSetDevice(ctx->device));
  pgpu_spr *s = new pgpu_spr();
  s->ctx = ctx;
  s->precision = precision;
  s->R = m->n_rates;
  s->RT = s->R <= 1 ? 1 : s->R <= 2 ? 2 : s->R <= 4 ? 4 : 8;
  s->NP = SPR_NT / s->RT;
  s->n = n_tips;
  s->n_codes = codes->n_codes;
  s->n_pat = n_pat;
  s->np = (n_pat + s->NP - 1) / s->NP * s->NP;
  s->ld = ld_pat;
  s->W4 = (n_pat + 31) / 32;
  s->codes = tip_codes_dev;
  s->vbytes = precision == 32 ? 4 : 8;
  s->cbytes = (size_t)s->R * 16 * (precision == 32 ? 4 : 8);
  auto fail = [&](pgpu_status st) {
    pgpu_spr_destroy(s);
    return st;
  };
#define SPR_TRY(x)                  \
  do {                              \
    pgpu_status st_ = (x);          \
    if (st_ != PGPU_OK) return fail(st_); \
  } while (0)
  const int R = s->R, nc = s->n_codes;
  const int ne = 2 * n_tips - 3, nd = 2 * ne;
  // model block
  double *blk;
  SPR_TRY(dalloc_t(s, 16 + 4 + 2 * 8 + (size_t)nc * 4 + 16 + 16 + 4 + 2, &blk));
  s->Q = blk;
  s->pi = s->Q + 16;
  s->rates = s->pi + 4;
  s->probs = s->rates + 8;
  s->ctab = s->probs + 8;
  s->U = s->ctab + (size_t)nc * 4;
  s->Ui = s->U + 16;
  s->lam = s->Ui + 16;
  s->status = reinterpret_cast<int *>(s->lam + 4);
  std::vector<double> hb(16 + 4 + 16 + (size_t)nc * 4, 0.0);
  std::copy(m->Q, m->Q + 16, hb.begin());
  std::copy(m->pi, m->pi + 4, hb.begin() + 16);
  std::copy(m->rates, m->rates + R, hb.begin() + 20);
  std::copy(m->probs, m->probs + R, hb.begin() + 28);
  std::copy(codes->table, codes->table + (size_t)nc * 4, hb.begin() + 36);
  SPR_TRY(upload(s, blk, hb.data(), hb.size()));
  SPR_TRY(pgpu_launch_eig(ctx, s->Q, s->pi, 4, 1, s->U, s->lam, s->Ui, s->status));
  std::vector<float2> ph(12, make_float2(0.0f, 0.0f));
  for (int i = 0; i < 4 + R; ++i) {
    const double v = i < 4 ? m->pi[i] : m->probs[i - 4];
    ph[i] = make_float2((float)v, (float)(v - (double)(float)v));
  }
  SPR_TRY(dalloc_t(s, ph.size(), &s->pairs));
  SPR_TRY(upload(s, s->pairs, ph.data(), ph.size()));
  // the code table in the form's layout (store4)
  std::vector<double> cr((size_t)nc * 4);   // room for the widest form
  for (int c = 0; c < nc; ++c)
    for (int i = 0; i < 4; ++i) {
      const double v = codes->table[(size_t)c * 4 + i];
      float *f = reinterpret_cast<float *>(cr.data());
      if (s->precision == 64) {
        cr[(size_t)c * 4 + i] = v;
      } else if (s->precision == 32) {
        f[(size_t)c * 4 + i] = (float)v;
      } else {
        float *q = f + (size_t)c * 8 + (i >> 1) * 4 + (i & 1);
        q[0] = (float)v;
        q[2] = (float)(v - (double)q[0]);
      }
    }
  double *crd;
  SPR_TRY(dalloc_t(s, cr.size(), &crd));
  SPR_TRY(upload(s, crd, cr.data(), cr.size()));
  s->crows = crd;
  // state-set masks of the codes
  std::vector<uint8_t> cm(nc);
  for (int c = 0; c < nc; ++c) {
    uint8_t b = 0;
    for (int i = 0; i < 4; ++i)
      if (codes->table[(size_t)c * 4 + i] > 0.0) b |= (uint8_t)(1u << i);
    cm[c] = b;
  }
  SPR_TRY(dalloc_t(s, (size_t)nc, &s->cmask));
  SPR_TRY(upload(s, s->cmask, cm.data(), cm.size()));
  // weights: FP64 and float-pair copies padded with zeros; integer bit planes for Fitch
  std::vector<double> wh(s->np, 0.0);
  if (weights_dev) {
    if (cudaMemcpy(wh.data(), weights_dev, n_pat * 8, cudaMemcpyDeviceToHost) != cudaSuccess) {
      (void)cudaGetLastError();
      return fail(pgpu_set_err(ctx, PGPU_ERR_CUDA, "spr: weights_dev is not readable device memory"));
    }
  } else {
    std::fill(wh.begin(), wh.begin() + n_pat, 1.0);
  }
  uint64_t wmax = 0;
  for (size_t i = 0; i < n_pat; ++i) {
    if (!(wh[i] >= 0.0) || wh[i] > 1e9) return fail(pgpu_set_err(ctx, PGPU_ERR_ARG, "spr: weight %zu is negative or too large", i));
    s->wtot += wh[i];
    wmax = std::max<uint64_t>(wmax, (uint64_t)llround(wh[i]));
  }
  std::vector<float2> w2h(s->np);
  for (size_t i = 0; i < s->np; ++i) w2h[i] = make_float2((float)wh[i], (float)(wh[i] - (double)(float)wh[i]));
  SPR_TRY(dalloc_t(s, s->np, &s->w));
  SPR_TRY(upload(s, s->w, wh.data(), wh.size()));
  SPR_TRY(dalloc_t(s, s->np, &s->w2));
  SPR_TRY(upload(s, s->w2, w2h.data(), w2h.size()));
  std::vector<float> w3h(s->np);
  bool rest = false;
  for (size_t i = 0; i < s->np; ++i) {
    w3h[i] = (float)(wh[i] - (double)w2h[i].x - (double)w2h[i].y);
    rest |= w3h[i] != 0.0f;
  }
  if (rest) {
    SPR_TRY(dalloc_t(s, s->np, &s->w3));
    SPR_TRY(upload(s, s->w3, w3h.data(), w3h.size()));
  }
  s->n_planes = 1;
  while ((wmax >> s->n_planes) != 0) ++s->n_planes;
  std::vector<uint32_t> planes((size_t)s->n_planes * s->W4, 0u);
  for (size_t i = 0; i < n_pat; ++i) {
    const uint64_t wi = (uint64_t)llround(wh[i]);
    for (int b = 0; b < s->n_planes; ++b)
      if ((wi >> b) & 1u) planes[(size_t)b * s->W4 + i / 32] |= 1u << (i % 32);
  }
  SPR_TRY(dalloc_t(s, (size_t)s->n_planes * s->W4, &s->planes));
  SPR_TRY(upload(s, s->planes, planes.data(), planes.size()));
  // logarithm table of the pair form
  std::vector<float4> lt(64);
  ff_log_table(lt.data(), [](double c) { return std::log(c); });
  SPR_TRY(dalloc_t(s, 64, &s->logtab));
  SPR_TRY(upload(s, s->logtab, lt.data(), lt.size()));
  // pool and tables
  const size_t vec = (size_t)nd * s->np * R * 4 * s->vbytes;
  SPR_TRY(dalloc(s, vec, &s->L));
  SPR_TRY(dalloc(s, vec, &s->M));
  SPR_TRY(dalloc(s, vec, &s->H));
  SPR_TRY(dalloc_t(s, (size_t)nd * s->np, &s->sc));
  SPR_TRY(dalloc(s, 2 * (size_t)ne * s->cbytes, &s->Dfull));
  const size_t tt = (size_t)n_tips * R * nc * 4 * s->vbytes;
  SPR_TRY(dalloc(s, tt, &s->tipfull));
  SPR_TRY(dalloc(s, tt, &s->tiphalf));
  SPR_TRY(dalloc_t(s, 2 * (size_t)ne + 2 * (size_t)n_tips, &s->elen));
  SPR_TRY(dalloc_t(s, (size_t)ne, &s->newlen));
  SPR_TRY(dalloc_t(s, (size_t)nd, &s->ops));
  SPR_TRY(dalloc_t(s, (size_t)nd, &s->half_list));
  SPR_TRY(dalloc_t(s, (size_t)n_tips, &s->tips));
  SPR_TRY(dalloc_t(s, s->np / s->NP, &s->pool_part));
  SPR_TRY(dalloc_t(s, 1, &s->tree_lnl));
  SPR_TRY(dalloc_t(s, s->np, &s->site_lnl));
  SPR_TRY(dalloc_t(s, (size_t)nd * s->W4, &s->F));
  SPR_TRY(dalloc_t(s, (size_t)nd + 1, &s->cntF));
  SPR_TRY(dalloc_t(s, (size_t)nd + 1, &s->lenF));
  SPR_TRY(dalloc_t(s, (size_t)nd * 4, &s->summ));
  const size_t max_moves = (size_t)nd * 2 * n_tips, max_prunes = (size_t)nd;
  SPR_TRY(dalloc_t(s, max_moves, &s->ins));
  SPR_TRY(dalloc_t(s, max_prunes, &s->join));
  int st = 0;
  if (cudaStreamSynchronize(ctx->stream) != cudaSuccess ||
      cudaMemcpy(&st, s->status, sizeof(int), cudaMemcpyDeviceToHost) != cudaSuccess) {
    (void)cudaGetLastError();
    return fail(pgpu_set_err(ctx, PGPU_ERR_CUDA, "spr: set-up failed on the device"));
  }
  SPR_TRY(pgpu_check_flag(ctx, "spr_create"));
  if (st != 0) return fail(pgpu_set_err(ctx, (pgpu_status)st, "spr: the rate matrix could not be diagonalised"));
#undef SPR_TRY
  *out = s;
  return PGPU_OK;
}

void pgpu_spr_destroy(pgpu_spr *s) {
  if (!s) return;
  if (s->ctx) cudaSetDevice(s->ctx->device);
  for (void *p : s->owned) cudaFree(p);
  delete s;
}

pgpu_status pgpu_spr_set_tree(pgpu_spr *s, const pgpu_tree *tree) {
  if (!s) return PGPU_ERR_ARG;
  if (!tree || tree->n_tips != s->n)
    return pgpu_set_err(s->ctx, PGPU_ERR_ARG, "spr: tree must have %d tips", s->n);
  SprTopo T;
  PGPU_TRY(spr_from_rooted(s->ctx, tree, &T));
  s->T = std::move(T);
  invalidate(s);
  return PGPU_OK;
}

pgpu_status pgpu_spr_get_tree(pgpu_spr *s, int32_t *left, int32_t *right, double *brlen) {
  if (!s || !left || !right || !brlen) return PGPU_ERR_ARG;
  if (s->T.n == 0) return pgpu_set_err(s->ctx, PGPU_ERR_ARG, "spr: no tree set");
  spr_to_rooted(s->T, left, right, brlen);
  return PGPU_OK;
}

pgpu_status pgpu_spr_lnl(pgpu_spr *s, double *lnl, double *site_lnl) {
  if (!s || !lnl) return PGPU_ERR_ARG;
  if (s->T.n == 0) return pgpu_set_err(s->ctx, PGPU_ERR_ARG, "spr: no tree set");
  PGPU_CUDA(s->ctx, cudaSetDevice(s->ctx->device));
  PGPU_TRY(ensure_pool(s));
  double *h = reinterpret_cast<double *>(s->ctx->h_pinned);
  PGPU_CUDA(s->ctx, cudaMemcpyAsync(h, s->tree_lnl, 8, cudaMemcpyDeviceToHost, s->ctx->stream));
  if (site_lnl)
    PGPU_CUDA(s->ctx, cudaMemcpyAsync(site_lnl, s->site_lnl, s->n_pat * 8, cudaMemcpyDeviceToHost, s->ctx->stream));
  PGPU_TRY(sync_check(s, "spr_lnl"));
  *lnl = *h;
  return PGPU_OK;
}

pgpu_status pgpu_spr_n_moves(pgpu_spr *s, size_t *n_moves) {
  if (!s || !n_moves) return PGPU_ERR_ARG;
  if (s->T.n == 0) return pgpu_set_err(s->ctx, PGPU_ERR_ARG, "spr: no tree set");
  PGPU_CUDA(s->ctx, cudaSetDevice(s->ctx->device));
  PGPU_TRY(ensure_plan(s));
  *n_moves = s->all.moves.size();
  return PGPU_OK;
}

pgpu_status pgpu_spr_moves(pgpu_spr *s, int32_t *p, int32_t *u, int32_t *c, int32_t *y, size_t cap) {
  if (!s || !p || !u || !c || !y) return PGPU_ERR_ARG;
  size_t nm = 0;
  PGPU_TRY(pgpu_spr_n_moves(s, &nm));
  if (cap < nm) return pgpu_set_err(s->ctx, PGPU_ERR_ARG, "spr: %zu moves, room for %zu", nm, cap);
  const int n = s->n;
  std::vector<int32_t> l(n - 1), r(n - 1), ids(2 * n - 2);
  std::vector<double> b(2 * n - 2);
  spr_to_rooted(s->T, l.data(), r.data(), b.data(), ids.data());
  for (size_t i = 0; i < nm; ++i) {
    const SprMove &mv = s->all.moves[i];
    const int dp = s->all.prunes[mv.prune].dp;
    p[i] = ids[s->T.dsrc(dp)];
    u[i] = ids[s->T.ddst(dp)];
    c[i] = ids[s->T.dsrc(mv.dc)];
    y[i] = ids[s->T.ddst(mv.dc)];
  }
  return PGPU_OK;
}

pgpu_status pgpu_spr_scan(pgpu_spr *s, double *lnl_dev) {
  if (!s || !lnl_dev) return PGPU_ERR_ARG;
  if (s->T.n == 0) return pgpu_set_err(s->ctx, PGPU_ERR_ARG, "spr: no tree set");
  PGPU_CUDA(s->ctx, cudaSetDevice(s->ctx->device));
  PGPU_TRY(ensure_pool(s, true));
  PGPU_TRY(ensure_plan(s));
  PGPU_TRY(run_scan(s, s->all, s->all_d, lnl_dev));
  return sync_check(s, "spr_scan");
}

pgpu_status pgpu_spr_score(pgpu_spr *s, const int64_t *move_idx, size_t k, double *lnl) {
  if (!s || (k && (!move_idx || !lnl))) return PGPU_ERR_ARG;
  if (s->T.n == 0) return pgpu_set_err(s->ctx, PGPU_ERR_ARG, "spr: no tree set");
  PGPU_CUDA(s->ctx, cudaSetDevice(s->ctx->device));
  if (k) PGPU_TRY(ensure_pool(s, k >= (size_t)s->T.n_dedges()));
  PGPU_TRY(ensure_plan(s));
  if (k == 0) return PGPU_OK;
  const size_t nm = s->all.moves.size();
  std::vector<int32_t> dp(k), dc(k);
  for (size_t i = 0; i < k; ++i) {
    if (move_idx[i] < 0 || (size_t)move_idx[i] >= nm)
      return pgpu_set_err(s->ctx, PGPU_ERR_ARG, "spr: move index %lld out of range", (long long)move_idx[i]);
    const SprMove &mv = s->all.moves[move_idx[i]];
    dp[i] = s->all.prunes[mv.prune].dp;
    dc[i] = mv.dc;
  }
  PGPU_TRY(spr_plan_selected(s->ctx, s->T, s->pp, dp.data(), dc.data(), (int)k, &s->sel));
  PGPU_TRY(upload_plan(s, s->sel, &s->sel_d));
  const size_t ns = s->sel.moves.size();
  double *out_dev;
  PGPU_TRY(pgpu_buf(s->ctx, BUF_OUT, std::max<size_t>(ns, 1) * 8, reinterpret_cast<void **>(&out_dev)));
  PGPU_TRY(run_scan(s, s->sel, s->sel_d, out_dev));
  std::vector<double> got(ns);
  PGPU_CUDA(s->ctx, cudaMemcpyAsync(got.data(), out_dev, ns * 8, cudaMemcpyDeviceToHost, s->ctx->stream));
  PGPU_TRY(sync_check(s, "spr_score"));
  // emitted order -> caller's order (the same move may be asked for twice)
  for (size_t i = 0; i < k; ++i) lnl[i] = NAN;
  for (size_t j = 0; j < ns; ++j) {
    const SprMove &mv = s->sel.moves[j];
    const int pdp = s->sel.prunes[mv.prune].dp;
    for (size_t i = 0; i < k; ++i)
      if (dp[i] == pdp && dc[i] == mv.dc) lnl[i] = got[j];
  }
  return PGPU_OK;
}

pgpu_status pgpu_spr_fitch(pgpu_spr *s, uint64_t *len_dev, uint64_t *tree_len) {
  if (!s || !len_dev) return PGPU_ERR_ARG;
  if (s->T.n == 0) return pgpu_set_err(s->ctx, PGPU_ERR_ARG, "spr: no tree set");
  PGPU_CUDA(s->ctx, cudaSetDevice(s->ctx->device));
  PGPU_TRY(run_fitch_scan(s));
  const size_t nm = s->all.moves.size();
  if (nm) {
    spr_fitch_moves_kernel<<<(unsigned)((nm + 255) / 256), 256, 0, s->ctx->stream>>>(
        s->all_d.moves, s->all_d.prunes, nm, s->lenF, s->ins, s->join,
        reinterpret_cast<unsigned long long *>(len_dev));
    PGPU_TRY(pgpu_after_launch(s->ctx, "spr_fitch_moves_kernel"));
  }
  uint64_t *h = reinterpret_cast<uint64_t *>(s->ctx->h_pinned);
  PGPU_CUDA(s->ctx, cudaMemcpyAsync(h, s->lenF + s->T.n_dedges(), 8, cudaMemcpyDeviceToHost, s->ctx->stream));
  PGPU_TRY(sync_check(s, "spr_fitch"));
  if (tree_len) *tree_len = *h;
  return PGPU_OK;
}

pgpu_status pgpu_spr_features(pgpu_spr *s, float *X_dev) {
  if (!s || !X_dev) return PGPU_ERR_ARG;
  if (s->T.n == 0) return pgpu_set_err(s->ctx, PGPU_ERR_ARG, "spr: no tree set");
  PGPU_CUDA(s->ctx, cudaSetDevice(s->ctx->device));
  PGPU_TRY(run_fitch_scan(s));
  if (!s->summ_valid) {
    SummaryArgs a;
    a.L = s->L;
    a.probs = s->probs;
    a.weights = s->w2;
    a.wd = s->w;
    a.out = s->summ;
    a.np = s->np;
    a.n_pat = s->n_pat;
    a.R = s->R;
    a.RT = s->RT;
    a.rt_shift = s->RT == 1 ? 0 : s->RT == 2 ? 1 : s->RT == 4 ? 2 : 3;
    a.inv_w = s->wtot > 0 ? 1.0 / s->wtot : 0.0;
    const unsigned nd = (unsigned)s->T.n_dedges();
    if (s->precision == 32) spr_summary_kernel<Fp32><<<nd, 256, 0, s->ctx->stream>>>(a);
    else if (s->precision == 48) spr_summary_kernel<Ff32><<<nd, 256, 0, s->ctx->stream>>>(a);
    else spr_summary_kernel<Fp64><<<nd, 256, 0, s->ctx->stream>>>(a);
    PGPU_TRY(pgpu_after_launch(s->ctx, "spr_summary_kernel"));
    s->summ_valid = true;
  }
  const size_t nm = s->all.moves.size();
  if (nm == 0) return sync_check(s, "spr_features");
  // edge lengths as doubles on the device: the first n_edges entries of elen
  FeatArgs f;
  f.moves = s->all_d.moves;
  f.prunes = s->all_d.prunes;
  int32_t *tc;
  PGPU_TRY(pgpu_buf(s->ctx, BUF_A, s->pp.tipcnt.size() * 4, reinterpret_cast<void **>(&tc)));
  PGPU_TRY(upload(s, tc, s->pp.tipcnt.data(), s->pp.tipcnt.size()));
  f.tipcnt = tc;
  f.len = s->elen;
  f.summ = s->summ;
  f.lenF = s->lenF;
  f.ins = s->ins;
  f.join = s->join;
  f.X = X_dev;
  f.n_moves = nm;
  f.n_tips = s->n;
  f.nd = s->T.n_dedges();
  f.wtot = s->wtot > 0 ? s->wtot : 1.0;
  spr_feature_kernel<<<(unsigned)((nm + 255) / 256), 256, 0, s->ctx->stream>>>(f);
  PGPU_TRY(pgpu_after_launch(s->ctx, "spr_feature_kernel"));
  return sync_check(s, "spr_features");
}

pgpu_status pgpu_spr_set_join_distance(pgpu_spr *s, int join_distance) {
  if (!s) return PGPU_ERR_ARG;
  if (join_distance < 0)
    return pgpu_set_err(s->ctx, PGPU_ERR_ARG, "spr: join distance %d < 0", join_distance);
  if (join_distance != s->join_distance) {
    s->join_distance = join_distance;
    s->plan_valid = false;
  }
  return PGPU_OK;
}

pgpu_status pgpu_spr_set_tbr_limits(pgpu_spr *s, int join_distance, int reroot_distance) {
  if (!s) return PGPU_ERR_ARG;
  if (join_distance < 0 || reroot_distance < 0)
    return pgpu_set_err(s->ctx, PGPU_ERR_ARG, "tbr: limits %d, %d must be >= 0", join_distance,
                        reroot_distance);
  if (join_distance != s->tbr_join || reroot_distance != s->tbr_reroot) {
    s->tbr_join = join_distance;
    s->tbr_reroot = reroot_distance;
    s->tbr_valid = false;
  }
  return PGPU_OK;
}

pgpu_status pgpu_spr_set_tbr_distance(pgpu_spr *s, int distance) {
  if (!s) return PGPU_ERR_ARG;
  if (distance < 0) return pgpu_set_err(s->ctx, PGPU_ERR_ARG, "tbr: distance %d < 0", distance);
  return pgpu_spr_set_tbr_limits(s, distance, distance);
}

pgpu_status pgpu_spr_set_tbr_budget(pgpu_spr *s, size_t bytes) {
  if (!s) return PGPU_ERR_ARG;
  s->tbr_budget = bytes ? bytes : size_t(2) << 30;
  return PGPU_OK;
}

pgpu_status pgpu_spr_tbr_n_moves(pgpu_spr *s, size_t *n_moves) {
  if (!s || !n_moves) return PGPU_ERR_ARG;
  if (s->T.n == 0) return pgpu_set_err(s->ctx, PGPU_ERR_ARG, "spr: no tree set");
  PGPU_CUDA(s->ctx, cudaSetDevice(s->ctx->device));
  PGPU_TRY(ensure_tbr(s));
  *n_moves = (size_t)s->tbr.n_moves;
  return PGPU_OK;
}

pgpu_status pgpu_spr_tbr_moves(pgpu_spr *s, int32_t *a, int32_t *b, int32_t *jc, int32_t *jy, int32_t *kc,
                               int32_t *ky, size_t cap) {
  if (!s || !a || !b || !jc || !jy || !kc || !ky) return PGPU_ERR_ARG;
  size_t nm = 0;
  PGPU_TRY(pgpu_spr_tbr_n_moves(s, &nm));
  if (cap < nm) return pgpu_set_err(s->ctx, PGPU_ERR_ARG, "tbr: %zu moves, room for %zu", nm, cap);
  const int n = s->n;
  std::vector<int32_t> l(n - 1), r(n - 1), ids(2 * n - 2);
  std::vector<double> bl(2 * n - 2);
  spr_to_rooted(s->T, l.data(), r.data(), bl.data(), ids.data());
  const SprPlan &P = s->tbr.emit;
  const std::vector<int64_t> &keep = s->tbr.keep;
  size_t m = 0;   // listed moves, in grid order
  for (const TbrCut &c : s->tbr.cuts) {
    const int ia = ids[s->T.ea[c.edge]], ib = ids[s->T.eb[c.edge]];
    for (int j = 0; j < c.nA; ++j) {
      const int dj = P.moves[P.prunes[c.pa].move_off + j].dc;
      for (int k = 0; k < c.nB; ++k) {
        if (!keep.empty() && (m >= keep.size() || keep[m] != c.grid_off + (int64_t)j * c.nB + k))
          continue;
        const int dk = P.moves[P.prunes[c.pb].move_off + k].dc;
        a[m] = ia;
        b[m] = ib;
        jc[m] = ids[s->T.dsrc(dj)];
        jy[m] = ids[s->T.ddst(dj)];
        kc[m] = ids[s->T.dsrc(dk)];
        ky[m] = ids[s->T.ddst(dk)];
        ++m;
      }
    }
  }
  return PGPU_OK;
}

pgpu_status pgpu_spr_tbr_scan(pgpu_spr *s, double *lnl_dev) {
  if (!s || !lnl_dev) return PGPU_ERR_ARG;
  if (s->T.n == 0) return pgpu_set_err(s->ctx, PGPU_ERR_ARG, "spr: no tree set");
  PGPU_CUDA(s->ctx, cudaSetDevice(s->ctx->device));
  PGPU_TRY(run_tbr_scan(s, lnl_dev));
  return sync_check(s, "pgpu_spr_tbr_scan");
}

pgpu_status pgpu_spr_tbr_apply(pgpu_spr *s, int64_t move_idx) {
  if (!s) return PGPU_ERR_ARG;
  size_t nm = 0;
  PGPU_TRY(pgpu_spr_tbr_n_moves(s, &nm));
  if (move_idx < 0 || (size_t)move_idx >= nm)
    return pgpu_set_err(s->ctx, PGPU_ERR_ARG, "tbr: move index %lld out of range", (long long)move_idx);
  const std::vector<TbrCut> &cuts = s->tbr.cuts;
  const int64_t g = s->tbr.keep.empty() ? move_idx : s->tbr.keep[(size_t)move_idx];
  size_t c = std::upper_bound(cuts.begin(), cuts.end(), g,
                              [](int64_t v, const TbrCut &x) { return v < x.grid_off; }) -
             cuts.begin() - 1;
  const TbrCut &x = cuts[c];
  const int64_t rel = g - x.grid_off;
  const SprPlan &P = s->tbr.emit;
  const int dj = P.moves[P.prunes[x.pa].move_off + (int)(rel / x.nB)].dc;
  const int dk = P.moves[P.prunes[x.pb].move_off + (int)(rel % x.nB)].dc;
  PGPU_TRY(tbr_apply(s->ctx, &s->T, x.edge, dj, dk));
  invalidate(s);
  return PGPU_OK;
}

pgpu_status pgpu_spr_apply(pgpu_spr *s, int64_t move_idx) {
  if (!s) return PGPU_ERR_ARG;
  size_t nm = 0;
  PGPU_TRY(pgpu_spr_n_moves(s, &nm));
  if (move_idx < 0 || (size_t)move_idx >= nm)
    return pgpu_set_err(s->ctx, PGPU_ERR_ARG, "spr: move index %lld out of range", (long long)move_idx);
  const SprMove mv = s->all.moves[move_idx];
  PGPU_TRY(spr_apply(s->ctx, &s->T, s->all.prunes[mv.prune].dp, mv.dc));
  invalidate(s);
  return PGPU_OK;
}

pgpu_status pgpu_spr_optimize(pgpu_spr *s, int passes, double tol, double *lnl_out) {
  if (!s) return PGPU_ERR_ARG;
  if (s->T.n == 0) return pgpu_set_err(s->ctx, PGPU_ERR_ARG, "spr: no tree set");
  PGPU_CUDA(s->ctx, cudaSetDevice(s->ctx->device));
  const int ne = s->T.n_edges();
  if (!s->S) PGPU_TRY(dalloc_t(s, (size_t)ne * s->np * s->R * 4, &s->S));
  double cur = 0.0;
  PGPU_TRY(pgpu_spr_lnl(s, &cur, nullptr));
  std::vector<double> old(s->T.len), nl(ne);
  for (int pass = 0; pass < passes; ++pass) {
    BlArgs a;
    a.L = s->L;
    a.U = s->U;
    a.Ui = s->Ui;
    a.lam = s->lam;
    a.pi = s->pi;
    a.rates = s->rates;
    a.probs = s->probs;
    a.w2 = s->w2;
    a.w3 = s->w3;
    a.S = s->S;
    a.len_in = s->elen;
    a.len_out = s->newlen;
    a.np = s->np;
    a.n_pat = s->n_pat;
    a.R = s->R;
    a.n_edges = ne;
    a.iters = 8;
    a.tol = 1e-6;
    a.tmin = 1e-8;
    a.tmax = 10.0;
    const dim3 g((unsigned)((s->np * s->R + 255) / 256), (unsigned)ne);
    if (s->precision == 32) bl_sumtab_pair_kernel<Fp32><<<g, 256, 0, s->ctx->stream>>>(a);
    else if (s->precision == 48) bl_sumtab_pair_kernel<Ff32><<<g, 256, 0, s->ctx->stream>>>(a);
    else bl_sumtab_kernel<<<g, 256, 0, s->ctx->stream>>>(a);
    PGPU_TRY(pgpu_after_launch(s->ctx, "bl_sumtab_kernel"));
    bl_newton_kernel<<<(unsigned)ne, 256, 0, s->ctx->stream>>>(a);
    PGPU_TRY(pgpu_after_launch(s->ctx, "bl_newton_kernel"));
    PGPU_CUDA(s->ctx, cudaMemcpyAsync(nl.data(), s->newlen, ne * 8, cudaMemcpyDeviceToHost, s->ctx->stream));
    PGPU_TRY(sync_check(s, "spr_optimize"));
    old = s->T.len;
    // take the joint Newton step; halve it until the likelihood rises
    double alpha = 1.0, got = cur;
    bool accepted = false;
    for (int tries = 0; tries < 10 && !accepted; ++tries, alpha *= 0.5) {
      for (int e = 0; e < ne; ++e) s->T.len[e] = old[e] + alpha * (nl[e] - old[e]);
      invalidate(s);
      PGPU_TRY(pgpu_spr_lnl(s, &got, nullptr));
      accepted = got > cur;
    }
    // the edges' steps interfere: take them a quarter of the edges at a time
    for (int g = 0; g < 4 && !accepted; ++g) {
      s->T.len = old;
      for (int e = g; e < ne; e += 4) s->T.len[e] = nl[e];
      invalidate(s);
      PGPU_TRY(pgpu_spr_lnl(s, &got, nullptr));
      accepted = got > cur;
    }
    if (!accepted) {   // no step improves: converged as far as Newton can see
      s->T.len = old;
      invalidate(s);
      PGPU_TRY(pgpu_spr_lnl(s, &got, nullptr));
      break;
    }
    const double gain = got - cur;
    cur = got;
    if (gain < tol) break;
  }
  if (lnl_out) *lnl_out = cur;
  return PGPU_OK;
}

pgpu_status pgpu_spr_lengths(pgpu_spr *s, double *len, int32_t *ea, int32_t *eb) {
  if (!s || !len) return PGPU_ERR_ARG;
  const int ne = s->T.n_edges();
  std::copy(s->T.len.begin(), s->T.len.end(), len);
  if (ea) std::copy(s->T.ea.begin(), s->T.ea.end(), ea);
  if (eb) std::copy(s->T.eb.begin(), s->T.eb.end(), eb);
  (void)ne;
  return PGPU_OK;
}

}  // extern "C"
