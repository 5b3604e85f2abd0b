// Likelihood_c one node at a time: the NodeData.S operator
// (lib/nodeData.ml:20-30) whose slot lib/likelihood_c.ml:14-21 leaves as
// `failwith "TODO"`.
//
//   m  (pgpu_lk)   the substitution model's eigen system (FP64, on the GPU),
//                  its rate classes, the tip-code table and the character
//                  block's pattern count and weights;
//   t  (pgpu_clv)  one node's conditional likelihoods on the device,
//                  [n_pat][R][S] in the storage type (float or double), a
//                  power-of-two exponent per pattern, the length of the
//                  branch above the node and that branch's P matrices.
//
// median_1/2/3 combine one, two or three neighbours: y = prod_k P(t_k) x_k
// per pattern and rate class.  Every result is normalised so that each
// pattern's largest entry lies in [1/2, 1): stored = true * 2^-E with an
// exact power of two e_p applied at the node and E summed over the subtree.
// The node's cost is what its own normalisation moved out of the
// likelihood, -ln 2 sum_p w_p e_p, and root_cost is
// -sum_p w_p log(sum_r probs_r sum_i pi_i stored).  The costs of all
// internal nodes plus the root's root_cost are then -lnL, which is how
// Node.Make1D sums node costs (lib/node.ml:191).
//
// One thread per (pattern, rate class): RL = the power of two >= R lanes
// per pattern, so a pattern's maximum is a shuffle over its lanes.  Loads
// of a child's vector are contiguous per thread and contiguous across the
// warp.  Integer weights make a node's cost an exact integer sum, one atomic
// add per CTA; with fractional weights each CTA writes a compensated partial
// and the last CTA adds them in CTA order, so costs are deterministic.
//
// Four states (clv_median4_kernel): a branch's P matrices are 16 numbers per
// rate class, formed on the host when its length is set and passed with the
// launch, and a leaf is its codes -- a CTA forms P x for every code in shared
// memory -- so a leaf is one copy, a branch length no device work, and a
// median one launch that reads n_pat bytes for a leaf instead of n_pat R S
// values.  Other state counts build P in a launch per branch and store
// leaves as vectors.
//
// Handles are allocated stream-ordered (cudaMallocAsync) on the context's
// stream; passing the node's previous value (the reference's `t option`)
// reuses its memory instead.
#include <algorithm>
#include <cmath>
#include <cstring>
#include <vector>

#include "pgpu_internal.cuh"
#include "forms.cuh"
#include "pmatrix.cuh"

using namespace pgpu_forms;

struct pgpu_lk {
  pgpu_ctx *ctx = nullptr;
  int S = 0, R = 0, RL = 1, n_codes = 0, precision = 64;
  size_t n_pat = 0;
  double *block = nullptr;   // U, Ui, lam, pi, rates, probs, code table, weights
  double *U = nullptr, *Ui = nullptr, *lam = nullptr, *pi = nullptr, *rates = nullptr,
         *probs = nullptr, *tab = nullptr, *weights = nullptr;
  int *status = nullptr;     // eigendecomposition status
  double2 *part = nullptr;   // per-CTA partial sums
  // integer weights (pattern counts): the node costs are summed exactly as
  // sum_p w_p e_p in int64 on the integer units, the FP64 units being slow
  bool int_w = false;
  int32_t *wint = nullptr;   // [n_pat] or null (all 1)
  unsigned *counter = nullptr;
  size_t n_cta = 0;
  long long live = 0;        // handles not yet destroyed
  double *zero = nullptr;    // a leaf's cost
  // four states: the eigen system on the host, the code table in the storage
  // type, and whether leaves stay codes (their rows fit shared memory)
  double hU[16] = {}, hUi[16] = {}, hlam[4] = {}, hrates[8] = {};
  void *tabv = nullptr;
  bool leaf_codes = false;
  int resident[3] = {};      // CTAs of clv_median4_kernel per SM, by neighbour count (0: not asked yet)
};

struct pgpu_clv {
  pgpu_lk *lk = nullptr;
  char *mem = nullptr;       // stream-ordered: scalars, P, codes
  char *vec = nullptr;       // stream-ordered: x, ex (allocated when first needed)
  void *x = nullptr;         // [n_pat][R][S]
  int32_t *ex = nullptr;     // [n_pat]
  void *P = nullptr;         // [R][S][S] of the branch above (not for 4 states)
  uint8_t *codes = nullptr;  // a leaf's codes (4 states)
  // [0], [1] the cost: a double in [0], or with integer weights an int64 in
  // [slot] (a median adds to the other slot, which the median before it
  // cleared); [2] root cost, [3] branch length
  double *scal = nullptr;
  int slot = 0;
  double P4[8][16];          // P of the branch above, 4 states
  double brlen = 0.0;
  bool has_P = false;
  bool leaf = false;
  bool expanded = false;     // a leaf whose vector is in x
  // a leaf with codes outside the table that nothing has read or reported yet:
  // the context's count of reports when it was made, else -1
  long long bad = -1;
};

namespace {

constexpr int CLV_THREADS = 256;

size_t al256(size_t x) { return (x + 255) & ~size_t(255); }

size_t vbytes(const pgpu_lk *lk) { return lk->precision == 32 ? 4 : 8; }

template <typename V> __device__ __forceinline__ V scale2(V v, int e);
template <> __device__ __forceinline__ float scale2<float>(float v, int e) {
  // v * 2^e, exact; e beyond a float exponent's range (a denormal maximum)
  // takes two steps
  if (e > 126) {
    v *= pow2f(126);
    e -= 126;
  } else if (e < -126) {
    v *= pow2f(-126);
    e += 126;
  }
  return v * pow2f(e);
}
template <> __device__ __forceinline__ double scale2<double>(double v, int e) { return ldexp(v, e); }

// Compensated sum of (s, c) over the CTA into part[blockIdx.x]; the last
// CTA adds all partials in order into *out (times `sign`) and resets the
// counter.
template <int NT>
__device__ __forceinline__ void cta_partial_and_finish(double s, double c, double2 *part,
                                                       unsigned *counter, double *out,
                                                       double sign) {
  __shared__ double2 red[NT / 32];
  __shared__ bool last;
  warp_csum(s, c);
  const int t = threadIdx.x, lane = t & 31;
  if (lane == 0) red[t >> 5] = make_double2(s, c);
  __syncthreads();
  if (t < 32) {
    double2 v = lane < NT / 32 ? red[lane] : make_double2(0.0, 0.0);
    double ss = v.x, cc = v.y;
    warp_csum(ss, cc);
    if (lane == 0) {
      part[blockIdx.x] = make_double2(ss, cc);
      __threadfence();
      last = atomicAdd(counter, 1u) == gridDim.x - 1;
    }
  }
  __syncthreads();
  if (!last) return;
  __threadfence();
  const double tot = csum_block<NT>(part, gridDim.x);
  if (t == 0) {
    *out = sign * tot;
    *counter = 0u;
  }
}

// An exact integer sum v over the CTA, added to *acc.
template <int NT>
__device__ __forceinline__ void cta_add_i64(long long v, long long *acc) {
  __shared__ long long red[NT / 32];
  const int t = threadIdx.x, lane = t & 31;
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  if (lane == 0) red[t >> 5] = v;
  __syncthreads();
  if (t < 32) {
    long long x = lane < NT / 32 ? red[lane] : 0;
#pragma unroll
    for (int o = NT / 64; o > 0; o >>= 1) x += __shfl_xor_sync(0xffffffffu, x, o);
    if (lane == 0 && x) atomicAdd(reinterpret_cast<unsigned long long *>(acc), (unsigned long long)x);
  }
}

// Leaf vectors: x[p][r][i] = code_tab[code_p][i] for every rate class.
template <typename V>
__global__ void __launch_bounds__(CLV_THREADS) clv_leaf_kernel(const uint8_t *codes,
                                                               const double *tab, int n_codes,
                                                               size_t n_pat, int S, int R,
                                                               V *x, int32_t *ex, int *flag) {
  const size_t g = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
  const size_t row = (size_t)R * S;
  if (g >= n_pat * row) return;
  const size_t p = g / row;
  const int i = (int)(g % row) % S;
  int c = codes[p];
  if (c >= n_codes) {
    atomicOr(flag, PGPU_FLAG_BADCODE);
    c = 0;
  }
  x[g] = (V)tab[c * S + i];
  if (g % row == 0) ex[p] = 0;
}

struct MedArgs {
  const void *x[3];
  const int32_t *ex[3];
  const void *P[3];
  void *y;
  int32_t *ey;
  const double *weights;
  double2 *part;
  unsigned *counter;
  double *cost;
  size_t n_pat;
  int n_ch, S, R, RL;
  int int_w;                 // integer weights: exact int64 cost sums
  const int32_t *wint;
  long long *acc, *acc_next;   // this median's sum (zero), and the one to clear
};

constexpr double NEG_LN2 = -0.69314718055994530942;

// 16-byte vector access to one (pattern, rate class) row of 4 states
template <typename V> struct Row4;
template <> struct Row4<float> {
  __device__ __forceinline__ static void load(const float *p, float *v) {
    const float4 q = __ldg(reinterpret_cast<const float4 *>(p));
    v[0] = q.x, v[1] = q.y, v[2] = q.z, v[3] = q.w;
  }
  __device__ __forceinline__ static void load_l2(const float *p, float *v) {
    const float4 q = __ldcg(reinterpret_cast<const float4 *>(p));
    v[0] = q.x, v[1] = q.y, v[2] = q.z, v[3] = q.w;
  }
  __device__ __forceinline__ static void load_shared(const float *p, float *v) {
    const float4 q = *reinterpret_cast<const float4 *>(p);
    v[0] = q.x, v[1] = q.y, v[2] = q.z, v[3] = q.w;
  }
  __device__ __forceinline__ static void store(float *p, const float *v) {
    *reinterpret_cast<float4 *>(p) = make_float4(v[0], v[1], v[2], v[3]);
  }
};
template <> struct Row4<double> {
  __device__ __forceinline__ static void load(const double *p, double *v) {
    const double2 a = __ldg(reinterpret_cast<const double2 *>(p));
    const double2 b = __ldg(reinterpret_cast<const double2 *>(p) + 1);
    v[0] = a.x, v[1] = a.y, v[2] = b.x, v[3] = b.y;
  }
  __device__ __forceinline__ static void load_l2(const double *p, double *v) {
    const double2 a = __ldcg(reinterpret_cast<const double2 *>(p));
    const double2 b = __ldcg(reinterpret_cast<const double2 *>(p) + 1);
    v[0] = a.x, v[1] = a.y, v[2] = b.x, v[3] = b.y;
  }
  __device__ __forceinline__ static void load_shared(const double *p, double *v) {
    const double2 a = reinterpret_cast<const double2 *>(p)[0], b = reinterpret_cast<const double2 *>(p)[1];
    v[0] = a.x, v[1] = a.y, v[2] = b.x, v[3] = b.y;
  }
  __device__ __forceinline__ static void store(double *p, const double *v) {
    reinterpret_cast<double2 *>(p)[0] = make_double2(v[0], v[1]);
    reinterpret_cast<double2 *>(p)[1] = make_double2(v[2], v[3]);
  }
};

// y = prod_k P_k x_k, normalised per pattern, for any S up to 64.  A grid of
// a few CTAs per SM strides over the (pattern, rate class) items, a warp at a
// time (the stride is a multiple of 32, so a pattern's RL lanes stay in one
// warp and one iteration); each thread keeps one cost sum and the CTA reduces
// it once at the end.
template <typename V>
__global__ void __launch_bounds__(CLV_THREADS) clv_median_kernel(const MedArgs a) {
  const int S = a.S, R = a.R, RL = a.RL;
  const int lane = threadIdx.x & 31;
  const size_t n_items = a.n_pat * (size_t)RL;
  const size_t stride = (size_t)gridDim.x * CLV_THREADS;
  V *y = static_cast<V *>(a.y);
  double s = 0.0, c = 0.0;
  long long iacc = 0;
  if (a.int_w && blockIdx.x == 0 && threadIdx.x == 0) *a.acc_next = 0;
  for (size_t base = (size_t)blockIdx.x * CLV_THREADS + (threadIdx.x & ~31); base < n_items;
       base += stride) {
    const size_t g = base + lane;
    const size_t p = g / RL;
    const int r = (int)(g % RL);
    const bool act = g < n_items && r < R;
    const size_t off = (p * R + r) * (size_t)S;
    // the pattern's first lane reads the children's exponents and its
    // weight up front, so their latency overlaps the rows' (loaded after the
    // vector stores below, they would wait on a second round trip)
    const bool lead = act && r == 0;
    int ex_sum = 0;
    long long wi = 0;
    double wd = 0.0;
    if (lead) {
      for (int k = 0; k < a.n_ch; ++k) ex_sum += __ldg(a.ex[k] + p);
      if (a.int_w) wi = a.wint ? (long long)__ldg(a.wint + p) : 1;
      else wd = a.weights ? __ldg(a.weights + p) : 1.0;
    }
    V m = (V)0;
    int e;
    if (act) {
      for (int i = 0; i < S; ++i) {
        V v = (V)1;
        for (int k = 0; k < a.n_ch; ++k) {
          const V *xs = static_cast<const V *>(a.x[k]) + off;
          const V *P = static_cast<const V *>(a.P[k]) + ((size_t)r * S + i) * S;
          V t = (V)0;
          for (int j = 0; j < S; ++j) t = fma(__ldg(P + j), xs[j], t);
          v *= t;
        }
        y[off + i] = v;
        m = v > m ? v : m;
      }
    }
    V mm = m;
    for (int o = 1; o < RL; o <<= 1) {
      const V q = __shfl_xor_sync(0xffffffffu, mm, o);
      mm = q > mm ? q : mm;
    }
    e = frexp_exp(mm);
    if (act)
      for (int i = 0; i < S; ++i) y[off + i] = scale2<V>(y[off + i], -e);
    // exponent bookkeeping and this node's cost, by the pattern's first lane
    if (lead) {
      a.ey[p] = e + ex_sum;
      if (a.int_w) {
        iacc += wi * e;
      } else {
        double t, err;
        two_sum(s, wd * (double)e, t, err);
        s = t;
        c += err;
      }
    }
  }
  // cost = -ln 2 * sum_p w_p e_p
  if (a.int_w) cta_add_i64<CLV_THREADS>(iacc, a.acc);
  else cta_partial_and_finish<CLV_THREADS>(s, c, a.part, a.counter, a.cost, NEG_LN2);
}

// The same for four states.  The next item's reads in flight while one is
// computed, P and the leaves' rows by code in shared memory.
// 100,003 patterns, 4 classes, float: 6.1 us a median over a 128-taxon tree (18
// at 446,427; 23 with internal neighbours only, more of them than L2 holds) against 14.4 us with vectors for leaves, P read per item and one
// item in flight; P in registers spills at 4 CTAs per SM (8.0 us), and at 2
// or 3 CTAs too few reads are in flight (8.3, 7.4).
template <typename V, int NCH>
struct Med4Args {
  const V *x[NCH];           // internal neighbours; null: a leaf
  const int32_t *ex[NCH];
  const uint8_t *codes[NCH];
  V P[NCH][8 * 16];
  V *y;
  int32_t *ey;
  const V *tab;              // [n_codes][4]
  const double *weights;
  double2 *part;
  unsigned *counter;
  double *cost;
  size_t n_pat;
  int R, RL, rl_shift, n_codes, int_w;   // RL = 1 << rl_shift
  const int32_t *wint;
  long long *acc, *acc_next;
};

template <typename V, int NCH>
__global__ void __launch_bounds__(CLV_THREADS, sizeof(V) == 4 ? 4 : 2) clv_median4_kernel(const __grid_constant__ Med4Args<V, NCH> a) {
  extern __shared__ __align__(16) unsigned char clv_sm[];
  V *sP = reinterpret_cast<V *>(clv_sm);            // [NCH][4 rows][R][4]: a warp's classes side by side
  V *rows = sP + NCH * a.R * 16;                    // per leaf neighbour [n_codes][R][4]
  const int R = a.R, RL = a.RL, tid = threadIdx.x, lane = tid & 31;
  const int n_rows = a.n_codes * R * 4;
#pragma unroll
  for (int k = 0; k < NCH; ++k)
    for (int i = tid; i < R * 16; i += CLV_THREADS) sP[k * R * 16 + (((i >> 2) & 3) * R + (i >> 4)) * 4 + (i & 3)] = a.P[k][i];
  __syncthreads();
  int n_leaf = 0;
#pragma unroll
  for (int k = 0; k < NCH; ++k)
    if (!a.x[k]) {
      for (int o = tid; o < n_rows; o += CLV_THREADS) {
        const int i = o & 3, r = (o >> 2) % R, c = (o >> 2) / R;
        V t = (V)0;
#pragma unroll
        for (int j = 0; j < 4; ++j) t = fma(sP[k * R * 16 + (i * R + r) * 4 + j], __ldg(a.tab + 4 * c + j), t);
        rows[n_leaf * n_rows + o] = t;
      }
      ++n_leaf;
    }
  __syncthreads();
  const size_t n_items = a.n_pat * (size_t)RL, stride = (size_t)gridDim.x * CLV_THREADS;
  // the stride is a multiple of RL, so a thread keeps its rate class
  const size_t first = (size_t)blockIdx.x * CLV_THREADS + tid;
  const int r = (int)(first & (RL - 1));
  const bool rate_on = r < R;
  // Launched while the kernel before drains (programmatic stream
  // serialisation): nothing above depends on it.  From here on its vectors
  // are read, past the read-only path, which may keep lines from before.
  asm volatile("griddepcontrol.wait;" ::: "memory");
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
  if (a.int_w && blockIdx.x == 0 && tid == 0) *a.acc_next = 0;
  double s = 0.0, c = 0.0;
  long long iacc = 0;
  // what one item reads; the next item's is on its way while one is computed
  struct Item {
    V x[NCH][4];
    uint32_t code[NCH];
    int ex;
    int32_t wi;
    double wd;
  };
  const bool lead = r == 0;   // the pattern's first lane keeps its exponents and cost
  auto fetch = [&](size_t g, Item &it) {
    it.ex = 0;
    it.wi = 1;
    it.wd = 1.0;
    if (g >= n_items || !rate_on) return;
    const size_t p = g >> a.rl_shift;
#pragma unroll
    for (int k = 0; k < NCH; ++k) {
      if (a.x[k]) Row4<V>::load_l2(a.x[k] + (p * R + r) * 4, it.x[k]);
      else it.code[k] = __ldcg(a.codes[k] + p);
      if (lead && a.x[k]) it.ex += __ldcg(a.ex[k] + p);
    }
    if (lead) {
      if (a.wint) it.wi = __ldg(a.wint + p);
      else if (!a.int_w && a.weights) it.wd = __ldg(a.weights + p);
    }
  };
  Item cur, next;
  size_t g = first;
  fetch(g, cur);
  // whole warps stay in the loop: RL lanes of a pattern share a warp
  for (size_t base = first - lane; base < n_items; base += stride) {
    const bool act = g < n_items && rate_on;
    fetch(g + stride, next);
    V acc[4] = {(V)1, (V)1, (V)1, (V)1}, m = (V)0;
    if (act) {
      int leaf = 0;
#pragma unroll
      for (int k = 0; k < NCH; ++k) {
        V t[4];
        if (a.x[k]) {
#pragma unroll
          for (int i = 0; i < 4; ++i) {
            V Pr[4];
            Row4<V>::load_shared(sP + k * R * 16 + (i * R + r) * 4, Pr);
            t[i] = (V)0;
#pragma unroll
            for (int j = 0; j < 4; ++j) t[i] = fma(Pr[j], cur.x[k][j], t[i]);
          }
        } else {
          Row4<V>::load_shared(
              rows + leaf * n_rows + (min(cur.code[k], (uint32_t)a.n_codes - 1u) * R + r) * 4, t);
          ++leaf;
        }
#pragma unroll
        for (int i = 0; i < 4; ++i) acc[i] *= t[i];
      }
#pragma unroll
      for (int i = 0; i < 4; ++i) m = acc[i] > m ? acc[i] : m;
    }
    for (int o = 1; o < RL; o <<= 1) {
      const V q = __shfl_xor_sync(0xffffffffu, m, o);
      m = q > m ? q : m;
    }
    const int e = frexp_exp(m);
    if (act) {
      const size_t p = g >> a.rl_shift;
      V out[4];
#pragma unroll
      for (int i = 0; i < 4; ++i) out[i] = scale2<V>(acc[i], -e);
      Row4<V>::store(a.y + (p * R + r) * 4, out);
      if (lead) {
        a.ey[p] = e + cur.ex;
        if (a.int_w) {
          iacc += (long long)cur.wi * e;
        } else {
          double t, err;
          two_sum(s, cur.wd * (double)e, t, err);
          s = t;
          c += err;
        }
      }
    }
    cur = next;
    g += stride;
  }
  if (a.int_w) cta_add_i64<CLV_THREADS>(iacc, a.acc);
  else cta_partial_and_finish<CLV_THREADS>(s, c, a.part, a.counter, a.cost, NEG_LN2);
}

// codes at or above n_codes become 0, as clv_leaf_kernel reads them
__global__ void __launch_bounds__(CLV_THREADS) clv_codes_kernel(uint8_t *codes, size_t n, int n_codes) {
  for (size_t i = (size_t)blockIdx.x * CLV_THREADS + threadIdx.x; i < n; i += (size_t)gridDim.x * CLV_THREADS)
    if (codes[i] >= n_codes) codes[i] = 0;
}

// root_cost: -sum_p w_p log(sum_r probs_r sum_i pi_i x[p][r][i]); the
// node costs carry every normalisation, so the root's own exponent E is
// left out (costs + root_cost = -lnL).  Grid-stride as the median kernel.
template <typename V>
__global__ void __launch_bounds__(CLV_THREADS) clv_root_kernel(
    const V *x, const int32_t *ex, const double *pi, const double *probs, const double *weights,
    size_t n_pat, int S, int R, int RL, double *site_lnl, double2 *part, unsigned *counter,
    double *out) {
  const int lane = threadIdx.x & 31;
  const size_t n_items = n_pat * (size_t)RL;
  const size_t stride = (size_t)gridDim.x * CLV_THREADS;
  double s = 0.0, c = 0.0;
  for (size_t base = (size_t)blockIdx.x * CLV_THREADS + (threadIdx.x & ~31); base < n_items;
       base += stride) {
    const size_t g = base + lane;
    const size_t p = g / RL;
    const int r = (int)(g % RL);
    const bool act = g < n_items && r < R;
    double v = 0.0;
    if (act) {
      const V *xs = x + (p * R + r) * (size_t)S;
      for (int i = 0; i < S; ++i) v = fma(pi[i], (double)xs[i], v);
      v *= probs[r];
    }
    for (int o = 1; o < RL; o <<= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    if (act && r == 0) {
      const double site = log(v);
      if (site_lnl) site_lnl[p] = site + (double)ex[p] * 0.69314718055994530942;
      double t, err;
      two_sum(s, weights ? weights[p] * site : site, t, err);
      s = t;
      c += err;
    }
  }
  cta_partial_and_finish<CLV_THREADS>(s, c, part, counter, out, -1.0);
}

// The same for four states, a thread per pattern: FP64 costs a warp the same
// however few of its lanes work (100,003 patterns, 4 classes: 38 us, 80
// with a lane per rate class).
template <typename V>
__global__ void __launch_bounds__(CLV_THREADS) clv_root4_kernel(
    const V *x, const int32_t *ex, const double *pi, const double *probs, const double *weights,
    size_t n_pat, int R, double *site_lnl, double2 *part, unsigned *counter, double *out) {
  double s = 0.0, c = 0.0;
  const double pi4[4] = {pi[0], pi[1], pi[2], pi[3]};
  for (size_t p = (size_t)blockIdx.x * CLV_THREADS + threadIdx.x; p < n_pat;
       p += (size_t)gridDim.x * CLV_THREADS) {
    double v = 0.0;
    for (int r = 0; r < R; ++r) {
      V xs[4];
      Row4<V>::load(x + (p * R + r) * 4, xs);
      double q = 0.0;
#pragma unroll
      for (int i = 0; i < 4; ++i) q = fma(pi4[i], (double)xs[i], q);
      v = fma(q, probs[r], v);
    }
    const double site = log(v);
    if (site_lnl) site_lnl[p] = site + (double)ex[p] * 0.69314718055994530942;
    double t, err;
    two_sum(s, weights ? weights[p] * site : site, t, err);
    s = t;
    c += err;
  }
  cta_partial_and_finish<CLV_THREADS>(s, c, part, counter, out, -1.0);
}

// costs of many nodes: out[i] = *src[i], or of the int64 there
__global__ void __launch_bounds__(256) clv_gather_kernel(const double *const *src, size_t n,
                                                        double *out, int int_w) {
  for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < n;
       i += (size_t)gridDim.x * blockDim.x)
    out[i] = int_w ? NEG_LN2 * (double)*reinterpret_cast<const long long *>(src[i]) : *src[i];
}

pgpu_status lk_err(pgpu_lk *lk, pgpu_status st, const char *msg) {
  return pgpu_set_err(lk->ctx, st, "%s", msg);
}

pgpu_status clv_malloc(pgpu_ctx *ctx, size_t bytes, char **out) {
  void *mem = nullptr;
  const cudaError_t e = cudaMallocAsync(&mem, bytes, ctx->stream);
  if (e != cudaSuccess) {
    (void)cudaGetLastError();
    return pgpu_set_err(ctx, e == cudaErrorMemoryAllocation ? PGPU_ERR_OOM : PGPU_ERR_CUDA,
                        "likelihood: node allocation of %zu bytes failed: %s", bytes, cudaGetErrorString(e));
  }
  *out = static_cast<char *>(mem);
  return PGPU_OK;
}

// A leaf's codes are looked at while they are copied; ctx->bad_leaves makes the
// next call that checks the error word report those outside the table.  A bad
// leaf that is overwritten or destroyed before such a call is not reported,
// unless something has read it.
void bad_leaf_read(pgpu_clv *t) { t->bad = -1; }
void bad_leaf_gone(pgpu_clv *t) {
  if (t->bad >= 0 && t->bad == t->lk->ctx->bad_reports) --t->lk->ctx->bad_leaves;
  t->bad = -1;
}

// Four maxima over the quarters of the codes: one is a chain of dependent
// operations (3.9 us per 100,000 codes on the host's cores, 1.1 with four;
// copying them takes 1.1).
bool codes_outside(const uint8_t *codes, size_t n, int n_codes) {
  uint8_t m0 = 0, m1 = 0, m2 = 0, m3 = 0;
  const size_t q = n / 4;
  for (size_t i = 0; i < q; ++i) {
    m0 = std::max(m0, codes[i]);
    m1 = std::max(m1, codes[q + i]);
    m2 = std::max(m2, codes[2 * q + i]);
    m3 = std::max(m3, codes[3 * q + i]);
  }
  for (size_t i = 4 * q; i < n; ++i) m0 = std::max(m0, codes[i]);
  return std::max(std::max(m0, m1), std::max(m2, m3)) >= n_codes;
}

// a handle for lk (or `reuse`, its memory taken over), without its vector
pgpu_status clv_alloc(pgpu_lk *lk, pgpu_clv *reuse, pgpu_clv **out) {
  pgpu_ctx *ctx = lk->ctx;
  if (reuse) {
    if (reuse->lk != lk)
      return lk_err(lk, PGPU_ERR_ARG, "likelihood: the reused node belongs to another model");
    *out = reuse;
    reuse->has_P = false;
    reuse->leaf = false;
    reuse->expanded = false;
    reuse->brlen = 0.0;
    bad_leaf_gone(reuse);
    return PGPU_OK;
  }
  const size_t pb = lk->S == 4 ? 0 : al256((size_t)lk->R * lk->S * lk->S * vbytes(lk));
  const size_t cb = lk->leaf_codes ? al256(lk->n_pat) : 0;
  pgpu_clv *t = new (std::nothrow) pgpu_clv();
  if (!t) return lk_err(lk, PGPU_ERR_OOM, "likelihood: host allocation failed");
  pgpu_status st = clv_malloc(ctx, 256 + pb + cb, &t->mem);
  if (st == PGPU_OK && cudaMemsetAsync(t->mem, 0, 32, ctx->stream) != cudaSuccess) {
    (void)cudaGetLastError();
    st = lk_err(lk, PGPU_ERR_CUDA, "likelihood: clearing a node failed");
  }
  if (st != PGPU_OK) {
    if (t->mem) cudaFreeAsync(t->mem, ctx->stream);
    delete t;
    return st;
  }
  t->lk = lk;
  t->scal = reinterpret_cast<double *>(t->mem);
  t->P = t->mem + 256;
  t->codes = reinterpret_cast<uint8_t *>(t->mem + 256 + pb);
  lk->live++;
  *out = t;
  return PGPU_OK;
}

// the node's vector memory
pgpu_status clv_vector(pgpu_clv *t) {
  if (t->vec) return PGPU_OK;
  pgpu_lk *lk = t->lk;
  const size_t xb = al256(lk->n_pat * lk->R * lk->S * vbytes(lk));
  PGPU_TRY(clv_malloc(lk->ctx, xb + al256(lk->n_pat * 4), &t->vec));
  t->x = t->vec;
  t->ex = reinterpret_cast<int32_t *>(t->vec + xb);
  return PGPU_OK;
}

void clv_free(pgpu_clv *t) {
  pgpu_ctx *ctx = t->lk->ctx;
  bad_leaf_gone(t);
  if (t->vec) cudaFreeAsync(t->vec, ctx->stream);
  cudaFreeAsync(t->mem, ctx->stream);
  t->lk->live--;
  delete t;
}

// a leaf's vector from its codes
pgpu_status clv_expand(pgpu_clv *t, const uint8_t *codes) {
  pgpu_lk *lk = t->lk;
  pgpu_ctx *ctx = lk->ctx;
  PGPU_TRY(clv_vector(t));
  const size_t n = lk->n_pat * lk->R * lk->S;
  const unsigned grid = (unsigned)((n + CLV_THREADS - 1) / CLV_THREADS);
  if (lk->precision == 32)
    clv_leaf_kernel<float><<<grid, CLV_THREADS, 0, ctx->stream>>>(codes, lk->tab, lk->n_codes, lk->n_pat, lk->S,
                                                                  lk->R, (float *)t->x, t->ex, ctx->d_flag);
  else
    clv_leaf_kernel<double><<<grid, CLV_THREADS, 0, ctx->stream>>>(codes, lk->tab, lk->n_codes, lk->n_pat,
                                                                   lk->S, lk->R, (double *)t->x, t->ex,
                                                                   ctx->d_flag);
  PGPU_TRY(pgpu_after_launch(ctx, "clv_leaf_kernel"));
  t->expanded = true;
  bad_leaf_read(t);
  return PGPU_OK;
}

const double *cost_at(const pgpu_clv *t) {
  return t->leaf ? t->lk->zero : t->scal + (t->lk->int_w ? t->slot : 0);
}

template <typename V, int NCH>
pgpu_status launch_median4(pgpu_lk *lk, pgpu_clv *t, pgpu_clv *const *ch) {
  pgpu_ctx *ctx = lk->ctx;
  Med4Args<V, NCH> a;
  int n_leaf = 0;
  for (int k = 0; k < NCH; ++k) {
    const bool vec = !ch[k]->leaf || ch[k]->expanded;
    a.x[k] = vec ? static_cast<const V *>(ch[k]->x) : nullptr;
    a.ex[k] = vec ? ch[k]->ex : nullptr;
    a.codes[k] = vec ? nullptr : ch[k]->codes;
    n_leaf += !vec;
    for (int i = 0; i < lk->R * 16; ++i) a.P[k][i] = (V)ch[k]->P4[i / 16][i % 16];
  }
  a.y = static_cast<V *>(t->x);
  a.ey = t->ex;
  a.tab = static_cast<const V *>(lk->tabv);
  a.weights = lk->weights;
  a.part = lk->part;
  a.counter = lk->counter;
  a.cost = t->scal;
  a.n_pat = lk->n_pat;
  a.R = lk->R;
  a.RL = lk->RL;
  a.rl_shift = lk->RL == 1 ? 0 : lk->RL == 2 ? 1 : lk->RL == 4 ? 2 : 3;
  a.n_codes = lk->n_codes;
  a.int_w = lk->int_w ? 1 : 0;
  a.wint = lk->wint;
  a.acc = reinterpret_cast<long long *>(t->scal + t->slot);
  a.acc_next = reinterpret_cast<long long *>(t->scal + (t->slot ^ 1));
  const size_t smem = sizeof(V) * (size_t)lk->R * (NCH * 16 + (size_t)n_leaf * lk->n_codes * 4);
  if (lk->resident[NCH - 1] == 0 || smem > 48 * 1024)
    PGPU_CUDA(ctx, cudaFuncSetAttribute(clv_median4_kernel<V, NCH>,
                                        cudaFuncAttributeMaxDynamicSharedMemorySize, 112 * 1024));
  // one wave of CTAs at most: each pays its prologue (P and the leaves' rows
  // to shared memory) once
  int &res = lk->resident[NCH - 1];
  if (res == 0) {
    const size_t most = sizeof(V) * (size_t)lk->R * NCH * (16 + (size_t)lk->n_codes * 4);
    PGPU_CUDA(ctx, cudaOccupancyMaxActiveBlocksPerMultiprocessor(
                       &res, clv_median4_kernel<V, NCH>, CLV_THREADS, lk->leaf_codes ? most : smem));
    res = std::max(res, 1);
  }
  const size_t want = (lk->n_pat * lk->RL + CLV_THREADS - 1) / CLV_THREADS;
  const size_t most_cta = std::min<size_t>(lk->n_cta, (size_t)res * std::max(ctx->num_sms, 1));
  cudaLaunchConfig_t c{};
  c.gridDim = dim3((unsigned)std::max<size_t>(std::min(want, most_cta), 1));
  c.blockDim = dim3(CLV_THREADS);
  c.dynamicSmemBytes = smem;
  c.stream = ctx->stream;
  cudaLaunchAttribute at{};
  at.id = cudaLaunchAttributeProgrammaticStreamSerialization;
  at.val.programmaticStreamSerializationAllowed = 1;
  c.attrs = &at;
  c.numAttrs = 1;
  PGPU_CUDA(ctx, cudaLaunchKernelEx(&c, clv_median4_kernel<V, NCH>, a));
  return pgpu_after_launch(ctx, "clv_median4_kernel");
}

pgpu_status check_cta(pgpu_lk *lk) {
  // grid of every per-pattern kernel: n_pat * RL threads
  const size_t n_cta = std::max<size_t>((lk->n_pat * lk->RL + CLV_THREADS - 1) / CLV_THREADS, 1);
  if (n_cta > 0x7fffffffu) return lk_err(lk, PGPU_ERR_LIMIT, "likelihood: too many patterns");
  return PGPU_OK;
}

pgpu_status median(pgpu_lk *lk, pgpu_clv *reuse, const pgpu_clv *const *nbr, int n_ch,
                   pgpu_clv **out) {
  if (!lk || !out) return PGPU_ERR_ARG;
  pgpu_ctx *ctx = lk->ctx;
  for (int k = 0; k < n_ch; ++k) {
    if (!nbr[k]) return lk_err(lk, PGPU_ERR_ARG, "likelihood: null neighbour");
    if (nbr[k]->lk != lk) return lk_err(lk, PGPU_ERR_ARG, "likelihood: neighbour of another model");
    if (!nbr[k]->has_P)
      return lk_err(lk, PGPU_ERR_ARG,
                    "likelihood: a neighbour has no branch length (pgpu_clv_set_brlen)");
    if (nbr[k] == reuse)
      return lk_err(lk, PGPU_ERR_ARG, "likelihood: the reused node is also a neighbour");
  }
  PGPU_CUDA(ctx, cudaSetDevice(ctx->device));
  pgpu_clv *const *ch = const_cast<pgpu_clv *const *>(nbr);
  pgpu_clv *t = nullptr;
  PGPU_TRY(clv_alloc(lk, reuse, &t));
  pgpu_status st = clv_vector(t);
  if (st != PGPU_OK) {
    if (!reuse) clv_free(t);
    return st;
  }
  if (lk->int_w) t->slot ^= 1;
  if (lk->S == 4) {
    for (int k = 0; k < n_ch; ++k)
      bad_leaf_read(ch[k]);
    if (lk->precision == 32)
      st = n_ch == 1 ? launch_median4<float, 1>(lk, t, ch)
                     : n_ch == 2 ? launch_median4<float, 2>(lk, t, ch) : launch_median4<float, 3>(lk, t, ch);
    else
      st = n_ch == 1 ? launch_median4<double, 1>(lk, t, ch)
                     : n_ch == 2 ? launch_median4<double, 2>(lk, t, ch) : launch_median4<double, 3>(lk, t, ch);
    PGPU_TRY(st);
    *out = t;
    return PGPU_OK;
  }
  MedArgs a{};
  for (int k = 0; k < n_ch; ++k) {
    a.x[k] = ch[k]->x;
    a.ex[k] = ch[k]->ex;
    a.P[k] = ch[k]->P;
  }
  a.y = t->x;
  a.ey = t->ex;
  a.weights = lk->weights;
  a.int_w = lk->int_w ? 1 : 0;
  a.wint = lk->wint;
  a.acc = reinterpret_cast<long long *>(t->scal + t->slot);
  a.acc_next = reinterpret_cast<long long *>(t->scal + (t->slot ^ 1));
  a.part = lk->part;
  a.counter = lk->counter;
  a.cost = t->scal;
  a.n_pat = lk->n_pat;
  a.n_ch = n_ch;
  a.S = lk->S;
  a.R = lk->R;
  a.RL = lk->RL;
  const unsigned grid = (unsigned)lk->n_cta;
  if (lk->precision == 32) clv_median_kernel<float><<<grid, CLV_THREADS, 0, ctx->stream>>>(a);
  else clv_median_kernel<double><<<grid, CLV_THREADS, 0, ctx->stream>>>(a);
  PGPU_TRY(pgpu_after_launch(ctx, "clv_median_kernel"));
  *out = t;
  return PGPU_OK;
}

}  // namespace

extern "C" {

pgpu_status pgpu_lk_create(pgpu_ctx *ctx, const pgpu_model *m, const pgpu_tip_codes *codes,
                           size_t n_pat, const double *weights, int precision, pgpu_lk **out) {
  if (!ctx || !out) return PGPU_ERR_ARG;
  *out = nullptr;
  if (!m || !m->Q || !m->pi || !m->rates || !m->probs)
    return pgpu_set_err(ctx, PGPU_ERR_ARG, "likelihood: null model field");
  if (m->n_states < 2 || m->n_states > 64)
    return pgpu_set_err(ctx, PGPU_ERR_LIMIT, "likelihood: 2..64 states are supported");
  if (m->n_rates < 1 || m->n_rates > 8)
    return pgpu_set_err(ctx, PGPU_ERR_LIMIT, "likelihood: 1..8 rate classes are supported");
  if (!codes || !codes->table || codes->n_codes < 1 || codes->n_codes > 256)
    return pgpu_set_err(ctx, PGPU_ERR_ARG, "likelihood: tip code table must have 1..256 rows");
  if (precision != 32 && precision != 64)
    return pgpu_set_err(ctx, PGPU_ERR_ARG, "likelihood: precision must be 32 or 64");
  if (n_pat == 0) return pgpu_set_err(ctx, PGPU_ERR_ARG, "likelihood: no patterns");
  PGPU_CUDA(ctx, cudaSetDevice(ctx->device));
  pgpu_lk *lk = new (std::nothrow) pgpu_lk();
  if (!lk) return pgpu_set_err(ctx, PGPU_ERR_OOM, "likelihood: host allocation failed");
  lk->ctx = ctx;
  lk->S = m->n_states;
  lk->R = m->n_rates;
  lk->RL = lk->R <= 1 ? 1 : lk->R <= 2 ? 2 : lk->R <= 4 ? 4 : 8;
  lk->n_codes = codes->n_codes;
  lk->precision = precision;
  lk->n_pat = n_pat;
  if (check_cta(lk) != PGPU_OK) {
    delete lk;
    return PGPU_ERR_LIMIT;
  }
  // the per-pattern kernels stride over the patterns with a few CTAs per SM
  const size_t want = (n_pat * lk->RL + CLV_THREADS - 1) / CLV_THREADS;
  lk->n_cta = std::max<size_t>(std::min<size_t>(want, (size_t)std::max(ctx->num_sms, 1) * 8), 1);
  const int S = lk->S, R = lk->R;
  const size_t SS = (size_t)S * S;
  // one block, every part on a 256-byte boundary (the partials are double2
  // and must be 16-byte aligned whatever the pattern count)
  size_t off = 0;
  auto take = [&](size_t bytes) {
    const size_t o = off;
    off += al256(bytes);
    return o;
  };
  const size_t oU = take(SS * 8), oUi = take(SS * 8), olam = take(S * 8), opi = take(S * 8),
               orates = take(R * 8), oprobs = take(R * 8),
               otab = take((size_t)codes->n_codes * S * 8), ow = take(n_pat * 8), oq = take(SS * 8),
               ost = take(64), opart = take(lk->n_cta * sizeof(double2)),
               owi = take(n_pat * 4), otabv = take((size_t)codes->n_codes * S * vbytes(lk)), ozero = take(8);
  const size_t bytes = off;
  void *blk = nullptr;
  cudaError_t e = cudaMalloc(&blk, bytes);
  if (e != cudaSuccess) {
    (void)cudaGetLastError();
    delete lk;
    return pgpu_set_err(ctx, PGPU_ERR_OOM, "likelihood: model allocation failed");
  }
  char *base = static_cast<char *>(blk);
  lk->block = reinterpret_cast<double *>(base);
  lk->U = reinterpret_cast<double *>(base + oU);
  lk->Ui = reinterpret_cast<double *>(base + oUi);
  lk->lam = reinterpret_cast<double *>(base + olam);
  lk->pi = reinterpret_cast<double *>(base + opi);
  lk->rates = reinterpret_cast<double *>(base + orates);
  lk->probs = reinterpret_cast<double *>(base + oprobs);
  lk->tab = reinterpret_cast<double *>(base + otab);
  double *w = reinterpret_cast<double *>(base + ow);
  double *q = reinterpret_cast<double *>(base + oq);
  lk->weights = weights ? w : nullptr;
  lk->status = reinterpret_cast<int *>(base + ost);
  lk->counter = reinterpret_cast<unsigned *>(lk->status + 4);
  lk->part = reinterpret_cast<double2 *>(base + opart);
  lk->tabv = base + otabv;
  lk->zero = reinterpret_cast<double *>(base + ozero);
  // a leaf neighbour's rows stay within a third of 96 KB
  lk->leaf_codes = S == 4 && (size_t)codes->n_codes * R * 4 * vbytes(lk) <= 32 * 1024;
  // integer weights, small enough that sum_p w_p e_p fits int64 (|e_p| <= 1074)
  std::vector<int32_t> wi;
  lk->int_w = true;
  if (weights) {
    wi.resize(n_pat);
    double wmax = 0.0;
    for (size_t i = 0; i < n_pat && lk->int_w; ++i) {
      const double v = weights[i];
      if (!(v >= 0.0) || v >= 2147483647.0 || v != std::floor(v)) lk->int_w = false;
      else wi[i] = (int32_t)v, wmax = std::max(wmax, v);
    }
    if (lk->int_w && (double)n_pat * std::max(wmax, 1.0) * 1100.0 >= 4.0e18) lk->int_w = false;
  }
  lk->wint = lk->int_w && weights ? reinterpret_cast<int32_t *>(base + owi) : nullptr;
  cudaStream_t s = ctx->stream;
  auto fail = [&](pgpu_status st) {
    cudaFree(blk);
    delete lk;
    return st;
  };
#define LK_CUDA(call)                                                                   \
  do {                                                                                  \
    cudaError_t e_ = (call);                                                            \
    if (e_ != cudaSuccess) {                                                            \
      (void)cudaGetLastError();                                                         \
      return fail(pgpu_set_err(ctx, PGPU_ERR_CUDA, "%s failed: %s", #call,              \
                               cudaGetErrorString(e_)));                                \
    }                                                                                   \
  } while (0)
  LK_CUDA(cudaMemcpyAsync(q, m->Q, SS * 8, cudaMemcpyHostToDevice, s));
  LK_CUDA(cudaMemcpyAsync(lk->pi, m->pi, S * 8, cudaMemcpyHostToDevice, s));
  LK_CUDA(cudaMemcpyAsync(lk->rates, m->rates, R * 8, cudaMemcpyHostToDevice, s));
  LK_CUDA(cudaMemcpyAsync(lk->probs, m->probs, R * 8, cudaMemcpyHostToDevice, s));
  LK_CUDA(cudaMemcpyAsync(lk->tab, codes->table, (size_t)codes->n_codes * S * 8,
                          cudaMemcpyHostToDevice, s));
  if (weights) LK_CUDA(cudaMemcpyAsync(w, weights, n_pat * 8, cudaMemcpyHostToDevice, s));
  if (lk->wint) LK_CUDA(cudaMemcpyAsync(lk->wint, wi.data(), n_pat * 4, cudaMemcpyHostToDevice, s));
  LK_CUDA(cudaMemsetAsync(lk->status, 0, 64, s));
  LK_CUDA(cudaMemsetAsync(lk->zero, 0, 8, s));
  std::vector<float> tabf;
  if (S == 4) {
    const size_t n = (size_t)codes->n_codes * 4;
    for (size_t i = 0; i < n && precision == 32; ++i) tabf.push_back((float)codes->table[i]);
    LK_CUDA(cudaMemcpyAsync(lk->tabv, precision == 32 ? (const void *)tabf.data() : codes->table,
                            n * vbytes(lk), cudaMemcpyHostToDevice, s));
  }
  pgpu_status st = pgpu_launch_eig(ctx, q, lk->pi, S, 1, lk->U, lk->lam, lk->Ui, lk->status);
  if (st != PGPU_OK) return fail(st);
  int *hst = reinterpret_cast<int *>(ctx->h_pinned);
  LK_CUDA(cudaMemcpyAsync(hst, lk->status, sizeof(int), cudaMemcpyDeviceToHost, s));
  if (S == 4) {
    LK_CUDA(cudaMemcpyAsync(lk->hU, lk->U, sizeof lk->hU, cudaMemcpyDeviceToHost, s));
    LK_CUDA(cudaMemcpyAsync(lk->hUi, lk->Ui, sizeof lk->hUi, cudaMemcpyDeviceToHost, s));
    LK_CUDA(cudaMemcpyAsync(lk->hlam, lk->lam, sizeof lk->hlam, cudaMemcpyDeviceToHost, s));
    std::copy(m->rates, m->rates + R, lk->hrates);
  }
  LK_CUDA(cudaStreamSynchronize(s));
#undef LK_CUDA
  if (*hst) {
    const int code = *hst;
    return fail(pgpu_set_err(ctx, code,
                             code == PGPU_ERR_NAN ? "likelihood: NaN or Inf in Q or pi"
                             : code == PGPU_ERR_NONREVERSIBLE
                                 ? "likelihood: Q is not reversible with respect to pi"
                                 : "likelihood: eigendecomposition did not converge"));
  }
  *out = lk;
  return PGPU_OK;
}

void pgpu_lk_destroy(pgpu_lk *lk) {
  if (!lk) return;
  cudaSetDevice(lk->ctx->device);
  cudaStreamSynchronize(lk->ctx->stream);
  cudaFree(lk->block);
  delete lk;
}

pgpu_status pgpu_clv_leaf(pgpu_lk *lk, pgpu_clv *reuse, const uint8_t *codes, pgpu_clv **out) {
  if (!lk || !codes || !out) return lk ? lk_err(lk, PGPU_ERR_ARG, "likelihood: null argument")
                                       : PGPU_ERR_ARG;
  pgpu_ctx *ctx = lk->ctx;
  PGPU_CUDA(ctx, cudaSetDevice(ctx->device));
  pgpu_clv *t = nullptr;
  PGPU_TRY(clv_alloc(lk, reuse, &t));
  const cudaStream_t s = ctx->stream;
  if (lk->leaf_codes) {
    // The codes themselves are the leaf.  Up to 1 MB they go through the pinned
    // staging blocks: a copy straight from pageable memory holds the caller up
    // (20 us against 9 at 100 KB).
    bool bad = false;
    if (lk->n_pat <= (size_t)1 << 20) {
      void *h;
      PGPU_TRY(pgpu_stage(ctx, lk->n_pat, &h, nullptr));
      uint8_t *to = static_cast<uint8_t *>(h);
      constexpr size_t block = 16 * 1024;   // looked at while it is in the first-level cache
      for (size_t i = 0; i < lk->n_pat; i += block) {
        const size_t k = std::min(block, lk->n_pat - i);
        std::memcpy(to + i, codes + i, k);
        bad |= codes_outside(codes + i, k, lk->n_codes);
      }
      PGPU_TRY(pgpu_stage_copy(ctx, t->codes, lk->n_pat));
    } else {
      PGPU_CUDA(ctx, cudaMemcpyAsync(t->codes, codes, lk->n_pat, cudaMemcpyHostToDevice, s));
      bad = codes_outside(codes, lk->n_pat, lk->n_codes);
    }
    if (bad) {
      const unsigned grid = (unsigned)std::min<size_t>((lk->n_pat + CLV_THREADS - 1) / CLV_THREADS, 1024);
      clv_codes_kernel<<<grid, CLV_THREADS, 0, s>>>(t->codes, lk->n_pat, lk->n_codes);
      PGPU_TRY(pgpu_after_launch(ctx, "clv_codes_kernel"));
      t->bad = ctx->bad_reports;
      ++ctx->bad_leaves;
    }
  } else {
    // the codes are copied into the context's tip buffer; later calls on the
    // stream are ordered after this leaf's kernel
    void *dc;
    PGPU_TRY(pgpu_buf(ctx, BUF_TIPS, std::max<size_t>(lk->n_pat, 16), &dc));
    PGPU_CUDA(ctx, cudaMemcpyAsync(dc, codes, lk->n_pat, cudaMemcpyHostToDevice, s));
    PGPU_TRY(clv_expand(t, (const uint8_t *)dc));
  }
  t->leaf = true;
  *out = t;
  return PGPU_OK;
}

pgpu_status pgpu_clv_set_brlen(pgpu_clv *t, double brlen) {
  if (!t) return PGPU_ERR_ARG;
  pgpu_lk *lk = t->lk;
  pgpu_ctx *ctx = lk->ctx;
  if (!(brlen >= 0.0) || !std::isfinite(brlen))
    return lk_err(lk, PGPU_ERR_ARG, "likelihood: branch length must be finite and >= 0");
  if (lk->S == 4) {
    // compose_kernel's arithmetic, 16 numbers per rate class
    for (int r = 0; r < lk->R; ++r) {
      const bool ident = !(brlen * lk->hrates[r] >= 1e-10);
      double e[4];
      for (int k = 0; k < 4; ++k) e[k] = ident ? 1.0 : std::exp(lk->hlam[k] * lk->hrates[r] * brlen);
      for (int i = 0; i < 4; ++i)
        for (int j = 0; j < 4; ++j) {
          double v = 0.0;
          for (int k = 0; k < 4; ++k) v = std::fma(lk->hU[4 * i + k] * e[k], lk->hUi[4 * k + j], v);
          t->P4[r][4 * i + j] = ident ? (i == j ? 1.0 : 0.0) : v;
        }
    }
    t->brlen = brlen;
    t->has_P = true;
    return PGPU_OK;
  }
  PGPU_CUDA(ctx, cudaSetDevice(ctx->device));
  void *h;
  PGPU_TRY(pgpu_stage(ctx, sizeof(double), &h, nullptr));
  *static_cast<double *>(h) = brlen;
  PGPU_TRY(pgpu_stage_copy(ctx, t->scal + 3, sizeof(double)));
  PGPU_TRY(pgpu_launch_compose(ctx, lk->U, lk->lam, lk->Ui, lk->S, t->scal + 3, 1, lk->rates, lk->R,
                               lk->precision == 64 ? (double *)t->P : nullptr,
                               lk->precision == 64 ? nullptr : (float *)t->P, false, lk->status,
                               P32_PLAIN));
  t->brlen = brlen;
  t->has_P = true;
  return PGPU_OK;
}

pgpu_status pgpu_clv_get_brlen(const pgpu_clv *t, double *brlen) {
  if (!t || !brlen) return PGPU_ERR_ARG;
  *brlen = t->brlen;
  return PGPU_OK;
}

pgpu_status pgpu_clv_median1(pgpu_lk *lk, pgpu_clv *reuse, const pgpu_clv *a, pgpu_clv **out) {
  const pgpu_clv *ch[1] = {a};
  return median(lk, reuse, ch, 1, out);
}

pgpu_status pgpu_clv_median2(pgpu_lk *lk, pgpu_clv *reuse, const pgpu_clv *a, const pgpu_clv *b,
                             pgpu_clv **out) {
  const pgpu_clv *ch[2] = {a, b};
  return median(lk, reuse, ch, 2, out);
}

pgpu_status pgpu_clv_median3(pgpu_lk *lk, pgpu_clv *reuse, const pgpu_clv *a, const pgpu_clv *b,
                             const pgpu_clv *c, pgpu_clv **out) {
  const pgpu_clv *ch[3] = {a, b, c};
  return median(lk, reuse, ch, 3, out);
}

pgpu_status pgpu_clv_cost(pgpu_clv *t, double *cost) {
  if (!t || !cost) return PGPU_ERR_ARG;
  pgpu_ctx *ctx = t->lk->ctx;
  PGPU_CUDA(ctx, cudaSetDevice(ctx->device));
  double *h = reinterpret_cast<double *>(ctx->h_pinned);
  PGPU_CUDA(ctx, cudaMemcpyAsync(h, cost_at(t), sizeof(double), cudaMemcpyDeviceToHost, ctx->stream));
  PGPU_TRY(pgpu_check_flag(ctx, "likelihood"));
  *cost = t->lk->int_w ? NEG_LN2 * (double)*reinterpret_cast<const long long *>(h) : *h;
  return PGPU_OK;
}

pgpu_status pgpu_clv_costs(pgpu_lk *lk, const pgpu_clv *const *nodes, size_t n, double *costs) {
  if (!lk || (n && (!nodes || !costs))) return PGPU_ERR_ARG;
  if (n == 0) return PGPU_OK;
  pgpu_ctx *ctx = lk->ctx;
  for (size_t i = 0; i < n; ++i)
    if (!nodes[i] || nodes[i]->lk != lk)
      return lk_err(lk, PGPU_ERR_ARG, "likelihood: a node is null or belongs to another model");
  PGPU_CUDA(ctx, cudaSetDevice(ctx->device));
  void *h, *d, *dout;
  PGPU_TRY(pgpu_stage(ctx, n * sizeof(double *), &h, &d));
  const double **src = static_cast<const double **>(h);
  for (size_t i = 0; i < n; ++i) src[i] = cost_at(nodes[i]);
  PGPU_TRY(pgpu_stage_commit(ctx, n * sizeof(double *)));
  PGPU_TRY(pgpu_buf(ctx, BUF_F, n * sizeof(double), &dout));
  const unsigned grid = (unsigned)std::min<size_t>((n + 255) / 256, 1024);
  clv_gather_kernel<<<grid, 256, 0, ctx->stream>>>(static_cast<const double *const *>(d), n,
                                                   static_cast<double *>(dout), lk->int_w ? 1 : 0);
  PGPU_TRY(pgpu_after_launch(ctx, "clv_gather_kernel"));
  PGPU_CUDA(ctx, cudaMemcpyAsync(costs, dout, n * sizeof(double), cudaMemcpyDeviceToHost, ctx->stream));
  return pgpu_check_flag(ctx, "likelihood");
}

pgpu_status pgpu_clv_root_cost(pgpu_clv *t, double *cost, double *site_lnl) {
  if (!t || !cost) return PGPU_ERR_ARG;
  pgpu_lk *lk = t->lk;
  pgpu_ctx *ctx = lk->ctx;
  PGPU_CUDA(ctx, cudaSetDevice(ctx->device));
  if (t->leaf && !t->expanded) PGPU_TRY(clv_expand(t, t->codes));
  void *dsl = nullptr;
  if (site_lnl) PGPU_TRY(pgpu_buf(ctx, BUF_SITECOST, lk->n_pat * 8, &dsl));
  const unsigned grid = (unsigned)lk->n_cta;
  if (lk->S == 4) {
    const unsigned g4 = (unsigned)std::min<size_t>((lk->n_pat + CLV_THREADS - 1) / CLV_THREADS, lk->n_cta);
    if (lk->precision == 32)
      clv_root4_kernel<float><<<g4, CLV_THREADS, 0, ctx->stream>>>(
          (const float *)t->x, t->ex, lk->pi, lk->probs, lk->weights, lk->n_pat, lk->R, (double *)dsl,
          lk->part, lk->counter, t->scal + 2);
    else
      clv_root4_kernel<double><<<g4, CLV_THREADS, 0, ctx->stream>>>(
          (const double *)t->x, t->ex, lk->pi, lk->probs, lk->weights, lk->n_pat, lk->R, (double *)dsl,
          lk->part, lk->counter, t->scal + 2);
  } else if (lk->precision == 32)
    clv_root_kernel<float><<<grid, CLV_THREADS, 0, ctx->stream>>>(
        (const float *)t->x, t->ex, lk->pi, lk->probs, lk->weights, lk->n_pat, lk->S, lk->R,
        lk->RL, (double *)dsl, lk->part, lk->counter, t->scal + 2);
  else
    clv_root_kernel<double><<<grid, CLV_THREADS, 0, ctx->stream>>>(
        (const double *)t->x, t->ex, lk->pi, lk->probs, lk->weights, lk->n_pat, lk->S, lk->R,
        lk->RL, (double *)dsl, lk->part, lk->counter, t->scal + 2);
  PGPU_TRY(pgpu_after_launch(ctx, "clv_root_kernel"));
  double *h = reinterpret_cast<double *>(ctx->h_pinned);
  PGPU_CUDA(ctx, cudaMemcpyAsync(h, t->scal + 2, sizeof(double), cudaMemcpyDeviceToHost, ctx->stream));
  if (site_lnl)
    PGPU_CUDA(ctx, cudaMemcpyAsync(site_lnl, dsl, lk->n_pat * 8, cudaMemcpyDeviceToHost, ctx->stream));
  PGPU_TRY(pgpu_check_flag(ctx, "likelihood"));
  *cost = *h;
  return PGPU_OK;
}

void pgpu_clv_destroy(pgpu_clv *t) {
  if (!t) return;
  pgpu_ctx *ctx = t->lk->ctx;
  cudaSetDevice(ctx->device);
  clv_free(t);
}

}  // extern "C"
