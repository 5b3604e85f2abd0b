// Batched likelihood of many trees, models and pattern sets of uneven size,
// for 20-state (protein) and 61-state (codon) models, on the tensor cores.
//
// Reference: the likelihood character is a stub in phylocaml
// (Likelihood_c.median_2, lib/likelihood_c.ml:15); P matrices follow
// MlModel.compose (lib/mlModel.ml:585-587, P[i][j] = Pr(j | i, t)).  Every
// variant is an independent (tree, model, patterns) problem.
//
// Design (one GB300, one launch for all variants):
//   setup kernels  the FP64 Jacobi eigen systems (pmatrix.cu), then per
//                  variant, internal branch and rate class the FP32 B operand
//                  B[n=i][k=j] = P(t r)[i][j] in the tcgen05 K-major
//                  core-matrix layout, and per tip branch the FP64-formed tip
//                  rows tab[c][i] = sum_j P[i][j] code_tab[c][j];
//   batch_tc_kernel  persistent, two CTAs per SM, over work items
//                  (variant, tile of 128 patterns).  A tile's conditional
//                  likelihood vectors live in tensor memory (TMEM lane =
//                  pattern, columns = states; the few that a CTA's half of
//                  TMEM has no room for, in global memory) and are the A operand of
//                  tcgen05.mma.kind::tf32 for internal children; D (FP32) is
//                  accumulated in TMEM.  Tip children need no MMA: their rows
//                  come from the staged tip table.  Rate classes are separate
//                  passes with their own power-of-two scalers, joined at the
//                  root with a log-sum-exp in FP64.
//     warp 8       producer and TMEM allocator: per postorder step,
//                  bulk-copies the B blocks of internal children, the
//                  tip-table blocks and tip-code rows of tip children into a
//                  shared ring slot, and publishes the step itself;
//     warps 9, 10  MMA issue, one per rate class of the pass (9 alone with one);
//     warps 0-7    epilogue: two warps per TMEM lane group of 32 patterns,
//                  each owning a share of the row (half the states, or a
//                  whole rate class when two share a pass); a thread reads
//                  its D columns (tcgen05.ld) or tip rows, forms the product,
//                  rescales, writes the parent's vector back into TMEM
//                  (tcgen05.st).
//   A step is a chain of latencies (MMAs about 1,100 cycles from one epilogue's
//   stores to the next one's loads, epilogue 700) that left an SM with one
//   codon chain or two protein chains two thirds idle.  Two CTAs per SM, each
//   with half of TMEM, run twice the chains; a tree that needs more stack than
//   its half spills a vector for the length of a subtree (13 of 127 steps on
//   codon Yule trees of 128 taxa, 3 or 4 on protein ones).  32 models, 128
//   taxa, 5,000 to 100,000 patterns: 10.2 ms against 15.9 with one CTA.
//   The MMA (tcgen05.commit -> mma_bar) and the epilogue (an mbarrier,
//   `stored`, after its TMEM stores) alternate per step, so a step's MMA
//   never reads a vector before it is written and no mbarrier phase can be
//   skipped.  With two rate classes per pass the two classes are separate
//   chains, each with its own mma_bar and stored barrier and its own four
//   epilogue warps: the MMAs of one class's next step run while the other
//   class's epilogue runs, and no warp waits for another to agree on a
//   rescaling exponent.
//   Every wait is bounded.  A barrier's parity tells neighbouring phases apart
//   only, so every warp that waits on one waits for each of its phases in turn.
//   Work items of one padded state count and number of rate classes per pass
//   are one launch of a kernel compiled for them; the launches are chained and
//   overlap at their ends.
//   batch_fp64_kernel  the FP64 comparison form on a sample of patterns.
#include <algorithm>
#include <cmath>
#include <type_traits>
#include <vector>

#include "forms.cuh"
#include "pgpu_internal.cuh"
#include "pmatrix.cuh"

using namespace pgpu_forms;

namespace {

constexpr int BT_M = 128;          // patterns per tile (TMEM lanes)
constexpr int BT_ST = 4;           // ring slots at most
constexpr int BT_EPI_WARPS = 8;    // epilogue warps, two per TMEM lane group
constexpr int BT_PARTS = BT_EPI_WARPS / 4;   // shares of a row (one per warp of a lane group)
constexpr int BT_EPI = 32 * BT_EPI_WARPS;
constexpr int bt_threads(int RP) { return BT_EPI + 32 + 32 * RP; }   // + the producer warp and an MMA warp per class
constexpr int BT_PRODUCER = BT_EPI_WARPS, BT_MMA = BT_EPI_WARPS + 1;   // the first of each
constexpr int BT_TMEM_COLS = 256;  // of a CTA: two share an SM
constexpr int BT_LIMIT_COLS = 512; // what a tree's depth is held against

// TMEM columns of a rate class's chain: SL stack slots of KP, then D of NP.
// D of the second of two internal children goes to the free slot above them;
// where it is wider than a slot its padding falls on columns that are free or
// that the first child's MMAs, issued after it, write.
template <int KP, int RP>
struct Cols {
  static constexpr int NP = (KP + 15) / 16 * 16;
  static constexpr int CH = BT_TMEM_COLS / RP;
  static constexpr int SL = (CH - NP) / KP < 15 ? (CH - NP) / KP : 15;
  static constexpr int D = SL * KP;
};
int stack_slots(int Kp, int Np, int RP) { return std::min((BT_TMEM_COLS / RP - Np) / Kp, 15); }

// A ring position, the parity of its barriers' current phase, and that of the
// barriers with a phase per step.
struct Ring {
  int slot = 0;
  uint32_t par = 0, par_step = 0;
  __device__ __forceinline__ void next(int n) {
    if (++slot == n) {
      slot = 0;
      par ^= 1u;
    }
    par_step ^= 1u;
  }
};

struct BVar {
  int n_tips, n_ops, S, R, n_codes;
  int Kp, Np, SpT, NCp;            // padded K (A columns), N (D columns), odd tip-row stride, padded code rows
  int RP;                          // rate classes per pass (1 or 2): their MMAs share a step
  int n_tiles;
  long long n_pat;
  long long ld;                    // tip-code row stride in bytes (n_tiles * 128)
  const uint8_t *codes;            // [n_tips][ld] device tip codes of this variant
  const double *weights;           // [n_pat] device weights or null
  long long pat_off;               // first pattern of the variant in the site outputs
  long long tile0;                 // the variant's first partial-sum slot (variant-major)
  long long ops_off;               // int4 entries into the ops array
  long long bmat_off;              // floats into the B array
  long long tip_off;               // floats into the tip-row array
  long long pi_off;                // doubles into the pi array
  long long brlen_off;             // doubles into the branch-length array ([2n-2])
  long long rates_off;             // doubles into the rates array ([R])
  long long ctab_off;              // doubles into the code-table array ([n_codes][S])
  int group, group_idx;            // eigen system: model group_idx of the group of this S
  double probs[4];
  float probsf[4];                 // probs rounded to float (the root's join)
};

// op.x = internal index k, op.y = first child, op.z = second child, op.w =
// four-bit fields: the stack slots of child a, child b and the result, the
// spill place + 1 that takes the result instead (0: none), the spill place + 1
// to bring back after the step, the slot it goes to, and the slot that takes D
// of child b when both children are internal
__host__ __device__ inline int op_field(int w, int k) { return (w >> (4 * k)) & 15; }
enum { OP_SA, OP_SB, OP_SO, OP_SPILL, OP_BACK, OP_BACK_SLOT, OP_DB };

__device__ __forceinline__ uint32_t su32(const void *p) {
  return static_cast<uint32_t>(__cvta_generic_to_shared(p));
}

// K-major, no-swizzle shared-memory descriptor: 8-row x 16-byte core
// matrices, K-adjacent ones LBO apart, 8-row groups SBO apart.
__device__ __forceinline__ uint64_t smem_desc(const void *base, uint32_t lbo, uint32_t sbo) {
  uint64_t d = 0;
  d |= (uint64_t)((su32(base) >> 4) & 0x3FFF);
  d |= (uint64_t)((lbo >> 4) & 0x3FFF) << 16;
  d |= (uint64_t)((sbo >> 4) & 0x3FFF) << 32;
  d |= (uint64_t)1 << 46;
  return d;
}

// byte offset of element (row n, col k) of a K-major core-matrix tile of
// 32-bit values with Kp columns
__host__ __device__ inline size_t cm_off(int n, int k, int Kp) {
  return (size_t)(n / 8) * (size_t)(Kp / 4) * 128 + (size_t)(k / 4) * 128 + (n % 8) * 16 + (k % 4) * 4;
}

// x rounded to the nearest TF32 value (10-bit mantissa, ties away from
// zero), as bits: the MMA then reads an unbiased operand instead of one
// whose low bits are dropped.  For a finite x >= 0 adding half a TF32 unit
// to the bit pattern rounds it (a carry out of the mantissa raises the
// exponent); the 13 bits below are not part of the operand and are left as
// they come (clearing them made the codon and protein batch 17.15 ms, not 16.5).
__device__ __forceinline__ uint32_t tf32_bits(float x) { return __float_as_uint(x) + 0x1000u; }

// W consecutive TMEM columns of this thread's lane (32x32b shape)
template <int W>
__device__ __forceinline__ void tmem_ld(uint32_t ta, float *v);
template <>
__device__ __forceinline__ void tmem_ld<4>(uint32_t ta, float *v) {
  uint32_t r[4];
  asm volatile("tcgen05.ld.sync.aligned.32x32b.x4.b32 {%0,%1,%2,%3}, [%4];"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3])
               : "r"(ta));
#pragma unroll
  for (int j = 0; j < 4; ++j) v[j] = __uint_as_float(r[j]);
}
template <>
__device__ __forceinline__ void tmem_ld<8>(uint32_t ta, float *v) {
  uint32_t r[8];
  asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]),
                 "=r"(r[7])
               : "r"(ta));
#pragma unroll
  for (int j = 0; j < 8; ++j) v[j] = __uint_as_float(r[j]);
}
template <>
__device__ __forceinline__ void tmem_ld<16>(uint32_t ta, float *v) {
  uint32_t r[16];
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, "
      "[%16];"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]),
        "=r"(r[7]), "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]),
        "=r"(r[14]), "=r"(r[15])
      : "r"(ta));
#pragma unroll
  for (int j = 0; j < 16; ++j) v[j] = __uint_as_float(r[j]);
}

// W consecutive TMEM columns of this thread's lane (32x32b shape)
template <int W>
__device__ __forceinline__ void tmem_st(uint32_t ta, const uint32_t *v);
template <>
__device__ __forceinline__ void tmem_st<4>(uint32_t ta, const uint32_t *v) {
  asm volatile("tcgen05.st.sync.aligned.32x32b.x4.b32 [%0], {%1,%2,%3,%4};" ::"r"(ta), "r"(v[0]), "r"(v[1]),
               "r"(v[2]), "r"(v[3])
               : "memory");
}
template <>
__device__ __forceinline__ void tmem_st<8>(uint32_t ta, const uint32_t *v) {
  asm volatile("tcgen05.st.sync.aligned.32x32b.x8.b32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8};" ::"r"(ta), "r"(v[0]),
               "r"(v[1]), "r"(v[2]), "r"(v[3]), "r"(v[4]), "r"(v[5]), "r"(v[6]), "r"(v[7])
               : "memory");
}
template <>
__device__ __forceinline__ void tmem_st<16>(uint32_t ta, const uint32_t *v) {
  asm volatile(
      "tcgen05.st.sync.aligned.32x32b.x16.b32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16};" ::"r"(
          ta),
      "r"(v[0]), "r"(v[1]), "r"(v[2]), "r"(v[3]), "r"(v[4]), "r"(v[5]), "r"(v[6]), "r"(v[7]), "r"(v[8]), "r"(v[9]),
      "r"(v[10]), "r"(v[11]), "r"(v[12]), "r"(v[13]), "r"(v[14]), "r"(v[15])
      : "memory");
}

__device__ __forceinline__ void two_sum_d(double a, double b, double &s, double &e) {
  s = a + b;
  const double bb = s - a;
  e = (a - (s - bb)) + (b - bb);
}

__device__ __forceinline__ void warp_csum_d(double &s, double &c) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    const double s2 = __shfl_xor_sync(0xffffffffu, s, o);
    const double c2 = __shfl_xor_sync(0xffffffffu, c, o);
    double t, e;
    two_sum_d(s, s2, t, e);
    s = t;
    c = c + c2 + e;
  }
}

struct BatchArgs {
  const BVar *vars;
  const int2 *work;               // [n_work] (variant, tile)
  long long n_work;
  const int4 *ops;
  const float *bmat;
  const float *tiptab;
  const double *pis;
  const float2 *pis2;             // pis as (hi, lo) float pairs
  const float4 *logtab;           // the float-pair logarithm's table (64 entries)
  double *site_lnl;               // [total patterns] or null
  double2 *partials;              // [n_work]
  int *flag;
  int slot_bytes;                 // ring slot size
  int n_st;                       // ring slots
  uint32_t *spill;                // [grid][n_spill][BT_SPILL_WORDS]
  int n_spill;
};
constexpr int BT_SPILL_WORDS = 64 * BT_M;   // the classes of a pass together have at most 64 states

// ring slot layout: [0,128) codes of child a, [128,256) codes of child b,
// then block a and block b (each the larger of a B block and a tip block)
__host__ __device__ inline int blk_bytes(const BVar &v) {
  const int b = v.Np * v.Kp * 4, t = v.NCp * v.SpT * 4;
  return ((b > t ? b : t) + 127) & ~127;
}


// What one epilogue step reads.  Shapes that follow from the padded state
// count are template parameters of the step; these are the rest, read from
// the variant once per work item.
struct EpiIn {
  uint32_t sl;               // the step's ring slot (shared-window address)
  int BB;                    // bytes of one child block in the slot
  int n_tips, n_codes;
  uint32_t chain;            // TMEM: stack slot 0 of this warp's class, at its lanes and share
  int m, n_live;             // pattern within the tile (TMEM lane), patterns of the tile
  bool last;
};

__device__ __forceinline__ float lds_f32(uint32_t a) {
  float v;
  asm volatile("ld.shared.f32 %0, [%1];" : "=f"(v) : "r"(a));
  return v;
}
__device__ __forceinline__ int lds_u8(uint32_t a) {
  uint32_t v;
  asm volatile("ld.shared.u8 %0, [%1];" : "=r"(v) : "r"(a));
  return (int)v;
}

// The share of a row that epilogue warp w owns (pt = w / 4): with one rate
// class per pass half of the states, with two the whole row of class pt, so
// that it needs no exchange with another warp.  Both are B columns wide; which
// of the two is a run-time offset, so that the warps run the same instructions
// from cache (a copy of every step for each took 16.0 ms where one took 12.0).
template <int KP, int RP>
struct Share {
  static_assert(BT_PARTS == 2, "two warps per lane group");
  static constexpr int PPR = BT_PARTS / RP;
  static constexpr int B = KP / PPR;
};

// a code outside the table counts as code 0, reported for lanes of patterns
__device__ __noinline__ int bad_code(int *flag, bool report) {
  if (report) atomicOr(flag, PGPU_FLAG_BADCODE);
  return 0;
}

// One postorder step for this warp's share of the row: the product of the
// two children (tip rows from the slot, or the MMA results from TMEM),
// rescaled by a power of two agreed with the other shares of the same rate
// class, written into the node's TMEM stack slot (or to its spill place).
// KP and RP are template parameters so that every index into the vectors is a
// compile-time constant and they stay in registers.
template <int KP, int RP>
__device__ __forceinline__ void epi_step(const BatchArgs &p, const BVar &vg, const EpiIn &in, const int4 op, int lane,
                                         int pt,
                                         int slot, uint64_t *empty, uint64_t *mma_bar, uint32_t mma_par,
                                         float (*xch)[BT_M], int &escale, bool &ok, ff &Lp) {
  using SH = Share<KP, RP>;
  constexpr int B = SH::B, PPR = SH::PPR;
  const int rate = RP == 2 ? pt : 0, e0 = RP == 2 ? 0 : pt * B;
  using C = Cols<KP, RP>;
  constexpr int SPT = KP | 1;
  const uint32_t chain = in.chain;
  float acc[B];
#pragma unroll
  for (int e = 0; e < B; ++e) acc[e] = 1.0f;
  // states S .. KP-1 need no masks: the tip rows and the B blocks are zero
  // there, so every vector's padding is a product of zeros
  const bool tips[2] = {op.y < in.n_tips, op.z < in.n_tips};
  // the tip rows first, while the MMAs of the other child run
  {
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      if (!ok || !tips[h]) continue;
      int code = lds_u8(in.sl + (uint32_t)(h * 128 + in.m));
      if (code >= in.n_codes) code = bad_code(p.flag, in.m < in.n_live && pt == 0);
      const uint32_t row = in.sl + 256 + (uint32_t)((h * RP + rate) * in.BB + (code * SPT + e0) * 4);
#pragma unroll
      for (int e = 0; e < B; ++e) acc[e] *= lds_f32(row + 4 * e);
    }
  }
  {
    const bool got = __all_sync(0xffffffffu, ok && mbar_wait_bounded_for(mma_bar, mma_par, p.flag));
    if (ok && !got) atomicOr(p.flag, PGPU_FLAG_TIMEOUT);
    ok = got;
  }
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
  {
    // TMEM loads of W columns: the widest of 16, 8, 4 that divides both the
    // first column and the width of the share
    constexpr int W = B % 16 == 0 ? 16 : B % 8 == 0 ? 8 : 4;
    auto load = [&](uint32_t col, int c0, int c1, float *d) {
#pragma unroll
      for (int c = c0; c < c1; c += W) tmem_ld<W>(chain + col + (uint32_t)c, &d[c - c0]);
    };
    // 16 columns or so at a time: two CTAs of these warps share the registers
    constexpr int CW = B <= 24 ? B : 16;
    static_assert(CW % W == 0 && B % W == 0, "a load's columns stay within its part of the row");
    auto times = [&](uint32_t col) {
#pragma unroll
      for (int c0 = 0; c0 < B; c0 += CW) {
        constexpr int c_all = CW;
        float d[c_all];
        const int c1 = c0 + CW < B ? c0 + CW : B;
        load(col, c0, c1, d);
        asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
        for (int e = c0; e < c1; ++e) acc[e] *= d[e - c0];
      }
    };
    if (ok && !(tips[0] && tips[1])) {
      if (!tips[0] && !tips[1]) {
        load(C::D, 0, B, acc);
        times((uint32_t)(op_field(op.w, OP_DB) * KP));
      } else {
        times(C::D);
      }
    }
  }
  __syncwarp();
  if (lane == 0) mbar_arrive(&empty[slot]);
  // rescale by an exact power of two per rate class; the shares agree
  float mx = 0.0f;
  {
    // three-way maxima in four chains
    float t[4] = {acc[0], acc[1], acc[2], acc[3]};
#pragma unroll
    for (int e = 4; e + 7 < B; e += 8)
#pragma unroll
      for (int k = 0; k < 4; ++k) t[k] = fmaxf(fmaxf(t[k], acc[e + 2 * k]), acc[e + 2 * k + 1]);
#pragma unroll
    for (int e = 4 + (B - 4) / 8 * 8; e < B; ++e) t[e & 3] = fmaxf(t[e & 3], acc[e]);
    mx = fmaxf(fmaxf(t[0], t[1]), fmaxf(t[2], t[3]));
  }
  float m2 = mx;
  if constexpr (PPR > 1) {
    xch[pt][in.m] = mx;
    // the exchange joins only the warps of this TMEM lane group that share
    // the rate class (named barrier 2 + lg + 4 rate); it also makes the
    // timeout verdict uniform over them, so they leave the step loop
    // together
    uint32_t all_ok;
    asm volatile(
        "{\n\t.reg .pred a, b;\n\tsetp.ne.u32 a, %1, 0;\n\t"
        "bar.red.and.pred b, %2, %3, a;\n\tselp.u32 %0, 1, 0, b;\n\t}"
        : "=r"(all_ok)
        : "r"((uint32_t)ok), "r"(2 + (in.m >> 5) + 4 * rate), "n"(PPR * 32)
        : "memory");
    ok = all_ok != 0;
    m2 = fmaxf(m2, xch[pt ^ 1][in.m]);
  } else {
    // this warp holds the whole row of its rate class
    ok = __all_sync(0xffffffffu, ok);
  }
  if (m2 < 0x1p-32f && m2 > 0.0f) {
    int ex;
    (void)frexpf(m2, &ex);
    escale += ex;
    const int k1 = min(-ex, 120), k2 = -ex - k1;
    const float f1 = __int_as_float((127 + k1) << 23), f2 = __int_as_float((127 + k2) << 23);
#pragma unroll
    for (int e = 0; e < B; ++e) acc[e] = acc[e] * f1 * f2;
  }
  {
    constexpr int WS = B % 16 == 0 ? 16 : B % 8 == 0 ? 8 : 4;
    // spill place 0, [state][lane], at this thread's
    auto place = [&]() {
      return p.spill + (size_t)blockIdx.x * p.n_spill * BT_SPILL_WORDS + (size_t)(rate * KP + e0) * BT_M + in.m;
    };
    if (const int sp = op_field(op.w, OP_SPILL)) {
      uint32_t *to = place() + (size_t)(sp - 1) * BT_SPILL_WORDS;
#pragma unroll
      for (int e = 0; e < B; ++e) to[e * BT_M] = tf32_bits(acc[e]);
    } else {
      const uint32_t col = chain + (uint32_t)(op_field(op.w, OP_SO) * KP);
#pragma unroll
      for (int c0 = 0; c0 < B; c0 += WS) {
        uint32_t v[WS];
#pragma unroll
        for (int e = 0; e < WS; ++e) v[e] = tf32_bits(acc[c0 + e]);
        tmem_st<WS>(col + (uint32_t)c0, v);
      }
    }
    if (const int sp = op_field(op.w, OP_BACK)) {   // each thread its own values
      const uint32_t *from = place() + (size_t)(sp - 1) * BT_SPILL_WORDS;
      const uint32_t col = chain + (uint32_t)(op_field(op.w, OP_BACK_SLOT) * KP);
#pragma unroll
      for (int c0 = 0; c0 < B; c0 += WS) {
        uint32_t v[WS];
#pragma unroll
        for (int e = 0; e < WS; ++e) v[e] = __ldcg(from + (c0 + e) * BT_M);
        tmem_st<WS>(col + (uint32_t)c0, v);
      }
    }
    if (in.last) {
      // sum_e pi_e x_e as a float pair: pi as (hi, lo), every product exact
      // with its cross term, the high parts added by an ordered Fast2Sum
      // (the terms are non-negative), all low parts in one float
      float hs = 0.0f, lo = 0.0f;
      const int S = vg.S;
      const float2 *pi2 = p.pis2 + vg.pi_off + e0;
#pragma unroll
      for (int e = 0; e < B; ++e)
        if (e0 + e < S) {
          const float2 pv = pi2[e];
          const float q = __fmul_rn(pv.x, acc[e]);
          float err = __fmaf_rn(pv.x, acc[e], -q);
          err = __fmaf_rn(pv.y, acc[e], err);
          const ff t = fast_two_sum(fmaxf(hs, q), fminf(hs, q));
          hs = t.h;
          lo = __fadd_rn(lo, __fadd_rn(t.l, err));
        }
      Lp = fast_two_sum(hs, lo);
    }
  }
}

// Shared state of the epilogue warps.
struct EpiShared {
  uint64_t *full, *empty;
  uint64_t *mma_bar;         // [RP]: per rate class of the pass; a phase per step
  uint64_t *stored;          // [RP]: the class's epilogue warps, likewise
  const int4 *slot_op;       // each ring slot's postorder step, written by the producer
  unsigned char *smem;
  float (*xch)[BT_M];        // [2][BT_PARTS]: per step parity and share, lane: max entry
  ff (*xchd)[BT_M];          // per share, lane: root likelihood (float pair)
  ff (*lnr)[BT_M];           // per rate class, lane: log root likelihood (float pair)
  double2 *red;
  uint32_t tmem;
};

// Every pass and postorder step of one work item (variant, tile) with
// compile-time shapes, for the epilogue warps: each step waits for
// its slot and its MMAs, runs the epilogue, and after its TMEM stores every
// warp arrives on `stored`, which the MMA warp waits for before the next
// step's MMAs.  A pass ends with the epilogue-wide verdict on timeouts, so
// the per-pass barriers below are reached by every warp alike.
template <int KP, int RP>
__device__ __forceinline__ void epi_item(const BatchArgs &p, const EpiShared &sh, const BVar &vg, const int2 wk,
                                         int tid, Ring &ring, bool &ok) {
  const int warp = tid >> 5, lane = tid & 31;
  const int lg = warp & 3, pt = warp >> 2;
  const int m = 32 * lg + lane;   // pattern within the tile
  constexpr int PPR = BT_PARTS / RP;
  const int my_rate = pt / PPR;
  // the share that combines its rate class's root likelihood
  const bool lead = pt % PPR == 0;
  // the variant's fields, once per item
  const int n_ops = vg.n_ops, R = vg.R;
  EpiIn in;
  in.BB = blk_bytes(vg);
  in.n_tips = vg.n_tips;
  in.n_codes = vg.n_codes;
  in.chain = sh.tmem + ((uint32_t)(32 * lg) << 16) +
             (uint32_t)(RP == 2 ? pt * Cols<KP, RP>::CH : pt * Share<KP, RP>::B);
  in.m = m;
  in.n_live = (int)min((long long)BT_M, vg.n_pat - (long long)wk.y * BT_M);
  const uint32_t smem0 = su32(sh.smem);
  ff Lp{0.0f, 0.0f};
  for (int r0 = 0; r0 < R && ok; r0 += RP) {
    int escale = 0;
    for (int i = 0; i < n_ops; ++i, ring.next(p.n_st)) {
      const int slot = ring.slot;
      const uint32_t par = ring.par;
      in.sl = smem0 + (uint32_t)(slot * p.slot_bytes);
      bool got = mbar_wait_bounded_for(&sh.full[slot], par, p.flag);
      got = __all_sync(0xffffffffu, got);
      if (!got) {
        ok = false;
        atomicOr(p.flag, PGPU_FLAG_TIMEOUT);
      }
      const int4 op = sh.slot_op[slot];
      uint64_t *const mma_bar = &sh.mma_bar[my_rate];
      const uint32_t mma_par = ring.par_step;
      in.last = i == n_ops - 1;
      // the max exchange is double-buffered by step parity: a group's next
      // write cannot meet a read of the previous step's values
      float(*xch)[BT_M] = sh.xch + ring.par_step * BT_PARTS;
      epi_step<KP, RP>(p, vg, in, op, lane, pt, slot, sh.empty, mma_bar, mma_par, xch, escale, ok, Lp);
      asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
      asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
      // this warp's vectors of the step are in TMEM and its D columns read
      __syncwarp();
      if (lane == 0) mbar_arrive(&sh.stored[my_rate]);
      if (!ok) break;
    }
    // one verdict for every epilogue warp before the barriers below
    {
      uint32_t all_ok;
      asm volatile(
          "{\n\t.reg .pred a, b;\n\tsetp.ne.u32 a, %1, 0;\n\t"
          "bar.red.and.pred b, 1, %2, a;\n\tselp.u32 %0, 1, 0, b;\n\t}"
          : "=r"(all_ok)
          : "r"((uint32_t)ok), "n"(BT_EPI)
          : "memory");
      ok = all_ok != 0;
    }
    if (!ok) break;
    // roots of this pass's rate classes: the shares of each meet
    sh.xchd[pt][m] = Lp;
    asm volatile("bar.sync 1, %0;" ::"n"(BT_EPI) : "memory");
    if (lead) {
      ff L{0.0f, 0.0f};
#pragma unroll
      for (int pp = my_rate * PPR; pp < my_rate * PPR + PPR; ++pp) L = ff_add(L, sh.xchd[pp][m]);
      // log(L 2^escale) in float pairs (no FP64 instruction: the FP64 pipe
      // of this GPU retires a warp's instruction in tens of cycles)
      sh.lnr[r0 + my_rate][m] = L.h > 0.0f ? ff_log(L, escale, p.logtab) : ff{-INFINITY, 0.0f};
    }
    asm volatile("bar.sync 1, %0;" ::"n"(BT_EPI) : "memory");
  }
  // join the rate classes: log sum_r probs[r] exp(lnr[r]), the largest
  // class's logarithm as a float pair plus the float logarithm of a sum in
  // [probs_min, 1]
  ff s{0.0f, 0.0f};
  const long long pat = (long long)wk.y * BT_M + m;
  if (ok && pat < vg.n_pat && pt == 0) {
    ff mx = sh.lnr[0][m];
    for (int r = 1; r < R; ++r)
      if (sh.lnr[r][m].h > mx.h) mx = sh.lnr[r][m];
    ff lnl = mx;
    if (mx.h != -INFINITY) {
      float sum = 0.0f;
      for (int r = 0; r < R; ++r) {
        const ff v = sh.lnr[r][m];
        sum += vg.probsf[r] * expf((v.h - mx.h) + (v.l - mx.l));
      }
      lnl = ff_add(mx, ff{logf(sum), 0.0f});
    }
    if (p.site_lnl) p.site_lnl[vg.pat_off + pat] = (double)lnl.h + (double)lnl.l;
    if (vg.weights) {
      const double w = vg.weights[pat];
      const float wh = (float)w;
      s = ff_mul(lnl, ff{wh, (float)(w - (double)wh)});
    } else {
      s = lnl;
    }
  }
  if (pt == 0) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) s = ff_add(s, ff_shfl_xor(s, o));
    if (lane == 0) sh.red[lg] = make_double2((double)s.h, (double)s.l);
  }
  asm volatile("bar.sync 1, %0;" ::"n"(BT_EPI) : "memory");
  if (tid == 0) {
    double ss = 0.0, cc = 0.0;
    for (int k = 0; k < 4; ++k) {
      double t, e;
      two_sum_d(ss, sh.red[k].x, t, e);
      ss = t;
      cc += e + sh.red[k].y;
    }
    // by (variant, tile), whatever order the work list runs in
    p.partials[vg.tile0 + wk.y] = make_double2(ss, cc);
  }
  asm volatile("bar.sync 1, %0;" ::"n"(BT_EPI) : "memory");
}

// An MMA warp's side of one work item: per step, once the slot is loaded, the
// step's tcgen05.mma for the internal children of rate class q.  They wait
// until the epilogue warps that write and read the class's columns have
// stored the previous step's vectors, and are committed to the class's
// mma_bar and the slot's empty barrier.  The
// warp stays converged: the descriptors are uniform and the elected thread,
// always the same, issues under a predicate (one thread issuing for both
// classes took 1,200 cycles of a step's 1,650).
template <int KP, int RP>
__device__ __forceinline__ void mma_item(const BatchArgs &p, const EpiShared &sh, const BVar &vg, const int q,
                                         const int lane, bool &first, Ring &ring, bool &ok) {
  using C = Cols<KP, RP>;
  constexpr int NP = C::NP;
  constexpr uint32_t LBO = 128, SBO = (uint32_t)(KP / 4) * 128;
  constexpr uint32_t IDESC = (1u << 4) | (2u << 7) | (2u << 10) | ((uint32_t)(NP >> 3) << 17) |
                             ((uint32_t)(BT_M >> 4) << 24);
  const int n_ops = vg.n_ops, R = vg.R, n_tips = vg.n_tips, BB16 = blk_bytes(vg) / 16;
  const uint64_t desc0 = smem_desc(sh.smem + 256, LBO, SBO);
  auto commit = [&](uint64_t *bar) {
    asm volatile(
        "{\n\t.reg .pred e;\n\telect.sync _|e, 0xffffffff;\n\t"
        "@e tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];\n\t}" ::"r"(su32(bar))
        : "memory");
  };
  for (int r0 = 0; r0 < R && ok; r0 += RP) {
    for (int i = 0; i < n_ops; ++i, ring.next(p.n_st)) {
      const int slot = ring.slot;
      const uint32_t par = ring.par;
      bool got = mbar_wait_bounded_for(&sh.full[slot], par, p.flag);
      // the epilogue warps of this class are done with the previous step
      if (!first) got = got && mbar_wait_bounded_for(&sh.stored[q], ring.par_step ^ 1u, p.flag);
      first = false;
      if (!__all_sync(0xffffffffu, got)) {
        ok = false;
        atomicOr(p.flag, PGPU_FLAG_TIMEOUT);
        return;
      }
      const int4 op = sh.slot_op[slot];
      const bool any = op.y >= n_tips || op.z >= n_tips;
      if (any) {
        const uint64_t slot_desc = desc0 + (uint32_t)slot * (uint32_t)(p.slot_bytes / 16);
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        const bool both = op.y >= n_tips && op.z >= n_tips;
#pragma unroll
        for (int h = 1; h >= 0; --h) {
          const int ch = h == 0 ? op.y : op.z;
          if (ch < n_tips) continue;
          const uint32_t a_col = (uint32_t)(q * C::CH + op_field(op.w, h == 0 ? OP_SA : OP_SB) * KP);
          const uint32_t d_col = (uint32_t)(q * C::CH + (both && h == 1 ? op_field(op.w, OP_DB) * KP : C::D));
          // the start address (16-byte units) is the descriptor's low field
          const uint64_t bd0 = slot_desc + (uint32_t)((h * RP + q) * BB16);
#pragma unroll
          for (int ks = 0; ks < KP / 8; ++ks) {
            const uint64_t bd = bd0 + (uint32_t)(ks * 2 * LBO / 16);
            asm volatile(
                "{\n\t.reg .pred e, q;\n\telect.sync _|e, 0xffffffff;\n\tsetp.ne.b32 q, %4, 0;\n\t"
                "@e tcgen05.mma.cta_group::1.kind::tf32 [%0], [%1], %2, %3, q;\n\t}" ::"r"(sh.tmem + d_col),
                "r"(sh.tmem + a_col + (uint32_t)(ks * 8)), "l"(bd), "r"(IDESC), "r"(ks > 0 ? 1u : 0u)
                : "memory");
          }
        }
        commit(&sh.mma_bar[q]);
        commit(&sh.empty[slot]);
      } else if (lane == 0) {
        mbar_arrive(&sh.mma_bar[q]);
        mbar_arrive(&sh.empty[slot]);
      }
      __syncwarp();
    }
  }
}

// One padded state count and number of rate classes per pass: a kernel of its
// own for each holds its instructions in cache and its vectors in registers
// (one kernel with a case for each took
// 11.3 ms on 16 protein and 16 codon models, two of these 10.2).
template <int KP, int RP>
__global__ void __launch_bounds__(bt_threads(RP), 2) batch_tc_kernel(const BatchArgs p) {
  extern __shared__ __align__(1024) unsigned char smem[];
  __shared__ uint64_t full[BT_ST], empty[BT_ST], mma_bar[RP], stored[RP];
  __shared__ int4 slot_op[BT_ST];
  __shared__ uint32_t tmem_base;
  __shared__ float xch[2 * BT_PARTS][BT_M];   // per step parity and share, lane: max entry
  __shared__ ff xchd[BT_PARTS][BT_M];   // per share, lane: root likelihood
  __shared__ ff lnr[4][BT_M];           // per rate class, lane: log root likelihood
  __shared__ double2 red[4];
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;

  // the next kernel of the chain may take SMs as they come free
  asm volatile("griddepcontrol.launch_dependents;");
  if (warp == BT_EPI_WARPS) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(
                     su32(&tmem_base)),
                 "r"(BT_TMEM_COLS));
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;");
  }
  if (tid == 0) {
    for (int s = 0; s < BT_ST; ++s) {
      mbar_init(&full[s], 1);
      mbar_init(&empty[s], RP + BT_EPI_WARPS);   // the MMA warps + the epilogue warps
    }
    for (int q = 0; q < RP; ++q) {
      mbar_init(&mma_bar[q], 1);
      mbar_init(&stored[q], BT_EPI_WARPS / RP);   // after a step's TMEM stores
    }
    fence_mbarrier_init();
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
  const uint32_t tmem = tmem_base;

  const EpiShared sh{full, empty, mma_bar, stored, slot_op, smem, xch, xchd, lnr, red, tmem};
  if (warp == BT_PRODUCER) {
    // ------------------------------------------------------------ producer
    if (lane == 0) {
      long long seq = 0;
      Ring ring;
      bool ok = true;
      for (long long w = blockIdx.x; w < p.n_work && ok; w += gridDim.x) {
        const int2 wk = __ldg(p.work + w);
        const BVar &v = p.vars[wk.x];
        const int BB = blk_bytes(v);
        const uint32_t bmat_bytes = (uint32_t)(v.Np * v.Kp * 4);
        const uint32_t tip_bytes = (uint32_t)(v.NCp * v.SpT * 4);
        const int R = v.R, n_ops = v.n_ops, n_tips = v.n_tips;
        const long long ops_off = v.ops_off, ld = v.ld, tip_off = v.tip_off, bmat_off = v.bmat_off;
        const uint8_t *codes = v.codes;
        const long long bstride = (long long)v.Np * v.Kp, tstride = (long long)v.NCp * v.SpT;
        for (int r0 = 0; r0 < R && ok; r0 += RP) {
          for (int i = 0; i < n_ops; ++i, ++seq, ring.next(p.n_st)) {
            const int slot = ring.slot;
            const int4 op = __ldg(p.ops + ops_off + i);
            if (seq >= p.n_st && !mbar_wait_bounded_for(&empty[slot], ring.par ^ 1u, p.flag)) {
              ok = false;
              break;
            }
            unsigned char *sl = smem + (size_t)slot * p.slot_bytes;
            uint32_t tx = 0;
            for (int h = 0; h < 2; ++h) {
              const int ch = h == 0 ? op.y : op.z;
              tx += ch < n_tips ? 128u + RP * tip_bytes : RP * bmat_bytes;
            }
            // the step itself, published by the arrive below (release)
            slot_op[slot] = op;
            mbar_arrive_expect_tx(&full[slot], tx);
            for (int h = 0; h < 2; ++h) {
              const int ch = h == 0 ? op.y : op.z;
              if (ch < n_tips)
                bulk_g2s(sl + h * 128, codes + (long long)ch * ld + (long long)wk.y * 128, 128u, &full[slot]);
              for (int q = 0; q < RP; ++q) {
                unsigned char *blk = sl + 256 + (size_t)(h * RP + q) * BB;
                if (ch < n_tips)
                  bulk_g2s(blk, p.tiptab + tip_off + ((long long)ch * R + r0 + q) * tstride, tip_bytes,
                           &full[slot]);
                else
                  bulk_g2s(blk, p.bmat + bmat_off + ((long long)(ch - n_tips) * R + r0 + q) * bstride,
                           bmat_bytes, &full[slot]);
              }
            }
          }
        }
      }
      // its last copies have arrived before it returns
      for (int s = 0; s < p.n_st; ++s)
        if (seq > s) (void)mbar_wait_bounded_for(&full[s], s < ring.slot ? ring.par : ring.par ^ 1u, p.flag);
    }
  } else if (warp >= BT_MMA) {
    // ------------------------------------------------------------ MMA issue
    const int q = warp - BT_MMA;
    Ring ring;
    bool ok = true, first = true;
    for (long long w = blockIdx.x; w < p.n_work && ok; w += gridDim.x)
      mma_item<KP, RP>(p, sh, p.vars[__ldg(p.work + w).x], q, lane, first, ring, ok);
    // the last MMAs finish before TMEM is released
    if (!first) (void)mbar_wait_bounded_for(&mma_bar[q], ring.par_step ^ 1u, p.flag);
  } else {
    // ------------------------------------------------------------ epilogue
    // warp w: TMEM lanes 32 (w % 4) .. 32 (w % 4) + 31, share w / 4 of the
    // row.
    Ring ring;
    bool ok = true;
    for (long long w = blockIdx.x; w < p.n_work && ok; w += gridDim.x) {
      const int2 wk = __ldg(p.work + w);
      epi_item<KP, RP>(p, sh, p.vars[wk.x], wk, tid, ring, ok);
    }
  }

  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
  if (warp == BT_EPI_WARPS)
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(BT_TMEM_COLS));
  // done only when the kernels before it in the chain are
  asm volatile("griddepcontrol.wait;" ::: "memory");
}

// Per variant: sum its tiles' (sum, compensation) pairs in tile order.
__global__ void __launch_bounds__(256) batch_finalize_kernel(const double2 *partials,
                                                            const long long *tile_base,
                                                            const int *n_tiles, int n_var, double *out) {
  const int v = blockIdx.x;
  if (v >= n_var) return;
  const double sum = pgpu_forms::csum_block<256>(partials + tile_base[v], n_tiles[v]);
  if (threadIdx.x == 0) out[v] = sum;
}

// Setup: for every branch of every variant of one state count S and every
// rate class, P = U diag(exp(lambda r t)) Ui in FP64 (shared memory), then
//   tip branch      tip rows tab[c][i] = sum_j P[i][j] code_tab[c][j]  (float)
//   internal branch B block B[n=i][k=j] = P[i][j] in the core-matrix layout
// Bound by FP64, which this GPU runs at 1/64 of the FP32 rate, so as little
// of it as gives the same values: U diag(e) is formed once per CTA; U and Ui
// come from a symmetric eigen system scaled by the frequencies, so that
// pi_i P_ij = pi_j P_ji and half the entries are summed; a tip row sums the
// states its code holds.  16 protein (4 classes) and 16 codon models, 254
// branches each: 1.26 ms against 5.04.
struct SetupArgs {
  const BVar *vars;
  const int *members;             // variants of this group
  const double *U, *lam, *Ui;     // group eigen systems [g][S][S], [g][S], [g][S][S]
  const int *status;              // [g]
  const double *brlen, *rates, *ctab, *pis;
  float *bmat, *tiptab;
  int *flag;
  int S;
};

__global__ void __launch_bounds__(256) batch_setup_kernel(const SetupArgs a) {
  extern __shared__ __align__(16) double P[];   // [S][S], then U diag(e) [S][S], Ui [S][S], e[S], pi[S], 1/pi[S]
  __shared__ unsigned long long holds[256];     // states of each code
  const int S = a.S, SS = S * S;
  const int vi = a.members[blockIdx.z];
  const BVar &v = a.vars[vi];
  const int c = blockIdx.x, r = blockIdx.y, tid = threadIdx.x, nt = blockDim.x;
  const int n_br = 2 * v.n_tips - 2;
  if (c >= n_br || r >= v.R) return;
  const int g = v.group_idx;
  if (a.status[g]) {
    if (c == 0 && r == 0 && tid == 0) atomicOr(a.flag, pgpu_model_flag(a.status[g]));
    return;
  }
  const double *U = a.U + (size_t)g * SS, *Ui = a.Ui + (size_t)g * SS, *lam = a.lam + (size_t)g * S;
  double *W = P + SS, *V = W + SS, *e = V + SS, *pi = e + S, *rpi = pi + S;
  const double t = a.brlen[v.brlen_off + c], rate = a.rates[v.rates_off + r];
  const bool ident = !(t * rate >= 1e-10);   // effective time: a rate-0 class gets I exactly
  const double *ct = a.ctab + v.ctab_off;
  for (int k = tid; k < S; k += nt) {
    e[k] = exp(lam[k] * rate * t);
    pi[k] = a.pis[v.pi_off + k];
    rpi[k] = 1.0 / pi[k];
  }
  if (c < v.n_tips)
    for (int code = tid >> 5; code < v.n_codes; code += nt >> 5) {
      const int lane = tid & 31;
      unsigned m[2];
      for (int h = 0; h < 2; ++h) {
        const int j = 32 * h + lane;
        m[h] = __ballot_sync(0xffffffffu, j < S && __double_as_longlong(ct[code * S + j]) != 0);
      }
      if (lane == 0) holds[code] = m[0] | (unsigned long long)m[1] << 32;
    }
  __syncthreads();
  if (ident) {
    for (int o = tid; o < SS; o += nt) P[o] = o / S == o % S ? 1.0 : 0.0;
  } else {
    for (int o = tid; o < SS; o += nt) {
      W[o] = U[o] * e[o % S];
      V[o] = Ui[o];
    }
    __syncthreads();
    // the entries on and above the diagonal: rows a and S - 1 - a together
    // are S + 1 of them
    for (int o = tid; o < S * (S + 1) / 2; o += nt) {
      const int q = o / (S + 1), m = o % (S + 1);
      const int i = m < S - q ? q : S - 1 - q, j = m < S - q ? q + m : m - 1;
      double x = 0.0;
      for (int k = 0; k < S; ++k) x = fma(W[i * S + k], V[k * S + j], x);
      x = fmax(x, 0.0);   // transition probabilities: clamp eigen-product noise below 0
      P[i * S + j] = x;
      if (i != j) P[j * S + i] = fmax(x * (pi[i] * rpi[j]), 0.0);
    }
  }
  __syncthreads();
  if (c < v.n_tips) {
    float *out = a.tiptab + v.tip_off + ((size_t)c * v.R + r) * v.NCp * v.SpT;
    for (int o = tid; o < v.NCp * v.SpT; o += nt) {
      const int code = o / v.SpT, i = o % v.SpT;
      float y = 0.0f;
      if (i < S && code < v.n_codes) {
        double x = 0.0;
        for (unsigned long long m = holds[code]; m; m &= m - 1) {
          const int j = __ffsll((long long)m) - 1;
          x = fma(P[i * S + j], ct[code * S + j], x);
        }
        y = (float)x;
      }
      out[o] = y;
    }
  } else {
    unsigned char *out = reinterpret_cast<unsigned char *>(
        a.bmat + v.bmat_off + ((size_t)(c - v.n_tips) * v.R + r) * (size_t)v.Np * v.Kp);
    for (int o = tid; o < v.Np * v.Kp; o += nt) {
      const int n = o / v.Kp, k = o % v.Kp;
      const float x = (n < S && k < S) ? (float)P[n * S + k] : 0.0f;   // P >= 0 after clamping
      *reinterpret_cast<uint32_t *>(out + cm_off(n, k, v.Kp)) = tf32_bits(x);
    }
  }
}

// The FP64 comparison form over the first `sample` patterns of every
// variant: one CTA per (variant, block of 32 patterns), thread = pattern,
// all rate classes and states in FP64; the stack of vectors in shared
// memory, each branch's P rebuilt in shared memory from the eigen system.
struct F64Args {
  const BVar *vars;
  const int4 *ops;
  const double *U, *lam, *Ui;     // per group, indexed through vars[].group / group_idx
  long long gU[8], gL[8];         // group bases (doubles) into U/Ui and lam
  const double *brlen, *rates, *ctab, *pis;
  double2 *partials;              // [n_var][blocks]
  int blocks;                     // blocks per variant
  long long sample;
  int max_depth;
};

constexpr int F64_NP = 32;

__global__ void __launch_bounds__(F64_NP) batch_fp64_kernel(const F64Args a) {
  extern __shared__ __align__(16) double sm[];
  const int vi = blockIdx.y, blk = blockIdx.x, tid = threadIdx.x;
  const BVar &v = a.vars[vi];
  const int S = v.S, SS = S * S, R = v.R;
  double *P = sm;                                   // [S][S]
  double *e = P + SS;                               // [S]
  double *stk = e + 64;                             // [depth][S][32]
  const long long n_use = min(a.sample, v.n_pat);
  const long long pat = (long long)blk * F64_NP + tid;
  const bool active = pat < n_use;
  const double *U = a.U + a.gU[v.group] + (size_t)v.group_idx * SS;
  const double *Ui = a.Ui + a.gU[v.group] + (size_t)v.group_idx * SS;
  const double *lam = a.lam + a.gL[v.group] + (size_t)v.group_idx * S;
  const double *ct = a.ctab + v.ctab_off;
  double lnr[4];
  double x[2][64];
  for (int r = 0; r < R; ++r) {
    int sp = 0;
    long long esc = 0;
    for (int i = 0; i < v.n_ops; ++i) {
      const int4 op = a.ops[v.ops_off + i];
      // pop the internal children (b above a)
      for (int h = 1; h >= 0; --h) {
        const int ch = h == 0 ? op.y : op.z;
        if (ch >= v.n_tips) {
          --sp;
          for (int j = 0; j < S; ++j) x[h][j] = stk[((size_t)sp * S + j) * F64_NP + tid];
        }
      }
      double out[64];
      for (int j = 0; j < S; ++j) out[j] = 1.0;
      for (int h = 0; h < 2; ++h) {
        const int ch = h == 0 ? op.y : op.z;
        __syncthreads();
        const double t = a.brlen[v.brlen_off + ch], rate = a.rates[v.rates_off + r];
        const bool ident = !(t * rate >= 1e-10);
        for (int k = tid; k < S; k += F64_NP) e[k] = exp(lam[k] * rate * t);
        __syncthreads();
        for (int o = tid; o < SS; o += F64_NP) {
          const int ii = o / S, jj = o % S;
          double y = 0.0;
          if (ident) y = ii == jj ? 1.0 : 0.0;
          else
            for (int k = 0; k < S; ++k) y = fma(U[ii * S + k] * e[k], Ui[k * S + jj], y);
          P[o] = fmax(y, 0.0);
        }
        __syncthreads();
        if (ch < v.n_tips) {
          int code = active ? v.codes[(long long)ch * v.ld + pat] : 0;
          if (code >= v.n_codes) code = 0;
          for (int j = 0; j < S; ++j) x[h][j] = ct[code * S + j];
        }
        for (int ii = 0; ii < S; ++ii) {
          double y = 0.0;
          for (int jj = 0; jj < S; ++jj) y = fma(P[ii * S + jj], x[h][jj], y);
          out[ii] *= y;
        }
      }
      double mx = 0.0;
      for (int j = 0; j < S; ++j) mx = fmax(mx, out[j]);
      if (mx > 0.0 && mx < 0x1p-256) {
        int ex;
        (void)frexp(mx, &ex);
        esc += ex;
        for (int j = 0; j < S; ++j) out[j] = ldexp(out[j], -ex);
      }
      if (i + 1 < v.n_ops) {
        for (int j = 0; j < S; ++j) stk[((size_t)sp * S + j) * F64_NP + tid] = out[j];
        ++sp;
      } else {
        double L = 0.0;
        for (int j = 0; j < S; ++j) L += a.pis[v.pi_off + j] * out[j];
        lnr[r] = log(L) + (double)esc * 0.69314718055994530942;
      }
    }
  }
  double s = 0.0, c = 0.0;
  if (active) {
    double mxl = -INFINITY;
    for (int r = 0; r < R; ++r) mxl = fmax(mxl, lnr[r]);
    double sum = 0.0;
    for (int r = 0; r < R; ++r) sum += v.probs[r] * exp(lnr[r] - mxl);
    const double lnl = mxl + log(sum);
    s = v.weights ? v.weights[pat] * lnl : lnl;
  }
  warp_csum_d(s, c);
  if (tid == 0) a.partials[(size_t)vi * a.blocks + blk] = make_double2(s, c);
}

}  // namespace

// ---------------------------------------------------------------------------
// host side
// ---------------------------------------------------------------------------

namespace {

// shared memory: what each of two CTAs on an SM may ask for beside the static
// part, and that part
constexpr size_t BT_SMEM_STATIC = 10 * 1024;
constexpr size_t BT_SMEM_PAIR = (228 * 1024) / 2 - 1024 - BT_SMEM_STATIC;

// Stack slots of a postorder schedule over `slots` slots, appended to ops;
// returns the spill places used.  A step whose children are both internal
// needs them in two slots and a third free; `need` is what a subtree takes
// above its own base.  The first child's vector keeps its slot while the
// second child's subtree is walked if that fits, else it is spilled and
// brought back by the step that ends that subtree.
int place_ops(const TreeSchedule &sch, int n, int slots, std::vector<int4> *ops) {
  const size_t first = ops->size(), m = sch.ops.size();
  std::vector<int> need(m), base(m, 0), place(m, 0), at(2 * n, -1);
  for (size_t i = 0; i < m; ++i) {
    const SchedOp &o = sch.ops[i];
    at[n + o.k] = (int)i;
    const int a = o.a >= n ? need[at[o.a]] : 0, b = o.b >= n ? need[at[o.b]] : 0;
    need[i] = a && b ? std::min(std::max(std::max(a, 1 + b), 3), slots) : std::max(std::max(a, b), 1);
    ops->push_back(make_int4(o.k, o.a, o.b, 0));
  }
  int used = 0;
  for (size_t i = m; i-- > 0;) {
    const SchedOp &o = sch.ops[i];
    const int x = base[i], ia = o.a >= n ? at[o.a] : -1, ib = o.b >= n ? at[o.b] : -1;
    int sa = x, sb = x, db = 0;
    if (ia >= 0) {
      base[ia] = x;
      place[ia] = place[i];
    }
    if (ib >= 0) {
      base[ib] = x;
      place[ib] = place[i];
    }
    if (ia >= 0 && ib >= 0) {
      db = x + 2;
      if (x + 1 + need[ib] <= slots) {
        base[ib] = sb = x + 1;
      } else {
        const int sp = place[i];
        used = std::max(used, sp + 1);
        place[ib] = sp + 1;
        sa = x + 1;
        (*ops)[first + ia].w |= (sp + 1) << (4 * OP_SPILL);
        (*ops)[first + ib].w |= (sp + 1) << (4 * OP_BACK) | sa << (4 * OP_BACK_SLOT);
      }
    }
    (*ops)[first + i].w |= sa << (4 * OP_SA) | sb << (4 * OP_SB) | x << (4 * OP_SO) | db << (4 * OP_DB);
  }
  return used;
}

}  // namespace

struct BatchLaunch {
  int Kp, RP, slot_bytes, n_st, grid;
  long long n_work, work0;
};

struct pgpu_batch {
  int n_var = 0;
  int max_depth = 0;
  long long n_work = 0, total_pat = 0;
  std::vector<BVar> hvars;
  std::vector<int> group_S;                     // state count of each group
  std::vector<std::vector<int>> group_members;  // variant ids per group
  // device
  BVar *vars = nullptr;
  int2 *work = nullptr;
  int4 *ops = nullptr;
  float *bmat = nullptr, *tiptab = nullptr;
  double *pis = nullptr, *brlen = nullptr, *rates = nullptr, *ctab = nullptr;
  float2 *pis2 = nullptr;
  float4 *logtab = nullptr;
  double *Q = nullptr, *U = nullptr, *Ui = nullptr, *lam = nullptr;
  int *status = nullptr, *members = nullptr;
  long long *tile_base = nullptr;
  int *n_tiles = nullptr;
  double2 *partials = nullptr;
  std::vector<long long> gQ, gL, gM;            // group bases (doubles, doubles, ints)
  std::vector<BatchLaunch> launches;
  int n_spill = 0;
  size_t lim_smem = 0;                          // what a run may ask for
  uint32_t *spill = nullptr;
};

namespace {

template <typename T>
pgpu_status upload(pgpu_ctx *ctx, T **dst, const std::vector<T> &src) {
  const size_t bytes = std::max<size_t>(src.size() * sizeof(T), 16);
  PGPU_CUDA(ctx, cudaMalloc(reinterpret_cast<void **>(dst), bytes));
  if (!src.empty())
    PGPU_CUDA(ctx, cudaMemcpy(*dst, src.data(), src.size() * sizeof(T), cudaMemcpyHostToDevice));
  return PGPU_OK;
}

// words of spill places: the launches overlap at their ends, so each has its own
size_t launch_spill(const pgpu_batch *b) {
  size_t ctas = 0;
  for (const BatchLaunch &l : b->launches) ctas += l.grid;
  return ctas * b->n_spill * BT_SPILL_WORDS;
}

template <int KP, int RP>
pgpu_status launch_tc(pgpu_ctx *ctx, const BatchArgs &a, const BatchLaunch &l, bool chained) {
  auto kernel = batch_tc_kernel<KP, RP>;
  // at least 72 KB, so that no third CTA waits on an SM for TMEM columns
  const size_t smem = std::max<size_t>((size_t)l.n_st * l.slot_bytes, 72 * 1024);
  PGPU_CUDA(ctx, cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
  // without it the driver may leave room for one CTA only
  PGPU_CUDA(ctx, cudaFuncSetAttribute(kernel, cudaFuncAttributePreferredSharedMemoryCarveout,
                                      cudaSharedmemCarveoutMaxShared));
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3((unsigned)l.grid);
  cfg.blockDim = dim3(bt_threads(RP));
  cfg.dynamicSmemBytes = smem;
  cfg.stream = ctx->stream;
  cudaLaunchAttribute at[1];
  at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  at[0].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = at;
  cfg.numAttrs = chained ? 1 : 0;
  PGPU_CUDA(ctx, cudaLaunchKernelEx(&cfg, kernel, a));
  return pgpu_after_launch(ctx, "batch_tc_kernel");
}

pgpu_status launch_tc(pgpu_ctx *ctx, const BatchArgs &a, const BatchLaunch &l, bool chained) {
  if (l.RP == 2) {
    switch (l.Kp) {
      case 8: return launch_tc<8, 2>(ctx, a, l, chained);
      case 16: return launch_tc<16, 2>(ctx, a, l, chained);
      case 24: return launch_tc<24, 2>(ctx, a, l, chained);
      default: return launch_tc<32, 2>(ctx, a, l, chained);
    }
  }
  switch (l.Kp) {
    case 8: return launch_tc<8, 1>(ctx, a, l, chained);
    case 16: return launch_tc<16, 1>(ctx, a, l, chained);
    case 24: return launch_tc<24, 1>(ctx, a, l, chained);
    case 32: return launch_tc<32, 1>(ctx, a, l, chained);
    case 40: return launch_tc<40, 1>(ctx, a, l, chained);
    case 48: return launch_tc<48, 1>(ctx, a, l, chained);
    case 56: return launch_tc<56, 1>(ctx, a, l, chained);
    default: return launch_tc<64, 1>(ctx, a, l, chained);
  }
}

void free_batch(pgpu_batch *b) {
  void *ptrs[] = {b->vars, b->work,   b->ops, b->bmat,   b->tiptab,  b->pis,      b->brlen,
                  b->rates, b->ctab,  b->Q,   b->U,      b->Ui,      b->lam,      b->status,
                  b->members, b->tile_base, b->n_tiles, b->partials, b->pis2, b->logtab, b->spill};
  for (void *p : ptrs)
    if (p) cudaFree(p);
  delete b;
}

}  // namespace

extern "C" {

pgpu_status pgpu_batch_create(pgpu_ctx *ctx, const pgpu_variant *vs, int n_var, pgpu_batch **out) {
  return pgpu_batch_create_opts(ctx, vs, n_var, nullptr, out);
}

pgpu_status pgpu_batch_create_opts(pgpu_ctx *ctx, const pgpu_variant *vs, int n_var,
                                   const pgpu_batch_options *opts, pgpu_batch **out) {
  if (!ctx || !out) return PGPU_ERR_ARG;
  *out = nullptr;
  const int rate_pairs = opts ? opts->rate_pairs : 1;
  const int order = opts ? opts->order : PGPU_BATCH_ORDER_VARIANT;
  if (order != PGPU_BATCH_ORDER_VARIANT && order != PGPU_BATCH_ORDER_COST)
    return pgpu_set_err(ctx, PGPU_ERR_ARG, "batch: unknown work order %d", order);
  if (!vs || n_var < 1) return pgpu_set_err(ctx, PGPU_ERR_ARG, "batch: no variants");
  PGPU_CUDA(ctx, cudaSetDevice(ctx->device));
  pgpu_batch *b = new pgpu_batch();
  b->n_var = n_var;
  std::vector<int4> ops;
  std::vector<int2> work;
  std::vector<double> pis, brl, rts, ctab, Qg;
  std::vector<long long> tile_base;
  std::vector<int> ntiles, members;
  long long bm_off = 0, tt_off = 0, pat_off = 0;
  size_t lim_blk = 0;
  auto fail = [&](pgpu_status st, const char *msg, int v) {
    free_batch(b);
    return pgpu_set_err(ctx, st, "batch: variant %d: %s", v, msg);
  };
  for (int vi = 0; vi < n_var; ++vi) {
    const pgpu_variant &x = vs[vi];
    const pgpu_model &m = x.model;
    if (!x.tree.brlen || !m.Q || !m.pi || !m.rates || !m.probs || !x.codes.table || !x.tip_codes)
      return fail(PGPU_ERR_ARG, "null field", vi);
    if (m.n_states < 2 || m.n_states > 64) return fail(PGPU_ERR_LIMIT, "2..64 states", vi);
    if (m.n_rates < 1 || m.n_rates > 4) return fail(PGPU_ERR_LIMIT, "1..4 rate classes", vi);
    if (x.codes.n_codes < 1 || x.codes.n_codes > 255) return fail(PGPU_ERR_ARG, "1..255 codes", vi);
    if (x.tree.n_tips < 2 || x.tree.n_tips > 255) return fail(PGPU_ERR_LIMIT, "2..255 tips", vi);
    const long long nt = (long long)((x.n_pat + BT_M - 1) / BT_M);
    if (x.ld_pat % 128 != 0 || (long long)x.ld_pat < nt * BT_M || ((uintptr_t)x.tip_codes & 15))
      return fail(PGPU_ERR_ARG, "ld_pat must be a multiple of 128 covering the padded tiles", vi);
    TreeSchedule sch;
    pgpu_status st = pgpu_build_schedule(ctx, &x.tree, &sch);
    if (st != PGPU_OK) {
      free_batch(b);
      return st;
    }
    const int n = x.tree.n_tips, S = m.n_states, R = m.n_rates;
    BVar v{};
    v.n_tips = n;
    v.n_ops = n - 1;
    v.S = S;
    v.R = R;
    v.n_codes = x.codes.n_codes;
    v.Kp = (S + 7) / 8 * 8;
    v.Np = (S + 15) / 16 * 16;
    v.SpT = v.Kp | 1;                     // odd row stride (distinct codes, distinct banks), entries S.. zero
    v.NCp = (x.codes.n_codes + 3) / 4 * 4; // rows padded so a block is a multiple of 16 bytes
    v.n_tiles = (int)nt;
    v.n_pat = (long long)x.n_pat;
    v.ld = (long long)x.ld_pat;
    v.codes = x.tip_codes;
    v.weights = x.weights;
    v.pat_off = pat_off;
    v.ops_off = (long long)ops.size();
    v.bmat_off = bm_off;
    v.tip_off = tt_off;
    v.pi_off = (long long)pis.size();
    v.brlen_off = (long long)brl.size();
    v.rates_off = (long long)rts.size();
    v.ctab_off = (long long)ctab.size();
    for (int r = 0; r < 4; ++r) {
      v.probs[r] = r < R ? m.probs[r] : 0.0;
      v.probsf[r] = (float)v.probs[r];
    }
    if (sch.max_depth > (BT_LIMIT_COLS - 2 * v.Np) / v.Kp)
      return fail(PGPU_ERR_LIMIT, "tree too deep for the TMEM stack", vi);
    const size_t blk = (std::max<size_t>((size_t)v.Np * v.Kp * 4, (size_t)v.NCp * v.SpT * 4) + 127) & ~size_t(127);
    // two rate classes per pass: their chains overlap, and two ring slots of
    // both still let two CTAs share an SM
    const bool pairs = rate_pairs && R % 2 == 0 && v.Kp <= 32;
    v.RP = pairs && 2 * (256 + 4 * blk) <= BT_SMEM_PAIR ? 2 : 1;
    // what the engine accepts is reckoned with one CTA per SM and its stack
    const bool lim_pairs = pairs && (BT_LIMIT_COLS - 4 * v.Np) / (2 * v.Kp) >= sch.max_depth;
    lim_blk = std::max(lim_blk, (lim_pairs ? 2 : 1) * blk);
    b->max_depth = std::max(b->max_depth, sch.max_depth);
    b->n_spill = std::max(b->n_spill, place_ops(sch, n, stack_slots(v.Kp, v.Np, v.RP), &ops));
    v.tile0 = (long long)work.size();
    for (long long t = 0; t < nt; ++t) work.push_back(make_int2(vi, (int)t));
    tile_base.push_back((long long)work.size() - nt);
    ntiles.push_back((int)nt);
    pis.insert(pis.end(), m.pi, m.pi + S);
    brl.insert(brl.end(), x.tree.brlen, x.tree.brlen + 2 * n - 2);
    rts.insert(rts.end(), m.rates, m.rates + R);
    ctab.insert(ctab.end(), x.codes.table, x.codes.table + (size_t)v.n_codes * S);
    bm_off += (long long)(n - 2) * R * v.Np * v.Kp;
    tt_off += (long long)n * R * v.NCp * v.SpT;
    bm_off = (bm_off + 3) / 4 * 4;
    tt_off = (tt_off + 3) / 4 * 4;
    pat_off += v.n_pat;
    // eigen group by state count
    int g = -1;
    for (size_t k = 0; k < b->group_S.size(); ++k)
      if (b->group_S[k] == S) g = (int)k;
    if (g < 0) {
      g = (int)b->group_S.size();
      b->group_S.push_back(S);
      b->group_members.emplace_back();
    }
    v.group = g;
    v.group_idx = (int)b->group_members[g].size();
    b->group_members[g].push_back(vi);
    b->hvars.push_back(v);
  }
  if (b->group_S.size() > 8) return fail(PGPU_ERR_LIMIT, "at most 8 distinct state counts", 0);
  // group layout of Q / pi / eigen arrays
  std::vector<double> Qall, PIall;
  long long q_acc = 0, l_acc = 0;
  for (size_t g = 0; g < b->group_S.size(); ++g) {
    const int S = b->group_S[g];
    b->gQ.push_back(q_acc);
    b->gL.push_back(l_acc);
    b->gM.push_back((long long)members.size());
    for (int vi : b->group_members[g]) {
      Qall.insert(Qall.end(), vs[vi].model.Q, vs[vi].model.Q + (size_t)S * S);
      PIall.insert(PIall.end(), vs[vi].model.pi, vs[vi].model.pi + S);
      members.push_back(vi);
    }
    q_acc += (long long)b->group_members[g].size() * S * S;
    l_acc += (long long)b->group_members[g].size() * S;
  }
  b->lim_smem = std::max<size_t>(BT_ST * (256 + 2 * lim_blk), 120 * 1024);
  // A launch per padded state count and rate classes per pass, those with the
  // longest items first; its ring takes what its variants need, two CTAs per SM
  // where two slots or more fit in half of the shared memory.
  std::vector<BatchLaunch> launches;
  for (const BVar &v : b->hvars) {
    const int slot_bytes = 256 + 2 * v.RP * blk_bytes(v);
    auto it = std::find_if(launches.begin(), launches.end(),
                           [&](const BatchLaunch &l) { return l.Kp == v.Kp && l.RP == v.RP; });
    if (it == launches.end()) it = launches.insert(it, BatchLaunch{v.Kp, v.RP, 0, BT_ST, 1, 0, 0});
    it->slot_bytes = std::max(it->slot_bytes, slot_bytes);
  }
  std::stable_sort(launches.begin(), launches.end(), [](const BatchLaunch &x, const BatchLaunch &y) {
    return x.RP * x.Kp > y.RP * y.Kp;
  });
  std::vector<int2> all;
  all.swap(work);
  work.reserve(all.size());
  for (BatchLaunch &l : launches) {
    l.work0 = (long long)work.size();
    const int per_sm = 2 * (size_t)l.slot_bytes <= BT_SMEM_PAIR ? 2 : 1;
    l.n_st = (int)std::min<size_t>(BT_ST, (per_sm == 2 ? BT_SMEM_PAIR : ctx->smem_optin - BT_SMEM_STATIC) / l.slot_bytes);
    std::vector<int2> mine;
    for (const int2 &w : all) {
      const BVar &v = b->hvars[w.x];
      if (v.Kp == l.Kp && v.RP == l.RP) mine.push_back(w);
    }
    l.n_work = (long long)mine.size();
    l.grid = (int)std::min<long long>(std::max(per_sm * ctx->num_sms, 1), std::max<long long>(l.n_work, 1));
    if (order == PGPU_BATCH_ORDER_COST && !mine.empty()) {
      // Largest items first, dealt back and forth over the persistent CTAs
      // (CTA c runs items c, c + G, c + 2G, ...), so every CTA's total is close
      // to the mean.  An item's cost is its postorder steps times its passes.
      const long long G = l.grid;
      std::vector<size_t> idx(mine.size());
      for (size_t i = 0; i < idx.size(); ++i) idx[i] = i;
      auto cost = [&](size_t i) {
        const BVar &v = b->hvars[mine[i].x];
        return (long long)(v.R / v.RP) * v.n_ops;
      };
      std::stable_sort(idx.begin(), idx.end(), [&](size_t x, size_t y) { return cost(x) > cost(y); });
      std::vector<std::vector<int2>> per(G);
      for (size_t r = 0; r < idx.size(); ++r) {
        const long long round = (long long)r / G, pos = (long long)r % G;
        per[round % 2 == 0 ? pos : G - 1 - pos].push_back(mine[idx[r]]);
      }
      // CTA c's k-th item goes to position k G + c; the last, partial round
      // is packed to the front of its row
      mine.clear();
      const size_t rounds = (idx.size() + G - 1) / G;
      for (size_t k = 0; k < rounds; ++k)
        for (long long c = 0; c < G; ++c)
          if (k < per[c].size()) mine.push_back(per[c][k]);
    }
    work.insert(work.end(), mine.begin(), mine.end());
  }
  b->launches = launches;
  b->n_work = (long long)work.size();
  b->total_pat = pat_off;
  pgpu_status st = PGPU_OK;
  if (st == PGPU_OK) st = upload(ctx, &b->vars, b->hvars);
  if (st == PGPU_OK) st = upload(ctx, &b->work, work);
  if (st == PGPU_OK) st = upload(ctx, &b->ops, ops);
  if (st == PGPU_OK) st = upload(ctx, &b->pis, pis);
  std::vector<float2> pis2(pis.size());
  for (size_t i = 0; i < pis.size(); ++i) {
    const float h = (float)pis[i];
    pis2[i] = make_float2(h, (float)(pis[i] - (double)h));
  }
  std::vector<float4> lt(64);
  ff_log_table(lt.data(), [](double c) { return std::log(c); });
  if (st == PGPU_OK) st = upload(ctx, &b->pis2, pis2);
  if (st == PGPU_OK) st = upload(ctx, &b->logtab, lt);
  if (st == PGPU_OK) st = upload(ctx, &b->brlen, brl);
  if (st == PGPU_OK) st = upload(ctx, &b->rates, rts);
  if (st == PGPU_OK) st = upload(ctx, &b->ctab, ctab);
  if (st == PGPU_OK) st = upload(ctx, &b->Q, Qall);
  if (st == PGPU_OK) st = upload(ctx, &b->tile_base, tile_base);
  if (st == PGPU_OK) st = upload(ctx, &b->n_tiles, ntiles);
  if (st == PGPU_OK) st = upload(ctx, &b->members, members);
  std::vector<double> pig(PIall);
  double *dpig = nullptr;
  if (st == PGPU_OK) st = upload(ctx, &dpig, pig);
  auto alloc = [&](void **p, size_t bytes) -> pgpu_status {
    PGPU_CUDA(ctx, cudaMalloc(p, std::max<size_t>(bytes, 16)));
    return PGPU_OK;
  };
  if (st == PGPU_OK) st = alloc((void **)&b->spill, launch_spill(b) * 4);
  if (st == PGPU_OK) st = alloc((void **)&b->bmat, (size_t)bm_off * 4);
  if (st == PGPU_OK) st = alloc((void **)&b->tiptab, (size_t)tt_off * 4);
  if (st == PGPU_OK) st = alloc((void **)&b->U, (size_t)q_acc * 8);
  if (st == PGPU_OK) st = alloc((void **)&b->Ui, (size_t)q_acc * 8);
  if (st == PGPU_OK) st = alloc((void **)&b->lam, (size_t)l_acc * 8);
  if (st == PGPU_OK) st = alloc((void **)&b->status, (size_t)n_var * 4);
  if (st == PGPU_OK) st = alloc((void **)&b->partials, (size_t)std::max<long long>(b->n_work, 1) * 16);
  // the eigen systems depend on the models only: solved once here
  if (st == PGPU_OK) {
    for (size_t g = 0; g < b->group_S.size() && st == PGPU_OK; ++g) {
      const int S = b->group_S[g];
      st = pgpu_launch_eig(ctx, b->Q + b->gQ[g], dpig + b->gL[g], S,
                           (int)b->group_members[g].size(), b->U + b->gQ[g], b->lam + b->gL[g],
                           b->Ui + b->gQ[g], b->status + b->gM[g]);
    }
  }
  if (st == PGPU_OK) {
    std::vector<int> hst(n_var, 0);
    cudaError_t e = cudaStreamSynchronize(ctx->stream);
    if (e == cudaSuccess) e = cudaMemcpy(hst.data(), b->status, (size_t)n_var * 4, cudaMemcpyDeviceToHost);
    if (e != cudaSuccess) st = pgpu_set_err(ctx, PGPU_ERR_CUDA, "batch: %s", cudaGetErrorString(e));
    for (int k = 0; k < n_var && st == PGPU_OK; ++k)
      if (hst[k]) st = pgpu_set_err(ctx, hst[k], "batch: model %d failed its eigendecomposition (%d)", k, hst[k]);
  }
  if (dpig) cudaFree(dpig);
  if (st != PGPU_OK) {
    free_batch(b);
    return st;
  }
  *out = b;
  return PGPU_OK;
}

void pgpu_batch_destroy(pgpu_batch *b) {
  if (b) free_batch(b);
}

pgpu_status pgpu_batch_run(pgpu_ctx *ctx, pgpu_batch *b, double *lnl_dev, double *site_lnl_dev) {
  if (!ctx || !b || !lnl_dev) return PGPU_ERR_ARG;
  PGPU_CUDA(ctx, cudaSetDevice(ctx->device));
  // B blocks and tip rows for every branch (FP64 P from the eigen systems)
  for (size_t g = 0; g < b->group_S.size(); ++g) {
    const int S = b->group_S[g];
    SetupArgs a;
    a.vars = b->vars;
    a.members = b->members + b->gM[g];
    a.U = b->U + b->gQ[g];
    a.lam = b->lam + b->gL[g];
    a.Ui = b->Ui + b->gQ[g];
    a.status = b->status + b->gM[g];
    a.brlen = b->brlen;
    a.rates = b->rates;
    a.ctab = b->ctab;
    a.pis = b->pis;
    a.bmat = b->bmat;
    a.tiptab = b->tiptab;
    a.flag = ctx->d_flag;
    a.S = S;
    int max_tips = 0, max_R = 0;
    for (int vi : b->group_members[g]) {
      max_tips = std::max(max_tips, b->hvars[vi].n_tips);
      max_R = std::max(max_R, b->hvars[vi].R);
    }
    const size_t smem = sizeof(double) * (3 * (size_t)S * S + 3 * S);
    PGPU_CUDA(ctx, cudaFuncSetAttribute(batch_setup_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                        (int)std::max<size_t>(smem, 1024)));
    batch_setup_kernel<<<dim3(2 * max_tips - 2, max_R, (unsigned)b->group_members[g].size()), 256, smem,
                         ctx->stream>>>(a);
    PGPU_TRY(pgpu_after_launch(ctx, "batch_setup_kernel"));
  }
  BatchArgs a;
  a.vars = b->vars;
  a.ops = b->ops;
  a.bmat = b->bmat;
  a.tiptab = b->tiptab;
  a.pis = b->pis;
  a.pis2 = b->pis2;
  a.logtab = b->logtab;
  a.site_lnl = site_lnl_dev;
  a.partials = b->partials;
  a.flag = ctx->d_flag;
  a.n_spill = b->n_spill;
  if (b->lim_smem > ctx->smem_optin)
    return pgpu_set_err(ctx, PGPU_ERR_LIMIT, "batch: %zu bytes of shared memory needed", b->lim_smem);
  // independent of one another: each after the first starts on the SMs that the
  // one before leaves
  uint32_t *spill = b->spill;
  for (size_t k = 0; k < b->launches.size(); ++k) {
    const BatchLaunch &l = b->launches[k];
    a.work = b->work + l.work0;
    a.n_work = l.n_work;
    a.slot_bytes = l.slot_bytes;
    a.n_st = l.n_st;
    a.spill = spill;
    spill += (size_t)l.grid * b->n_spill * BT_SPILL_WORDS;
    PGPU_TRY(launch_tc(ctx, a, l, k > 0));
  }
  batch_finalize_kernel<<<b->n_var, 256, 0, ctx->stream>>>(b->partials, b->tile_base,
                                                                        b->n_tiles, b->n_var, lnl_dev);
  return pgpu_after_launch(ctx, "batch_finalize_kernel");
}

pgpu_status pgpu_batch_run_fp64(pgpu_ctx *ctx, pgpu_batch *b, size_t sample, double *lnl_dev) {
  if (!ctx || !b || !lnl_dev || sample == 0) return PGPU_ERR_ARG;
  PGPU_CUDA(ctx, cudaSetDevice(ctx->device));
  F64Args a;
  a.vars = b->vars;
  a.ops = b->ops;
  a.U = b->U;
  a.Ui = b->Ui;
  a.lam = b->lam;
  for (size_t g = 0; g < 8; ++g) {
    a.gU[g] = g < b->gQ.size() ? b->gQ[g] : 0;
    a.gL[g] = g < b->gL.size() ? b->gL[g] : 0;
  }
  a.brlen = b->brlen;
  a.rates = b->rates;
  a.ctab = b->ctab;
  a.pis = b->pis;
  long long max_pat = 0;
  int max_S = 0;
  for (const BVar &v : b->hvars) {
    max_pat = std::max(max_pat, std::min<long long>(v.n_pat, (long long)sample));
    max_S = std::max(max_S, v.S);
  }
  a.blocks = (int)((max_pat + F64_NP - 1) / F64_NP);
  a.sample = (long long)sample;
  a.max_depth = b->max_depth;
  double2 *dpart = nullptr;
  PGPU_TRY(pgpu_buf(ctx, BUF_D, (size_t)a.blocks * b->n_var * sizeof(double2), (void **)&dpart));
  a.partials = dpart;
  const size_t smem = sizeof(double) * ((size_t)max_S * max_S + 64 + (size_t)b->max_depth * max_S * F64_NP);
  if (smem > ctx->smem_optin) return pgpu_set_err(ctx, PGPU_ERR_LIMIT, "batch fp64: tree too deep");
  PGPU_CUDA(ctx, cudaFuncSetAttribute(batch_fp64_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                      (int)std::max<size_t>(smem, 48 * 1024)));
  batch_fp64_kernel<<<dim3(a.blocks, b->n_var), F64_NP, smem, ctx->stream>>>(a);
  PGPU_TRY(pgpu_after_launch(ctx, "batch_fp64_kernel"));
  // per variant: blocks * F64_NP patterns, partials at [v * blocks]
  std::vector<long long> base(b->n_var);
  std::vector<int> cnt(b->n_var, a.blocks);
  for (int v = 0; v < b->n_var; ++v) base[v] = (long long)v * a.blocks;
  long long *dbase = nullptr;
  int *dcnt = nullptr;
  PGPU_TRY(pgpu_buf(ctx, BUF_E, base.size() * 8, (void **)&dbase));
  PGPU_TRY(pgpu_buf(ctx, BUF_F, cnt.size() * 4, (void **)&dcnt));
  PGPU_CUDA(ctx, cudaMemcpyAsync(dbase, base.data(), base.size() * 8, cudaMemcpyHostToDevice, ctx->stream));
  PGPU_CUDA(ctx, cudaMemcpyAsync(dcnt, cnt.data(), cnt.size() * 4, cudaMemcpyHostToDevice, ctx->stream));
  batch_finalize_kernel<<<b->n_var, 256, 0, ctx->stream>>>(dpart, dbase, dcnt,
                                                                        b->n_var, lnl_dev);
  return pgpu_after_launch(ctx, "batch_finalize_kernel");
}

long long pgpu_batch_work_items(const pgpu_batch *b) { return b ? b->n_work : 0; }
long long pgpu_batch_patterns(const pgpu_batch *b) { return b ? b->total_pat : 0; }

}  // extern "C"
