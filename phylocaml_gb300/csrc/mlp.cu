// The learned SPR ranking: a BF16 multilayer perceptron 64 -> 256 -> 256 ->
// 256 -> 1 (GELU) with FP32 accumulation, trained by AdamW on (move, dlnL)
// pairs.  phylocaml has no learned component; this is the proposal model that
// orders SPR moves (lib/treeNeighborhoods.ml:27-75 leaves the search itself
// as a TODO).
//
// Forward:  h1 = gelu(W1 xn + b1), h2 = gelu(W2 h1 + b2), h3 = gelu(W3 h2 + b3),
//           y = w4 . h3 + b4, xn = (x - mu) / sd in BF16.
// Backward: dz3 = dy w4 * gelu'(z3); dW3 = dz3^T h2; dz2 = (dz3 W3) * gelu'(z2);
//           dW2 = dz2^T h1; dz1 = (dz2 W2) * gelu'(z1); dW1 = dz1^T xn;
//           db_l = sum over rows of dz_l; dw4 = dy^T h3; db4 = sum dy.
//
// Every product is C[M x N] = A[M x K] B[N x K]^T on the tensor cores, A and
// B in BF16 and D in TMEM (FP32): tcgen05.mma.kind::f16, M = 128, K = 16, K
// always in ascending order, so how N is cut over CTAs changes no bit.  Every
// operand lies in global memory as the tensor cores read it from shared
// memory (packed_at): tiles of 128 rows x 64 of K, 16 KB each, in 8 x 16-byte
// core matrices, so a tile is one bulk copy and no thread touches operands.
//
// Ranking (mlp_forward_kernel): a CTA takes 128 rows through all four layers;
// the hidden vectors stay in shared memory and 16 KB weight tiles stream
// through a ring.  Two CTAs share an SM, one's tensor work under the other's
// GELUs.  Bound by the GELUs (768 erff a row).
// Training (mlp_tile_kernel): a batch of 1,024 rows is small, so what counts
// is latency: a layer is cut into 128 x 32 tiles over 64 CTAs, and one step
// is seven launches: three layers, the output layer with the loss gradient,
// two back-propagated layers, and all weight gradients with their AdamW
// updates and new BF16 copies.
#include <cuda_bf16.h>

#include <algorithm>
#include <cmath>
#include <random>
#include <vector>

#include "pgpu_internal.cuh"

namespace {

constexpr int IN = 64, HID = 256;
constexpr int GM = 128;           // rows of an operand tile
constexpr int GK = 64;            // K of an operand tile
constexpr uint32_t TILE_BYTES = GM * GK * 2;   // 16 KB
constexpr int TN = 32;            // columns per CTA of the training kernels
constexpr int TST = 8;            // training ring: stages of one A tile and TN rows of B
constexpr uint32_t TB_BYTES = TN * GK * 2, TSTAGE = TILE_BYTES + TB_BYTES;
constexpr int FR = 3;             // ranking ring: weight tiles
constexpr int MLP_NT = 256;       // threads: two per row, half the columns each
constexpr size_t FWD_SMEM = (size_t)HID / GK * TILE_BYTES + (size_t)FR * TILE_BYTES;   // 112 KB: 2 CTAs/SM

// parameter offsets in the flat FP32 vector
constexpr size_t OFF_W1 = 0, OFF_B1 = OFF_W1 + (size_t)HID * IN, OFF_W2 = OFF_B1 + HID,
                 OFF_B2 = OFF_W2 + (size_t)HID * HID, OFF_W3 = OFF_B2 + HID,
                 OFF_B3 = OFF_W3 + (size_t)HID * HID, OFF_W4 = OFF_B3 + HID, OFF_B4 = OFF_W4 + HID,
                 N_PARAMS = OFF_B4 + 1;

// element (r, k) of a K-major operand with K columns in all
__host__ __device__ __forceinline__ size_t packed_at(size_t r, size_t k, size_t K) {
  return ((r / GM) * (K / GK) + k / GK) * (size_t)(GM * GK) + (r % GM) / 8 * (8 * GK) + k % GK / 8 * 64 +
         r % 8 * 8 + k % 8;
}

__device__ __forceinline__ uint32_t su32(const void *p) {
  return static_cast<uint32_t>(__cvta_generic_to_shared(p));
}

__device__ __forceinline__ uint64_t smem_desc(const void *base, uint32_t lbo, uint32_t sbo) {
  uint64_t d = 0;
  d |= (uint64_t)((su32(base) >> 4) & 0x3FFF);
  d |= (uint64_t)((lbo >> 4) & 0x3FFF) << 16;
  d |= (uint64_t)((sbo >> 4) & 0x3FFF) << 32;
  d |= (uint64_t)1 << 46;
  return d;
}

__device__ __forceinline__ void tmem_ld16(uint32_t ta, float *v) {
  uint32_t r[16];
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, "
      "[%16];"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]),
        "=r"(r[7]), "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]),
        "=r"(r[14]), "=r"(r[15])
      : "r"(ta));
  asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
  for (int j = 0; j < 16; ++j) v[j] = __uint_as_float(r[j]);
}

__device__ __forceinline__ float gelu(float z) { return 0.5f * z * (1.0f + erff(z * 0.70710678118654752f)); }
__device__ __forceinline__ float dgelu(float z) {
  return 0.5f * (1.0f + erff(z * 0.70710678118654752f)) + z * 0.39894228040143268f * expf(-0.5f * z * z);
}

// core matrices of a 128 x 64 tile: 128 bytes from one 8 of K to the next,
// 1,024 bytes from one 8 rows to the next
constexpr uint32_t LBO = 128, SBO = (GK / 8) * 128;

__device__ __forceinline__ uint32_t mma_idesc(int n) {
  uint32_t d = 0;
  d |= 1u << 4;                     // D f32
  d |= 1u << 7;                     // A bf16
  d |= 1u << 10;                    // B bf16
  d |= (uint32_t)(n >> 3) << 17;
  d |= (uint32_t)(GM >> 4) << 24;
  return d;
}

// the four K = 16 steps of one operand tile; first: D starts at zero
__device__ __forceinline__ void mma_tile(uint32_t tmem, const unsigned char *a, const unsigned char *b,
                                         uint32_t idesc, bool first) {
#pragma unroll
  for (int ks = 0; ks < GK / 16; ++ks) {
    const uint64_t ad = smem_desc(a + ks * 2 * LBO, LBO, SBO);
    const uint64_t bd = smem_desc(b + ks * 2 * LBO, LBO, SBO);
    const uint32_t acc = first && ks == 0 ? 0u : 1u;
    asm volatile(
        "{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}" ::"r"(tmem),
        "l"(ad), "l"(bd), "r"(idesc), "r"(acc));
  }
}
__device__ __forceinline__ void mma_commit(uint64_t *bar) {
  asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(su32(bar))
               : "memory");
}
__device__ __forceinline__ void tc_fence_before() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void tc_fence_after() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }

template <int COLS>
__device__ __forceinline__ void tmem_alloc(uint32_t *base) {
  asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(su32(base)), "n"(COLS));
  asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;");
}
template <int COLS>
__device__ __forceinline__ void tmem_free(uint32_t tmem) {
  asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "n"(COLS));
}

__device__ __forceinline__ void st_bf16x8(unsigned char *dst, const __nv_bfloat16 *v) {
  *reinterpret_cast<uint4 *>(dst) = *reinterpret_cast<const uint4 *>(v);
}

// rows row0 .. row0 + 127 of (X - mu) / sd as BF16 into a packed 128 x 64
// tile in shared memory, rows from n on zero; XT (or null) gets the packed
// transpose [64][kt]
__device__ __forceinline__ void stage_norm(const float *X, size_t n, size_t row0, const float *mu,
                                           const float *inv_sd, unsigned char *tile, __nv_bfloat16 *XT,
                                           size_t kt) {
  for (int i = threadIdx.x; i < GM * (IN / 8); i += MLP_NT) {
    const int r = i >> 3, kv = i & 7;
    const size_t row = row0 + r;
    __align__(16) __nv_bfloat16 b[8];
#pragma unroll
    for (int j = 0; j < 8; ++j) {
      const int k = kv * 8 + j;
      b[j] = __float2bfloat16_rn(row < n ? (X[row * IN + k] - mu[k]) * inv_sd[k] : 0.0f);
      if (XT) XT[packed_at(k, row, kt)] = b[j];
    }
    st_bf16x8(tile + (r >> 3) * SBO + kv * LBO + (r & 7) * 16, b);
  }
}

struct NetView {   // device pointers of one network
  const float *p, *mu, *inv_sd;
  const __nv_bfloat16 *W[3];
};

// ---- ranking: 128 rows per CTA through every layer ------------------------
// 257,048 rows: 0.30 ms; the three-launch form, which wrote each hidden
// layer to memory and read it back, took 1.8 ms.
__global__ void __launch_bounds__(MLP_NT, 2) mlp_forward_kernel(const NetView net, const float *X, size_t n,
                                                                float *y, int *flag) {
  extern __shared__ __align__(1024) unsigned char smem[];
  __shared__ uint64_t full[FR], done[FR], layer_bar;
  __shared__ uint32_t tbase;
  unsigned char *sH = smem;                                      // [HID / GK] tiles of 128 x 64
  unsigned char *ring = smem + HID / GK * TILE_BYTES;
  const int tid = threadIdx.x, warp = tid >> 5;
  const size_t row0 = (size_t)blockIdx.x * GM;
  if (warp == 0) tmem_alloc<HID>(&tbase);
  if (tid == 0) {
    for (int i = 0; i < FR; ++i) {
      mbar_init(&full[i], 1);
      mbar_init(&done[i], 1);
    }
    mbar_init(&layer_bar, 1);
    fence_mbarrier_init();
  }
  // weight tile u of the sequence W1 (2 tiles), W2, W3 (8 each: the first
  // 128 outputs' four K tiles, then the other 128's)
  constexpr int U1 = 2, U2 = 8, UN = U1 + 2 * U2;
  auto fetch = [&](int u) {
    const __nv_bfloat16 *w = u < U1 ? net.W[0] + (size_t)u * GM * GK
                                    : net.W[u < U1 + U2 ? 1 : 2] + (size_t)((u - U1) % U2) * GM * GK;
    mbar_arrive_expect_tx(&full[u % FR], TILE_BYTES);
    bulk_g2s(ring + (u % FR) * TILE_BYTES, w, TILE_BYTES, &full[u % FR]);
  };
  stage_norm(X, n, row0, net.mu, net.inv_sd, sH, nullptr, 0);
  fence_proxy_async_smem();
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = tbase;
  const uint32_t idesc = mma_idesc(GM);
  int fetched = 0;
  bool ok = true;
  if (tid == 0)
    for (; fetched < FR; ++fetched) fetch(fetched);
  const uint32_t lane_base = tmem + ((uint32_t)(32 * (warp & 3)) << 16);
  const int r = (warp & 3) * 32 + (tid & 31), half = (warp >> 2) * (HID / 2);
#pragma unroll 1
  for (int l = 0; l < 3; ++l) {
    if (tid == 0) {
      const int u0 = l == 0 ? 0 : l == 1 ? U1 : U1 + U2, nu = l == 0 ? U1 : U2, nk = nu / 2;
      for (int i = 0; i < nu && ok; ++i) {
        const int u = u0 + i, sl = u % FR;
        ok = mbar_wait_bounded(&full[sl], (u / FR) & 1, flag);
        if (!ok) break;
        mma_tile(tmem + (uint32_t)(i / nk) * GM, sH + (i % nk) * TILE_BYTES, ring + sl * TILE_BYTES, idesc,
                 i % nk == 0);
        mma_commit(&done[sl]);
        // refill the slot of the tile before this one, whose MMAs ran while
        // this one's were queued; the layer's last slot waits for the next
        if (u > 0 && fetched < UN && fetched - FR < u) {
          ok = mbar_wait_bounded(&done[(u - 1) % FR], ((u - 1) / FR) & 1, flag);
          if (ok) fetch(fetched++);
        }
      }
      mma_commit(&layer_bar);
    }
    ok = mbar_wait_bounded(&layer_bar, l & 1, flag) && ok;
    tc_fence_after();
    // GELU: thread = (row, half of the columns); the vectors go back to
    // shared memory as the next layer's A operand
    const float *bias = net.p + (l == 0 ? OFF_B1 : l == 1 ? OFF_B2 : OFF_B3);
#pragma unroll 1
    for (int c0 = half; c0 < half + HID / 2; c0 += 16) {
      float v[16];
      tmem_ld16(lane_base + (uint32_t)c0, v);
      __align__(16) __nv_bfloat16 hb[16];
#pragma unroll
      for (int j = 0; j < 16; j += 4) {
        const float4 b = __ldg(reinterpret_cast<const float4 *>(bias + c0 + j));
        hb[j] = __float2bfloat16_rn(gelu(v[j] + b.x));
        hb[j + 1] = __float2bfloat16_rn(gelu(v[j + 1] + b.y));
        hb[j + 2] = __float2bfloat16_rn(gelu(v[j + 2] + b.z));
        hb[j + 3] = __float2bfloat16_rn(gelu(v[j + 3] + b.w));
      }
      unsigned char *dst = sH + (c0 / GK) * TILE_BYTES + (r >> 3) * SBO + (c0 % GK / 8) * LBO + (r & 7) * 16;
      st_bf16x8(dst, hb);
      st_bf16x8(dst + LBO, hb + 8);
    }
    fence_proxy_async_smem();
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
  }
  // the output layer: one sum per row, columns in ascending order
  if (tid < GM && row0 + tid < n) {
    float ysum = 0.0f;
    for (int c = 0; c < HID; c += 8) {
      __align__(16) __nv_bfloat16 hb[8];
      *reinterpret_cast<uint4 *>(hb) = *reinterpret_cast<const uint4 *>(
          sH + (c / GK) * TILE_BYTES + (tid >> 3) * SBO + (c % GK / 8) * LBO + (tid & 7) * 16);
#pragma unroll
      for (int j = 0; j < 8; ++j) ysum = fmaf(__bfloat162float(hb[j]), __ldg(net.p + OFF_W4 + c + j), ysum);
    }
    y[row0 + tid] = ysum + __ldg(net.p + OFF_B4);
  }
  if (tid == 0 && !ok)   // no copy may be in flight when the CTA leaves
    for (int u = max(0, fetched - FR); u < fetched; ++u)
      (void)mbar_wait_bounded(&full[u % FR], (u / FR) & 1, flag);
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  if (warp == 0) tmem_free<HID>(tmem);
}

struct AdamArgs {
  float *p, *m, *v;
  float lr, b1, b2, eps, wd, c1, c2;   // c1 = 1 - b1^t, c2 = 1 - b2^t
};

// one AdamW update of a parameter from its old p, m and v; decay: decoupled
// weight decay (the matrices and w4; biases are not decayed)
__device__ __forceinline__ void adamw(const AdamArgs &a, float &p, float &m, float &v, float g, bool decay) {
  // the roundings are written out, so that every kernel that updates agrees
  m = fmaf(1.0f - a.b1, g, __fmul_rn(a.b1, m));
  v = fmaf(__fmul_rn(1.0f - a.b2, g), g, __fmul_rn(a.b2, v));
  if (decay) p -= a.lr * a.wd * p;
  p -= a.lr * (m / a.c1) / (sqrtf(v / a.c2) + a.eps);
}

__device__ __forceinline__ void adamw_at(const AdamArgs &a, size_t i, float g, bool decay) {
  float p = a.p[i], m = a.m[i], v = a.v[i];
  adamw(a, p, m, v, g, decay);
  a.p[i] = p, a.m[i] = m, a.v[i] = v;
}

// A training step's kernels run back to back on one stream: each is launched
// while the one before drains (programmatic stream serialisation) and waits
// here, its barriers and tensor memory set up, until that one's writes are
// visible.  What such a kernel reads goes through plain loads: the read-only
// path may keep lines from before the wait.
__device__ __forceinline__ void wait_previous() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
__device__ __forceinline__ void let_next() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }

template <typename... P, typename... A>
cudaError_t launch_chained(void (*kern)(P...), dim3 grid, int threads, size_t smem, cudaStream_t st, A... args) {
  cudaLaunchConfig_t c{};
  c.gridDim = grid;
  c.blockDim = dim3((unsigned)threads);
  c.dynamicSmemBytes = smem;
  c.stream = st;
  cudaLaunchAttribute at{};
  at.id = cudaLaunchAttributeProgrammaticStreamSerialization;
  at.val.programmaticStreamSerializationAllowed = 1;
  c.attrs = &at;
  c.numAttrs = 1;
  return cudaLaunchKernelEx(&c, kern, args...);
}

// ---- training: one 128 x TN tile of a product per CTA ----------------------
// TILE_NORM   layer 1: A is the normalised input, staged from X
// TILE_GELU   layers 2, 3
//             z = C + b, h = gelu(z): z, packed h and packed h^T
// TILE_DGELU  dz = C gelu'(z): packed dz and dz^T
enum { TILE_NORM = 0, TILE_GELU = 1, TILE_DGELU = 2 };

struct TileArgs {
  const __nv_bfloat16 *A, *B;   // packed [M][K], [N][K]
  int K;
  const float *bias;
  float *Z;                     // [M][256]
  __nv_bfloat16 *H, *HT;        // packed [M][256], [256][rows]
  int rows;                     // M
  // TILE_NORM
  const float *X, *mu, *inv_sd;
  size_t n;
  __nv_bfloat16 *XT;            // packed [64][rows]
  int *flag;
};

// A and B tiles through a ring of bulk copies, the MMAs issued as they land;
// one thread does both.  On return every thread may read D (128 x TN) in TMEM.
__device__ __forceinline__ bool tile_product(const __nv_bfloat16 *A, const __nv_bfloat16 *B, int n_chunks,
                                             unsigned char *ring, uint64_t *full, uint64_t *done,
                                             uint64_t *last, uint32_t tmem, bool a_staged, int *flag) {
  bool ok = true;
  if (threadIdx.x == 0) {
    const uint32_t idesc = mma_idesc(TN);
    auto fetch = [&](int ch) {
      unsigned char *st = ring + (size_t)(ch % TST) * TSTAGE;
      uint64_t *bar = &full[ch % TST];
      mbar_arrive_expect_tx(bar, a_staged ? TB_BYTES : TSTAGE);
      if (!a_staged) bulk_g2s(st, A + (size_t)ch * GM * GK, TILE_BYTES, bar);
      bulk_g2s(st + TILE_BYTES, B + (size_t)ch * GM * GK, TB_BYTES, bar);
    };
    int fetched = 0;
    for (; fetched < min(TST, n_chunks); ++fetched) fetch(fetched);
    for (int ch = 0; ch < n_chunks && ok; ++ch) {
      const int s = ch % TST;
      ok = mbar_wait_bounded(&full[s], (ch / TST) & 1, flag);
      if (!ok) break;
      const unsigned char *st = ring + (size_t)s * TSTAGE;
      mma_tile(tmem, st, st + TILE_BYTES, idesc, ch == 0);
      mma_commit(&done[s]);
      if (ch > 0 && fetched < n_chunks) {   // refill the slot of the chunk before
        ok = mbar_wait_bounded(&done[(ch - 1) % TST], ((ch - 1) / TST) & 1, flag);
        if (ok) fetch(fetched++);
      }
    }
    if (!ok)
      for (int ch = max(0, fetched - TST); ch < fetched; ++ch)
        (void)mbar_wait_bounded(&full[ch % TST], (ch / TST) & 1, flag);
    mma_commit(last);
  }
  ok = mbar_wait_bounded(last, 0, flag) && ok;
  tc_fence_after();
  return ok;
}

__device__ __forceinline__ void tile_setup(uint64_t *full, uint64_t *done, uint64_t *last, uint32_t *tbase) {
  if (threadIdx.x < 32) tmem_alloc<TN>(tbase);
  if (threadIdx.x == 0) {
    for (int i = 0; i < TST; ++i) {
      mbar_init(&full[i], 1);
      mbar_init(&done[i], 1);
    }
    mbar_init(last, 1);
    fence_mbarrier_init();
  }
}

// rows of B in tile order: TN rows from n0 on
__device__ __forceinline__ const __nv_bfloat16 *b_rows(const __nv_bfloat16 *B, int n0, int K) {
  return B + (size_t)(n0 / GM) * (K / GK) * (GM * GK) + (size_t)(n0 % GM) * GK;
}

template <int EPI>
__global__ void __launch_bounds__(MLP_NT) mlp_tile_kernel(const TileArgs a) {
  extern __shared__ __align__(1024) unsigned char smem[];
  __shared__ uint64_t full[TST], done[TST], last;
  __shared__ uint32_t tbase;
  const int tid = threadIdx.x, warp = tid >> 5;
  const int row0 = blockIdx.x * GM, n0 = blockIdx.y * TN;
  tile_setup(full, done, &last, &tbase);
  wait_previous();
  let_next();
  if (EPI == TILE_NORM) {
    stage_norm(a.X, a.n, row0, a.mu, a.inv_sd, smem, n0 == 0 ? a.XT : nullptr, a.rows);
    fence_proxy_async_smem();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = tbase;
  const int nk = a.K / GK;
  const bool ok = tile_product(EPI == TILE_NORM ? nullptr : a.A + (size_t)blockIdx.x * nk * (GM * GK),
                               b_rows(a.B, n0, a.K), nk, smem, full, done, &last, tmem, EPI == TILE_NORM,
                               a.flag);
  const int r = (warp & 3) * 32 + (tid & 31), c0 = (warp >> 2) * (TN / 2);
  const int row = row0 + r, col = n0 + c0;
  float v[16];
  tmem_ld16(tmem + ((uint32_t)(32 * (warp & 3)) << 16) + (uint32_t)c0, v);
  if (ok) {
    __align__(16) __nv_bfloat16 hb[16];
    float4 *z4 = reinterpret_cast<float4 *>(a.Z + (size_t)row * HID + col);
#pragma unroll
    for (int j = 0; j < 16; j += 4) {
      float z[4];
      if (EPI == TILE_DGELU) {
        const float4 q = z4[j / 4];
        z[0] = q.x, z[1] = q.y, z[2] = q.z, z[3] = q.w;
      } else {
        const float4 b = *reinterpret_cast<const float4 *>(a.bias + col + j);
        z[0] = v[j] + b.x, z[1] = v[j + 1] + b.y, z[2] = v[j + 2] + b.z, z[3] = v[j + 3] + b.w;
        z4[j / 4] = make_float4(z[0], z[1], z[2], z[3]);
      }
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        hb[j + i] = __float2bfloat16_rn(EPI == TILE_DGELU ? v[j + i] * dgelu(z[i]) : gelu(z[i]));
        a.HT[packed_at(col + j + i, row, a.rows)] = hb[j + i];
      }
    }
    *reinterpret_cast<uint4 *>(a.H + packed_at(row, col, HID)) = reinterpret_cast<const uint4 *>(hb)[0];
    *reinterpret_cast<uint4 *>(a.H + packed_at(row, col + 8, HID)) = reinterpret_cast<const uint4 *>(hb)[1];
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  if (warp == 0) tmem_free<TN>(tmem);
}

// Output layer and its gradient, 32 rows per CTA: y = h3 . w4 + b4 (columns
// in ascending order), dy = 2 sw (y - t) / sum sw (rows from n on: 0), and
// dz3 = dy w4 gelu'(z3), packed, with its transpose.
__global__ void __launch_bounds__(MLP_NT) mlp_out_kernel(const float *p, const __nv_bfloat16 *H3T,
                                                         const float *Z3, const float *t, const float *sw,
                                                         int n, int rows, float *y, float *dy,
                                                         __nv_bfloat16 *DZ, __nv_bfloat16 *DZT) {
  __shared__ double red[MLP_NT / 32];
  __shared__ float sdy[32];
  __shared__ float sh[HID][32];   // h3 of this CTA's rows
  constexpr int NW = MLP_NT / 32;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int r = blockIdx.x * 32 + lane;
  wait_previous();
  let_next();
#pragma unroll
  for (int i = 0; i < HID / NW; ++i) {
    const int c = warp * (HID / NW) + i;
    sh[c][lane] = __bfloat162float(H3T[packed_at(c, r, rows)]);
  }
  // thread = (row, columns 8 warp + 64 q .. + 7): the pre-activations are
  // on their way while warp 0 forms the outputs
  float z[HID / 64][8];
#pragma unroll
  for (int q = 0; q < HID / 64; ++q) {
    const float4 *src = reinterpret_cast<const float4 *>(Z3 + (size_t)r * HID + q * 64 + warp * 8);
    const float4 u = src[0], v = src[1];
    z[q][0] = u.x, z[q][1] = u.y, z[q][2] = u.z, z[q][3] = u.w;
    z[q][4] = v.x, z[q][5] = v.y, z[q][6] = v.z, z[q][7] = v.w;
  }
  if (sw) {   // every CTA sums the weights in the same order
    double s = 0.0;
    for (int i = tid; i < n; i += MLP_NT) s += (double)sw[i];
    for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
    if (lane == 0) red[warp] = s;
  }
  __syncthreads();
  if (warp == 0) {
    double W = (double)n;
    if (sw) {
      W = 0.0;
      for (int w = 0; w < NW; ++w) W += red[w];
    }
    const double inv = W > 0 ? 1.0 / W : 0.0;
    float ysum = 0.0f;
#pragma unroll 16
    for (int c = 0; c < HID; ++c) ysum = fmaf(sh[c][lane], p[OFF_W4 + c], ysum);
    const float yr = ysum + p[OFF_B4];
    float g = 0.0f;
    if (r < n) g = (float)(2.0 * (sw ? (double)sw[r] : 1.0) * ((double)yr - (double)t[r]) * inv);
    y[r] = yr;
    dy[r] = g;
    sdy[lane] = g;
  }
  __syncthreads();
#pragma unroll
  for (int q = 0; q < HID / 64; ++q) {
    const int c = q * 64 + warp * 8;
    __align__(16) __nv_bfloat16 b[8];
#pragma unroll
    for (int j = 0; j < 8; ++j) {
      const float g = r < n ? sdy[lane] * p[OFF_W4 + c + j] * dgelu(z[q][j]) : 0.0f;
      b[j] = __float2bfloat16_rn(g);
      DZT[packed_at(c + j, r, rows)] = b[j];
    }
    *reinterpret_cast<uint4 *>(DZ + packed_at(r, c, HID)) = *reinterpret_cast<const uint4 *>(b);
  }
}

// ---- all weight gradients of a step, and their updates ---------------------
// CTAs 0 .. 35: a 128 x TN tile of dW3, dW2 (16 each) or dW1 (4), K the
// batch's rows; the next 128: eight rows each of db3, db2, db1 and dw4; the
// last: db4 and the loss.  Gradients go to G (when set) or straight into
// AdamW and the packed BF16 copies, W for the layers and W^T for
// back-propagation.
constexpr int WG_TILES = 36, WG_SUMS = 4 * HID / (MLP_NT / 32);

struct GradArgs {
  const __nv_bfloat16 *DZT[3], *HT[4];   // packed, [256][rows] ([64][rows] for HT[0], the input)
  const float *y, *t, *sw, *dy;
  int n, rows;
  float *G;                 // flat gradient, or null: update
  AdamArgs adam;
  __nv_bfloat16 *W[3], *WT[3];
  float *loss;
  int *flag;
};

__global__ void __launch_bounds__(MLP_NT) mlp_grad_kernel(const GradArgs a) {
  extern __shared__ __align__(1024) unsigned char smem[];
  __shared__ uint64_t full[TST], done[TST], last;
  __shared__ uint32_t tbase;
  __shared__ double red[3][MLP_NT / 32];
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int blk = blockIdx.x;
  auto give = [&](size_t i, float g, bool decay) {
    if (a.G) a.G[i] = g;
    else adamw_at(a.adam, i, g, decay);
  };
  if (blk < WG_TILES) {
    const int l = blk < 16 ? 2 : blk < 32 ? 1 : 0;
    const int i = blk < 32 ? blk & 15 : blk - 32, K_in = l == 0 ? IN : HID, nt = K_in / TN;
    const int row0 = i / nt * GM, n0 = i % nt * TN;
    const size_t woff = l == 0 ? OFF_W1 : l == 1 ? OFF_W2 : OFF_W3;
    tile_setup(full, done, &last, &tbase);
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = tbase;
    // this thread's parameters, on their way during the product
    const int r = (warp & 3) * 32 + lane, c0 = (warp >> 2) * (TN / 2);
    const int o = row0 + r, k0 = n0 + c0;
    const size_t at = woff + (size_t)o * K_in + k0;   // a multiple of 4
    wait_previous();
    let_next();
    float4 P[4], Mo[4], Vo[4];
    if (!a.G) {
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        P[j] = reinterpret_cast<const float4 *>(a.adam.p + at)[j];
        Mo[j] = reinterpret_cast<const float4 *>(a.adam.m + at)[j];
        Vo[j] = reinterpret_cast<const float4 *>(a.adam.v + at)[j];
      }
    }
    const int nk = a.rows / GK;
    const bool ok = tile_product(a.DZT[l] + (size_t)(row0 / GM) * nk * (GM * GK), b_rows(a.HT[l], n0, a.rows),
                                 nk, smem, full, done, &last, tmem, false, a.flag);
    float v[16];
    tmem_ld16(tmem + ((uint32_t)(32 * (warp & 3)) << 16) + (uint32_t)c0, v);
    if (ok && a.G) {
#pragma unroll
      for (int j = 0; j < 4; ++j)
        reinterpret_cast<float4 *>(a.G + at)[j] = make_float4(v[4 * j], v[4 * j + 1], v[4 * j + 2], v[4 * j + 3]);
    } else if (ok) {
      __align__(16) __nv_bfloat16 wb[16];
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        adamw(a.adam, P[j].x, Mo[j].x, Vo[j].x, v[4 * j], true);
        adamw(a.adam, P[j].y, Mo[j].y, Vo[j].y, v[4 * j + 1], true);
        adamw(a.adam, P[j].z, Mo[j].z, Vo[j].z, v[4 * j + 2], true);
        adamw(a.adam, P[j].w, Mo[j].w, Vo[j].w, v[4 * j + 3], true);
        reinterpret_cast<float4 *>(a.adam.p + at)[j] = P[j];
        reinterpret_cast<float4 *>(a.adam.m + at)[j] = Mo[j];
        reinterpret_cast<float4 *>(a.adam.v + at)[j] = Vo[j];
        wb[4 * j] = __float2bfloat16_rn(P[j].x), wb[4 * j + 1] = __float2bfloat16_rn(P[j].y);
        wb[4 * j + 2] = __float2bfloat16_rn(P[j].z), wb[4 * j + 3] = __float2bfloat16_rn(P[j].w);
      }
      if (l > 0) {
#pragma unroll
        for (int j = 0; j < 16; ++j) a.WT[l][packed_at(k0 + j, o, HID)] = wb[j];
      }
      *reinterpret_cast<uint4 *>(a.W[l] + packed_at(o, k0, K_in)) = reinterpret_cast<const uint4 *>(wb)[0];
      *reinterpret_cast<uint4 *>(a.W[l] + packed_at(o, k0 + 8, K_in)) = reinterpret_cast<const uint4 *>(wb)[1];
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    if (warp == 0) tmem_free<TN>(tmem);
  } else if (blk < WG_TILES + WG_SUMS) {
    // one warp per sum over the rows
    const int q = (blk - WG_TILES) * (MLP_NT / 32) + warp, which = q / HID, j = q % HID;
    const __nv_bfloat16 *T = which < 3 ? a.DZT[2 - which] : a.HT[3];
    wait_previous();
    let_next();
    float acc = 0.0f;
#pragma unroll 16
    for (int r = lane; r < a.rows; r += 32)
      acc = fmaf(__bfloat162float(T[packed_at(j, r, a.rows)]), which < 3 ? 1.0f : a.dy[r], acc);
    for (int o = 16; o > 0; o >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, o);
    const size_t off = which == 0 ? OFF_B3 : which == 1 ? OFF_B2 : which == 2 ? OFF_B1 : OFF_W4;
    if (lane == 0) give(off + j, acc, which == 3);
  } else {
    // loss = sum sw (y - t)^2 / sum sw and db4 = sum dy
    wait_previous();
    let_next();
    double s[3] = {0.0, 0.0, 0.0};
    for (int i = tid; i < a.n; i += MLP_NT) {
      const double w = a.sw ? (double)a.sw[i] : 1.0, e = (double)a.y[i] - (double)a.t[i];
      s[0] += w;
      s[1] += w * e * e;
      s[2] += (double)a.dy[i];
    }
#pragma unroll
    for (int k = 0; k < 3; ++k) {
      for (int o = 16; o > 0; o >>= 1) s[k] += __shfl_xor_sync(0xffffffffu, s[k], o);
      if (lane == 0) red[k][warp] = s[k];
    }
    __syncthreads();
    if (tid == 0) {
      double S[3] = {0.0, 0.0, 0.0};
      for (int k = 0; k < 3; ++k)
        for (int w = 0; w < MLP_NT / 32; ++w) S[k] += red[k][w];
      *a.loss = (float)(S[1] * (S[0] > 0 ? 1.0 / S[0] : 0.0));
      give(OFF_B4, (float)S[2], false);
    }
  }
}

// column mean and 1/sd of X [n][64] (FP64 sums; sd floored at 1e-6)
__global__ void __launch_bounds__(256) mlp_colstats_kernel(const float *X, size_t n, float *mu,
                                                           float *inv_sd) {
  __shared__ double red[2][8];
  const int k = blockIdx.x;
  double s = 0.0, s2 = 0.0;
  for (size_t r = threadIdx.x; r < n; r += 256) {
    const double v = X[r * IN + k];
    s += v;
    s2 += v * v;
  }
  for (int o = 16; o > 0; o >>= 1) {
    s += __shfl_xor_sync(0xffffffffu, s, o);
    s2 += __shfl_xor_sync(0xffffffffu, s2, o);
  }
  if ((threadIdx.x & 31) == 0) {
    red[0][threadIdx.x >> 5] = s;
    red[1][threadIdx.x >> 5] = s2;
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    double S = 0, S2 = 0;
    for (int w = 0; w < 8; ++w) {
      S += red[0][w];
      S2 += red[1][w];
    }
    const double m = n ? S / (double)n : 0.0;
    const double var = n ? fmax(S2 / (double)n - m * m, 0.0) : 1.0;
    mu[k] = (float)m;
    inv_sd[k] = (float)(1.0 / fmax(sqrt(var), 1e-6));
  }
}

// packed BF16 weights W [out][in] and W^T [in][out] from the FP32 master copy
__global__ void mlp_pack_kernel(const float *p, __nv_bfloat16 *W1, __nv_bfloat16 *W2, __nv_bfloat16 *W2T,
                                __nv_bfloat16 *W3, __nv_bfloat16 *W3T) {
  const size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i < (size_t)HID * IN) W1[packed_at(i / IN, i % IN, IN)] = __float2bfloat16_rn(p[OFF_W1 + i]);
  if (i < (size_t)HID * HID) {
    const size_t o = i / HID, k = i % HID;
    const __nv_bfloat16 b2 = __float2bfloat16_rn(p[OFF_W2 + i]);
    const __nv_bfloat16 b3 = __float2bfloat16_rn(p[OFF_W3 + i]);
    W2[packed_at(o, k, HID)] = b2;
    W2T[packed_at(k, o, HID)] = b2;
    W3[packed_at(o, k, HID)] = b3;
    W3T[packed_at(k, o, HID)] = b3;
  }
}

size_t pad_to(size_t x, size_t m) { return (x + m - 1) / m * m; }

}  // namespace

struct pgpu_mlp {
  pgpu_ctx *ctx = nullptr;
  int max_batch = 0, bpad = 0;   // bpad: rows padded to 128
  long long step = 0;
  float *p = nullptr, *m = nullptr, *v = nullptr, *g = nullptr;   // flat [N_PARAMS]
  __nv_bfloat16 *W[3] = {}, *WT[3] = {};                          // packed copies (no W1^T)
  float *mu = nullptr, *inv_sd = nullptr, *loss = nullptr;
  // training scratch (bpad rows); HT[0] is the normalised input's transpose
  __nv_bfloat16 *H[3] = {}, *HT[4] = {}, *DZ[3] = {}, *DZT[3] = {};
  float *Z[3] = {}, *y = nullptr, *dy = nullptr;
  std::vector<void *> owned;
};

namespace {

pgpu_status malloc_own(pgpu_mlp *n, size_t bytes, void **p) {
  PGPU_CUDA(n->ctx, cudaMalloc(p, std::max<size_t>(bytes, 16)));
  n->owned.push_back(*p);
  return PGPU_OK;
}
template <typename T>
pgpu_status mo(pgpu_mlp *n, size_t count, T **p) {
  void *v;
  PGPU_TRY(malloc_own(n, count * sizeof(T), &v));
  *p = static_cast<T *>(v);
  return PGPU_OK;
}

pgpu_status pack(pgpu_mlp *nn) {
  mlp_pack_kernel<<<(HID * HID + 255) / 256, 256, 0, nn->ctx->stream>>>(nn->p, nn->W[0], nn->W[1], nn->WT[1],
                                                                        nn->W[2], nn->WT[2]);
  return pgpu_after_launch(nn->ctx, "mlp_pack_kernel");
}

template <int EPI>
pgpu_status tile(pgpu_mlp *nn, const TileArgs &a) {
  constexpr int smem = TST * TSTAGE;
  PGPU_CUDA(nn->ctx, cudaFuncSetAttribute(mlp_tile_kernel<EPI>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem));
  PGPU_CUDA(nn->ctx, launch_chained(mlp_tile_kernel<EPI>, dim3((unsigned)(a.rows / GM), HID / TN), MLP_NT, smem,
                                    nn->ctx->stream, a));
  return pgpu_after_launch(nn->ctx, "mlp_tile_kernel");
}

}  // namespace

extern "C" {

long long pgpu_mlp_n_params(void) { return (long long)N_PARAMS; }

pgpu_status pgpu_mlp_create(pgpu_ctx *ctx, uint64_t seed, int max_batch, pgpu_mlp **out) {
  if (!ctx || !out || max_batch < 1) return PGPU_ERR_ARG;
  *out = nullptr;
  PGPU_CUDA(ctx, cudaSetDevice(ctx->device));
  pgpu_mlp *nn = new pgpu_mlp();
  nn->ctx = ctx;
  nn->max_batch = max_batch;
  nn->bpad = (int)pad_to((size_t)max_batch, GM);
  auto fail = [&](pgpu_status st) {
    pgpu_mlp_destroy(nn);
    return st;
  };
#define MLP_TRY(x)                        \
  do {                                    \
    pgpu_status st_ = (x);                \
    if (st_ != PGPU_OK) return fail(st_); \
  } while (0)
  MLP_TRY(mo(nn, N_PARAMS, &nn->p));
  MLP_TRY(mo(nn, N_PARAMS, &nn->m));
  MLP_TRY(mo(nn, N_PARAMS, &nn->v));
  MLP_TRY(mo(nn, N_PARAMS, &nn->g));
  MLP_TRY(mo(nn, (size_t)HID * IN, &nn->W[0]));
  for (int l = 1; l < 3; ++l) {
    MLP_TRY(mo(nn, (size_t)HID * HID, &nn->W[l]));
    MLP_TRY(mo(nn, (size_t)HID * HID, &nn->WT[l]));
  }
  MLP_TRY(mo(nn, IN, &nn->mu));
  MLP_TRY(mo(nn, IN, &nn->inv_sd));
  MLP_TRY(mo(nn, 8, &nn->loss));
  const size_t B = nn->bpad;
  MLP_TRY(mo(nn, B * GM, &nn->HT[0]));   // 64 rows in tiles of 128
  for (int l = 0; l < 3; ++l) {
    MLP_TRY(mo(nn, B * HID, &nn->H[l]));
    MLP_TRY(mo(nn, B * HID, &nn->HT[l + 1]));
    MLP_TRY(mo(nn, B * HID, &nn->Z[l]));
    MLP_TRY(mo(nn, B * HID, &nn->DZ[l]));
    MLP_TRY(mo(nn, B * HID, &nn->DZT[l]));
  }
  MLP_TRY(mo(nn, B, &nn->y));
  MLP_TRY(mo(nn, B, &nn->dy));
  // He-uniform initial weights (seeded host RNG), zero biases
  std::vector<float> h(N_PARAMS, 0.0f);
  std::mt19937_64 rng(seed);
  auto fill = [&](size_t off, int fan_out, int fan_in) {
    const float lim = std::sqrt(6.0f / (float)fan_in);
    std::uniform_real_distribution<float> u(-lim, lim);
    for (size_t i = 0; i < (size_t)fan_out * fan_in; ++i) h[off + i] = u(rng);
  };
  fill(OFF_W1, HID, IN);
  fill(OFF_W2, HID, HID);
  fill(OFF_W3, HID, HID);
  {
    const float lim = std::sqrt(3.0f / (float)HID);
    std::uniform_real_distribution<float> u(-lim, lim);
    for (int i = 0; i < HID; ++i) h[OFF_W4 + i] = u(rng);
  }
  std::vector<float> ones(IN, 1.0f), zeros(IN, 0.0f);
  if (cudaMemcpy(nn->p, h.data(), N_PARAMS * 4, cudaMemcpyHostToDevice) != cudaSuccess ||
      cudaMemset(nn->m, 0, N_PARAMS * 4) != cudaSuccess || cudaMemset(nn->v, 0, N_PARAMS * 4) != cudaSuccess ||
      cudaMemcpy(nn->mu, zeros.data(), IN * 4, cudaMemcpyHostToDevice) != cudaSuccess ||
      cudaMemcpy(nn->inv_sd, ones.data(), IN * 4, cudaMemcpyHostToDevice) != cudaSuccess) {
    (void)cudaGetLastError();
    return fail(pgpu_set_err(ctx, PGPU_ERR_CUDA, "mlp: initial copies failed"));
  }
  MLP_TRY(pack(nn));
#undef MLP_TRY
  *out = nn;
  return PGPU_OK;
}

void pgpu_mlp_destroy(pgpu_mlp *nn) {
  if (!nn) return;
  if (nn->ctx) cudaSetDevice(nn->ctx->device);
  for (void *p : nn->owned) cudaFree(p);
  delete nn;
}

pgpu_status pgpu_mlp_get_params(pgpu_mlp *nn, float *host) {
  if (!nn || !host) return PGPU_ERR_ARG;
  PGPU_CUDA(nn->ctx, cudaMemcpyAsync(host, nn->p, N_PARAMS * 4, cudaMemcpyDeviceToHost, nn->ctx->stream));
  PGPU_CUDA(nn->ctx, cudaStreamSynchronize(nn->ctx->stream));
  return PGPU_OK;
}

pgpu_status pgpu_mlp_set_params(pgpu_mlp *nn, const float *host) {
  if (!nn || !host) return PGPU_ERR_ARG;
  PGPU_CUDA(nn->ctx, cudaMemcpyAsync(nn->p, host, N_PARAMS * 4, cudaMemcpyHostToDevice, nn->ctx->stream));
  PGPU_TRY(pack(nn));
  PGPU_CUDA(nn->ctx, cudaStreamSynchronize(nn->ctx->stream));
  return PGPU_OK;
}

pgpu_status pgpu_mlp_get_norm(pgpu_mlp *nn, float *mu, float *inv_sd) {
  if (!nn || !mu || !inv_sd) return PGPU_ERR_ARG;
  PGPU_CUDA(nn->ctx, cudaMemcpyAsync(mu, nn->mu, IN * 4, cudaMemcpyDeviceToHost, nn->ctx->stream));
  PGPU_CUDA(nn->ctx, cudaMemcpyAsync(inv_sd, nn->inv_sd, IN * 4, cudaMemcpyDeviceToHost, nn->ctx->stream));
  PGPU_CUDA(nn->ctx, cudaStreamSynchronize(nn->ctx->stream));
  return PGPU_OK;
}

// feature normalisation from the column statistics of X_dev [n][64]
pgpu_status pgpu_mlp_fit_norm(pgpu_mlp *nn, const float *X_dev, size_t n) {
  if (!nn || !X_dev) return PGPU_ERR_ARG;
  mlp_colstats_kernel<<<IN, 256, 0, nn->ctx->stream>>>(X_dev, n, nn->mu, nn->inv_sd);
  return pgpu_after_launch(nn->ctx, "mlp_colstats_kernel");
}

pgpu_status pgpu_mlp_forward(pgpu_mlp *nn, const float *X_dev, size_t n, float *y_dev) {
  if (!nn || !X_dev || !y_dev) return PGPU_ERR_ARG;
  if (n == 0) return PGPU_OK;
  if (n > (size_t)1 << 30) return pgpu_set_err(nn->ctx, PGPU_ERR_LIMIT, "mlp: too many rows");
  PGPU_CUDA(nn->ctx, cudaSetDevice(nn->ctx->device));
  const NetView net{nn->p, nn->mu, nn->inv_sd, {nn->W[0], nn->W[1], nn->W[2]}};
  PGPU_CUDA(nn->ctx, cudaFuncSetAttribute(mlp_forward_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                          (int)FWD_SMEM));
  mlp_forward_kernel<<<(unsigned)((n + GM - 1) / GM), MLP_NT, FWD_SMEM, nn->ctx->stream>>>(net, X_dev, n, y_dev,
                                                                                           nn->ctx->d_flag);
  return pgpu_after_launch(nn->ctx, "mlp_forward_kernel");
}

// Gradients of the weighted squared loss: into the flat vector nn->g
// (adam null), or straight into the parameters.
static pgpu_status mlp_backprop(pgpu_mlp *nn, const float *X_dev, const float *t_dev, const float *sw_dev,
                                size_t n, float *loss_host, const AdamArgs *adam) {
  if (n == 0 || n > (size_t)nn->max_batch)
    return pgpu_set_err(nn->ctx, PGPU_ERR_ARG, "mlp: batch of %zu rows (1..%d)", n, nn->max_batch);
  const int B = (int)pad_to(n, GM);   // rows from n on are zero
  cudaStream_t st = nn->ctx->stream;
  const size_t boff[3] = {OFF_B1, OFF_B2, OFF_B3};
  for (int l = 0; l < 3; ++l) {
    TileArgs a{};
    a.A = l == 0 ? nullptr : nn->H[l - 1];
    a.B = nn->W[l];
    a.K = l == 0 ? IN : HID;
    a.bias = nn->p + boff[l];
    a.Z = nn->Z[l];
    a.H = nn->H[l];
    a.HT = nn->HT[l + 1];
    a.rows = B;
    a.X = X_dev;
    a.mu = nn->mu;
    a.inv_sd = nn->inv_sd;
    a.n = n;
    a.XT = nn->HT[0];
    a.flag = nn->ctx->d_flag;
    if (l == 0) PGPU_TRY(tile<TILE_NORM>(nn, a));
    else PGPU_TRY(tile<TILE_GELU>(nn, a));
  }
  PGPU_CUDA(nn->ctx, launch_chained(mlp_out_kernel, dim3((unsigned)(B / 32)), MLP_NT, 0, st, (const float *)nn->p,
                                    (const __nv_bfloat16 *)nn->HT[3], (const float *)nn->Z[2], t_dev, sw_dev,
                                    (int)n, B, nn->y, nn->dy, nn->DZ[2], nn->DZT[2]));
  PGPU_TRY(pgpu_after_launch(nn->ctx, "mlp_out_kernel"));
  for (int l = 2; l > 0; --l) {   // dz_{l-1} = (dz_l W_l) * gelu'(z_{l-1})
    TileArgs a{};
    a.A = nn->DZ[l];
    a.B = nn->WT[l];
    a.K = HID;
    a.Z = nn->Z[l - 1];
    a.H = nn->DZ[l - 1];
    a.HT = nn->DZT[l - 1];
    a.rows = B;
    a.flag = nn->ctx->d_flag;
    PGPU_TRY(tile<TILE_DGELU>(nn, a));
  }
  GradArgs g{};
  for (int l = 0; l < 3; ++l) {
    g.DZT[l] = nn->DZT[l];
    g.W[l] = nn->W[l];
    g.WT[l] = nn->WT[l];
  }
  for (int l = 0; l < 4; ++l) g.HT[l] = nn->HT[l];
  g.y = nn->y;
  g.t = t_dev;
  g.sw = sw_dev;
  g.dy = nn->dy;
  g.n = (int)n;
  g.rows = B;
  if (adam) g.adam = *adam;
  else g.G = nn->g;
  g.loss = nn->loss;
  g.flag = nn->ctx->d_flag;
  constexpr int smem = TST * TSTAGE;
  PGPU_CUDA(nn->ctx, cudaFuncSetAttribute(mlp_grad_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, smem));
  PGPU_CUDA(nn->ctx, launch_chained(mlp_grad_kernel, dim3(WG_TILES + WG_SUMS + 1), MLP_NT, smem, st, g));
  PGPU_TRY(pgpu_after_launch(nn->ctx, "mlp_grad_kernel"));
  if (loss_host) PGPU_CUDA(nn->ctx, cudaMemcpyAsync(loss_host, nn->loss, 4, cudaMemcpyDeviceToHost, st));
  return PGPU_OK;
}

pgpu_status pgpu_mlp_grads(pgpu_mlp *nn, const float *X_dev, const float *t_dev, const float *sw_dev,
                           size_t n, float *grad_host, float *loss_host) {
  if (!nn || !X_dev || !t_dev || !grad_host) return PGPU_ERR_ARG;
  PGPU_CUDA(nn->ctx, cudaSetDevice(nn->ctx->device));
  PGPU_TRY(mlp_backprop(nn, X_dev, t_dev, sw_dev, n, loss_host, nullptr));
  PGPU_CUDA(nn->ctx, cudaMemcpyAsync(grad_host, nn->g, N_PARAMS * 4, cudaMemcpyDeviceToHost, nn->ctx->stream));
  return pgpu_check_flag(nn->ctx, "mlp_grads");
}

pgpu_status pgpu_mlp_train_step(pgpu_mlp *nn, const float *X_dev, const float *t_dev, const float *sw_dev,
                                size_t n, float lr, float weight_decay, float *loss_host) {
  if (!nn || !X_dev || !t_dev) return PGPU_ERR_ARG;
  PGPU_CUDA(nn->ctx, cudaSetDevice(nn->ctx->device));
  const double step = (double)(nn->step + 1);
  AdamArgs a;
  a.p = nn->p;
  a.m = nn->m;
  a.v = nn->v;
  a.lr = lr;
  a.b1 = 0.9f;
  a.b2 = 0.999f;
  a.eps = 1e-8f;
  a.wd = weight_decay;
  a.c1 = (float)(1.0 - std::pow(0.9, step));
  a.c2 = (float)(1.0 - std::pow(0.999, step));
  PGPU_TRY(mlp_backprop(nn, X_dev, t_dev, sw_dev, n, loss_host, &a));
  nn->step += 1;
  if (loss_host) {
    return pgpu_check_flag(nn->ctx, "mlp_train_step");
  }
  return PGPU_OK;
}

}  // extern "C"
