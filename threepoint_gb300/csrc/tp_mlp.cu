// The b_kappa surrogate network on the 5th-generation tensor cores: a
// multilayer perceptron 8 -> 256 -> 256 -> 256 -> 256 -> 1 (SiLU after the
// hidden layers) trained and evaluated with BF16 operands and FP32
// accumulation. Every layer is one GEMM C = A B^T (A [M x K], B [N x K], both
// BF16 with K contiguous) on tcgen05: a CTA computes 128 x N tiles (N <= 256)
// into tensor memory from 64-wide K slabs staged in shared memory in the
// 128-byte-swizzled K-major layout by asynchronous copies; one thread issues
// the MMAs and commits them to an mbarrier; sixteen warps read the accumulator
// back (tcgen05.ld) and apply the layer's epilogue (bias, SiLU or its
// derivative, BF16 row-major and transposed copies for the next layer and the
// weight gradients, the last layer's dot product). The layers (K <= 256) keep
// the whole weight matrix in shared memory and run persistently over the row
// tiles, the next tile's rows loading during the epilogue; weight gradients
// are a GEMM over the batch (K = batch) with a ring of four slabs, split into
// K slices whose FP32 partials a second kernel sums in a fixed order.
//
// Every mbarrier wait has an iteration limit: on expiry the kernel raises an
// error flag, waits (bounded) for its committed MMAs, frees its tensor memory
// and skips the epilogue.
#include <cuda_bf16.h>
#include <cuda_runtime.h>
#include <math.h>
#include <stdint.h>

#include <string>
#include <vector>

#include "tp_capi_internal.h"
#include "tp_kernels.cuh"

namespace tp {

constexpr int MLP_IN = 8;       // features
constexpr int MLP_IN_PAD = 64;  // first layer's K (one 64-wide slab, zero padded)
constexpr int MLP_W = 256;      // hidden width
constexpr int GEMM_NT = 512;    // threads of a GEMM CTA: four warps per 32 TMEM lanes
constexpr int GEMM_BM = 128;    // rows per CTA tile
constexpr int GEMM_BK = 64;     // K per slab (one 128-byte swizzle atom of BF16)
constexpr int MBAR_SPIN = 1 << 22;

enum GemmEpi : int {
  EPI_BIAS = 1,        // z += bias[col]
  EPI_DSILU = 2,       // z *= silu'(zin[row, col])
  EPI_STORE_Z = 4,     // zout[row, col] = z (FP32)
  EPI_SILU = 8,        // h = silu(z), else h = z
  EPI_STORE_H = 16,    // h_bf16[row, col]
  EPI_STORE_HT = 32,   // ht_bf16[col, row]
  EPI_STORE_F32 = 64,  // out_f32[split][row, col] = h
  EPI_DOT = 128,       // y[row] = sum_col h w5[col] + b5
};

struct GemmArgs {
  const __nv_bfloat16* A;
  int lda;
  const __nv_bfloat16* B;
  int ldb;
  int M, N, K;  // M % 128 == 0, N % 32 == 0 and 32 <= N <= 256, K % 64 == 0
  int kslices;  // grid.y; each CTA row covers K / kslices (a multiple of 64)
  int flags;
  const float* bias;
  const float* zin;
  int ldzin;
  float* zout;
  int ldz;
  __nv_bfloat16* h;
  int ldh;
  __nv_bfloat16* ht;
  int ldht;
  float* out;
  int ldo;
  long long split_stride;
  const float* w5;
  const float* b5;  // device scalar
  float* y;
  unsigned* err;  // bit 0: an mbarrier wait reached its limit
  int spin;       // limit of the main loops' waits (the drain's is MBAR_SPIN)
};

// ---- tcgen05 / mbarrier primitives (inline PTX) -----------------------------
__device__ __forceinline__ void mbar_init(uint32_t a, unsigned count) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(a), "r"(count) : "memory");
}
__device__ __forceinline__ bool mbar_wait(uint32_t a, uint32_t parity, int limit) {
  uint32_t ok = 0;
  for (int it = 0; it < limit && !ok; ++it)
    asm volatile(
        "{\n .reg .pred p;\n mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n selp.u32 %0, 1, 0, p;\n}\n"
        : "=r"(ok)
        : "r"(a), "r"(parity)
        : "memory");
  return ok != 0;
}
__device__ __forceinline__ void tc_fence_before() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void tc_fence_after() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }

// K-major operand tile in the 128-byte swizzle: rows of 64 BF16 (128 bytes),
// 8-row atoms of 1024 bytes (stride 1024), 1024-byte aligned base; the K
// step of 16 elements inside the atom advances the start address by 32 bytes
__device__ __forceinline__ uint64_t smem_desc_sw128(uint32_t addr) {
  return (uint64_t)((addr >> 4) & 0x3FFFu) | ((uint64_t)1 << 16) | ((uint64_t)(1024 >> 4) << 32) |
         ((uint64_t)1 << 46) | ((uint64_t)2 << 61);
}
// kind::f16 instruction descriptor: D FP32, A and B BF16, both K-major, M = 128
__host__ __device__ constexpr uint32_t idesc_bf16_m128(int n) {
  return (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(n >> 3) << 17) | ((uint32_t)(128 >> 4) << 24);
}

__device__ __forceinline__ void tc_mma(uint32_t d_tmem, uint64_t a, uint64_t b, uint32_t idesc, uint32_t acc) {
  asm volatile(
      "{\n .reg .pred p;\n setp.ne.b32 p, %4, 0;\n tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n}\n" ::"r"(
          d_tmem),
      "l"(a), "l"(b), "r"(idesc), "r"(acc)
      : "memory");
}
__device__ __forceinline__ void tc_commit(uint32_t mbar) {
  asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(mbar)
               : "memory");
}
// 32 consecutive accumulator columns of this warp's 32 lanes (one row per lane)
__device__ __forceinline__ void tc_ld32(uint32_t taddr, float* v) {
  uint32_t r[32];
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x32.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16,%17,%18,%19,%"
      "20,%21,%22,%23,%24,%25,%26,%27,%28,%29,%30,%31}, [%32];"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]),
        "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15]), "=r"(r[16]),
        "=r"(r[17]), "=r"(r[18]), "=r"(r[19]), "=r"(r[20]), "=r"(r[21]), "=r"(r[22]), "=r"(r[23]), "=r"(r[24]),
        "=r"(r[25]), "=r"(r[26]), "=r"(r[27]), "=r"(r[28]), "=r"(r[29]), "=r"(r[30]), "=r"(r[31])
      : "r"(taddr)
      : "memory");
  asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
  for (int i = 0; i < 32; ++i) v[i] = __uint_as_float(r[i]);
}

__device__ __forceinline__ void tc_st32(uint32_t taddr, const float* v) {
  asm volatile(
      "tcgen05.st.sync.aligned.32x32b.x32.b32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16,%17,%18,%19,"
      "%20,%21,%22,%23,%24,%25,%26,%27,%28,%29,%30,%31,%32};" ::"r"(taddr),
      "r"(__float_as_uint(v[0])), "r"(__float_as_uint(v[1])), "r"(__float_as_uint(v[2])), "r"(__float_as_uint(v[3])),
      "r"(__float_as_uint(v[4])), "r"(__float_as_uint(v[5])), "r"(__float_as_uint(v[6])), "r"(__float_as_uint(v[7])),
      "r"(__float_as_uint(v[8])), "r"(__float_as_uint(v[9])), "r"(__float_as_uint(v[10])), "r"(__float_as_uint(v[11])),
      "r"(__float_as_uint(v[12])), "r"(__float_as_uint(v[13])), "r"(__float_as_uint(v[14])), "r"(__float_as_uint(v[15])),
      "r"(__float_as_uint(v[16])), "r"(__float_as_uint(v[17])), "r"(__float_as_uint(v[18])), "r"(__float_as_uint(v[19])),
      "r"(__float_as_uint(v[20])), "r"(__float_as_uint(v[21])), "r"(__float_as_uint(v[22])), "r"(__float_as_uint(v[23])),
      "r"(__float_as_uint(v[24])), "r"(__float_as_uint(v[25])), "r"(__float_as_uint(v[26])), "r"(__float_as_uint(v[27])),
      "r"(__float_as_uint(v[28])), "r"(__float_as_uint(v[29])), "r"(__float_as_uint(v[30])), "r"(__float_as_uint(v[31]))
      : "memory");
  asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
}
// eight words, a whole 32-byte sector, a lane
__device__ __forceinline__ void st8(void* p, const uint32_t* r) {
  asm volatile("st.global.v8.b32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8};" ::"l"(p), "r"(r[0]), "r"(r[1]), "r"(r[2]),
               "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7])
               : "memory");
}
__device__ __forceinline__ void st8(float* p, const float* v) {
  uint32_t r[8];
#pragma unroll
  for (int i = 0; i < 8; ++i) r[i] = __float_as_uint(v[i]);
  st8((void*)p, r);
}
__device__ __forceinline__ void ld8(float* v, const float* p) {
  uint32_t r[8];
  asm volatile("ld.global.v8.b32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7])
               : "l"(p)
               : "memory");
#pragma unroll
  for (int i = 0; i < 8; ++i) v[i] = __uint_as_float(r[i]);
}

__device__ __forceinline__ float silu_f(float z) { return z / (1.f + __expf(-z)); }
__device__ __forceinline__ float silu_grad_f(float z) {
  const float s = 1.f / (1.f + __expf(-z));
  return s * (1.f + z * (1.f - s));
}

// copy one 64-wide K slab of `rows` rows (K-major, 16-byte chunks) into the
// swizzled layout, asynchronously
__device__ __forceinline__ void load_slab(uint32_t dst, const __nv_bfloat16* src, int ld, int rows, int k0) {
  const int chunks = rows * 8;
  for (int q = threadIdx.x; q < chunks; q += GEMM_NT) {
    const int r = q >> 3, c = q & 7;
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dst + r * 128 + ((c ^ (r & 7)) << 4)),
                 "l"(src + (size_t)r * ld + k0 + 8 * c)
                 : "memory");
  }
}
__device__ __forceinline__ void load_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N>
__device__ __forceinline__ void load_wait() {
  asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory");
}

// four MMAs of one 64-wide slab (K order: slabs ascending, 16 at a time)
__device__ __forceinline__ void mma_slab(uint32_t tmem, uint32_t a0, uint32_t b0, uint32_t idesc, bool first) {
#pragma unroll
  for (int kk = 0; kk < GEMM_BK / 16; ++kk)
    tc_mma(tmem, smem_desc_sw128(a0 + 32 * kk), smem_desc_sw128(b0 + 32 * kk), idesc, !first || kk != 0);
}

constexpr size_t GEMM_SLAB_A = (size_t)GEMM_BM * GEMM_BK * 2;
constexpr size_t GEMM_SLAB_B = (size_t)MLP_W * GEMM_BK * 2;
constexpr int GEMM_KMAX = 256, GEMM_STAGES = 4;             // k_gemm_rows' K; k_gemm_ring's slabs in flight
constexpr size_t GEMM_SMEM = 1024 + GEMM_STAGES * (GEMM_SLAB_A + GEMM_SLAB_B) + 64;
static_assert(GEMM_STAGES * GEMM_BK >= GEMM_KMAX, "k_gemm_rows holds every slab of A and B");

// The epilogue of the 128 x N tile at row m0 in tensor memory: warp w takes
// the 32 rows of lanes 32 (w % 4) and every fourth 32-column chunk from w / 4
// on, a row a lane. Row-major operands and results move a 32-byte sector a
// lane and instruction: whole sectors without a pass through shared memory, so
// that sixteen warps fit beside the slabs.
__device__ __forceinline__ void gemm_epilogue(const GemmArgs& g, uint32_t tmem, int m0) {
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, quad = warp & 3, part = warp >> 2;
  const int row = m0 + quad * 32 + lane;
  const uint32_t tw = tmem + ((uint32_t)(quad * 32) << 16);
  const int f = g.flags, nch = g.N / 32;
  for (int c = part; c < nch; c += GEMM_NT / 128) {
    const int c0 = 32 * c;
    float v[32], zin[32];
    if (f & EPI_DSILU) {
#pragma unroll
      for (int q = 0; q < 4; ++q) ld8(zin + 8 * q, g.zin + (size_t)row * g.ldzin + c0 + 8 * q);
    }
    tc_ld32(tw + (uint32_t)c0, v);
#pragma unroll
    for (int q = 0; q < 4; ++q) {
      float z[8];
#pragma unroll
      for (int i = 0; i < 8; ++i) {
        const int j = 8 * q + i;
        z[i] = v[j];
        if (f & EPI_BIAS) z[i] += g.bias[c0 + j];
        if (f & EPI_DSILU) z[i] *= silu_grad_f(zin[j]);
        v[j] = (f & EPI_SILU) ? silu_f(z[i]) : z[i];
      }
      if (f & EPI_STORE_Z) st8(g.zout + (size_t)row * g.ldz + c0 + 8 * q, z);
    }
    if (f & EPI_STORE_HT) {
      // two rows (this lane's and its neighbour's) of one column a lane
#pragma unroll
      for (int j = 0; j < 32; j += 2) {
        const float other = __shfl_xor_sync(0xffffffffu, (lane & 1) ? v[j] : v[j + 1], 1);
        const __nv_bfloat162 p = (lane & 1) ? __floats2bfloat162_rn(other, v[j + 1]) : __floats2bfloat162_rn(v[j], other);
        *reinterpret_cast<__nv_bfloat162*>(g.ht + (size_t)(c0 + j + (lane & 1)) * g.ldht + (row & ~1)) = p;
      }
    }
    if (f & EPI_STORE_F32) {
      float* o = g.out + (size_t)blockIdx.y * g.split_stride + (size_t)row * g.ldo + c0;
      if (((size_t)g.out & 31) == 0 && g.ldo % 8 == 0) {  // (split_stride is a multiple of 8)
#pragma unroll
        for (int q = 0; q < 4; ++q) st8(o + 8 * q, v + 8 * q);
      } else {  // a caller's matrix of any alignment
#pragma unroll
        for (int j = 0; j < 32; ++j) o[j] = v[j];
      }
    }
    if (f & EPI_STORE_H) {
#pragma unroll
      for (int q = 0; q < 2; ++q) {
        uint32_t r[8];
#pragma unroll
        for (int i = 0; i < 8; ++i) {
          const __nv_bfloat162 p = __floats2bfloat162_rn(v[16 * q + 2 * i], v[16 * q + 2 * i + 1]);
          r[i] = *reinterpret_cast<const uint32_t*>(&p);
        }
        st8(g.h + (size_t)row * g.ldh + c0 + 16 * q, r);
      }
    }
    if (f & EPI_DOT) tc_st32(tw + (uint32_t)c0, v);
  }
  if (f & EPI_DOT) {
    // one chain over the columns of a row, from the results put back in tensor memory
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    if (part == 0) {
      float dot = 0.f;
      for (int c = 0; c < nch; ++c) {
        float v[32];
        tc_ld32(tw + (uint32_t)(32 * c), v);
#pragma unroll
        for (int j = 0; j < 32; ++j) dot = fmaf(v[j], g.w5[32 * c + j], dot);
      }
      g.y[row] = dot + *g.b5;
    }
  }
}

// shared memory of a GEMM CTA: slabs (1024-byte aligned), barriers
struct GemmSmem {
  uint32_t a, b;  // slab s of A at a + s GEMM_SLAB_A, of B at b + s GEMM_SLAB_B
  uint64_t* bars;
  uint32_t* tmem;
  __device__ __forceinline__ GemmSmem(char* raw) {
    char* base = raw + ((1024u - (smem_u32(raw) & 1023u)) & 1023u);
    a = smem_u32(base);
    b = a + GEMM_STAGES * GEMM_SLAB_A;
    bars = (uint64_t*)(base + GEMM_STAGES * (GEMM_SLAB_A + GEMM_SLAB_B));
    tmem = (uint32_t*)(bars + GEMM_STAGES);
  }
};
__device__ __forceinline__ int tmem_cols(int N) { return N <= 32 ? 32 : N <= 64 ? 64 : N <= 128 ? 128 : 256; }
__device__ __forceinline__ void gemm_begin(const GemmSmem& m, int N) {
  if (threadIdx.x == 0) {
    for (int s = 0; s < GEMM_STAGES; ++s) mbar_init(smem_u32(&m.bars[s]), 1);
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (threadIdx.x < 32) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(m.tmem)),
                 "r"(tmem_cols(N))
                 : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
}
__device__ __forceinline__ void gemm_end(const GemmArgs& g, uint32_t tmem, bool ok) {
  if (!ok && threadIdx.x == 0 && g.err) atomicOr(g.err, 1u);
  tc_fence_before();
  __syncthreads();
  if (threadIdx.x < 32)
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(tmem_cols(g.N)) : "memory");
}

// K <= GEMM_KMAX: B stays in shared memory, the CTA walks the row tiles
// blockIdx.x, + gridDim.x, ...; the next tile's rows of A are copied while this
// tile's epilogue runs. The epilogue's stores bound it (HBM: 167 MB for a
// training layer of 65536 rows, 25 us): 177 -> 62 us for that layer with sixteen
// warps on the accumulator, 100 us with eight and a shared-memory transpose,
// against one tile a CTA whose loads, MMAs and epilogue wait for one another
__global__ void __launch_bounds__(GEMM_NT, 1) k_gemm_rows(GemmArgs g) {
  extern __shared__ __align__(16) char smem_raw[];
  const GemmSmem m(smem_raw);
  gemm_begin(m, g.N);
  const uint32_t tmem = *m.tmem, bar = smem_u32(&m.bars[0]), idesc = idesc_bf16_m128(g.N);
  const int nslab = g.K / GEMM_BK, ntile = g.M / GEMM_BM;
  auto load_a = [&](int t) {
    for (int s = 0; s < nslab; ++s)
      load_slab(m.a + s * GEMM_SLAB_A, g.A + (size_t)t * GEMM_BM * g.lda, g.lda, GEMM_BM, s * GEMM_BK);
    load_commit();
  };
  for (int s = 0; s < nslab; ++s) load_slab(m.b + s * GEMM_SLAB_B, g.B, g.ldb, g.N, s * GEMM_BK);
  if ((int)blockIdx.x < ntile) load_a(blockIdx.x);
  bool ok = true;
  uint32_t parity = 0;
  for (int t = blockIdx.x; t < ntile; t += gridDim.x) {
    load_wait<0>();
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    tc_fence_before();  // the previous epilogue's accumulator reads
    __syncthreads();
    if (threadIdx.x == 0) {
      tc_fence_after();
      for (int s = 0; s < nslab; ++s) mma_slab(tmem, m.a + s * GEMM_SLAB_A, m.b + s * GEMM_SLAB_B, idesc, s == 0);
      tc_commit(bar);
    }
    ok = mbar_wait(bar, parity, g.spin);
    ok = __syncthreads_and(ok);
    if (!ok) {
      mbar_wait(bar, parity, MBAR_SPIN);  // the tile's MMAs still read shared memory
      break;
    }
    parity ^= 1;
    tc_fence_after();
    if (t + (int)gridDim.x < ntile) load_a(t + gridDim.x);
    gemm_epilogue(g, tmem, t * GEMM_BM);
  }
  load_wait<0>();
  gemm_end(g, tmem, ok);
}

// Any K: a ring of GEMM_STAGES slabs of A and B; blockIdx.x the row tile,
// blockIdx.y the K slice. The copies of three slabs are in flight while the
// tensor core works on the fourth (a 256 x 256 weight gradient over 65536 rows
// in 64 slices: 222 -> 25 us, against two slabs and a wait after each load)
__global__ void __launch_bounds__(GEMM_NT, 1) k_gemm_ring(GemmArgs g) {
  extern __shared__ __align__(16) char smem_raw[];
  const GemmSmem m(smem_raw);
  gemm_begin(m, g.N);
  const uint32_t tmem = *m.tmem, idesc = idesc_bf16_m128(g.N);
  const int m0 = blockIdx.x * GEMM_BM, kper = g.K / g.kslices, kbeg = blockIdx.y * kper, nslab = kper / GEMM_BK;
  auto load = [&](int s) {  // a group a slab, empty past the end
    if (s < nslab) {
      const int b = s % GEMM_STAGES;
      load_slab(m.a + b * GEMM_SLAB_A, g.A + (size_t)m0 * g.lda, g.lda, GEMM_BM, kbeg + s * GEMM_BK);
      load_slab(m.b + b * GEMM_SLAB_B, g.B, g.ldb, g.N, kbeg + s * GEMM_BK);
    }
    load_commit();
  };
  for (int s = 0; s < GEMM_STAGES - 1; ++s) load(s);
  bool ok = true;
  int last = 0;  // the last slab whose MMAs are committed
  for (int s = 0; s < nslab; ++s) {
    load_wait<GEMM_STAGES - 2>();  // slab s has landed
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    __syncthreads();
    if (threadIdx.x == 0) {
      tc_fence_after();
      const int b = s % GEMM_STAGES;
      mma_slab(tmem, m.a + b * GEMM_SLAB_A, m.b + b * GEMM_SLAB_B, idesc, s == 0);
      tc_commit(smem_u32(&m.bars[b]));
    }
    last = s;
    // slab s - 1's buffer is free once its MMAs are done: slab s + 3 goes there
    if (s > 0) {
      ok = mbar_wait(smem_u32(&m.bars[(s - 1) % GEMM_STAGES]), ((s - 1) / GEMM_STAGES) & 1, g.spin);
      ok = __syncthreads_and(ok);
      if (!ok) break;
    }
    load(s + GEMM_STAGES - 1);
  }
  // MMAs complete in order: this wait covers all of them, after an expired one too
  const uint32_t bar = smem_u32(&m.bars[last % GEMM_STAGES]), parity = (last / GEMM_STAGES) & 1;
  if (ok) ok = mbar_wait(bar, parity, g.spin);
  ok = __syncthreads_and(ok);
  if (!ok) mbar_wait(bar, parity, MBAR_SPIN);
  load_wait<0>();
  tc_fence_after();
  if (ok) gemm_epilogue(g, tmem, m0);
  gemm_end(g, tmem, ok);
}

// ---- element-wise and reduction kernels of the training step ---------------

// features [n][8] (FP32) -> X [Mpad][64] and the first 8 rows of XT [64][Mpad]
// (BF16, zero padded; the caller clears the other rows); one thread a row, so
// that both are written in whole sectors
__global__ void k_mlp_pack(const float* x, long n, int mpad, __nv_bfloat16* X, __nv_bfloat16* XT) {
  const int r = blockIdx.x * blockDim.x + threadIdx.x;
  if (r >= mpad) return;
  alignas(16) __nv_bfloat16 v[MLP_IN];
#pragma unroll
  for (int c = 0; c < MLP_IN; ++c) {
    v[c] = __float2bfloat16_rn(r < n ? x[(size_t)r * MLP_IN + c] : 0.f);
    XT[(size_t)c * mpad + r] = v[c];
  }
  uint4* o = reinterpret_cast<uint4*>(X + (size_t)r * MLP_IN_PAD);
  o[0] = *reinterpret_cast<const uint4*>(v);
#pragma unroll
  for (int q = 1; q < MLP_IN_PAD / 8; ++q) o[q] = make_uint4(0, 0, 0, 0);
}

// dy = 2 (y - t) / n (0 on padding rows); per-block partial sums of (y - t)^2
__global__ void k_mlp_loss(const float* y, const float* t, long n, int mpad, float* dy, double* part) {
  __shared__ double red[256];
  const long i = (long)blockIdx.x * blockDim.x + threadIdx.x;
  double e2 = 0;
  if (i < mpad) {
    float d = 0.f;
    if (i < n) {
      d = y[i] - t[i];
      e2 = (double)d * d;
    }
    dy[i] = i < n ? 2.f * d / (float)n : 0.f;
  }
  red[threadIdx.x] = e2;
  __syncthreads();
  for (int o = blockDim.x / 2; o > 0; o >>= 1) {
    if (threadIdx.x < o) red[threadIdx.x] += red[threadIdx.x + o];
    __syncthreads();
  }
  if (threadIdx.x == 0) part[blockIdx.x] = red[0];
}

// sum of nparts doubles in a fixed order (one thread, from shared memory)
__global__ void k_sum_fixed(const double* part, int nparts, long n, float* loss) {
  __shared__ double sp[1024];
  double s = 0;
  for (int i0 = 0; i0 < nparts; i0 += 1024) {
    const int m = min(1024, nparts - i0);
    __syncthreads();
    for (int i = threadIdx.x; i < m; i += blockDim.x) sp[i] = part[i0 + i];
    __syncthreads();
    if (threadIdx.x == 0) {
#pragma unroll 8
      for (int i = 0; i < m; ++i) s += sp[i];
    }
  }
  if (threadIdx.x == 0) *loss = (float)(s / (double)n);
}

// dW5[j] = sum_b dy[b] h4[b][j], db5 = sum_b dy[b] in 32 chains (b mod 32)
// whose sums a butterfly adds: one block a chain and 64 columns, a thread a
// column, so that 128 blocks read whole row pieces. A chain is serial, so its
// rows are copied ahead, three of four stages of 32 rows in flight (335 -> 34
// us for 65536 rows, against one warp a column)
constexpr int LG_COLS = 64, LG_ROWS = 32, LG_STAGES = 4;
__global__ void __launch_bounds__(LG_COLS) k_mlp_last_grad(const float* dy, const float* h4, int mpad, float* part) {
  __shared__ __align__(16) float sh[LG_STAGES][LG_ROWS][LG_COLS];
  __shared__ float sd[LG_STAGES][LG_ROWS];
  const int l = blockIdx.x, c0 = blockIdx.y * LG_COLS, tid = threadIdx.x;
  const int nrow = mpad / 32, ns = (nrow + LG_ROWS - 1) / LG_ROWS;
  auto load = [&](int k) {  // a group a stage, empty past the end
    if (k < ns) {
      const int b = k % LG_STAGES, n = min(LG_ROWS, nrow - k * LG_ROWS);
      for (int q = tid; q < n * (LG_COLS / 4); q += LG_COLS) {
        const int r = q / (LG_COLS / 4), c = 4 * (q % (LG_COLS / 4));
        asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(smem_u32(&sh[b][r][c])),
                     "l"(h4 + (size_t)((k * LG_ROWS + r) * 32 + l) * MLP_W + c0 + c)
                     : "memory");
      }
      if (tid < n)
        asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"(smem_u32(&sd[b][tid])),
                     "l"(dy + (k * LG_ROWS + tid) * 32 + l)
                     : "memory");
    }
    load_commit();
  };
  for (int k = 0; k < LG_STAGES - 1; ++k) load(k);
  float s = 0.f, sb = 0.f;
  for (int k = 0; k < ns; ++k) {
    load_wait<LG_STAGES - 2>();
    __syncthreads();  // stage k has landed and stage k - 1 is read
    load(k + LG_STAGES - 1);
    const int b = k % LG_STAGES, n = min(LG_ROWS, nrow - k * LG_ROWS);  // a multiple of 4
#pragma unroll 4
    for (int r = 0; r < n; ++r) {
      const float d = sd[b][r];
      s += d * sh[b][r][tid];
      sb += d;
    }
  }
  load_wait<0>();
  part[(c0 + tid) * 32 + l] = s;
  if (c0 + tid == 0) part[MLP_W * 32 + l] = sb;
}
__global__ void k_mlp_last_sum(const float* part, float* gw5, float* gb5) {
  const int w = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5), lane = threadIdx.x & 31;
  if (w > MLP_W) return;
  float s = part[w * 32 + lane];
  for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
  if (lane == 0) {
    if (w < MLP_W)
      gw5[w] = s;
    else
      *gb5 = s;
  }
}

// dZ4 = dy w5 silu'(Z4): row-major and transposed BF16, in 64 x 64 tiles
// through shared memory so that both are written in 128-byte pieces (155 ->
// 43 us for 65536 rows)
__global__ void __launch_bounds__(256) k_mlp_dz4(const float* dy, const float* w5, const float* z4, int mpad,
                                                 __nv_bfloat16* dz, __nv_bfloat16* dzt) {
  __shared__ float t[64][65];
  const int r0 = blockIdx.x * 64, c0 = blockIdx.y * 64;  // mpad % 128 == 0
  const int c = threadIdx.x & 63;
  const float w = w5[c0 + c];
#pragma unroll
  for (int q = threadIdx.x >> 6; q < 64; q += 4) {
    const size_t i = (size_t)(r0 + q) * MLP_W + c0 + c;
    const float v = dy[r0 + q] * w * silu_grad_f(z4[i]);
    dz[i] = __float2bfloat16_rn(v);
    t[q][c] = v;
  }
  __syncthreads();
  const int lane = threadIdx.x & 31;
#pragma unroll
  for (int q = threadIdx.x >> 5; q < 64; q += 8)
    *reinterpret_cast<__nv_bfloat162*>(dzt + (size_t)(c0 + q) * mpad + r0 + 2 * lane) =
        __floats2bfloat162_rn(t[2 * lane][q], t[2 * lane + 1][q]);
}

// bias gradient: db[j] = sum_b dZ[b][j] from the transposed copy (row j
// contiguous over the batch) in 32 chains (b mod 32) and a butterfly; a block a
// row, its segments copied to shared memory ahead of the one warp that sums
// (114 -> 16 us for 65536 columns, against one warp a row reading them itself)
constexpr int RS_SEG = 4096;
__global__ void __launch_bounds__(256) k_mlp_rowsum(const __nv_bfloat16* dzt, int mpad, float* db) {
  __shared__ __align__(16) __nv_bfloat16 seg[2][RS_SEG];
  const __nv_bfloat16* row = dzt + (size_t)blockIdx.x * mpad;
  const int lane = threadIdx.x & 31, ns = (mpad + RS_SEG - 1) / RS_SEG;
  auto load = [&](int k) {
    if (k < ns) {
      const int n = min(RS_SEG, mpad - k * RS_SEG);  // a multiple of 128
      for (int i = 8 * threadIdx.x; i < n; i += 8 * 256)
        asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(smem_u32(&seg[k & 1][i])), "l"(row + k * RS_SEG + i)
                     : "memory");
    }
    load_commit();
  };
  float s = 0.f;
  load(0);
  for (int k = 0; k < ns; ++k) {
    load(k + 1);
    load_wait<1>();
    __syncthreads();
    if (threadIdx.x < 32) {
      const int n = min(RS_SEG, mpad - k * RS_SEG);
#pragma unroll 16
      for (int b = lane; b < n; b += 32) s += __bfloat162float(seg[k & 1][b]);
    }
    __syncthreads();
  }
  if (threadIdx.x < 32) {
    for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
    if (lane == 0) db[blockIdx.x] = s;
  }
}

// out[i] = sum_s part[s][i] in a fixed order
__global__ void k_split_reduce(const float* part, int slices, long count, long stride, float* out) {
  const long i = (long)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= count) return;
  float s = 0.f;
  for (int k = 0; k < slices; ++k) s += part[(size_t)k * stride + i];
  out[i] = s;
}

// Adam (Kingma & Ba 2015, bias-corrected) on the FP32 master copy, then the
// BF16 copies the GEMMs read: wb [rows][ld] and optionally its transpose
// wt [cols][256]; cols <= ld, the padding columns stay zero. All parameters in
// one launch: seg lists the weight matrices, the rest (biases, the last layer)
// has no copies.
struct AdamSeg {
  long first, count;
  int cols, ld;
  __nv_bfloat16 *wb, *wt;
};
struct AdamSegs {
  AdamSeg s[4];
};
__global__ void k_mlp_adam(float* w, const float* g, float* m, float* v, long count, float lr, float b1, float b2,
                           float eps, float c1, float c2, AdamSegs segs) {
  const long p = (long)blockIdx.x * blockDim.x + threadIdx.x;
  if (p >= count) return;
  const float gi = g[p];
  const float mi = b1 * m[p] + (1.f - b1) * gi;
  const float vi = b2 * v[p] + (1.f - b2) * gi * gi;
  m[p] = mi;
  v[p] = vi;
  const float wi = w[p] - lr * (mi / c1) / (sqrtf(vi / c2) + eps);
  w[p] = wi;
#pragma unroll
  for (int k = 0; k < 4; ++k) {
    const AdamSeg& s = segs.s[k];
    const long i = p - s.first;
    if (i < 0 || i >= s.count) continue;
    const int r = (int)(i / s.cols), c = (int)(i % s.cols);
    s.wb[(size_t)r * s.ld + c] = __float2bfloat16_rn(wi);
    if (s.wt) s.wt[(size_t)c * MLP_W + r] = __float2bfloat16_rn(wi);
  }
}

// BF16 copies of an FP32 weight matrix (after set_params)
__global__ void k_mlp_cast(const float* w, long count, int cols, __nv_bfloat16* w_bf, int ld_bf, __nv_bfloat16* wt_bf,
                           int rows) {
  const long i = (long)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= count) return;
  const int r = (int)(i / cols), c = (int)(i % cols);
  w_bf[(size_t)r * ld_bf + c] = __float2bfloat16_rn(w[i]);
  if (wt_bf) wt_bf[(size_t)c * rows + r] = __float2bfloat16_rn(w[i]);
}

}  // namespace tp

// ---------------------------------------------------------------------------
// host side: the network's device state and its C ABI
// ---------------------------------------------------------------------------
using namespace tp;

namespace {

// FP32 master parameters and Adam moments, flat: W1 [256][8], b1, W2..W4
// [256][256], b2..b4, W5 [1][256], b5 (the host API's FP64 layout)
constexpr long P_W1 = 0, P_B1 = P_W1 + (long)MLP_W * MLP_IN;
constexpr long P_W2 = P_B1 + MLP_W, P_B2 = P_W2 + (long)MLP_W * MLP_W;
constexpr long P_W3 = P_B2 + MLP_W, P_B3 = P_W3 + (long)MLP_W * MLP_W;
constexpr long P_W4 = P_B3 + MLP_W, P_B4 = P_W4 + (long)MLP_W * MLP_W;
constexpr long P_W5 = P_B4 + MLP_W, P_B5 = P_W5 + MLP_W;
constexpr long P_COUNT = P_B5 + 1;
const long P_W[5] = {P_W1, P_W2, P_W3, P_W4, P_W5};
const long P_B[5] = {P_B1, P_B2, P_B3, P_B4, P_B5};
const int L_IN[5] = {MLP_IN, MLP_W, MLP_W, MLP_W, MLP_W};
const int L_OUT[5] = {MLP_W, MLP_W, MLP_W, MLP_W, 1};

int round_up(long n, int m) { return (int)((n + m - 1) / m * m); }

}  // namespace

struct tp_mlp {
  int device = 0;
  cudaStream_t stream = nullptr;
  int max_rows = 0;  // padded batch capacity (multiple of 128)
  int kslices_max = 1;
  long adam_t = 0;
  std::string err;
  float *p = nullptr, *g = nullptr, *m = nullptr, *v = nullptr;  // [P_COUNT]
  __nv_bfloat16* wb[4] = {};  // W1 [256][64] (padded), W2..W4 [256][256]
  __nv_bfloat16* wt[4] = {};  // transposes of W2..W4 (index 1..3; [0] unused)
  __nv_bfloat16 *X = nullptr, *XT = nullptr;
  float* Z[4] = {};
  __nv_bfloat16* H[3] = {};
  __nv_bfloat16* HT[3] = {};
  float* H4 = nullptr;
  float *y = nullptr, *t = nullptr, *dy = nullptr, *xin = nullptr;
  __nv_bfloat16* dZ[2] = {};
  __nv_bfloat16* dZT[2] = {};
  float* split = nullptr;  // [kslices][256][256]
  double* lpart = nullptr;
  float* loss = nullptr;
  unsigned* d_err = nullptr;
  int spin = MBAR_SPIN;  // limit of the GEMMs' waits
};

static int mlp_fail(tp_mlp* m, int st, const std::string& msg) {
  if (m) m->err = msg;
  return st;
}
static int mlp_cuda(tp_mlp* m, cudaError_t e, const char* where) {
  if (e == cudaSuccess) return TP_OK;
  return mlp_fail(m, TP_ERR_CUDA, std::string(where) + ": " + cudaGetErrorString(e));
}

template <class T>
static cudaError_t dmalloc(T** p, size_t count) {
  return cudaMalloc((void**)p, sizeof(T) * (count ? count : 1));
}

static cudaError_t gemm(tp_mlp* m, GemmArgs a) {
  static thread_local int attr_dev = -1, sms = 0;
  if (attr_dev != m->device) {
    cudaError_t e = cudaFuncSetAttribute(k_gemm_rows, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)GEMM_SMEM);
    if (e == cudaSuccess)
      e = cudaFuncSetAttribute(k_gemm_ring, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)GEMM_SMEM);
    if (e == cudaSuccess) e = cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, m->device);
    if (e != cudaSuccess) return e;
    attr_dev = m->device;
  }
  if (a.M % GEMM_BM || a.N % 32 || a.N < 32 || a.N > MLP_W || a.K % GEMM_BK || a.kslices < 1 ||
      (a.K / a.kslices) % GEMM_BK || a.K % a.kslices)
    return cudaErrorInvalidValue;
  if (a.M > 0 && a.K <= 0) return cudaSuccess;  // nothing to sum
  a.err = m->d_err;
  a.spin = m->spin;
  const int tiles = a.M / GEMM_BM;
  // B in shared memory while it fits; else (and for K slices) the slab ring
  if (a.kslices == 1 && a.K <= GEMM_KMAX)
    k_gemm_rows<<<tiles < sms ? tiles : sms, GEMM_NT, GEMM_SMEM, m->stream>>>(a);
  else
    k_gemm_ring<<<dim3(tiles, a.kslices), GEMM_NT, GEMM_SMEM, m->stream>>>(a);
  return cudaGetLastError();
}

static GemmArgs gemm_args(const __nv_bfloat16* A, int lda, const __nv_bfloat16* B, int ldb, int M, int N, int K) {
  GemmArgs a{};
  a.A = A;
  a.lda = lda;
  a.B = B;
  a.ldb = ldb;
  a.M = M;
  a.N = N;
  a.K = K;
  a.kslices = 1;
  return a;
}

// BF16 copies of the weights from the FP32 masters
static cudaError_t mlp_cast_all(tp_mlp* m) {
  for (int l = 0; l < 4; ++l) {
    const long cnt = (long)L_OUT[l] * L_IN[l];
    k_mlp_cast<<<(unsigned)((cnt + 255) / 256), 256, 0, m->stream>>>(
        m->p + P_W[l], cnt, L_IN[l], m->wb[l], l == 0 ? MLP_IN_PAD : MLP_W, l == 0 ? nullptr : m->wt[l], MLP_W);
  }
  return cudaGetLastError();
}

// forward over `rows` (multiple of 128) packed rows; training also keeps the
// pre-activations and transposed activations for the backward pass
static cudaError_t mlp_forward_dev(tp_mlp* m, int rows, bool train) {
  cudaError_t e = cudaSuccess;
  const __nv_bfloat16* a = m->X;
  int lda = MLP_IN_PAD;
  for (int l = 0; l < 4 && e == cudaSuccess; ++l) {
    GemmArgs g = gemm_args(a, lda, m->wb[l], l == 0 ? MLP_IN_PAD : MLP_W, rows, MLP_W, l == 0 ? MLP_IN_PAD : MLP_W);
    g.bias = m->p + P_B[l];
    g.flags = EPI_BIAS | EPI_SILU;
    if (train) {
      g.flags |= EPI_STORE_Z;
      g.zout = m->Z[l];
      g.ldz = MLP_W;
    }
    if (l < 3) {
      g.flags |= EPI_STORE_H;
      g.h = m->H[l];
      g.ldh = MLP_W;
      if (train) {
        g.flags |= EPI_STORE_HT;
        g.ht = m->HT[l];
        g.ldht = rows;
      }
    } else {
      g.flags |= EPI_DOT;
      g.w5 = m->p + P_W5;
      g.b5 = m->p + P_B5;
      g.y = m->y;
      if (train) {
        g.flags |= EPI_STORE_F32;
        g.out = m->H4;
        g.ldo = MLP_W;
      }
    }
    e = gemm(m, g);
    a = m->H[l < 3 ? l : 0];
    lda = MLP_W;
  }
  return e;
}

static int mlp_check(tp_mlp* m) {
  unsigned h = 0;
  cudaError_t e = cudaMemcpyAsync(&h, m->d_err, sizeof(unsigned), cudaMemcpyDeviceToHost, m->stream);
  if (e == cudaSuccess) e = cudaStreamSynchronize(m->stream);
  if (e != cudaSuccess) return mlp_cuda(m, e, "mlp");
  if (h) {
    cudaMemsetAsync(m->d_err, 0, sizeof(unsigned), m->stream);
    return mlp_fail(m, TP_ERR_CUDA, "mlp: a tensor-core wait reached its iteration limit");
  }
  return TP_OK;
}

// gradients of the mean squared error into m->g (forward included)
static cudaError_t mlp_backward_dev(tp_mlp* m, long n, int rows) {
  cudaError_t e = cudaSuccess;
  const int nb = (rows + 255) / 256;
  k_mlp_loss<<<nb, 256, 0, m->stream>>>(m->y, m->t, n, rows, m->dy, m->lpart);
  k_sum_fixed<<<1, 256, 0, m->stream>>>(m->lpart, nb, n, m->loss);
  // (the chains' sums go through the slice buffer, free until the first GEMM below)
  k_mlp_last_grad<<<dim3(32, MLP_W / LG_COLS), LG_COLS, 0, m->stream>>>(m->dy, m->H4, rows, m->split);
  k_mlp_last_sum<<<(MLP_W + 1 + 7) / 8, 256, 0, m->stream>>>(m->split, m->g + P_W5, m->g + P_B5);
  k_mlp_dz4<<<dim3(rows / 64, MLP_W / 64), 256, 0, m->stream>>>(m->dy, m->p + P_W5, m->Z[3], rows, m->dZ[0], m->dZT[0]);
  e = cudaGetLastError();
  // K slices of the weight-gradient GEMMs: 1024 batch rows each (at most the
  // allocated partial buffers)
  int ks = rows / 1024;
  if (ks < 1) ks = 1;
  while (ks > m->kslices_max || rows % ks || (rows / ks) % GEMM_BK) --ks;
  int cur = 0;
  for (int l = 3; l >= 0 && e == cudaSuccess; --l) {
    const int in = l == 0 ? MLP_IN_PAD : MLP_W;
    // dW_l = dZ_l^T H_{l-1}: A = dZT [256][rows], B = H_{l-1}^T [in][rows]
    GemmArgs g = gemm_args(m->dZT[cur], rows, l == 0 ? m->XT : m->HT[l - 1], rows, MLP_W, in, rows);
    g.kslices = ks;
    g.flags = EPI_STORE_F32;
    g.out = ks > 1 ? m->split : m->g + P_W[l];
    g.ldo = in;
    g.split_stride = (long long)MLP_W * in;
    if (l == 0) {  // W1's gradient has 8 real columns of the 64 computed
      g.out = m->split;
    }
    e = gemm(m, g);
    if (e != cudaSuccess) break;
    if (l == 0) {
      // sum the slices into [256][64], then keep the 8 real columns
      k_split_reduce<<<(unsigned)(((long)MLP_W * in + 255) / 256), 256, 0, m->stream>>>(
          m->split, ks, (long)MLP_W * in, (long)MLP_W * in, m->split + (size_t)ks * MLP_W * in);
      e = cudaMemcpy2DAsync(m->g + P_W1, sizeof(float) * MLP_IN, m->split + (size_t)ks * MLP_W * in,
                            sizeof(float) * in, sizeof(float) * MLP_IN, MLP_W, cudaMemcpyDeviceToDevice, m->stream);
    } else if (ks > 1) {
      k_split_reduce<<<(unsigned)(((long)MLP_W * in + 255) / 256), 256, 0, m->stream>>>(
          m->split, ks, (long)MLP_W * in, (long)MLP_W * in, m->g + P_W[l]);
    }
    k_mlp_rowsum<<<MLP_W, 256, 0, m->stream>>>(m->dZT[cur], rows, m->g + P_B[l]);
    if (e == cudaSuccess) e = cudaGetLastError();
    if (l == 0 || e != cudaSuccess) break;
    // dZ_{l-1} = (dZ_l W_l) * silu'(Z_{l-1}): B = W_l^T [in][out]
    GemmArgs d = gemm_args(m->dZ[cur], MLP_W, m->wt[l], MLP_W, rows, MLP_W, MLP_W);
    d.flags = EPI_DSILU | EPI_STORE_H | EPI_STORE_HT;
    d.zin = m->Z[l - 1];
    d.ldzin = MLP_W;
    d.h = m->dZ[cur ^ 1];
    d.ldh = MLP_W;
    d.ht = m->dZT[cur ^ 1];
    d.ldht = rows;
    e = gemm(m, d);
    cur ^= 1;
  }
  return e;
}

static cudaError_t mlp_adam_dev(tp_mlp* m, float lr) {
  const float b1 = 0.9f, b2 = 0.999f, eps = 1e-8f;
  m->adam_t++;
  const float c1 = 1.f - powf(b1, (float)m->adam_t), c2 = 1.f - powf(b2, (float)m->adam_t);
  AdamSegs segs;
  for (int l = 0; l < 4; ++l)
    segs.s[l] = {P_W[l], (long)L_OUT[l] * L_IN[l], L_IN[l], l == 0 ? MLP_IN_PAD : MLP_W, m->wb[l], l == 0 ? nullptr : m->wt[l]};
  k_mlp_adam<<<(unsigned)((P_COUNT + 255) / 256), 256, 0, m->stream>>>(m->p, m->g, m->m, m->v, P_COUNT, lr, b1, b2, eps,
                                                                      c1, c2, segs);
  return cudaGetLastError();
}

static cudaError_t mlp_pack(tp_mlp* m, const float* x, long n, int rows) {
  cudaError_t e = cudaMemsetAsync(m->XT + (size_t)MLP_IN * rows, 0,
                                  sizeof(__nv_bfloat16) * (size_t)(MLP_IN_PAD - MLP_IN) * rows, m->stream);
  if (e != cudaSuccess) return e;
  k_mlp_pack<<<(rows + 127) / 128, 128, 0, m->stream>>>(x, n, rows, m->X, m->XT);
  return cudaGetLastError();
}

static cudaError_t mlp_upload_x(tp_mlp* m, const double* x, long n, int rows) {
  std::vector<float> xf((size_t)n * MLP_IN);
  for (size_t i = 0; i < xf.size(); ++i) xf[i] = (float)x[i];
  cudaError_t e = cudaMemcpyAsync(m->xin, xf.data(), sizeof(float) * xf.size(), cudaMemcpyHostToDevice, m->stream);
  if (e == cudaSuccess) e = cudaStreamSynchronize(m->stream);  // xf leaves scope
  if (e == cudaSuccess) {
    e = mlp_pack(m, m->xin, n, rows);
  }
  return e;
}

extern "C" long tp_mlp_param_count(void) { return P_COUNT; }

extern "C" void tp_mlp_destroy(tp_mlp* m);

extern "C" int tp_mlp_create(int device, int max_batch, tp_mlp** out) {
  if (!out || max_batch < 1 || max_batch > (1 << 22)) return TP_ERR_ARG;
  *out = nullptr;
  tp_mlp* m = new tp_mlp();
  m->device = device;
  m->max_rows = round_up(max_batch, 1024);
  m->kslices_max = m->max_rows / 1024;
  const size_t R = (size_t)m->max_rows;
  cudaError_t e = cudaSetDevice(device);
  if (e == cudaSuccess) e = cudaStreamCreateWithFlags(&m->stream, cudaStreamNonBlocking);
  for (float** q : {&m->p, &m->g, &m->m, &m->v})
    if (e == cudaSuccess) e = dmalloc(q, P_COUNT);
  if (e == cudaSuccess) e = dmalloc(&m->wb[0], (size_t)MLP_W * MLP_IN_PAD);
  for (int l = 1; l < 4; ++l) {
    if (e == cudaSuccess) e = dmalloc(&m->wb[l], (size_t)MLP_W * MLP_W);
    if (e == cudaSuccess) e = dmalloc(&m->wt[l], (size_t)MLP_W * MLP_W);
  }
  if (e == cudaSuccess) e = dmalloc(&m->X, R * MLP_IN_PAD);
  if (e == cudaSuccess) e = dmalloc(&m->XT, R * MLP_IN_PAD);
  for (int l = 0; l < 4; ++l)
    if (e == cudaSuccess) e = dmalloc(&m->Z[l], R * MLP_W);
  for (int l = 0; l < 3; ++l) {
    if (e == cudaSuccess) e = dmalloc(&m->H[l], R * MLP_W);
    if (e == cudaSuccess) e = dmalloc(&m->HT[l], R * MLP_W);
  }
  if (e == cudaSuccess) e = dmalloc(&m->H4, R * MLP_W);
  for (float** q : {&m->y, &m->t, &m->dy})
    if (e == cudaSuccess) e = dmalloc(q, R);
  if (e == cudaSuccess) e = dmalloc(&m->xin, R * MLP_IN);
  for (int i = 0; i < 2; ++i) {
    if (e == cudaSuccess) e = dmalloc(&m->dZ[i], R * MLP_W);
    if (e == cudaSuccess) e = dmalloc(&m->dZT[i], R * MLP_W);
  }
  if (e == cudaSuccess) e = dmalloc(&m->split, (size_t)(m->kslices_max + 1) * MLP_W * MLP_W);
  if (e == cudaSuccess) e = dmalloc(&m->lpart, R / 256 + 1);
  if (e == cudaSuccess) e = dmalloc(&m->loss, 1);
  if (e == cudaSuccess) e = dmalloc(&m->d_err, 1);
  // zero everything the padding relies on (padded weight columns, moments)
  if (e == cudaSuccess) e = cudaMemsetAsync(m->wb[0], 0, sizeof(__nv_bfloat16) * MLP_W * MLP_IN_PAD, m->stream);
  for (float* q : {m->p, m->g, m->m, m->v})
    if (e == cudaSuccess) e = cudaMemsetAsync(q, 0, sizeof(float) * P_COUNT, m->stream);
  if (e == cudaSuccess) e = cudaMemsetAsync(m->d_err, 0, sizeof(unsigned), m->stream);
  if (e == cudaSuccess) e = cudaStreamSynchronize(m->stream);
  if (e != cudaSuccess) {
    tp_mlp_destroy(m);
    return TP_ERR_CUDA;
  }
  *out = m;
  return TP_OK;
}

extern "C" void tp_mlp_destroy(tp_mlp* m) {
  if (!m) return;
  cudaSetDevice(m->device);
  if (m->stream) cudaStreamSynchronize(m->stream);
  for (void* q : {(void*)m->p, (void*)m->g, (void*)m->m, (void*)m->v, (void*)m->X, (void*)m->XT, (void*)m->H4,
                  (void*)m->y, (void*)m->t, (void*)m->dy, (void*)m->xin, (void*)m->split, (void*)m->lpart,
                  (void*)m->loss, (void*)m->d_err})
    cudaFree(q);
  for (int l = 0; l < 4; ++l) {
    cudaFree(m->wb[l]);
    cudaFree(m->wt[l]);
    cudaFree(m->Z[l]);
  }
  for (int l = 0; l < 3; ++l) {
    cudaFree(m->H[l]);
    cudaFree(m->HT[l]);
  }
  for (int i = 0; i < 2; ++i) {
    cudaFree(m->dZ[i]);
    cudaFree(m->dZT[i]);
  }
  if (m->stream) cudaStreamDestroy(m->stream);
  delete m;
}

extern "C" const char* tp_mlp_last_error(const tp_mlp* m) { return m ? m->err.c_str() : ""; }

extern "C" int tp_mlp_set_params(tp_mlp* m, const double* params) {
  if (!m || !params) return TP_ERR_ARG;
  cudaSetDevice(m->device);
  std::vector<float> f(P_COUNT);
  for (long i = 0; i < P_COUNT; ++i) f[i] = (float)params[i];
  cudaError_t e = cudaMemcpyAsync(m->p, f.data(), sizeof(float) * P_COUNT, cudaMemcpyHostToDevice, m->stream);
  for (float* q : {m->m, m->v})
    if (e == cudaSuccess) e = cudaMemsetAsync(q, 0, sizeof(float) * P_COUNT, m->stream);
  if (e == cudaSuccess) e = mlp_cast_all(m);
  if (e == cudaSuccess) e = cudaStreamSynchronize(m->stream);
  m->adam_t = 0;
  return mlp_cuda(m, e, "mlp set_params");
}

extern "C" int tp_mlp_get_params(tp_mlp* m, double* params) {
  if (!m || !params) return TP_ERR_ARG;
  cudaSetDevice(m->device);
  std::vector<float> f(P_COUNT);
  cudaError_t e = cudaMemcpyAsync(f.data(), m->p, sizeof(float) * P_COUNT, cudaMemcpyDeviceToHost, m->stream);
  if (e == cudaSuccess) e = cudaStreamSynchronize(m->stream);
  if (e != cudaSuccess) return mlp_cuda(m, e, "mlp get_params");
  for (long i = 0; i < P_COUNT; ++i) params[i] = f[i];
  return TP_OK;
}

// y[n] for features x[n][8] (host buffers), in batches of the capacity
extern "C" int tp_mlp_forward(tp_mlp* m, const double* x, long n, double* y) {
  if (!m || !x || !y || n < 0) return TP_ERR_ARG;
  cudaSetDevice(m->device);
  std::vector<float> yf;
  for (long s = 0; s < n; s += m->max_rows) {
    const long c = n - s < m->max_rows ? n - s : m->max_rows;
    const int rows = round_up(c, GEMM_BM);
    cudaError_t e = mlp_upload_x(m, x + s * MLP_IN, c, rows);
    if (e == cudaSuccess) e = mlp_forward_dev(m, rows, false);
    if (e != cudaSuccess) return mlp_cuda(m, e, "mlp forward");
    yf.resize(c);
    e = cudaMemcpyAsync(yf.data(), m->y, sizeof(float) * c, cudaMemcpyDeviceToHost, m->stream);
    if (e != cudaSuccess) return mlp_cuda(m, e, "mlp forward");
    const int st = mlp_check(m);
    if (st) return st;
    for (long i = 0; i < c; ++i) y[s + i] = yf[i];
  }
  return TP_OK;
}

// loss and gradients (flat FP64, the parameter layout) of the mean squared
// error on one batch, without an update
extern "C" int tp_mlp_gradients(tp_mlp* m, const double* x, const double* t, long n, double* grads, double* loss) {
  if (!m || !x || !t || n < 1 || n > m->max_rows) return TP_ERR_ARG;
  cudaSetDevice(m->device);
  const int rows = round_up(n, GEMM_BM);
  cudaError_t e = mlp_upload_x(m, x, n, rows);
  std::vector<float> tf(n);
  for (long i = 0; i < n; ++i) tf[i] = (float)t[i];
  if (e == cudaSuccess) e = cudaMemcpyAsync(m->t, tf.data(), sizeof(float) * n, cudaMemcpyHostToDevice, m->stream);
  if (e == cudaSuccess) e = mlp_forward_dev(m, rows, true);
  if (e == cudaSuccess) e = mlp_backward_dev(m, n, rows);
  std::vector<float> gf(P_COUNT);
  float lf = 0.f;
  if (e == cudaSuccess) e = cudaMemcpyAsync(gf.data(), m->g, sizeof(float) * P_COUNT, cudaMemcpyDeviceToHost, m->stream);
  if (e == cudaSuccess) e = cudaMemcpyAsync(&lf, m->loss, sizeof(float), cudaMemcpyDeviceToHost, m->stream);
  if (e != cudaSuccess) return mlp_cuda(m, e, "mlp gradients");
  const int st = mlp_check(m);
  if (st) return st;
  if (grads)
    for (long i = 0; i < P_COUNT; ++i) grads[i] = gf[i];
  if (loss) *loss = lf;
  return TP_OK;
}

// one Adam step on one batch given in device memory (x [n][8], t [n], FP32),
// asynchronous on the network's stream; *loss_dev receives the batch's loss
extern "C" int tp_mlp_train_step_device(tp_mlp* m, const float* x_dev, const float* t_dev, long n, float lr,
                                        float* loss_dev) {
  if (!m || !x_dev || !t_dev || n < 1 || n > m->max_rows) return TP_ERR_ARG;
  cudaSetDevice(m->device);
  const int rows = round_up(n, GEMM_BM);
  cudaError_t e = cudaMemcpyAsync(m->xin, x_dev, sizeof(float) * n * MLP_IN, cudaMemcpyDeviceToDevice, m->stream);
  if (e == cudaSuccess) e = cudaMemcpyAsync(m->t, t_dev, sizeof(float) * n, cudaMemcpyDeviceToDevice, m->stream);
  if (e == cudaSuccess) {
    e = mlp_pack(m, m->xin, n, rows);
  }
  if (e == cudaSuccess) e = mlp_forward_dev(m, rows, true);
  if (e == cudaSuccess) e = mlp_backward_dev(m, n, rows);
  if (e == cudaSuccess) e = mlp_adam_dev(m, lr);
  if (e == cudaSuccess && loss_dev)
    e = cudaMemcpyAsync(loss_dev, m->loss, sizeof(float), cudaMemcpyDeviceToDevice, m->stream);
  return mlp_cuda(m, e, "mlp train step");
}

// status of the asynchronous steps so far (synchronises the stream)
extern "C" int tp_mlp_set_wait_limit(tp_mlp* m, int iterations) {
  if (!m) return TP_ERR_ARG;
  m->spin = iterations < 0 ? MBAR_SPIN : iterations;
  return TP_OK;
}

extern "C" int tp_mlp_sync(tp_mlp* m) {
  if (!m) return TP_ERR_ARG;
  cudaSetDevice(m->device);
  return mlp_check(m);
}

extern "C" void* tp_mlp_stream(const tp_mlp* m) { return m ? (void*)m->stream : nullptr; }

// C = A B^T (BF16 operands with K contiguous, FP32 result, device pointers) on
// the network's stream: M % 128 == 0, N % 32 == 0 with 32 <= N <= 256,
// K % 64 == 0; the tensor-core GEMM every layer uses
extern "C" int tp_gemm_bf16_device(tp_mlp* m, const void* A, int lda, const void* B, int ldb, float* C, int ldc,
                                   int M, int N, int K) {
  if (!m || !A || !B || !C || lda % 8 || ldb % 8 || lda < K || ldb < K || ldc < N) return TP_ERR_ARG;
  if (((uintptr_t)A | (uintptr_t)B) % 16 || (uintptr_t)C % 4)
    return mlp_fail(m, TP_ERR_ARG, "gemm: A and B must be 16-byte aligned");  // copied in 16-byte pieces
  cudaSetDevice(m->device);
  GemmArgs g = gemm_args((const __nv_bfloat16*)A, lda, (const __nv_bfloat16*)B, ldb, M, N, K);
  g.flags = EPI_STORE_F32;
  g.out = C;
  g.ldo = ldc;
  cudaError_t e = gemm(m, g);
  if (e == cudaErrorInvalidValue) return mlp_fail(m, TP_ERR_ARG, "gemm: unsupported shape");
  if (e != cudaSuccess) return mlp_cuda(m, e, "gemm");
  return mlp_check(m);
}
