// Large-batch predict as ONE tensor-core kernel: the vote sums of every
// (sample, class) from the clauses' action bits and the samples' literal bits.
//
// For 0/1 operands the number of a clause's included literals that a sample
// satisfies is the dot product of their bit rows, so its failed-literal count
// is F = L - a.x with L the clause's literal count (capi.c:97-122).  0 and 1
// are exact in 4-bit floats (e2m1) and every partial sum is an integer below
// 2^24, exact in fp32, so the products run on the block-scaled 4-bit kind of
// tcgen05.mma (all scales 1), at twice the rate of 8-bit operands and half
// their bytes.
//
// k_votes: clusters of two CTAs, persistent over tiles of 256 samples x 240
// clauses.  Each CTA holds 128 of the tile's samples and 120 of its clauses;
// the leader issues cta_group::2 MMAs over both (each SM reads each operand
// byte once per pair: the L2 traffic of a 256 x 256 tile, without multicast).
//   warp 0     TMA producer: 128-byte (256-literal) steps through a ring of
//              6 stages, 128-byte swizzle, both CTAs' copies counted on the
//              leader's barrier
//   warp 1     (leader) four MMAs of K = 64 per step; commits free the stage in
//              both CTAs
//   warp 2     TMEM: 2 x 240 accumulator columns (a tile's epilogue runs
//              under the next tile's products) and 32 columns of scale factors
//   warps 4-7  epilogue: a thread per sample walks the tile's columns, forms
//              the votes max(0, min(L, tol) - F), or tol for an empty clause,
//              signed by clause parity (capi.c:110-118, 148-161), and adds its
//              class sums; products never leave the SM
// Every wait is bounded; one that runs out sets *err and ends the kernel.
#include <cuda.h>
#include <cuda_runtime.h>
#include <stdint.h>

#include <algorithm>
#include <atomic>

#include "tm_device.cuh"

namespace tmb {

namespace {

constexpr uint32_t VT_M = 256, VT_N = 240;         // samples, clauses per pair of CTAs
constexpr uint32_t VT_KB = 128;                    // bytes of a row per stage
constexpr uint32_t VT_STAGES = 6;
constexpr uint32_t VT_A = VT_M / 2 * VT_KB, VT_B = VT_N / 2 * VT_KB;
constexpr uint32_t VT_STAGE = VT_A + VT_B;
constexpr uint32_t VT_SF = 2 * VT_N;               // TMEM column of the scale factors
constexpr uint32_t VT_SMEM = VT_STAGES * VT_STAGE + 1024 + 4096;
constexpr uint32_t VT_GROUP = 8;                   // sample tiles walked per clause tile

__device__ __forceinline__ uint32_t cluster_rank() {
  uint32_t r;
  asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
  return r;
}
__device__ __forceinline__ uint32_t cluster_id() {
  uint32_t r;
  asm volatile("mov.u32 %0, %%clusterid.x;" : "=r"(r));
  return r;
}
__device__ __forceinline__ uint32_t cluster_count() {
  uint32_t r;
  asm volatile("mov.u32 %0, %%nclusterid.x;" : "=r"(r));
  return r;
}
__device__ __forceinline__ void cluster_sync() {
  asm volatile("barrier.cluster.arrive.release.aligned;\n barrier.cluster.wait.acquire.aligned;" ::
                   : "memory");
}
// shared-memory address of the same variable in CTA `rank` of the cluster
__device__ __forceinline__ uint32_t map_rank(uint32_t addr, uint32_t rank) {
  uint32_t r;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(addr), "r"(rank));
  return r;
}
__device__ __forceinline__ void arrive_cluster(uint32_t addr) {
  asm volatile("mbarrier.arrive.release.cluster.shared::cluster.b64 _, [%0];" ::"r"(addr) : "memory");
}
__device__ __forceinline__ void expect_tx(uint64_t *bar, uint32_t bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_u32(bar)),
               "r"(bytes)
               : "memory");
}
// bounded wait at cluster scope (the other CTA's arrivals and copies count)
__device__ __forceinline__ bool wait_cluster(uint64_t *bar, uint32_t parity) {
  const uint32_t a = smem_u32(bar);
  for (uint32_t it = 0; it < TM_WAIT_LIMIT; it++) {
    uint32_t done;
    asm volatile(
        "{\n .reg .pred p;\n"
        " mbarrier.try_wait.parity.acquire.cluster.shared::cta.b64 p, [%1], %2;\n"
        " selp.u32 %0, 1, 0, p;\n}\n"
        : "=r"(done)
        : "r"(a), "r"(parity)
        : "memory");
    if (done) return true;
  }
  return false;
}
// one tile of a 2-D byte tensor into this CTA's shared memory, counted on a
// barrier of the leader CTA
__device__ __forceinline__ void tma_tile(const CUtensorMap *map, uint32_t dst, uint32_t bar,
                                         int32_t x, int32_t y) {
  asm volatile(
      "cp.async.bulk.tensor.2d.shared::cluster.global.tile.mbarrier::complete_tx::bytes."
      "cta_group::2 [%0], [%1, {%3, %4}], [%2];" ::"r"(dst),
      "l"(map), "r"(bar), "r"(x), "r"(y)
      : "memory");
}
// K-major operand, rows of 128 bytes, 128-byte swizzle: 1,024 bytes from one
// group of eight rows to the next
__device__ __forceinline__ uint64_t operand_desc(uint32_t addr) {
  return (uint64_t)((addr & 0x3FFFFu) >> 4) | (uint64_t)1 << 16 | (uint64_t)(1024 >> 4) << 32 |
         (uint64_t)1 << 46 | (uint64_t)2 << 61;
}
// e2m1 x e2m1 -> f32, M = 256, N = 240, UE8M0 scales, both operands K-major
constexpr uint32_t VT_IDESC = 1u << 7 | 1u << 10 | (VT_N >> 3) << 17 | 1u << 23 | (VT_M >> 4) << 24;

__device__ __forceinline__ void mma_fp4(uint32_t d, uint64_t a, uint64_t b, uint32_t sf, bool acc) {
  asm volatile(
      "{\n .reg .pred p;\n setp.ne.u32 p, %5, 0;\n"
      " tcgen05.mma.cta_group::2.kind::mxf4.block_scale.scale_vec::2X [%0], %1, %2, %3, [%4], [%6], p;\n}"
      ::"r"(d), "l"(a), "l"(b), "r"(VT_IDESC), "r"(sf), "r"((uint32_t)acc), "r"(sf + 16)
      : "memory");
}
// the MMAs issued so far, when done, arrive on this barrier of both CTAs
__device__ __forceinline__ void commit_both(uint64_t *bar) {
  asm volatile(
      "tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.multicast::cluster.b64 "
      "[%0], %1;" ::"r"(smem_u32(bar)),
      "h"((uint16_t)3)
      : "memory");
}
__device__ __forceinline__ void tmem_ld8(uint32_t addr, uint32_t (&v)[8]) {
  asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
               : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]),
                 "=r"(v[6]), "=r"(v[7])
               : "r"(addr));
}

struct VotesTiles {
  uint32_t samples, rows;   // samples, clause rows (classes x clauses)
  uint32_t st, ct;          // tiles of samples, of clause rows
  uint32_t steps;           // K steps
};

// tile t: groups of VT_GROUP sample tiles, in a group clause tile by clause
// tile, so that the tiles running at once share their rows in L2
__device__ __forceinline__ void tile_at(const VotesTiles &T, uint32_t t, uint32_t &s, uint32_t &c) {
  const uint32_t per = VT_GROUP * T.ct, gr = t / per, in = t - gr * per;
  const uint32_t w = T.st - gr * VT_GROUP < VT_GROUP ? T.st - gr * VT_GROUP : VT_GROUP;
  c = in / w;
  s = gr * VT_GROUP + in - c * w;
}

__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(256, 1)
    k_votes(const __grid_constant__ CUtensorMap xmap, const __grid_constant__ CUtensorMap amap,
            const VotesTiles T, const int32_t *__restrict__ lits, uint32_t clauses,
            uint32_t classes, uint32_t tol, int32_t *__restrict__ sums,
            const uint32_t *__restrict__ gate, uint32_t *__restrict__ err) {
  if (gate && *gate == 0) return;  // a search machine that stopped training (both CTAs alike)
  extern __shared__ uint8_t raw[];
  uint8_t *buf = (uint8_t *)(((uintptr_t)raw + 1023) & ~(uintptr_t)1023);
  uint8_t *tail = buf + VT_STAGES * VT_STAGE;
  uint64_t *full = (uint64_t *)tail, *empty = full + VT_STAGES;
  uint64_t *acc_full = empty + VT_STAGES, *acc_empty = acc_full + 2;
  uint32_t *tmem_at = (uint32_t *)(acc_empty + 2), *bad = tmem_at + 1, *stop = bad + 1;
  float *dtab = (float *)(tail + 256);  // [2][VT_N]: L - min(L, tol), -tol for an empty clause
  const uint32_t tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const uint32_t rank = cluster_rank();
  if (tid == 0) {
    for (uint32_t i = 0; i < VT_STAGES; i++) {
      mbar_init(&full[i], 1);
      mbar_init(&empty[i], 1);
    }
    for (uint32_t i = 0; i < 2; i++) {
      mbar_init(&acc_full[i], 1);
      mbar_init(&acc_empty[i], 8);  // four epilogue warps of each CTA
    }
    mbar_fence_init();
    *bad = 0;
    *stop = 0;
  }
  if (warp == 2) {
    asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], 512;" ::"r"(
                     smem_u32(tmem_at))
                 : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;");
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  cluster_sync();
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
  const uint32_t tmem = *tmem_at;
  if (warp >= 4) {
    // scale factors: 1.0 (exponent 127) in every byte of the 32 columns
    const uint32_t one = 0x7F7F7F7Fu, at = tmem + ((warp - 4) * 32u << 16) + VT_SF;
#pragma unroll
    for (uint32_t c = 0; c < 32; c += 8)
      asm volatile("tcgen05.st.sync.aligned.32x32b.x8.b32 [%0], {%1, %1, %1, %1, %1, %1, %1, %1};" ::"r"(
                       at + c),
                   "r"(one)
                   : "memory");
    asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  cluster_sync();
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
  const uint32_t tiles = T.st * T.ct, first = cluster_id(), stride = cluster_count();

  if (warp == 0) {
    if (lane == 0) {
      uint32_t k = 0;  // steps issued
      bool ok = true;
      for (uint32_t t = first; t < tiles && ok; t += stride) {
        uint32_t s, c;
        tile_at(T, t, s, c);
        const int32_t xr = (int32_t)(s * VT_M + rank * (VT_M / 2));
        const int32_t ar = (int32_t)(c * VT_N + rank * (VT_N / 2));
        for (uint32_t i = 0; i < T.steps; i++, k++) {
          const uint32_t sl = k % VT_STAGES, ph = (k / VT_STAGES) & 1u;
          if (k >= VT_STAGES && !wait_cluster(&empty[sl], ph ^ 1u)) {
            ok = false;
            break;
          }
          const uint32_t bar = map_rank(smem_u32(&full[sl]), 0);
          if (rank == 0) expect_tx(&full[sl], 2 * VT_STAGE);
          const uint32_t dst = smem_u32(buf + sl * VT_STAGE);
          tma_tile(&xmap, dst, bar, (int32_t)(i * VT_KB), xr);
          tma_tile(&amap, dst + VT_A, bar, (int32_t)(i * VT_KB), ar);
        }
      }
      if (!ok) *bad = 1;
      // this CTA's copies in flight, before it leaves: the stages still full
      // are freed by the leader's last commits
      const uint32_t last = k < VT_STAGES ? k : VT_STAGES;
      for (uint32_t q = 0; ok && q < last; q++) {
        const uint32_t kk = k - last + q;
        if (!wait_cluster(&empty[kk % VT_STAGES], (kk / VT_STAGES) & 1u)) {
          *bad = 1;
          break;
        }
      }
    }
  } else if (warp == 1 && rank == 0) {
    if (lane == 0) {
      uint32_t k = 0, it = 0;
      bool ok = true;
      for (uint32_t t = first; t < tiles && ok; t += stride, it++) {
        const uint32_t b = it & 1u, ph = (it >> 1) & 1u;
        if (it >= 2 && !wait_cluster(&acc_empty[b], ph ^ 1u)) {
          ok = false;
          break;
        }
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        for (uint32_t i = 0; i < T.steps; i++, k++) {
          const uint32_t sl = k % VT_STAGES;
          if (!wait_cluster(&full[sl], (k / VT_STAGES) & 1u)) {
            ok = false;
            break;
          }
          asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
          const uint32_t at = smem_u32(buf + sl * VT_STAGE);
          const uint64_t da = operand_desc(at), db = operand_desc(at + VT_A);
#pragma unroll
          for (uint32_t q = 0; q < 4; q++)  // 64 literals = 32 bytes each
            mma_fp4(tmem + b * VT_N, da + 2 * q, db + 2 * q, tmem + VT_SF, i > 0 || q > 0);
          commit_both(&empty[sl]);
        }
        if (ok) commit_both(&acc_full[b]);
      }
      if (!ok) *bad = 1;
    }
  } else if (warp >= 4) {
    const uint32_t q = warp - 4, row = q * 32 + lane;  // this thread's sample of the CTA
    uint32_t it = 0;
    bool dead = false;  // a wait ran out: no more waits, tables or outputs
    for (uint32_t t = first; t < tiles && !dead; t += stride, it++) {
      uint32_t s, c;
      tile_at(T, t, s, c);
      const uint32_t b = it & 1u, ph = (it >> 1) & 1u;
      const uint32_t r0 = c * VT_N;
      // the other half of the epilogue's threads is done with this buffer of
      // the table: they passed the barrier below of the tile in between
      float *d = dtab + b * VT_N;
      for (uint32_t i = row; i < VT_N; i += 128) {
        float v = 0.0f;
        if (r0 + i < T.rows) {
          const int32_t L = lits[r0 + i];
          v = L == 0 ? -(float)tol : (float)(L - (L < (int32_t)tol ? L : (int32_t)tol));
        }
        d[i] = v;
      }
      // one wait, shared by the four warps, so that they go on (or stop) together
      if (row == 0 && !wait_cluster(&acc_full[b], ph)) *stop = *bad = 1;
      asm volatile("bar.sync 1, 128;" ::: "memory");
      dead = *(volatile uint32_t *)stop != 0;  // written by row 0 alone, between these barriers
      asm volatile("bar.sync 1, 128;" ::: "memory");
      if (dead) break;
      wait_cluster(&acc_full[b], ph);  // done: the acquire of this thread
      asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
      const uint32_t sample = s * VT_M + rank * (VT_M / 2) + row;
      const bool mine = sample < T.samples;
      const uint32_t at = tmem + (q * 32u << 16) + b * VT_N;
      uint32_t h = r0 / clauses, left = clauses - (r0 - h * clauses);  // class, rows left of it
      float acc = 0.0f;
      for (uint32_t col = 0; col < VT_N; col += 8) {
        uint32_t v[8];
        tmem_ld8(at + col, v);
        const float4 d0 = *(const float4 *)(d + col), d1 = *(const float4 *)(d + col + 4);
        // (the values pass through the wait, so that none is used before it)
        asm volatile("tcgen05.wait::ld.sync.aligned;"
                     : "+r"(v[0]), "+r"(v[1]), "+r"(v[2]), "+r"(v[3]), "+r"(v[4]), "+r"(v[5]),
                       "+r"(v[6]), "+r"(v[7])::"memory");
        const float dd[8] = {d0.x, d0.y, d0.z, d0.w, d1.x, d1.y, d1.z, d1.w};
#pragma unroll
        for (int i = 0; i < 8; i += 2) {
          acc += fmaxf(__uint_as_float(v[i]) - dd[i], 0.0f);
          acc -= fmaxf(__uint_as_float(v[i + 1]) - dd[i + 1], 0.0f);
        }
        left -= 8;  // classes have a multiple of 8 clauses
        if (left == 0 || col + 8 == VT_N) {
          if (mine && acc != 0.0f) atomicAdd(&sums[(uint64_t)sample * classes + h], __float2int_rn(acc));
          acc = 0.0f;
          h++;
          left = clauses;
          if (r0 + col + 8 >= T.rows) break;
        }
      }
      asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
      __syncwarp();
      if (lane == 0) arrive_cluster(map_rank(smem_u32(&acc_empty[b]), 0));
    }
  }
  __syncwarp();
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  if (tid == 0 && *bad) atomicExch(err, 1u);
  // neither CTA leaves, nor frees TMEM, while the other still uses the pair's
  cluster_sync();
  if (warp == 2)
    asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, 512;" ::"r"(tmem));
}

// 8 bits -> 8 four-bit floats: bit i to 1.0 (code 2) or 0 in nibble i
__device__ __forceinline__ uint32_t spread8(uint32_t b) {
  b = (b | b << 12) & 0x000F000Fu;
  b = (b | b << 6) & 0x03030303u;
  return ((b | b << 3) & 0x11111111u) << 1;
}

// rows x W words (stride `stride` words) -> rows x 16 W bytes of 4-bit
// floats; the last word of a row is ANDed with `last_mask`.  Bound by HBM: a
// word in, 16 bytes out.
__global__ void k_expand_fp4(const uint32_t *__restrict__ src, uint64_t rows, uint32_t stride,
                             uint32_t W, uint32_t last_mask, uint8_t *__restrict__ dst) {
  const uint64_t total = rows * W;
  for (uint64_t t = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; t < total;
       t += (uint64_t)gridDim.x * blockDim.x) {
    const uint64_t r = t / W;
    const uint32_t w = (uint32_t)(t - r * W);
    uint32_t v = src[r * stride + w];
    if (w == W - 1) v &= last_mask;
    ((uint4 *)dst)[t] = make_uint4(spread8(v & 0xFFu), spread8((v >> 8) & 0xFFu),
                                   spread8((v >> 16) & 0xFFu), spread8(v >> 24));
  }
}

// The same from byte rows of any alignment (the reference's sample layout);
// `zero` is cleared in the same launch (the vote sums of the predict).  Bits
// past a row's bytes are zero.
__global__ void k_expand_fp4_bytes(const uint8_t *__restrict__ src, uint64_t rows,
                                   uint32_t row_bytes, uint32_t W, uint8_t *__restrict__ dst,
                                   uint32_t *__restrict__ zero, uint64_t zero_words) {
  const uint64_t t0 = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
  const uint64_t step = (uint64_t)gridDim.x * blockDim.x;
  for (uint64_t t = t0; t < zero_words; t += step) zero[t] = 0;
  const uint64_t total = rows * W;
  const bool words = ((row_bytes | (uint32_t)(uintptr_t)src) & 3) == 0;
  for (uint64_t t = t0; t < total; t += step) {
    const uint64_t r = t / W;
    const uint32_t w = (uint32_t)(t - r * W);
    const uint8_t *p = src + r * row_bytes + 4 * w;
    uint32_t v = 0;
    if (words) {
      v = *(const uint32_t *)p;
    } else {
#pragma unroll
      for (uint32_t b = 0; b < 4; b++)
        if (4 * w + b < row_bytes) v |= (uint32_t)p[b] << (8 * b);
    }
    ((uint4 *)dst)[t] = make_uint4(spread8(v & 0xFFu), spread8((v >> 8) & 0xFFu),
                                   spread8((v >> 16) & 0xFFu), spread8(v >> 24));
  }
}

typedef CUresult (*EncodeFn)(CUtensorMap *, CUtensorMapDataType, cuuint32_t, void *,
                             const cuuint64_t *, const cuuint64_t *, const cuuint32_t *,
                             const cuuint32_t *, CUtensorMapInterleave, CUtensorMapSwizzle,
                             CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

EncodeFn encode_fn() {
  static std::atomic<void *> fn{nullptr};
  void *p = fn.load();
  if (!p) {
    cudaDriverEntryPointQueryResult q;
    if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &p, cudaEnableDefault, &q) != cudaSuccess ||
        q != cudaDriverEntryPointSuccess)
      return nullptr;
    fn.store(p);
  }
  return (EncodeFn)p;
}

// rows of `bytes` bytes, boxes of VT_KB bytes x `box` rows; reads past either
// end give zeros
bool encode_rows(CUtensorMap *map, const void *base, uint64_t rows, uint64_t bytes, uint32_t box) {
  EncodeFn fn = encode_fn();
  if (!fn) return false;
  const cuuint64_t dims[2] = {bytes, rows}, strides[1] = {bytes};
  const cuuint32_t boxes[2] = {VT_KB, box}, steps[2] = {1, 1};
  return fn(map, CU_TENSOR_MAP_DATA_TYPE_UINT8, 2, (void *)base, dims, strides, boxes, steps,
            CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B,
            CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

}  // namespace

cudaError_t launch_expand_fp4(const uint32_t *src, uint64_t rows, uint32_t stride, uint32_t W,
                              uint32_t last_mask, uint8_t *dst, cudaStream_t st) {
  if (!rows || !W) return cudaSuccess;
  const uint64_t b = (rows * W + 255) / 256;
  k_expand_fp4<<<(unsigned)(b < 148 * 16 ? b : 148 * 16), 256, 0, st>>>(src, rows, stride, W,
                                                                        last_mask, dst);
  return cudaGetLastError();
}

cudaError_t launch_expand_fp4_bytes(const uint8_t *src, uint64_t rows, uint32_t row_bytes,
                                    uint32_t W, uint8_t *dst, uint32_t *zero, uint64_t zero_words,
                                    cudaStream_t st) {
  const uint64_t work = rows * W > zero_words ? rows * W : zero_words;
  if (!work) return cudaSuccess;
  const uint64_t b = (work + 255) / 256;
  k_expand_fp4_bytes<<<(unsigned)(b < 148 * 16 ? b : 148 * 16), 256, 0, st>>>(
      src, rows, row_bytes, W, dst, zero, zero_words);
  return cudaGetLastError();
}

cudaError_t launch_votes(int dev, int sms, const uint8_t *act4, const uint8_t *x4, uint32_t classes,
                         uint32_t clauses, uint32_t W, uint32_t tol, const int32_t *lits, uint32_t n,
                         int32_t *sums, const uint32_t *gate, uint32_t *err, cudaStream_t st) {
  const uint64_t rows = (uint64_t)classes * clauses, bytes = 16ull * W;
  static std::atomic<uint64_t> ready{0};  // devices whose shared-memory limit is raised
  if (!(ready.load() >> (dev & 63) & 1u)) {
    const cudaError_t e =
        cudaFuncSetAttribute(k_votes, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)VT_SMEM);
    if (e != cudaSuccess) return e;
    ready.fetch_or(1ull << (dev & 63));
  }
  const uint32_t span = tmb_votes_span(rows);
  for (uint64_t s0 = 0; s0 < n; s0 += span) {
    CUtensorMap xmap, amap;
    VotesTiles T;
    T.samples = (uint32_t)std::min<uint64_t>(span, n - s0);
    if (!encode_rows(&xmap, x4 + s0 * bytes, T.samples, bytes, VT_M / 2) ||
        !encode_rows(&amap, act4, rows, bytes, VT_N / 2))
      return cudaErrorInvalidValue;
    T.rows = (uint32_t)rows;
    T.st = (uint32_t)(((uint64_t)T.samples + VT_M - 1) / VT_M);
    T.ct = (uint32_t)((rows + VT_N - 1) / VT_N);
    T.steps = (uint32_t)((bytes + VT_KB - 1) / VT_KB);
    const uint64_t tiles = (uint64_t)T.st * T.ct;
    const uint64_t pairs = (uint64_t)sms / 2 < tiles ? (uint64_t)sms / 2 : tiles;
    k_votes<<<(unsigned)(2 * pairs), 256, VT_SMEM, st>>>(xmap, amap, T, lits, clauses, classes, tol,
                                                         sums + s0 * classes, gate, err);
    const cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) return e;
  }
  return cudaSuccess;
}

}  // namespace tmb

// Samples per launch against `rows` clause rows: all of them, unless the launch
// counts 2^31 tiles and more (the kernel's tile numbers, and their last step
// past the end, have 32 bits); then whole tiles, at least one.
uint32_t tmb_votes_span(uint64_t rows) {
  const uint64_t ct = (rows + tmb::VT_N - 1) / tmb::VT_N, most = ((1ull << 31) - 1) / (ct ? ct : 1);
  const uint64_t span = (most ? most : 1) * tmb::VT_M;
  return span < (1ull << 31) ? (uint32_t)span : 1u << 31;
}
