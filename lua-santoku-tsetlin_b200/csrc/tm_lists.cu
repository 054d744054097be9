// Large dense predicts of machines whose clauses hold few literals (capi.c:85-133,
// 907-999): bit-sliced over the samples.
//
// A clause row of 8,192 literals holds about a hundred, and every product of the
// tensor-core kernel with the others is a multiplication by zero.  Here each
// clause is a list of its literals, and a literal of 32 samples is one word:
//
//   k_list_plan     per group of 32 clauses the longest list, its place in the
//                   lists, and the most a counter has to hold
//   k_list_fill     action rows -> lists (once per state of the automata)
//   k_slice_bytes   byte rows -> failing literals, [tile][literal][TW words]
//   k_list_votes    a CTA holds one tile of samples in shared memory; a lane
//                   takes one clause of a group, adds the words of its literals
//                   in bit-sliced counters (16 literals per carry), subtracts
//                   them from the clause's literal count and adds the votes in
//                   bit-sliced sums, which are formed into numbers once per class
//
// Bound by LOP3 (62 % of the ALU pipe: 30 per 16 literals and sample word, 45
// per clause) and the shared-memory reads beside it (a literal is one read of
// 4 TW bytes per lane, rows in random banks).  Tiles of TW x 32 samples, as
// wide as shared memory allows: a wide read spends fewer clocks and fewer
// address instructions per byte.  Predicts of 20,000 samples, tensor-core
// kernel -> lists: 256 x 1,024 clauses of 8,192 literals, 32 of them included
// 12.4 -> 2.5 ms (2-word tiles 2.8), 110 included 12.4 -> 6.6 ms; 20 x 2,048
// clauses of 32,768 literals, 32 included 7.5 -> 0.70 ms, 110 included 7.5 ->
// 1.66 ms.
#include <algorithm>
#include <atomic>

#include "tm_device.cuh"

namespace tmb {

namespace {

__device__ __forceinline__ void copy16(void *dst, const void *src) {
  const uint32_t d = (uint32_t)__cvta_generic_to_shared(dst);
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(d), "l"(src) : "memory");
}
__device__ __forceinline__ void copies_done() {
  asm volatile("cp.async.wait_all;" ::: "memory");
}

constexpr int SL_ACC = 12;     // planes of the vote sums kept between flushes
// threads of k_list_votes: as many warps as its registers (166, 114 and 80 a
// thread) leave room for (one-word tiles with 384 threads 0.86 ms, 768 0.70)
__host__ __device__ constexpr int list_threads(int tw) { return tw == 4 ? 384 : (tw == 2 ? 512 : 768); }
constexpr uint32_t SL_SMEM = 224 * 1024;

__device__ __forceinline__ uint32_t x3(uint32_t a, uint32_t b, uint32_t c) { return a ^ b ^ c; }
__device__ __forceinline__ uint32_t m3(uint32_t a, uint32_t b, uint32_t c) {
  return (a & b) | (c & (a | b));
}

// a lane's clause c of class h: its literal count, and the most it votes
__device__ __forceinline__ uint32_t list_count(const int32_t *lits, uint32_t h, uint32_t c,
                                               uint32_t clauses) {
  return c < clauses ? (uint32_t)lits[(uint64_t)h * clauses + c] : 0;
}
__device__ __forceinline__ uint32_t list_cap(uint32_t L, uint32_t c, uint32_t clauses,
                                             uint32_t tol) {
  return c < clauses ? (L == 0 || L > tol ? tol : L) : 0;
}

// A warp per group: groups[g] = {first block of 16 literals, blocks | need <<
// 16}, need the largest literal count or vote (65,535: that or more).
// tot[0] counts blocks, tot[1] is the largest need.
__global__ void k_list_plan(const int32_t *__restrict__ lits, uint32_t classes, uint32_t clauses,
                            uint32_t gpc, uint32_t tol, uint2 *__restrict__ groups,
                            uint32_t *__restrict__ tot) {
  const uint32_t lane = threadIdx.x & 31;
  const uint64_t ng = (uint64_t)classes * gpc;
  for (uint64_t g = ((uint64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5; g < ng;
       g += ((uint64_t)gridDim.x * blockDim.x) >> 5) {
    const uint32_t h = (uint32_t)(g / gpc), j = (uint32_t)(g - (uint64_t)h * gpc);
    const uint32_t L = list_count(lits, h, j * 32 + lane, clauses);
    const uint32_t mx = __reduce_max_sync(0xFFFFFFFFu, L);
    const uint32_t mc = __reduce_max_sync(0xFFFFFFFFu, list_cap(L, j * 32 + lane, clauses, tol));
    if (lane == 0) {
      const uint32_t blocks = (mx + 15) / 16, need = mx > mc ? mx : mc;
      const uint32_t off = atomicAdd(&tot[0], blocks);
      atomicMax(&tot[1], need);
      groups[g] = make_uint2(off, (blocks & 0xFFFFu) | (need < 0xFFFFu ? need : 0xFFFFu) << 16);
    }
  }
}

// A warp per clause slot (32 per group): the numbers of the row's literals into
// the lane's places of the group's blocks, the rest filled with `pad`, the
// tile row in which nothing fails.  Block b: two halves of 32 lanes x 8 numbers.
__global__ void k_list_fill(const uint32_t *__restrict__ act, uint32_t classes, uint32_t clauses,
                            uint32_t gpc, uint32_t Wp, uint32_t W, uint32_t last_mask,
                            const uint2 *__restrict__ groups, uint32_t pad,
                            uint16_t *__restrict__ lists) {
  const uint32_t lane = threadIdx.x & 31;
  const uint64_t total = (uint64_t)classes * gpc * 32;
  for (uint64_t i = ((uint64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5; i < total;
       i += ((uint64_t)gridDim.x * blockDim.x) >> 5) {
    const uint64_t g = i >> 5;
    const uint32_t slot = (uint32_t)i & 31u;
    const uint32_t h = (uint32_t)(g / gpc), c = (uint32_t)(g - (uint64_t)h * gpc) * 32 + slot;
    const uint2 gi = groups[g];
    const uint32_t room = (gi.y & 0xFFFFu) * 16;
    uint16_t *dst = lists + ((uint64_t)gi.x * 64 + slot) * 8;
    auto put = [&](uint32_t p, uint32_t v) {
      if (p < room) dst[(uint64_t)(p >> 3) * 256 + (p & 7)] = (uint16_t)v;
    };
    uint32_t pos = 0;
    if (c < clauses) {
      const uint4 *row = (const uint4 *)(act + ((uint64_t)h * clauses + c) * Wp);
      for (uint32_t w0 = 0; w0 < W; w0 += 128) {
        const uint32_t w = w0 + 4 * lane;
        uint4 q = make_uint4(0, 0, 0, 0);
        if (w < Wp) q = row[w >> 2];
        uint32_t a[4] = {q.x, q.y, q.z, q.w};
        uint32_t cnt = 0;
#pragma unroll
        for (int k = 0; k < 4; k++) {
          if (w + k >= W) a[k] = 0;
          else if (w + k + 1 == W) a[k] &= last_mask;
          cnt += __popc(a[k]);
        }
        uint32_t inc = cnt;
#pragma unroll
        for (int d = 1; d < 32; d <<= 1) {
          const uint32_t t = __shfl_up_sync(0xFFFFFFFFu, inc, d);
          if (lane >= (uint32_t)d) inc += t;
        }
        uint32_t p = pos + inc - cnt;
#pragma unroll
        for (int k = 0; k < 4; k++)
          for (uint32_t v = a[k]; v; v &= v - 1) put(p++, 32 * (w + k) + __ffs(v) - 1);
        pos += __shfl_sync(0xFFFFFFFFu, inc, 31);
      }
    }
    for (uint32_t p = pos + lane; p < room; p += 32) put(p, pad);
  }
}

// Byte rows -> tiles.  A CTA turns 32 words of a tile's TW x 32 samples: lane
// j of a warp ends up with literal 32 w + j of 32 samples (a bit transpose in
// five exchanges).  Row 32 W of a tile is all zeros.  The launch also clears
// `zero` (vote sums).
template <int TW>
__global__ void __launch_bounds__(256)
    k_slice_bytes(const uint8_t *__restrict__ src, uint32_t n, uint32_t row_bytes, uint32_t W,
                  uint32_t Kp, uint32_t *__restrict__ dst, uint32_t *__restrict__ zero,
                  uint64_t zero_words) {
  __shared__ uint32_t sm[TW * 32][33];
  const uint32_t lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const uint32_t w0 = blockIdx.x * 32, tile = blockIdx.y;
  const uint64_t cta = (uint64_t)blockIdx.y * gridDim.x + blockIdx.x;
  for (uint64_t i = cta * 256 + threadIdx.x; i < zero_words;
       i += (uint64_t)gridDim.x * gridDim.y * 256)
    zero[i] = 0;
  const bool words = ((row_bytes | (uint32_t)(uintptr_t)src) & 3) == 0;
  for (uint32_t r = warp; r < TW * 32; r += 8) {
    const uint32_t s = tile * (TW * 32) + r, w = w0 + lane;
    uint32_t v = 0xFFFFFFFFu;
    if (s < n && w < W) {
      const uint8_t *row = src + (uint64_t)s * row_bytes;
      if (words) {
        v = ((const uint32_t *)row)[w];
      } else {
        v = 0;
#pragma unroll
        for (uint32_t b = 0; b < 4; b++)
          if (4 * w + b < row_bytes) v |= (uint32_t)row[4 * w + b] << (8 * b);
      }
    }
    sm[r][lane] = ~v;
  }
  __syncthreads();
  uint32_t *out = dst + (uint64_t)tile * Kp * TW;
  for (uint32_t k = warp; k < 32 && w0 + k < W; k += 8) {
    uint32_t v[TW];
#pragma unroll
    for (int t = 0; t < TW; t++) {
      uint32_t x = sm[t * 32 + lane][k], m = 0x0000FFFFu;
#pragma unroll
      for (int j = 16; j; j >>= 1) {
        const uint32_t y = __shfl_xor_sync(0xFFFFFFFFu, x, j);
        x = (lane & j) ? (x & ~m) | ((y >> j) & m) : (x & m) | ((y << j) & ~m);
        m ^= m << (j >> 1);
      }
      v[t] = x;
    }
    uint32_t *p = out + (uint64_t)((w0 + k) * 32 + lane) * TW;
    if (TW == 4) *(uint4 *)p = make_uint4(v[0], v[TW > 1 ? 1 : 0], v[TW > 2 ? 2 : 0], v[TW - 1]);
    else if (TW == 2) *(uint2 *)p = make_uint2(v[0], v[TW - 1]);
    else *p = v[0];
  }
  if (blockIdx.x == 0)
    for (uint32_t i = threadIdx.x; i < (Kp - 32 * W) * TW; i += 256)
      out[(uint64_t)32 * W * TW + i] = 0;
}

template <int TW>
struct Words {
  uint32_t w[TW];
};
template <int TW>
__device__ __forceinline__ Words<TW> tile_row(const uint32_t *xs, uint32_t i) {
  Words<TW> r;
  if constexpr (TW == 4) {
    const uint4 v = *(const uint4 *)(xs + 4 * i);
    r.w[0] = v.x, r.w[1] = v.y, r.w[2] = v.z, r.w[3] = v.w;
  } else if constexpr (TW == 2) {
    const uint2 v = *(const uint2 *)(xs + 2 * i);
    r.w[0] = v.x, r.w[1] = v.y;
  } else {
    r.w[0] = xs[i];
  }
  return r;
}
// a += b + c bit by bit; returns the carries
template <int TW>
__device__ __forceinline__ Words<TW> full_add(Words<TW> &a, const Words<TW> &b,
                                              const Words<TW> &c) {
  Words<TW> r;
#pragma unroll
  for (int t = 0; t < TW; t++) {
    r.w[t] = m3(a.w[t], b.w[t], c.w[t]);
    a.w[t] = x3(a.w[t], b.w[t], c.w[t]);
  }
  return r;
}

// The votes of one clause per lane, added to acc: P counter planes (literal
// counts and votes below 2^P).  n0, n1: the first block of the group's lists
// at lp, on return the one at `next`.
template <int TW, int P>
__device__ __forceinline__ void list_group(const uint32_t *xs, const uint4 *lp, const uint4 *next,
                                           uint4 &n0, uint4 &n1, uint32_t blocks, uint32_t cap,
                                           Words<TW> (&acc)[SL_ACC]) {
  Words<TW> f[P];
#pragma unroll
  for (int b = 0; b < P; b++)
#pragma unroll
    for (int t = 0; t < TW; t++) f[b].w[t] = 0;
  // eight literals into f[0..2]; returns the carries of weight 8
  auto eight = [&](const uint4 &q) {
    const uint32_t i[4] = {q.x, q.y, q.z, q.w};
    Words<TW> v[8];
#pragma unroll
    for (int k = 0; k < 4; k++) {
      v[2 * k] = tile_row<TW>(xs, i[k] & 0xFFFFu);
      v[2 * k + 1] = tile_row<TW>(xs, i[k] >> 16);
    }
    const Words<TW> a2 = full_add(f[0], v[0], v[1]), b2 = full_add(f[0], v[2], v[3]);
    const Words<TW> a4 = full_add(f[1], a2, b2);
    const Words<TW> c2 = full_add(f[0], v[4], v[5]), d2 = full_add(f[0], v[6], v[7]);
    const Words<TW> b4 = full_add(f[1], c2, d2);
    return full_add(f[2], a4, b4);
  };
#pragma unroll 1
  for (uint32_t b = 0; b < blocks; b++) {
    const uint4 q0 = n0, q1 = n1;
    lp = b + 1 < blocks ? lp + 64 : next;
    n0 = __ldg(lp);
    n1 = __ldg(lp + 32);
    const Words<TW> a8 = eight(q0), b8 = eight(q1);
    Words<TW> c = full_add(f[3], a8, b8);
#pragma unroll
    for (int p = 4; p < P; p++)
#pragma unroll
      for (int t = 0; t < TW; t++) {
        const uint32_t k = f[p].w[t] & c.w[t];
        f[p].w[t] ^= c.w[t];
        c.w[t] = k;
      }
  }
  if (!blocks) {
    n0 = __ldg(next);
    n1 = __ldg(next + 32);
  }
  // votes (capi.c:110-118): cap - failed, zero where that is negative
  uint32_t m[P];
#pragma unroll
  for (int b = 0; b < P; b++) m[b] = 0u - ((cap >> b) & 1u);
#pragma unroll
  for (int t = 0; t < TW; t++) {
    uint32_t d[P], br = 0;
#pragma unroll
    for (int b = 0; b < P; b++) {
      d[b] = x3(m[b], f[b].w[t], br);
      br = m3(~m[b], f[b].w[t], br);
    }
    uint32_t c = 0;
#pragma unroll
    for (int b = 0; b < SL_ACC; b++) {
      const uint32_t v = b < P ? d[b < P ? b : 0] & ~br : 0u, o = acc[b].w[t];
      acc[b].w[t] = x3(o, v, c);
      c = m3(o, v, c);
    }
  }
}

// Grid: tiles x parts, the parts of one tile's groups `tiles` blocks apart.
template <int TW>
__global__ void __launch_bounds__(list_threads(TW), 1)
    k_list_votes(const uint4 *__restrict__ lists, const uint2 *__restrict__ groups,
                 const int32_t *__restrict__ lits, uint32_t classes, uint32_t clauses, uint32_t gpc,
                 uint32_t tol, uint32_t tiles, uint32_t parts, const uint32_t *__restrict__ slices,
                 uint32_t Kp, uint32_t n, int32_t *__restrict__ sums) {
  extern __shared__ __align__(16) uint32_t xs[];
  constexpr int NT = list_threads(TW);
  const uint32_t lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const uint32_t tile = blockIdx.x % tiles, part = blockIdx.x / tiles;
  {
    const uint4 *src = (const uint4 *)(slices + (uint64_t)tile * Kp * TW);
    const uint32_t q = Kp * TW / 4;
    for (uint32_t i = threadIdx.x; i < q; i += NT) copy16((uint4 *)xs + i, src + i);
  }
  // this warp's groups
  const uint64_t ng = (uint64_t)classes * gpc, shares = (uint64_t)parts * (NT / 32);
  const uint64_t me = (uint64_t)part * (NT / 32) + warp;
  uint64_t g = ng * me / shares;
  const uint64_t ge = ng * (me + 1) / shares;
  copies_done();
  __syncthreads();
  Words<TW> acc[SL_ACC];
#pragma unroll
  for (int b = 0; b < SL_ACC; b++)
#pragma unroll
    for (int t = 0; t < TW; t++) acc[b].w[t] = 0;
  uint32_t h = (uint32_t)(g / gpc), j = (uint32_t)(g - (uint64_t)h * gpc), used = 0;
  // the next group's place, literal counts and first block are read while one
  // is counted (a group with no literals names a readable block all the same)
  uint2 gn = make_uint2(0, 0);
  uint32_t Ln = 0;
  if (g < ge) {
    gn = __ldg(&groups[g]);
    Ln = list_count(lits, h, j * 32 + lane, clauses);
  }
  uint4 n0 = __ldg(lists + (uint64_t)gn.x * 64 + lane);
  uint4 n1 = __ldg(lists + (uint64_t)gn.x * 64 + lane + 32);
  while (g < ge) {
    const uint2 gi = gn;
    const uint32_t need = gi.y >> 16, blocks = gi.y & 0xFFFFu;
    const uint32_t cap = list_cap(Ln, j * 32 + lane, clauses, tol);
    const bool ends = ++j == gpc;
    if (g + 1 < ge) {
      gn = __ldg(&groups[g + 1]);
      Ln = list_count(lits, h + ends, (ends ? 0 : j * 32) + lane, clauses);
    }
    const uint4 *lp = lists + (uint64_t)gi.x * 64 + lane;
    const uint4 *next = lists + (uint64_t)gn.x * 64 + lane;
    if (need < 128) list_group<TW, 7>(xs, lp, next, n0, n1, blocks, cap, acc);
    else list_group<TW, 10>(xs, lp, next, n0, n1, blocks, cap, acc);
    used += need < tol ? need : tol;
    g++;
    const uint32_t after = gn.y >> 16;
    if (g < ge && !ends && used + (after < tol ? after : tol) < 1u << SL_ACC) continue;
    // the sums of the lanes of one parity (a class's clauses vote for it and
    // against it in turn), then of both, and one number per sample
#pragma unroll
    for (int t = 0; t < TW; t++) {
      uint32_t s[SL_ACC + 4];
#pragma unroll
      for (int b = 0; b < SL_ACC; b++) {
        s[b] = acc[b].w[t];
        acc[b].w[t] = 0;
      }
#pragma unroll
      for (int d = 0; d < 4; d++) {
        uint32_t c = 0;
#pragma unroll
        for (int b = 0; b < SL_ACC + d; b++) {
          const uint32_t o = __shfl_xor_sync(0xFFFFFFFFu, s[b], 2 << d), a = s[b];
          s[b] = x3(a, o, c);
          c = m3(a, o, c);
        }
        s[SL_ACC + d] = c;
      }
      int32_t v = 0;
#pragma unroll
      for (int b = 0; b < SL_ACC + 4; b++) {
        const uint32_t o = __shfl_xor_sync(0xFFFFFFFFu, s[b], 1);
        v += (int32_t)(((s[b] >> lane) & 1u) << b) - (int32_t)(((o >> lane) & 1u) << b);
      }
      if (lane & 1) v = -v;
      const uint32_t sample = (tile * TW + t) * 32 + lane;
      if (sample < n && v != 0) atomicAdd(&sums[(uint64_t)sample * classes + h], v);
    }
    used = 0;
    if (ends) {
      h++;
      j = 0;
    }
  }
}

uint32_t list_kp(uint32_t W) { return 32 * W + 4; }

template <int TW>
cudaError_t run_tw(const ListVotes &v, cudaStream_t st) {
  const uint32_t Kp = list_kp(v.W), tiles = (v.n + TW * 32 - 1) / (TW * 32);
  k_slice_bytes<TW><<<dim3((v.W + 31) / 32, tiles), 256, 0, st>>>(
      v.rows, v.n, v.row_bytes, v.W, Kp, v.slices, (uint32_t *)v.sums,
      (uint64_t)v.n * v.classes);
  static std::atomic<uint64_t> ready{0};  // devices whose shared-memory limit is raised
  if (!(ready.load() >> (v.device & 63) & 1u)) {
    const cudaError_t e = cudaFuncSetAttribute(
        k_list_votes<TW>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)SL_SMEM);
    if (e != cudaSuccess) return e;
    ready.fetch_or(1ull << (v.device & 63));
  }
  // eight waves of CTAs level out the last one, if a warp's share of a tile
  // stays eight groups or more; few tiles are split until every SM has a CTA
  const uint32_t gpc = (v.clauses + 31) / 32;
  const uint64_t ng = (uint64_t)v.classes * gpc, warps = list_threads(TW) / 32;
  uint64_t parts = std::min<uint64_t>(((uint64_t)v.sms * 8 + tiles - 1) / tiles, ng / (warps * 8));
  const uint64_t fill = ((uint64_t)v.sms + tiles - 1) / tiles;
  parts = std::max(parts, std::min<uint64_t>(fill, (ng + warps - 1) / warps));
  k_list_votes<TW><<<(unsigned)(tiles * parts), list_threads(TW), (size_t)Kp * TW * 4, st>>>(
      (const uint4 *)v.lists, (const uint2 *)v.groups, v.lits, v.classes, v.clauses, gpc, v.tol,
      tiles, (uint32_t)parts, v.slices, Kp, v.n, v.sums);
  return cudaGetLastError();
}

}  // namespace

// Words per tile row for rows of W words: the widest that fits (0: none).
int list_tile_words(uint32_t W) {
  for (int tw = 4; tw; tw >>= 1)
    if ((uint64_t)list_kp(W) * tw * 4 <= SL_SMEM && 32ull * W < 0xFFFFu) return tw;
  return 0;
}

uint64_t list_slice_bytes(uint32_t W, uint64_t n) {
  const uint64_t tw = list_tile_words(W);
  return (n + tw * 32 - 1) / (tw * 32) * list_kp(W) * tw * 4;
}

cudaError_t launch_list_plan(const int32_t *lits, uint32_t classes, uint32_t clauses, uint32_t tol,
                             void *groups, uint32_t *tot, cudaStream_t st) {
  const uint64_t ng = (uint64_t)classes * ((clauses + 31) / 32), b = (ng + 7) / 8;
  k_list_plan<<<(unsigned)(b < 148 * 8 ? b : 148 * 8), 256, 0, st>>>(
      lits, classes, clauses, (clauses + 31) / 32, tol, (uint2 *)groups, tot);
  return cudaGetLastError();
}

cudaError_t launch_list_fill(const uint32_t *act, uint32_t classes, uint32_t clauses,
                             const ClassDev &c, const void *groups, void *lists, cudaStream_t st) {
  const uint64_t warps = (uint64_t)classes * ((clauses + 31) / 32) * 32, b = (warps + 7) / 8;
  k_list_fill<<<(unsigned)(b < 148 * 32 ? b : 148 * 32), 256, 0, st>>>(
      act + c.act_off, classes, clauses, (clauses + 31) / 32, c.Wp, c.W, c.emask,
      (const uint2 *)groups, 32 * c.W, (uint16_t *)lists);
  return cudaGetLastError();
}

cudaError_t launch_list_votes(const ListVotes &v, cudaStream_t st) {
  switch (list_tile_words(v.W)) {
    case 4: return run_tw<4>(v, st);
    case 2: return run_tw<2>(v, st);
    case 1: return run_tw<1>(v, st);
  }
  return cudaErrorInvalidValue;
}

}  // namespace tmb
