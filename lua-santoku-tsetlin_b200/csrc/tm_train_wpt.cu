// The fused train kernels for units of 8-bit automata whose rows have at most
// 1,024 words (capi.c:85-243 evaluation and feedback, automata.h:88-742
// updates).  A unit's actions, and the count planes of rows up to 64 words (256
// in k_train_spec), stay on its SM while it trains; the count planes of wider
// rows stay in global memory, in L2 as far as the resident units' planes fit.
//
//   k_train_wpt   every thread owns WPT consecutive words of all eight clauses
//   k_train_spec  few units: eight warps evaluate eight samples at once
//
// What bounds them: integer issue (LOP3 at half rate, POPC at an eighth) and the
// dependent chain of one sample's step.  Hence:
//   - saturation is decided before any plane is written: a carry chain of one
//     LOP3 per plane finds the bits that would overflow, then one LOP3 per
//     plane applies the update to the others (count_step and its kin);
//   - one body of update code serves all eight clauses, the planes addressed
//     in shared memory, or for rows above 64 words in global memory (L2): eight
//     unrolled bodies (automata in registers) were 77 KB of code and half the
//     warps waited for instructions (search rows: 127 ms against 69 ms);
//   - a sample's row words go straight to the thread that owns them by 4- to
//     16-byte asynchronous copies, three samples ahead: no mbarrier stands
//     between a copy and its use;
//   - the failed-literal counts of two clauses share one 32-bit word, so a
//     warp reduces eight clauses in four __reduce_add_sync;
//   - the chance draws are turned into vote thresholds (feedback fires when
//     the signed chunk vote is below the threshold) for a group of samples at
//     once, outside the dependent chain;
//   - a unit of one warp needs no CTA barrier at all; larger units add their
//     counts into a rotating shared accumulator and pass one barrier per
//     sample (a second one when the sample has Type Ib clauses), every warp
//     taking the same decisions from it.
// Measured (train calls, B200, before -> after): search rows of 49 words, 28.5M
// active steps, 44.7 -> 26 ms (narrow rows 34.7 -> 17.4 ms); plain classifier
// 8,000 samples x 10 epochs, 320 units, 15.0 -> 2.8 ms; encoder rows of 256
// words 190 -> 113 ms; sparse classifier rows of 1,024 words 127 -> 90 ms.
// The same rules and draws as k_train, so the same automata bit for bit.
#include <math.h>

#include "tm_device.cuh"

namespace tmb {

namespace {

constexpr int M7 = 7;      // count planes (8 state bits)
constexpr int RING = 4;    // sample rows in flight per thread (3 ahead)
constexpr int SC = 2;      // positions a thread examines per scan of the epoch order

template <int WPT>
struct WVec;
template <>
struct WVec<1> {
  __device__ static void ld(const uint32_t *p, uint32_t (&v)[1]) { v[0] = *p; }
  __device__ static void st(uint32_t *p, const uint32_t (&v)[1]) { *p = v[0]; }
};
template <>
struct WVec<4> {
  __device__ static void ld(const uint32_t *p, uint32_t (&v)[4]) {
    const uint4 t = *(const uint4 *)p;
    v[0] = t.x;
    v[1] = t.y;
    v[2] = t.z;
    v[3] = t.w;
  }
  __device__ static void st(uint32_t *p, const uint32_t (&v)[4]) {
    *(uint4 *)p = make_uint4(v[0], v[1], v[2], v[3]);
  }
};
template <>
struct WVec<2> {
  __device__ static void ld(const uint32_t *p, uint32_t (&v)[2]) {
    const uint2 t = *(const uint2 *)p;
    v[0] = t.x;
    v[1] = t.y;
  }
  __device__ static void st(uint32_t *p, const uint32_t (&v)[2]) {
    *(uint2 *)p = make_uint2(v[0], v[1]);
  }
};

// asynchronous copy of a thread's own row words (4, 8 or 16 bytes)
template <int BYTES>
__device__ __forceinline__ void cp_async_words(void *dst, const void *src) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], %2;\n" ::"r"(smem_u32(dst)), "l"(src),
               "n"(BYTES)
               : "memory");
}
__device__ __forceinline__ void cp_commit() { asm volatile("cp.async.commit_group;\n" ::: "memory"); }
template <int N>
__device__ __forceinline__ void cp_wait() {
  asm volatile("cp.async.wait_group %0;\n" ::"n"(N) : "memory");
}

// philox with the key taken as new at every call: its ten round keys are then
// computed there instead of being kept in (and spilled from) registers
// across the sample loop.
__device__ __forceinline__ void draw4(uint32_t c0, uint32_t c1, uint32_t c2, uint32_t c3,
                                      uint64_t key, uint32_t *o) {
  asm volatile("" : "+l"(key));
  philox(c0, c1, c2, c3, key, o);
}

// The updates below run on a thread's WPT words plane by plane, so that the
// words' carry chains (one dependent LOP3 per plane) overlap.

// +1 on the bits of `c0` outside `dm`, -1 on those inside it, both saturating
// (automata.h:88-318).  A decrement is an increment of the complement, so the
// carry runs through p ^ dm; bits whose carry leaves the action plane are
// saturated and keep every plane.
template <int N>
__device__ __forceinline__ void count_step(uint32_t (&p)[M7][N], uint32_t (&a)[N],
                                           const uint32_t (&c0)[N], const uint32_t (&dm)[N],
                                           const uint32_t (&am)[N]) {
  uint32_t c[M7 + 1][N], keep[N];
#pragma unroll
  for (int q = 0; q < N; q++) c[0][q] = c0[q];
#pragma unroll
  for (int b = 0; b < M7; b++)
#pragma unroll
    for (int q = 0; q < N; q++) c[b + 1][q] = c[b][q] & (p[b][q] ^ dm[q]);
#pragma unroll
  for (int q = 0; q < N; q++) {
    const uint32_t ca = c[M7][q] & am[q];
    keep[q] = ~(ca & (a[q] ^ dm[q]));
    a[q] ^= ca & keep[q];
  }
#pragma unroll
  for (int b = 0; b < M7; b++)
#pragma unroll
    for (int q = 0; q < N; q++) p[b][q] ^= c[b][q] & keep[q];
}

// +1 on bits whose automaton is not included (action 0 with one include bit,
// so the carry into the action plane never saturates)
template <int N>
__device__ __forceinline__ void count_inc0(uint32_t (&p)[M7][N], uint32_t (&a)[N], uint32_t (&c)[N],
                                           const uint32_t (&am)[N]) {
#pragma unroll
  for (int b = 0; b < M7; b++)
#pragma unroll
    for (int q = 0; q < N; q++) {
      const uint32_t t = c[q] & p[b][q];
      p[b][q] ^= c[q];
      c[q] = t;
    }
#pragma unroll
  for (int q = 0; q < N; q++) a[q] ^= c[q] & am[q];
}

// -1 on bits with action 0: the action plane stays, a borrow that reaches it
// means the count was zero
template <int N>
__device__ __forceinline__ void count_dec0(uint32_t (&p)[M7][N], const uint32_t (&d)[N],
                                           const uint32_t (&am)[N]) {
  uint32_t c[M7 + 1][N], keep[N];
#pragma unroll
  for (int q = 0; q < N; q++) c[0][q] = d[q];
#pragma unroll
  for (int b = 0; b < M7; b++)
#pragma unroll
    for (int q = 0; q < N; q++) c[b + 1][q] = c[b][q] & ~p[b][q];
#pragma unroll
  for (int q = 0; q < N; q++) keep[q] = ~(c[M7][q] & am[q]);
#pragma unroll
  for (int b = 0; b < M7; b++)
#pragma unroll
    for (int q = 0; q < N; q++) p[b][q] ^= c[b][q] & keep[q];
}

// Saturating subtraction of m0 + 2 m1 per bit (Type Ib picks counted in two
// binary levels): a two-bit subtractor, then the borrow through the higher
// planes; bits whose borrow leaves the action plane end at zero.
template <int N>
__device__ __forceinline__ void count_sub(uint32_t (&p)[M7][N], uint32_t (&a)[N],
                                          const uint32_t (&m0)[N], const uint32_t (&m1)[N],
                                          const uint32_t (&am)[N]) {
  uint32_t r[M7 + 1][N], keep[N];
#pragma unroll
  for (int q = 0; q < N; q++) r[1][q] = m0[q] & ~p[0][q];
#pragma unroll
  for (int q = 0; q < N; q++)
    r[2][q] = (~p[1][q] & (m1[q] | r[1][q])) | (m1[q] & r[1][q]);
#pragma unroll
  for (int b = 2; b < M7; b++)
#pragma unroll
    for (int q = 0; q < N; q++) r[b + 1][q] = r[b][q] & ~p[b][q];
#pragma unroll
  for (int q = 0; q < N; q++) {
    const uint32_t ra = r[M7][q] & am[q];
    keep[q] = ~(ra & ~a[q]);
    a[q] &= ~ra;
    p[0][q] = (p[0][q] ^ m0[q]) & keep[q];
    p[1][q] = (p[1][q] ^ m1[q] ^ r[1][q]) & keep[q];
  }
#pragma unroll
  for (int b = 2; b < M7; b++)
#pragma unroll
    for (int q = 0; q < N; q++) p[b][q] = (p[b][q] ^ r[b][q]) & keep[q];
}

// automata.h:499-512: action AND the top include_bits - 1 count planes
template <int N>
__device__ __forceinline__ uint32_t included(const uint32_t (&p)[M7][N], uint32_t a, int q,
                                             uint32_t ib) {
#pragma unroll
  for (int b = 0; b < M7; b++)
    if (b + (int)ib > M7) a &= p[b][q];
  return a;
}

// Vote thresholds of sample `ent` (index | positive << 31) for the eight
// clauses.  Clause c's draw d fires iff floor(d 2T / 2^32) < T - v for a
// positive sample, T + v for a negative one, v clamped to [-T, T]
// (capi.c:217-242): iff v (or -v) < T - floor(d 2T / 2^32), a value in
// (-T, T], so the clamp never decides.
__device__ __forceinline__ void vote_thresholds(uint32_t ent, uint32_t ee, uint32_t g, uint32_t T,
                                                uint64_t seed, int32_t *out) {
  const uint32_t s = ent & 0x7FFFFFFFu;
  uint32_t d[8];
  draw4(s, ee, g, ST_CH0, seed, d);
  draw4(s, ee, g, ST_CH1, seed, d + 4);
  int32_t t[8];
#pragma unroll
  for (int c = 0; c < 8; c++) {
    // draw 2p decides Type I of pair p, draw 2p + 1 Type II; a positive
    // sample gives Type I to the even clause
    const uint32_t dd = ((ent >> 31) != 0) == ((c & 1) == 0) ? d[c & ~1] : d[c | 1];
    int64_t v = (int64_t)T - (int64_t)bounded64(dd, 2ull * T);
    v = v > INT32_MAX ? INT32_MAX : (v <= INT32_MIN ? INT32_MIN + 1 : v);
    t[c] = T ? (int32_t)v : INT32_MIN;
  }
  *(int4 *)out = make_int4(t[0], t[1], t[2], t[3]);
  *(int4 *)(out + 4) = make_int4(t[4], t[5], t[6], t[7]);
}

// The picks of every Type Ib clause of `ibm` (capi.c:181-190), spread over
// the unit's threads: counted per bit in two binary levels of the clause's
// slot, larger counts as overflow entries worth 4 each (saturating
// subtraction is order-free).  The four level-0 exchanges of a draw are
// issued together; only draws that carry go on.
template <uint32_t NT, uint32_t SW>
__device__ __forceinline__ void draw_picks(uint32_t ibm, uint32_t sp, uint32_t ee, uint32_t g,
                                           uint64_t seed, uint32_t npk, uint32_t nq,
                                           uint32_t input_bits, uint32_t *lev, uint16_t *ovf,
                                           uint32_t *oc, uint32_t ovf_cap) {
  uint32_t clist = 0, nib = 0;
  for (uint32_t cm = ibm; cm; cm &= cm - 1, nib++)
    clist |= (uint32_t)(__ffs(cm) - 1) << (4 * nib);
  const uint32_t total = nib * nq;
  for (uint32_t it = threadIdx.x; it < total; it += NT) {
    const uint32_t slot = (it >= nq) + (it >= 2 * nq) + (it >= 3 * nq);
    const uint32_t q = it - slot * nq, c = (clist >> (4 * slot)) & 15u;
    uint32_t *l0 = lev + slot * (2 * SW), *l1 = l0 + SW;
    uint32_t r[4], mk[4], old[4];
    draw4(sp, ee, g, ST_IB | (c << 20) | q, seed, r);
#pragma unroll
    for (uint32_t z = 0; z < 4; z++) {
      r[z] = __umulhi(r[z], input_bits);
      mk[z] = 1u << (r[z] & 31);
    }
    if (4 * q + 4 > npk) {  // the last draw may hold fewer than 4 picks
#pragma unroll
      for (uint32_t z = 1; z < 4; z++) mk[z] = 4 * q + z < npk ? mk[z] : 0u;
    }
#pragma unroll
    for (uint32_t z = 0; z < 4; z++) old[z] = atomicXor(&l0[r[z] >> 5], mk[z]);
#pragma unroll
    for (uint32_t z = 0; z < 4; z++) mk[z] &= old[z];
    if (mk[0] | mk[1] | mk[2] | mk[3]) {
      // (all four again, without a branch per pick: most warps carry somewhere)
#pragma unroll
      for (uint32_t z = 0; z < 4; z++) old[z] = atomicXor(&l1[r[z] >> 5], mk[z]);
#pragma unroll
      for (uint32_t z = 0; z < 4; z++) mk[z] &= old[z];
      if (mk[0] | mk[1] | mk[2] | mk[3]) {
#pragma unroll
        for (uint32_t z = 0; z < 4; z++)
          if (mk[z]) {
            const uint32_t k = atomicAdd(&oc[slot], 1u);
            if (k < ovf_cap) ovf[slot * ovf_cap + k] = (uint16_t)r[z];
          }
      }
    }
  }
}

// Overflow entries (each worth 4) of one clause that lie in words [first, first
// + words), those of the calling warp: their bits into the level-1 words `l1`,
// which the warp's lanes have read and cleared.  A lane takes every 32nd entry
// from `at` on and stops at a bit that is set already: it waits until the
// caller has subtracted and cleared what there is.  (Rows of 24,000 literals at
// specificity 1.2, 250 entries per clause, 800 units: 121.8 ms with every entry
// subtracted from every word, 16.3 ms this way.)
__device__ __forceinline__ void take_overflow(const uint16_t *entries, uint32_t n, uint32_t &at,
                                              uint32_t first, uint32_t words, uint32_t *l1) {
  __syncwarp();
  while (at < n) {
    const uint32_t e = entries[at], w = e >> 5, bit = 1u << (e & 31);
    if (w - first < words && (atomicOr(&l1[w], bit) & bit)) break;
    at += 32;
  }
  __syncwarp();
}

// samples whose vote thresholds are held at a time
__host__ __device__ constexpr uint32_t wpt_group(uint32_t NT) { return NT < 64 ? NT : 64; }

// Samples listed before a unit starts on them: enough that the threshold
// pass (one sample per thread) and the row copies' start-up weigh little.
__host__ __device__ constexpr uint32_t wpt_fill(uint32_t NT) {
  return NT == 32 ? 96 : (NT == 64 ? 128 : NT);
}

// Shared-memory layout of a unit (byte offsets): NT threads, SW words per
// row slot, IBS Type Ib slots.
struct WptLayout {
  uint32_t planes, ring, list, thr, acc, lev, ovf, misc, total;
};
__host__ __device__ constexpr WptLayout wpt_layout(uint32_t NT, uint32_t SW, int RP, int IBS,
                                                   uint32_t ovf_cap) {
  WptLayout L{};
  uint32_t at = 0;
  auto take = [&](uint32_t bytes) {
    const uint32_t r = at;
    at += (bytes + 15) / 16 * 16;
    return r;
  };
  L.planes = take((8 - RP) * 8 * SW * 4);
  L.ring = take(RING * SW * 4);
  L.list = take((wpt_fill(NT) + SC * NT) * 4);
  L.thr = take(wpt_group(NT) * 8 * 4);
  L.acc = take(NT == 32 ? 0 : 3 * 16 * 4);  // the one-warp form adds nothing up
  L.lev = take(IBS * 2 * SW * 4);
  L.misc = take((NT == 32 ? 8 : 64) * 4);
  L.ovf = take(IBS * ovf_cap * 2);
  L.total = at;
  return L;
}

}  // namespace

// misc: [0] unit, [8..39] live counts of a scan, [48..55] overflow counts (2 parities x 4)
// NT threads per unit (32: the one-warp form) of WPT words, SW words per
// row slot (at most NT * WPT, at least the widest row).  The first RP count
// planes are held in registers, the last GP in global memory, the others and
// the actions in shared memory; IBS Type Ib clauses are drawn at a time; MINB
// CTAs per SM the registers are sized for; OV for launches whose Type Ib
// clauses meet overflow entries at all often (WPT_OVF): a warp hands them to
// the lanes they concern, where the other form, cheaper without entries,
// subtracts each from every word.
template <int NT, int WPT, int SW, int RP, int GP, int IBS, int MINB, bool OV>
__global__ void __launch_bounds__(NT, MINB)
    k_train_wpt(const TrainDev *__restrict__ machines, const WorkItem *__restrict__ work,
                uint32_t nwork, uint32_t *__restrict__ counter, uint32_t e_begin, uint32_t e_end,
                uint32_t ovf_cap, uint32_t *__restrict__ err) {
  constexpr bool ONE = NT == 32;
  constexpr uint32_t NW = NT / 32;
  constexpr uint32_t TG = wpt_group(NT);
  // planes in shared memory: count planes RP .. 6 - GP, then the actions
  constexpr int SP = 8 - RP - GP;
  constexpr int G0 = M7 - GP;  // first count plane that stays in global memory
  constexpr uint32_t FULL = 0xFFFFFFFFu;
  extern __shared__ __align__(128) uint8_t smem[];
  const WptLayout o = wpt_layout(NT, SW, RP + GP, IBS, ovf_cap);
  const uint32_t tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const uint32_t w0 = tid * WPT;  // this thread's first word
  // threads past the row slots own no words: they load word 0's (under masks
  // that are zero) and store nothing
  const uint32_t ws = w0 < SW ? w0 : 0;
  uint32_t *splanes = (uint32_t *)(smem + o.planes) + ws;
  uint32_t *ring = (uint32_t *)(smem + o.ring) + ws;
  uint32_t *list = (uint32_t *)(smem + o.list);
  int32_t *thr = (int32_t *)(smem + o.thr);
  uint32_t *acc = (uint32_t *)(smem + o.acc);
  uint32_t *lev = (uint32_t *)(smem + o.lev);
  uint16_t *ovf = (uint16_t *)(smem + o.ovf);
  uint32_t *misc = (uint32_t *)(smem + o.misc);
  uint32_t *ocnt = misc + (ONE ? 0 : 48);  // overflow counts (2 parities x 4)
  auto sync = [] {
    if constexpr (ONE) __syncwarp();
    else __syncthreads();
  };
  for (uint32_t i = tid; i < IBS * 2 * SW; i += NT) lev[i] = 0;
  if (tid < 8) ocnt[tid] = 0;
  // lane c of every warp decides clause c (lanes above 8 repeat them)
  const uint32_t cl = lane & 7;
  const int32_t sign = lane < 8 ? ((lane & 1) ? -1 : 1) : 0;
  uint32_t step = 0;  // parity of the overflow counts, ring slot
  uint32_t ab = 0;    // accumulator of this step

  while (true) {
    uint32_t u = 0;
    if (tid == 0) {
      // the next unit, passing over those of machines whose gate is closed
      u = atomicAdd(counter, 1u);
      while (u < nwork) {
        const uint32_t *gt = machines[work[u].m].gate;
        if (!gt || *gt) break;
        u = atomicAdd(counter, 1u);
      }
      if (!ONE) misc[0] = u;
    }
    if (ONE) {
      u = __shfl_sync(FULL, u, 0);
    } else {
      if (tid < 48) acc[tid] = 0;
      __syncthreads();
      u = misc[0];
      __syncthreads();
    }
    if (u >= nwork) break;
    const WorkItem wi = work[u];
    const TrainDev &M = machines[wi.m];
    const ClassDev C = M.cls[wi.h];
    const uint32_t Wp = C.Wp, W = C.W;
    const uint32_t g = wi.h * M.clause_chunks + wi.k;
    uint32_t *gact = M.act + C.act_off + (uint64_t)wi.k * 8 * Wp + w0;
    uint32_t *gcnt = M.cnt + C.cnt_off + (uint64_t)wi.k * 8 * M7 * Wp + w0;
    // the count planes that stay in global memory are read and written in
    // place; threads without words of their own read word 0's and store nothing
    uint32_t *gpl = M.cnt + C.cnt_off + (uint64_t)wi.k * 8 * M7 * Wp + (w0 < Wp ? w0 : 0);
    __builtin_assume(__isGlobal(gpl));
    // ---- the unit's automata onto the SM ------------------------------------
    uint32_t pl[8][RP > 0 ? RP : 1][WPT];
    const bool mine = w0 < Wp;  // Wp is a multiple of 4, so of WPT
#pragma unroll
    for (int c = 0; c < 8; c++)
#pragma unroll
      for (int b = 0; b < 8; b++) {
        if (b >= G0 && b < M7) continue;
        uint32_t t[WPT] = {};
        if (mine) WVec<WPT>::ld(b < M7 ? gcnt + (c * M7 + b) * Wp : gact + c * Wp, t);
        if (b < RP) {
#pragma unroll
          for (int q = 0; q < WPT; q++) pl[c][b < RP ? b : 0][q] = t[q];
        } else if (w0 < SW) {
          WVec<WPT>::st(splanes + (c * SP + (b < M7 ? b - RP : SP - 1)) * SW, t);
        }
      }
    uint32_t vm[WPT], em[WPT], am[WPT];
#pragma unroll
    for (int q = 0; q < WPT; q++) {
      vm[q] = word_mask(w0 + q, W, C.vmask);
      em[q] = word_mask(w0 + q, W, C.emask);
      am[q] = word_mask(w0 + q, W, C.amask);
    }
    // this thread's words of clause c, c known at run time (one body of update
    // code for all eight clauses keeps the kernel in the instruction cache):
    // the register planes through a branch to the clause's registers (the
    // empty asm keeps it a branch: selects would read all eight), the others
    // by address
#define TM_CLAUSES(X) X(0) X(1) X(2) X(3) X(4) X(5) X(6) X(7)
    auto gather = [&](uint32_t c, uint32_t (&p)[M7][WPT], uint32_t (&a)[WPT]) {
      const uint32_t *base = splanes + c * (SP * SW);
      const uint32_t *gbase = gpl + c * (M7 * Wp);
#pragma unroll
      for (int b = RP; b < 8; b++) {
        uint32_t t[WPT];
        if (b >= G0 && b < M7) {
          WVec<WPT>::ld(gbase + b * Wp, t);
        } else {
          WVec<WPT>::ld(base + (b < M7 ? b - RP : SP - 1) * SW, t);
        }
#pragma unroll
        for (int q = 0; q < WPT; q++) {
          if (b < M7) p[b < M7 ? b : 0][q] = t[q];
          else a[q] = t[q];
        }
      }
      if constexpr (RP > 0) {
#define TM_IN(K)                                                                         \
  case K:                                                                                \
    asm volatile("");                                                                    \
    _Pragma("unroll") for (int q = 0; q < WPT; q++)                                      \
        _Pragma("unroll") for (int b = 0; b < RP; b++) p[b][q] = pl[K][b][q];            \
    break;
        switch (c) { TM_CLAUSES(TM_IN) }
#undef TM_IN
      }
    };
    auto scatter = [&](uint32_t c, const uint32_t (&p)[M7][WPT], const uint32_t (&a)[WPT]) {
      uint32_t *base = splanes + c * (SP * SW);
      uint32_t *gbase = gpl + c * (M7 * Wp);
      if (mine) {
#pragma unroll
        for (int b = RP; b < 8; b++) {
          uint32_t t[WPT];
#pragma unroll
          for (int q = 0; q < WPT; q++) t[q] = b < M7 ? p[b < M7 ? b : 0][q] : a[q];
          if (b >= G0 && b < M7) WVec<WPT>::st(gbase + b * Wp, t);
          else WVec<WPT>::st(base + (b < M7 ? b - RP : SP - 1) * SW, t);
        }
      }
      if constexpr (RP > 0) {
#define TM_OUT(K)                                                                        \
  case K:                                                                                \
    asm volatile("");                                                                    \
    _Pragma("unroll") for (int q = 0; q < WPT; q++)                                      \
        _Pragma("unroll") for (int b = 0; b < RP; b++) pl[K][b][q] = p[b][q];            \
    break;
        switch (c) { TM_CLAUSES(TM_OUT) }
#undef TM_OUT
      }
    };
    // this warp's share of clause c's literal count
    auto lits_of = [&](const uint32_t (&a)[WPT]) {
      uint32_t l = 0;
#pragma unroll
      for (int q = 0; q < WPT; q++) l += __popc(a[q] & em[q]);
      return __reduce_add_sync(FULL, l);
    };
    const uint32_t tol = M.tol, maxlit = M.maxlit, ib = M.ib, n = M.n, type = M.type;
    const uint64_t seed = M.seed;
    const uint32_t npk = C.s_picks, nq = (npk + 3) >> 2, input_bits = C.input_bits;
    const uint32_t ep_end = e_end < M.epochs ? e_end : M.epochs;
    const uint32_t *xbase = M.x + C.x_off + w0;
    // literal counts: lane c's clause; in the multi-warp form each warp's
    // share waits in lane 4 + c for the next exchange
    uint32_t dirty = 0xFFu, L = 0, lval = 0, incM = 0;
    int32_t cap = 0;
#pragma unroll
    for (int c = 0; c < 8; c++) {
      uint32_t a[WPT];
      WVec<WPT>::ld(splanes + (c * SP + SP - 1) * SW, a);
      const uint32_t l = lits_of(a);
      if (ONE) L = cl == (uint32_t)c ? l : L;
      else lval = lane == 4u + c ? l : lval;
    }
    auto settle = [&]() {  // the vote cap of lane c's clause, and the increment mask
      cap = (int32_t)(L == 0 || L > tol ? tol : L);
      incM = __ballot_sync(FULL, L <= maxlit);
    };
    if (ONE) settle();
    uint64_t nsteps = 0;

    for (uint32_t e = e_begin; e < ep_end; e++) {
      const uint32_t ee = M.epoch_base + e;
      const uint32_t *perm = M.perm + (uint64_t)(e - e_begin) * n;
      uint32_t at = 0;  // next position of the epoch order
      while (at < n) {
        // ---- the next samples this unit trains on ---------------------------
        // Skip decisions (capi.c:215) do not depend on the automata: scan
        // positions until the list holds enough samples, in order.
        uint32_t cnt = 0;
        while (at < n && cnt < wpt_fill(NT)) {
          uint32_t s[SC], y[SC], bal[SC];
#pragma unroll
          for (int j = 0; j < SC; j++) {
            const uint32_t i = at + j * NT + tid;
            s[j] = i < n ? perm[i] : FULL;
          }
#pragma unroll
          for (int j = 0; j < SC; j++) {
            y[j] = 0;
            if (s[j] != FULL) {
              if (type == 0) y[j] = (uint32_t)M.labels[s[j]] == wi.h;
              else y[j] = (M.codes[(uint64_t)s[j] * M.code_bytes + (wi.h >> 3)] >> (wi.h & 7)) & 1u;
            }
          }
#pragma unroll
          for (int j = 0; j < SC; j++) {
            bool live = s[j] != FULL;
            if (live && type == 0 && !y[j]) {
              uint32_t r[4];
              draw4(s[j], ee, g, ST_NEG, seed, r);
              live = (uint64_t)r[0] >= M.thr_neg;
            }
            bal[j] = __ballot_sync(FULL, live);
          }
          const uint32_t below = (1u << lane) - 1u;
          if (ONE) {
#pragma unroll
            for (int j = 0; j < SC; j++) {
              if ((bal[j] >> lane) & 1u) list[cnt + __popc(bal[j] & below)] = s[j] | (y[j] << 31);
              cnt += __popc(bal[j]);
            }
          } else {
            if (lane == 0)
#pragma unroll
              for (int j = 0; j < SC; j++) misc[8 + j * NW + warp] = __popc(bal[j]);
            __syncthreads();
            // order: scan j, then warp, then lane
            const uint32_t own = lane < SC * NW ? misc[8 + lane] : 0;
            uint32_t inc = own;
#pragma unroll
            for (int d = 1; d < 32; d <<= 1) {
              const uint32_t t = __shfl_up_sync(FULL, inc, d);
              if (lane >= (uint32_t)d) inc += t;
            }
#pragma unroll
            for (int j = 0; j < SC; j++) {
              const uint32_t off = __shfl_sync(FULL, inc - own, j * NW + warp);
              if ((bal[j] >> lane) & 1u)
                list[cnt + off + __popc(bal[j] & below)] = s[j] | (y[j] << 31);
            }
            cnt += __shfl_sync(FULL, inc, 31);
            __syncthreads();
          }
          at += SC * NT;
        }
        sync();
        nsteps += cnt;
        // rows of the first samples of the list
        auto fetch = [&](uint32_t a) {
          if (a < cnt && mine)
            cp_async_words<WPT * 4>(ring + ((step + a) & (RING - 1)) * SW,
                                    xbase + (uint64_t)(list[a] & 0x7FFFFFFFu) * Wp);
          cp_commit();
        };
        if (cnt) {
#pragma unroll
          for (uint32_t a = 0; a < RING - 1; a++) fetch(a);
        }
        for (uint32_t g0 = 0; g0 < cnt; g0 += TG) {
          // ---- vote thresholds of a group of samples --------------------------
          if (g0) sync();
          if (tid < TG && g0 + tid < cnt) vote_thresholds(list[g0 + tid], ee, g, M.T, seed, thr + tid * 8);
          sync();
          const uint32_t ge = cnt - g0 < TG ? cnt - g0 : TG;
          // ---- sequential per-sample steps ------------------------------------
          for (uint32_t a = 0; a < ge; a++) {
            fetch(g0 + a + RING - 1);
            const uint32_t ent = list[g0 + a];
            const int32_t tc = thr[a * 8 + cl];
            const uint32_t par = (step + g0 + a) & 1u;
            cp_wait<RING - 1>();
            uint32_t x[WPT];
            WVec<WPT>::ld(ring + ((step + g0 + a) & (RING - 1)) * SW, x);
            // failed literals of the eight clauses, two per word
            uint32_t pk[4];
#pragma unroll
            for (int c = 0; c < 8; c += 2) {
              uint32_t f0 = 0, f1 = 0, a0[WPT], a1[WPT];
              WVec<WPT>::ld(splanes + (c * SP + SP - 1) * SW, a0);
              WVec<WPT>::ld(splanes + ((c + 1) * SP + SP - 1) * SW, a1);
#pragma unroll
              for (int q = 0; q < WPT; q++) {
                f0 += __popc(a0[q] & em[q] & ~x[q]);
                f1 += __popc(a1[q] & em[q] & ~x[q]);
              }
              pk[c >> 1] = __reduce_add_sync(FULL, f0 + (f1 << 16));
            }
            uint32_t pr = (lane & 2) ? ((lane & 1) ? pk[3] : pk[2]) : ((lane & 1) ? pk[1] : pk[0]);
            if (ONE) {
              pr = (lane & 4) ? ((lane & 2) ? pk[3] : pk[2]) : ((lane & 2) ? pk[1] : pk[0]);
            } else {
              // accumulator ab is zero since step - 2; the one of step + 2
              // was read before this step's barrier and is cleared after it
              if (lane < 12) atomicAdd(&acc[ab * 16 + lane], lane < 4 ? pr : lval);
              __syncthreads();
              const uint32_t *A = acc + ab * 16;
              pr = A[cl >> 1];
              if (dirty) {
                const uint32_t l = A[4 + cl];
                if ((dirty >> cl) & 1u) L = l;
                settle();
              }
              const uint32_t nx2 = ab == 0 ? 2 : ab - 1;
              if (tid < 16) acc[nx2 * 16 + tid] = 0;
              // the previous step's overflow counts, for the next step
              if (tid < 4) ocnt[(par ^ 1u) * 4 + tid] = 0;
              ab = ab == 2 ? 0 : ab + 1;
            }
            const uint32_t F = (lane & 1) ? pr >> 16 : pr & 0xFFFFu;
            // votes (capi.c:110-118), signed by clause parity (:148-161)
            int32_t vote = cap - (int32_t)F;
            vote = vote < 0 ? 0 : vote;
            const int32_t v = (int32_t)__reduce_add_sync(FULL, (uint32_t)(vote * sign));
            const bool pa = ent >> 31;
            const uint32_t fm = __ballot_sync(FULL, (pa ? v : -v) < tc) & 0xFFu;
            const uint32_t vt = __ballot_sync(FULL, vote > 0);
            const uint32_t t1 = pa ? 0x55u : 0xAAu;  // Type I clauses
            const uint32_t ibm = fm & t1 & ~vt;      // Type Ib (capi.c:181-190)
            const uint32_t fbm = fm & vt;            // Type Ia and II
            dirty = 0;
            if (!(ibm | fbm)) continue;
            const uint32_t sp = ent & 0x7FFFFFFFu;
            uint32_t *oc = ocnt + par * 4;
            // feedback, Type Ib clauses in rounds of at most IBS, the first with
            // the Type Ia and II clauses
            uint32_t rest = ibm, grp, todo = fbm;
            do {
              grp = 0;
#pragma unroll
              for (int k = 0; k < IBS; k++) {
                grp |= rest & (0u - rest);
                rest &= rest - 1u;
              }
              if constexpr (IBS == 4) rest = 0;  // a sample has at most one Type I clause per pair
              todo |= grp;
              if (grp) {
                if (ONE) __syncwarp();
                draw_picks<NT, SW>(grp, sp, ee, g, seed, npk, nq, input_bits, lev, ovf, oc, ovf_cap);
                sync();
              }
#pragma unroll 1
              for (uint32_t cm = todo; cm; cm &= cm - 1) {
                const uint32_t c = __ffs(cm) - 1;
                uint32_t p[M7][WPT], ac[WPT];
                gather(c, p, ac);
                const bool is1 = (t1 >> c) & 1u;
                bool changed = true;  // false: the action plane is as it was
                if ((grp >> c) & 1u) {
                  const uint32_t slot = __popc(grp & ((1u << c) - 1u));
                  uint32_t *l0 = lev + slot * (2 * SW) + ws, *l1 = l0 + SW;
                  uint32_t m0[WPT], m1[WPT];
                  WVec<WPT>::ld(l0, m0);
                  WVec<WPT>::ld(l1, m1);
                  if (mine) {
                    const uint32_t zero[WPT] = {};
                    WVec<WPT>::st(l0, zero);
                    WVec<WPT>::st(l1, zero);
                  } else {
#pragma unroll
                    for (int q = 0; q < WPT; q++) m0[q] = m1[q] = 0;
                  }
                  // an overflow entry is worth 4: twice a level-1 count
                  if constexpr (OV) {
                    const uint32_t no = min(oc[slot], ovf_cap);
                    uint32_t next = lane;  // this lane's next entry
                    for (uint32_t t = 0;; t++) {
                      count_sub(p, ac, m0, m1, am);
                      if (t & 1u) continue;
                      if (!__any_sync(FULL, next < no)) break;
                      take_overflow(ovf + slot * ovf_cap, no, next, warp * 32 * WPT, 32 * WPT,
                                    lev + slot * (2 * SW) + SW);
                      WVec<WPT>::ld(l1, m1);
                      if (mine) {
                        const uint32_t zero[WPT] = {};
                        WVec<WPT>::st(l1, zero);
                      }
#pragma unroll
                      for (int q = 0; q < WPT; q++) {
                        m0[q] = 0;
                        m1[q] = mine ? m1[q] : 0;
                      }
                    }
                  } else {
                    const uint32_t no = 2 * min(oc[slot], ovf_cap);
                    for (uint32_t t = 0;; t++) {
                      count_sub(p, ac, m0, m1, am);
                      if (t >= no) break;
                      const uint32_t bit = ovf[slot * ovf_cap + (t >> 1)];
#pragma unroll
                      for (int q = 0; q < WPT; q++) {
                        m0[q] = 0;
                        m1[q] = (bit >> 5) == w0 + q ? 1u << (bit & 31) : 0u;
                      }
                    }
                  }
                } else {
                  // Type Ia (capi.c:177-180): inc where x = 1 (if L <= maximum),
                  // dec where x = 0 and not included.  Type II (capi.c:192-196):
                  // inc where x = 0 and not included.
                  const bool incx = is1 && ((incM >> c) & 1u);
                  uint32_t nx[WPT];
                  if (ib == 1 && !incx) {
#pragma unroll
                    for (int q = 0; q < WPT; q++) nx[q] = ~(x[q] | ac[q]) & vm[q];
                    if (is1) count_dec0(p, nx, am);
                    else count_inc0(p, ac, nx, am);
                    changed = !is1;
                  } else {
                    uint32_t c0[WPT], dm[WPT];
#pragma unroll
                    for (int q = 0; q < WPT; q++) {
                      nx[q] = ~(x[q] | included(p, ac[q], q, ib)) & vm[q];
                      c0[q] = nx[q] | (incx ? x[q] & vm[q] : 0u);
                      dm[q] = is1 ? nx[q] : 0u;
                    }
                    count_step(p, ac, c0, dm, am);
                  }
                }
                scatter(c, p, ac);
                if (changed) {
                  dirty |= 1u << c;
                  const uint32_t l = lits_of(ac);
                  if (ONE) L = cl == c ? l : L;
                  else lval = lane == 4u + c ? l : lval;
                }
              }
              if (ONE && grp) {
                __syncwarp();
                if (lane < IBS) oc[lane] = 0;
              }
              if (rest) {
                // the slots are used again: every thread has read its levels, and
                // counts overflows apart
                sync();
                todo = 0;
                if (!ONE) oc += IBS;
              }
            } while (rest);
            if (ONE && dirty) settle();
          }
        }
        step += cnt;
        sync();
      }
    }
    // ---- the unit's automata back to global memory ----------------------------
    // (the row stride read again, so that the 64 addresses of the load above
    // are not kept, spilled, until here)
    uint32_t Wo = Wp;
    asm volatile("" : "+r"(Wo));
    if (mine) {
#pragma unroll
      for (int c = 0; c < 8; c++)
#pragma unroll
        for (int b = 0; b < 8; b++) {
          if (b >= G0 && b < M7) continue;
          uint32_t t[WPT];
          if (b < RP) {
#pragma unroll
            for (int q = 0; q < WPT; q++) t[q] = pl[c][b < RP ? b : 0][q];
          } else {
            WVec<WPT>::ld(splanes + (c * SP + (b < M7 ? b - RP : SP - 1)) * SW, t);
          }
          WVec<WPT>::st(b < M7 ? gcnt + (c * M7 + b) * Wo : gact + c * Wo, t);
        }
    }
    if (tid == 0 && nsteps) atomicAdd((unsigned long long *)(err + 2), (unsigned long long)nsteps);
  }
}

// ---------------------------------------------------------------------------
// k_train_spec: for launches of few units, whose time is the dependent chain
// of one unit's samples.  A CTA of eight warps holds a unit in shared memory
// and works in rounds: warp w evaluates sample b + w of the unit's list
// (votes and feedback decisions of all eight clauses) against the same
// automata, one barrier publishes the eight results, and the samples'
// feedback is applied in order, warp j updating clause j.  Evaluation reads
// only the action planes, so a sample's feedback leaves the later results
// valid unless it may move an action (Type II, Type Ib, Type Ia with
// increments or several include bits): then the round ends after that sample
// and the others are evaluated again.  Bit for bit the sequential rule.
// Rows arrive in a ring of SP_RING slots.
// ---------------------------------------------------------------------------
namespace {

constexpr int SPW = 8;              // warps per unit: samples per round, clauses
constexpr uint32_t SP_NT = 32 * SPW;
constexpr uint32_t SP_SC = 4;       // positions a thread examines per scan
constexpr uint32_t SP_FILL = 128;
constexpr uint32_t SP_RING = 32;    // sample rows held: at least two rounds ahead

struct SpecLayout {
  uint32_t planes, ring, list, thr, lev, ovf, misc, total;
};
__host__ __device__ constexpr SpecLayout spec_layout(uint32_t SW, uint32_t ovf_cap) {
  SpecLayout L{};
  uint32_t at = 0;
  auto take = [&](uint32_t bytes) {
    const uint32_t r = at;
    at += (bytes + 15) / 16 * 16;
    return r;
  };
  L.planes = take(8 * 8 * SW * 4);
  L.ring = take(SP_RING * SW * 4);
  L.list = take((SP_FILL + SP_SC * SP_NT) * 4);
  L.thr = take(SP_NT * 8 * 4);
  L.lev = take(4 * 2 * SW * 4);
  L.misc = take(96 * 4);
  L.ovf = take(4 * ovf_cap * 2);
  L.total = at;
  return L;
}

}  // namespace

// misc: [0] unit, [8..39] live counts of a scan, [48..55] overflow counts
// (2 parities x 4), [56..63] literal counts, [64..79] results (2 x 8)
template <int SW, int MINB, bool OV>
__global__ void __launch_bounds__(SP_NT, MINB)
    k_train_spec(const TrainDev *__restrict__ machines, const WorkItem *__restrict__ work,
                 uint32_t nwork, uint32_t *__restrict__ counter, uint32_t e_begin, uint32_t e_end,
                 uint32_t ovf_cap, uint32_t *__restrict__ err) {
  constexpr int NK = SW / 64;       // word pairs per lane
  // Rows above 128 words: while every first sample moves an action, one sample
  // at a time, each warp evaluating its own clause, without a barrier after the
  // update (80 units of 219-word rows 2.24 -> 1.87 ms, 76 encoder units of 191
  // words 4.86 -> 4.14 ms).  In narrower rows eight evaluations cost less than
  // the second exchange (333 units of 44 words 6.7 ms, 7.3 ms this way).
  constexpr bool ALONE = NK >= 4;
  constexpr uint32_t FULL = 0xFFFFFFFFu;
  // rows a round may need were issued two rounds before it
  constexpr uint32_t R = SP_RING;
  constexpr int AHEAD = 1;
  extern __shared__ __align__(128) uint8_t smem[];
  const SpecLayout o = spec_layout(SW, ovf_cap);
  uint32_t *planes = (uint32_t *)(smem + o.planes);  // [clause][count planes 0..6, action][SW]
  uint32_t *ring = (uint32_t *)(smem + o.ring);
  uint32_t *list = (uint32_t *)(smem + o.list);
  int32_t *thr = (int32_t *)(smem + o.thr);
  uint32_t *lev = (uint32_t *)(smem + o.lev);
  uint16_t *ovf = (uint16_t *)(smem + o.ovf);
  uint32_t *misc = (uint32_t *)(smem + o.misc);
  uint32_t *lits = misc + 56, *res = misc + 64;
  const uint32_t tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const uint32_t cl = lane & 7;  // lane c decides clause c
  const int32_t sign = lane < 8 ? ((lane & 1) ? -1 : 1) : 0;
  const uint32_t jbit = 1u << warp;
  uint32_t *own = planes + warp * (8 * SW) + 2 * lane;  // this warp's clause, this lane's words
  for (uint32_t i = tid; i < 8 * SW; i += SP_NT) lev[i] = 0;
  if (tid < 8) misc[48 + tid] = 0;
  uint32_t par = 0, opar = 0, win = SPW;

  while (true) {
    if (tid == 0) {
      // the next unit, passing over those of machines whose gate is closed
      uint32_t u = atomicAdd(counter, 1u);
      while (u < nwork) {
        const uint32_t *gt = machines[work[u].m].gate;
        if (!gt || *gt) break;
        u = atomicAdd(counter, 1u);
      }
      misc[0] = u;
    }
    __syncthreads();
    const uint32_t u = misc[0];
    if (u >= nwork) break;
    const WorkItem wi = work[u];
    const TrainDev &M = machines[wi.m];
    const ClassDev C = M.cls[wi.h];
    const uint32_t Wp = C.Wp, W = C.W;
    const uint32_t g = wi.h * M.clause_chunks + wi.k;
    uint32_t *gact = M.act + C.act_off + ((uint64_t)wi.k * 8 + warp) * Wp + 2 * lane;
    uint32_t *gcnt = M.cnt + C.cnt_off + ((uint64_t)wi.k * 8 + warp) * M7 * Wp + 2 * lane;
    // masks of this lane's words: only a row's last word and the words past
    // it have masks other than all ones
    uint32_t vm[NK][2], em[NK][2], am[NK][2];
#pragma unroll
    for (int k = 0; k < NK; k++)
#pragma unroll
      for (int q = 0; q < 2; q++) {
        const uint32_t w = 64 * k + 2 * lane + q;
        vm[k][q] = word_mask(w, W, C.vmask);
        em[k][q] = word_mask(w, W, C.emask);
        am[k][q] = word_mask(w, W, C.amask);
      }
    // ---- the unit's automata onto the SM: warp j loads clause j ---------------
    auto recount = [&]() {  // literal count of this warp's clause
      uint32_t l = 0;
#pragma unroll
      for (int k = 0; k < NK; k++) {
        const uint2 a = *(const uint2 *)(own + M7 * SW + 64 * k);
        l += __popc(a.x & em[k][0]) + __popc(a.y & em[k][1]);
      }
      l = __reduce_add_sync(FULL, l);
      if (lane == 0) lits[warp] = l;
      if (ALONE) __syncwarp();
    };
#pragma unroll
    for (int k = 0; k < NK; k++) {
      const bool mine = 64 * k + 2 * lane < Wp;
#pragma unroll
      for (int b = 0; b < 8; b++) {
        uint2 t = make_uint2(0, 0);
        if (mine) t = *(const uint2 *)((b < M7 ? gcnt + b * Wp : gact) + 64 * k);
        *(uint2 *)(own + b * SW + 64 * k) = t;
      }
    }
    recount();
    __syncthreads();
    const uint32_t tol = M.tol, maxlit = M.maxlit, ib = M.ib, n = M.n, type = M.type;
    const uint64_t seed = M.seed;
    const uint32_t npk = C.s_picks, nq = (npk + 3) >> 2, input_bits = C.input_bits;
    const uint32_t ep_end = e_end < M.epochs ? e_end : M.epochs;
    const uint32_t *xbase = M.x + C.x_off;
    uint64_t nsteps = 0;

    for (uint32_t e = e_begin; e < ep_end; e++) {
      const uint32_t ee = M.epoch_base + e;
      const uint32_t *perm = M.perm + (uint64_t)(e - e_begin) * n;
      uint32_t at = 0;  // next position of the epoch order
      while (at < n) {
        // ---- the next samples this unit trains on, in order -------------------
        uint32_t cnt = 0;
        while (at < n && cnt < SP_FILL) {
          uint32_t s[SP_SC], y[SP_SC], bal[SP_SC];
#pragma unroll
          for (uint32_t j = 0; j < SP_SC; j++) {
            const uint32_t i = at + j * SP_NT + tid;
            s[j] = i < n ? perm[i] : FULL;
          }
#pragma unroll
          for (uint32_t j = 0; j < SP_SC; j++) {
            y[j] = 0;
            if (s[j] != FULL) {
              if (type == 0) y[j] = (uint32_t)M.labels[s[j]] == wi.h;
              else y[j] = (M.codes[(uint64_t)s[j] * M.code_bytes + (wi.h >> 3)] >> (wi.h & 7)) & 1u;
            }
          }
#pragma unroll
          for (uint32_t j = 0; j < SP_SC; j++) {
            bool live = s[j] != FULL;
            if (live && type == 0 && !y[j]) {
              uint32_t r[4];
              draw4(s[j], ee, g, ST_NEG, seed, r);
              live = (uint64_t)r[0] >= M.thr_neg;
            }
            bal[j] = __ballot_sync(FULL, live);
            if (lane == 0) misc[8 + j * SPW + warp] = __popc(bal[j]);
          }
          __syncthreads();
          const uint32_t here = misc[8 + lane];  // SP_SC * SPW = 32 counts
#pragma unroll
          for (uint32_t j = 0; j < SP_SC; j++) {
            const uint32_t before = __reduce_add_sync(FULL, lane < j * SPW + warp ? here : 0);
            if ((bal[j] >> lane) & 1u)
              list[cnt + before + __popc(bal[j] & ((1u << lane) - 1u))] = s[j] | (y[j] << 31);
          }
          cnt += __reduce_add_sync(FULL, here);
          at += SP_SC * SP_NT;
          __syncthreads();
        }
        nsteps += cnt;
        // rows [from, to) of the list into their ring slots, by all threads
        auto fetch = [&](uint32_t from, uint32_t to) {
          constexpr uint32_t TR = NK >= 4 ? 32 : 16;  // threads per row
          const uint32_t q4 = Wp >> 2;
          for (uint32_t a = from + tid / TR; a < to; a += SP_NT / TR) {
            const uint32_t *src = xbase + (uint64_t)(list[a] & 0x7FFFFFFFu) * Wp;
            uint32_t *dst = ring + (a % R) * SW;
            for (uint32_t q = tid % TR; q < q4; q += TR) cp_async_words<16>(dst + 4 * q, src + 4 * q);
          }
          cp_commit();
        };
        uint32_t fetched = cnt < R ? cnt : R;
        fetch(0, fetched);
        for (uint32_t g0 = 0; g0 < cnt; g0 += SP_NT) {
          if (g0) __syncthreads();
          if (g0 + tid < cnt) vote_thresholds(list[g0 + tid], ee, g, M.T, seed, thr + tid * 8);
          if (!g0) cp_wait<0>();
          __syncthreads();
          const uint32_t ge = cnt - g0 < SP_NT ? cnt : g0 + SP_NT;
          for (uint32_t b = g0; b < ge;) {
            const uint32_t be = b + win < ge ? b + win : ge;  // the round's end
            // what sample a does (lane c holds clause c's vote, `few` if its
            // literals may grow): Type Ib clauses (capi.c:181-190), Type Ia and
            // II << 8, Type Ia increments << 16
            auto decide = [&](uint32_t a, int32_t vote, bool few) -> uint32_t {
              const bool pa = list[a] >> 31;
              const int32_t tc = thr[(a - g0) * 8 + cl];
              const int32_t v = (int32_t)__reduce_add_sync(FULL, (uint32_t)(vote * sign));
              const uint32_t fm = __ballot_sync(FULL, (pa ? v : -v) < tc) & 0xFFu;
              if (!fm) return 0;
              const uint32_t vt = __ballot_sync(FULL, vote > 0);
              const uint32_t inc = __ballot_sync(FULL, few);
              const uint32_t t1 = pa ? 0x55u : 0xAAu;  // Type I clauses
              return (fm & t1 & ~vt) | (fm & vt) << 8 | (fm & vt & t1 & inc & 0xFFu) << 16;
            };
            // votes (capi.c:110-118), signed by clause parity (:148-161)
            auto votes = [&](uint32_t L, uint32_t F) {
              const int32_t vote = (int32_t)(L == 0 || L > tol ? tol : L) - (int32_t)F;
              return vote < 0 ? 0 : vote;
            };
            uint32_t rs;  // lane w: what the round's sample w does
            const bool alone = ALONE && win == 1;
            if (alone) {
              // ---- one sample, each warp its own clause ---------------------------
              const uint32_t *xs = ring + (b % R) * SW + 2 * lane;
              uint32_t f = 0;
#pragma unroll
              for (int k = 0; k < NK; k++) {
                const uint2 x = *(const uint2 *)(xs + 64 * k);
                const uint2 t = *(const uint2 *)(own + M7 * SW + 64 * k);
                f += __popc(t.x & em[k][0] & ~x.x) + __popc(t.y & em[k][1] & ~x.y);
              }
              f = __reduce_add_sync(FULL, f);
              const uint32_t L = lits[warp];
              if (lane == 0)
                res[par * SPW + warp] = (uint32_t)votes(L, f) | (L <= maxlit ? 0x80000000u : 0u);
              cp_wait<AHEAD>();
              __syncthreads();
              const uint32_t rv = res[par * SPW + cl];
              const uint32_t r = decide(b, (int32_t)(rv & 0x7FFFFFFFu), rv >> 31);
              rs = cl == 0 ? r : 0;
            } else {
              // ---- this warp's sample of the round --------------------------------
              const uint32_t a = b + warp;
              uint32_t r = 0;
              if (a < be) {
                const uint32_t L = lits[cl];
                const uint32_t *xs = ring + (a % R) * SW + 2 * lane;
                uint32_t f[8] = {};
#pragma unroll
                for (int k = 0; k < NK; k++) {
                  uint2 x = *(const uint2 *)(xs + 64 * k);
                  x.x |= ~em[k][0];
                  x.y |= ~em[k][1];
#pragma unroll
                  for (int c = 0; c < 8; c++) {
                    const uint2 t =
                        *(const uint2 *)(planes + (c * 8 + M7) * SW + 2 * lane + 64 * k);
                    f[c] += __popc(t.x & ~x.x) + __popc(t.y & ~x.y);
                  }
                }
                uint32_t pk[4];
#pragma unroll
                for (int c = 0; c < 4; c++)
                  pk[c] = __reduce_add_sync(FULL, f[2 * c] + (f[2 * c + 1] << 16));
                const uint32_t pr =
                    (lane & 4) ? ((lane & 2) ? pk[3] : pk[2]) : ((lane & 2) ? pk[1] : pk[0]);
                r = decide(a, votes(L, (lane & 1) ? pr >> 16 : pr & 0xFFFFu), L <= maxlit);
              }
              if (lane == 0) res[par * SPW + warp] = r;
              cp_wait<AHEAD>();
              __syncthreads();
              rs = res[par * SPW + cl];
            }
            // rows behind this round are done with: refill their slots, eight at
            // a time while the rounds are single samples (a round that grows from
            // one sample reaches at most 15 rows within the two rounds that its
            // copies may take)
            if (!alone || b + R - fetched >= 8) {
              const uint32_t to = cnt - b < R ? cnt : b + R;
              fetch(fetched, to);
              fetched = to;
            } else {
              cp_commit();
            }
            // ---- feedback of the round's samples, in order -----------------------
            par ^= 1u;
            bool moved = false;
            uint32_t next = be;
            for (uint32_t pend = __ballot_sync(FULL, rs != 0) & 0xFFu; pend; pend &= pend - 1) {
              const uint32_t w = __ffs(pend) - 1;
              const uint32_t rw = __shfl_sync(FULL, rs, w);
              const uint32_t ent = list[b + w];
              const uint32_t ibm = rw & 0xFFu, fbm = (rw >> 8) & 0xFFu, incm = rw >> 16;
              const uint32_t t1 = (ent >> 31) ? 0x55u : 0xAAu;
              uint32_t *oc = misc + 48 + opar * 4;
              if (ibm) {
                draw_picks<SP_NT, SW>(ibm, ent & 0x7FFFFFFFu, ee, g, seed, npk, nq, input_bits, lev,
                                      ovf, oc, ovf_cap);
                __syncthreads();
                opar ^= 1u;
                if (tid < 4) misc[48 + opar * 4 + tid] = 0;  // for the next pass with picks
              }
              if ((ibm | fbm) & jbit) {
                const bool is1 = (t1 & jbit) != 0, incx = (incm & jbit) != 0;
                const uint32_t slot = __popc(ibm & (jbit - 1u));
                const uint32_t *xs = ring + ((b + w) % R) * SW + 2 * lane;
                // nonzero if the clause's actions may move.  Those of a Type Ia clause
                // without increments do not: other warps may be reading them for the
                // next round, so they are not written
                const uint32_t act_moves = ((ibm | incm | ~t1) & jbit) | (ib - 1u);
#pragma unroll 1
                for (int k = 0; k < NK; k++) {
                  uint32_t p[M7][2], ac[2], x[2], mv[2], ma[2];
#pragma unroll
                  for (int bb = 0; bb < M7; bb++) WVec<2>::ld(own + bb * SW + 64 * k, p[bb]);
                  WVec<2>::ld(own + M7 * SW + 64 * k, ac);
                  WVec<2>::ld(xs + 64 * k, x);
#pragma unroll
                  for (int q = 0; q < 2; q++) {
                    if (NK == 1) {
                      mv[q] = vm[0][q];
                      ma[q] = am[0][q];
                    } else {
                      mv[q] = word_mask(64 * k + 2 * lane + q, W, C.vmask);
                      ma[q] = word_mask(64 * k + 2 * lane + q, W, C.amask);
                    }
                  }
                  if (ibm & jbit) {
                    uint32_t *l0 = lev + slot * (2 * SW) + 2 * lane + 64 * k, *l1 = l0 + SW;
                    uint32_t m0[2], m1[2];
                    const uint32_t zero[2] = {};
                    WVec<2>::ld(l0, m0);
                    WVec<2>::ld(l1, m1);
                    WVec<2>::st(l0, zero);
                    WVec<2>::st(l1, zero);
                    // an overflow entry is worth 4: twice a level-1 count
                    if constexpr (OV) {
                      const uint32_t no = min(oc[slot], ovf_cap);
                      uint32_t next = lane;  // this lane's next entry
                      for (uint32_t t = 0;; t++) {
                        count_sub(p, ac, m0, m1, ma);
                        if (t & 1u) continue;
                        if (!__any_sync(FULL, next < no)) break;
                        take_overflow(ovf + slot * ovf_cap, no, next, 64 * k, 64,
                                      lev + slot * (2 * SW) + SW);
                        WVec<2>::ld(l1, m1);
                        WVec<2>::st(l1, zero);
                        m0[0] = m0[1] = 0;
                      }
                    } else {
                      const uint32_t no = 2 * min(oc[slot], ovf_cap);
                      for (uint32_t t = 0;; t++) {
                        count_sub(p, ac, m0, m1, ma);
                        if (t >= no) break;
                        const uint32_t bit = ovf[slot * ovf_cap + (t >> 1)];
#pragma unroll
                        for (int q = 0; q < 2; q++) {
                          m0[q] = 0;
                          m1[q] = (bit >> 5) == 64 * k + 2 * lane + q ? 1u << (bit & 31) : 0u;
                        }
                      }
                    }
                  } else {
                    // Type Ia (capi.c:177-180): inc where x = 1 (if L <=
                    // maximum), dec where x = 0 and not included.  Type II
                    // (capi.c:192-196): inc where x = 0 and not included.
                    uint32_t c0[2], dm[2];
#pragma unroll
                    for (int q = 0; q < 2; q++) {
                      const uint32_t nx = ~(x[q] | included(p, ac[q], q, ib)) & mv[q];
                      c0[q] = nx | (incx ? x[q] & mv[q] : 0u);
                      dm[q] = is1 ? nx : 0u;
                    }
                    count_step(p, ac, c0, dm, ma);
                  }
#pragma unroll
                  for (int bb = 0; bb < M7; bb++) WVec<2>::st(own + bb * SW + 64 * k, p[bb]);
                  if (act_moves) WVec<2>::st(own + M7 * SW + 64 * k, ac);
                }
              }
              if (ibm || incm || (fbm & ~t1) || ib > 1) {
                // an action may have moved: the later results no longer hold
                if ((ibm | fbm) & jbit) recount();
                next = b + w + 1;
                moved = true;
                if (!alone) __syncthreads();  // alone, a warp reads its own clause only
                break;
              }
            }
            // a round that ended early is followed by one that little longer
            // (evaluations thrown away take issue slots from other units), in
            // the ALONE form by one sample if its first one ended it; a full
            // one by one of twice its length
            const uint32_t done = next - b;
            const uint32_t grown = ALONE && moved && done == 1 ? 1
                                   : (next < be ? done + 1 : 2 * win);
            win = grown < SPW ? grown : SPW;
            b = next;
          }
        }
        cp_wait<0>();
        __syncthreads();
      }
    }
    // ---- the unit's automata back to global memory ----------------------------
#pragma unroll
    for (int k = 0; k < NK; k++) {
      if (64 * k + 2 * lane >= Wp) continue;
#pragma unroll
      for (int b = 0; b < 8; b++)
        *(uint2 *)((b < M7 ? gcnt + b * Wp : gact) + 64 * k) = *(const uint2 *)(own + b * SW + 64 * k);
    }
    if (tid == 0 && nsteps) atomicAdd((unsigned long long *)(err + 2), (unsigned long long)nsteps);
    __syncthreads();
  }
}

// ---- configurations ----------------------------------------------------------
// id (1-based).  k_train_wpt: W(threads per unit, words per thread, words
// per row slot, count planes in registers, count planes in global memory,
// Type Ib slots, CTAs per SM the registers are sized for); k_train_spec:
// S(words per row slot, CTAs per SM).
// Rows of up to 64 words keep every plane in shared memory (search rows: 26.2
// ms; with three planes in L2 and 16 units per SM 30.7).  Wider rows leave
// their count planes in L2, where the resident units' planes fit: the units
// that shared memory then holds hide more latency than the planes cost
// (256-word rows: 10 units of two warps 112 ms, 4 units of four warps with
// four planes in registers 156 ms; 128 words 37 / 51 ms; 512 words 53 / 71 ms;
// 1,024 words, two units with one plane in registers 90 ms, one unit with
// three 105 ms).
#define TM_WPT_CONFIGS(W, S)      \
  W(1, 256, 4, 1024, 1, 6, 4, 2)  \
  S(2, 256, 1)                    \
  W(3, 128, 4, 512, 0, 7, 2, 5)   \
  W(4, 64, 4, 256, 0, 7, 2, 10)   \
  S(5, 64, 3)                     \
  W(6, 32, 2, 64, 0, 0, 4, 16)    \
  W(7, 32, 2, 56, 0, 0, 4, 16)    \
  W(8, 32, 1, 32, 0, 0, 4, 20)    \
  S(9, 128, 2)                    \
  W(10, 32, 4, 128, 0, 7, 2, 20)  \
  W(11, 32, 2, 48, 0, 0, 4, 16)   \
  W(12, 32, 1, 24, 0, 0, 4, 20)

struct WptConfig {
  int id;
  bool spec;  // k_train_spec, else k_train_wpt
  int nt, sw, off;  // off: count planes not in shared memory
  int ibs;
};
static constexpr WptConfig kWpt[] = {
#define TM_W(ID, NT, WPT, SW, RP, GP, IBS, MINB) {ID, false, NT, SW, RP + GP, IBS},
#define TM_S(ID, SW, MINB) {ID, true, (int)SP_NT, SW, 0, 4},
    TM_WPT_CONFIGS(TM_W, TM_S)
#undef TM_W
#undef TM_S
};
constexpr int kWptCount = (int)(sizeof(kWpt) / sizeof(kWpt[0]));
constexpr bool wpt_in_order() {
  for (int i = 0; i < kWptCount; i++)
    if (kWpt[i].id != i + 1) return false;
  return true;
}
static_assert(wpt_in_order(), "a configuration's place is its id");

// The configuration that a launch of rows of at most Wpmax words runs for `id`:
// 7 serves rows of up to 64 words to callers that pin it, those above its own
// slots in the 64-word ones of 6.
static int wpt_slot(int id, uint32_t Wpmax) { return id == 7 && Wpmax > 56 ? 6 : id; }

static uint32_t wpt_ovf_cap(uint32_t smax) { return smax / 4 > 0 ? smax / 4 : 1; }

double wpt_overflow(uint32_t bits, uint32_t picks) {
  if (!bits) return 0.0;
  const double l = (double)picks / bits;
  return bits * (1.0 - exp(-l) * (1.0 + l + l * l / 2 + l * l * l / 6));
}

static size_t wpt_bytes(const WptConfig &k, uint32_t smax) {
  const uint32_t oc = wpt_ovf_cap(smax);
  return k.spec ? spec_layout(k.sw, oc).total
                : wpt_layout(k.nt, k.sw, k.off, k.ibs, oc).total;
}

template <class F>
static int wpt_occ(F kernel, int threads, size_t bytes) {
  raise_smem((const void *)kernel);
  int nb = 0;
  cudaOccupancyMaxActiveBlocksPerMultiprocessor(&nb, kernel, threads, bytes);
  return nb;
}

template <bool OV>
static int config_occ(int id, size_t bytes) {
  switch (id) {
#define TM_W(ID, NT, WPT, SW, RP, GP, IBS, MINB) \
  case ID: return wpt_occ(k_train_wpt<NT, WPT, SW, RP, GP, IBS, MINB, OV>, NT, bytes);
#define TM_S(ID, SW, MINB) \
  case ID: return wpt_occ(k_train_spec<SW, MINB, OV>, SP_NT, bytes);
    TM_WPT_CONFIGS(TM_W, TM_S)
#undef TM_W
#undef TM_S
  }
  return 0;
}

// Resident CTAs (units) per SM of configuration `id` for rows of at most
// Wpmax words (0 when it cannot hold them), and its shared memory.
int train_wpt_occupancy(int id, uint32_t Wpmax, uint32_t smax, bool many_ovf, size_t *smem_bytes) {
  if (id < 1 || id > kWptCount) return 0;
  id = wpt_slot(id, Wpmax);
  const WptConfig &k = kWpt[id - 1];
  if (Wpmax > (uint32_t)k.sw) return 0;
  const size_t bytes = wpt_bytes(k, smax);
  *smem_bytes = bytes;
  return many_ovf ? config_occ<true>(id, bytes) : config_occ<false>(id, bytes);
}

// The configurations worth a launch of `units` units on `sms` SMs, rows of at
// most Wpmax words (ids, best guess first; 0 to `max` of them).
//   k_train_wpt with the smallest row slot that holds the rows: smaller slots
//     hold more units per SM (rows of 49 words: 26.2 ms in 56-word slots,
//     27.5 ms in 64-word ones).
//   Up to 6 units per SM also:
//   k_train_spec for rows up to 256 words: with few units the chain of one
//     unit's samples is what takes the time (plain classifier, 320 units: 2.8 ms
//     against 6.6 ms), with many the evaluations it throws away (search rows,
//     15,000 units: 67.8 against 25.7 ms).
//   k_train_wpt with the next larger slot, whose units have twice the threads to
//     scan and to draw with (four words per thread, so for rows above 64 words:
//     encoder rows of 94 words, specificity 4, 800 units 35.3 ms with the two
//     choices above, 26.4 ms in 256-word slots; 4,800 units 18.2 against 24.5 ms
//     at specificity 5).
int wpt_choices(uint32_t Wpmax, uint32_t smax, uint32_t units, int sms, int optin, int *ids,
                int max) {
  auto smallest = [&](bool spec, int threads) {
    int best = 0;
    for (int id = 1; id <= kWptCount; id++) {
      const WptConfig &k = kWpt[id - 1];
      if (k.spec != spec || k.nt < threads || Wpmax > (uint32_t)k.sw) continue;
      if (wpt_bytes(k, smax) > (size_t)optin) continue;
      if (best && kWpt[best - 1].sw <= k.sw) continue;
      best = id;
    }
    return best;
  };
  const int first = smallest(false, 0);
  int pick[3] = {first, 0, 0}, n = 0;
  if (units <= 6u * (uint32_t)sms) {
    pick[1] = smallest(true, 0);
    if (first && Wpmax > 64) pick[2] = smallest(false, kWpt[first - 1].nt + 1);
  }
  for (int id : pick)
    if (id && n < max) ids[n++] = id;
  return n;
}

template <bool OV>
static void config_launch(int id, int grid, size_t bytes, cudaStream_t st,
                          const TrainDev *machines, const WorkItem *work, uint32_t nwork,
                          uint32_t *counter, uint32_t e_begin, uint32_t e_end, uint32_t ovf_cap,
                          uint32_t *err) {
  switch (id) {
#define TM_W(ID, NT, WPT, SW, RP, GP, IBS, MINB)                                 \
  case ID:                                                                       \
    k_train_wpt<NT, WPT, SW, RP, GP, IBS, MINB, OV><<<grid, NT, bytes, st>>>(    \
        machines, work, nwork, counter, e_begin, e_end, ovf_cap, err);           \
    break;
#define TM_S(ID, SW, MINB)                                                       \
  case ID:                                                                       \
    k_train_spec<SW, MINB, OV><<<grid, SP_NT, bytes, st>>>(                      \
        machines, work, nwork, counter, e_begin, e_end, ovf_cap, err);           \
    break;
    TM_WPT_CONFIGS(TM_W, TM_S)
#undef TM_W
#undef TM_S
  }
}

cudaError_t launch_train_wpt(int id, const TrainDev *machines, const WorkItem *work,
                             uint32_t nwork, uint32_t *counter, uint32_t e_begin, uint32_t e_end,
                             uint32_t Wpmax, uint32_t smax, bool many_ovf, int grid, uint32_t *err,
                             cudaStream_t st) {
  if (id < 1 || id > kWptCount) return cudaErrorInvalidValue;
  id = wpt_slot(id, Wpmax);
  if (Wpmax > (uint32_t)kWpt[id - 1].sw) return cudaErrorInvalidValue;
  const size_t bytes = wpt_bytes(kWpt[id - 1], smax);
  (many_ovf ? config_launch<true> : config_launch<false>)(id, grid, bytes, st, machines, work, nwork,
                                                          counter, e_begin, e_end,
                                                          wpt_ovf_cap(smax), err);
  return cudaGetLastError();
}

}  // namespace tmb
