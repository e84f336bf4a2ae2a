// canon_sparse.cuh -- one warp canonizes one graph of any size (n <= 65536).
//
// Same search as canon_warp64.cuh -- the reference's sequential DFS
// (src/sequential.cpp:216-670) step for step, bit-exact in canonical form,
// stored automorphisms and node count -- with data structures whose cost
// follows the work a step does rather than n:
//
//   * the ordered partition is elem[] / pos[] plus a two-level bitmap of cell
//     start positions; a vertex's cell is the last start at or before its
//     position, so splitting a cell only sets bits and swaps the moved
//     vertices, and backtracking (reconstruct_at_level) only clears bits;
//   * a refinement step touches only the neighbours of the splitter: counts
//     go to cnt[], touched vertices are grouped per cell by a counting sort,
//     and each split cell is rearranged by pairing its misplaced vertices
//     with the holes of the target region -- O(touched), the work nauty does;
//   * a leaf certificate is, per vertex, the sorted canonical positions of
//     its neighbours (O(m) words), compared row by row in canonical order
//     exactly like the upper-triangle compare (sequential.cpp:114-124);
//   * the target cell of a level is not stored: when the search is back at
//     that level the partition is the same, so its members are the cell at
//     the stored start position; orbit representatives live in a stack with
//     an entry per member, pushed when orbits first change at a level.  (With
//     an array of n per level, trees of more than 32 levels outgrew the first
//     pass and were searched twice: 45 of 48 trees of 257 to 1,000 vertices.)
//
// All state lives in a per-warp slot of device memory; the warp's pointers
// and scalars live in shared memory.  Each phase is one non-inlined function.
//
// A refinement step is a chain of dependent loads, so what bounds the kernel is
// the latency of one warp and, for the many-warp search, how many warps' state
// fits in shared memory.  Positions and vertices are 16-bit (n <= 65536), and a
// cell's level is not kept (see the log of cell starts): 6.5 bytes per vertex
// where 32-bit arrays with in_level took 16.4, so a graph of 4,096 vertices fits an
// SM's shared memory 8 times instead of 3.  When they were made, both changes took
// a batch of mixed graphs up to 256 vertices from 478 to 430 ms.
#pragma once
#include <cstdint>

#include "canon_warp64.cuh"
#include "gcl_device.cuh"

namespace gcl {

constexpr int kSpThreads = 128;
constexpr int kSpWarps = kSpThreads / 32;
constexpr uint32_t kNone = 0xffffffffu;

struct SpTc {
  uint32_t first, len, counter;
  int32_t last;   // last_num_aut_at_level
  uint32_t rslot;  // this level's representatives in W.reps, kNone = all v are reps
  uint32_t pad;
};

// Byte layout of one slot for graphs with at most n vertices and m2 CSR
// entries, representatives of `pool` target cells of n vertices (a target
// cell takes as many entries as it has vertices, so sparse searches reach far
// deeper), `cap` ring slots, and the fix state of `fixcap` entries of a shared
// store.
struct SpLayout {
  uint64_t u32n[13];  // offsets of the n-sized u32 arrays
  uint64_t elem, pos, cnt;
  uint64_t fcode, ccode, pool_owner;
  uint64_t stb, sts, act, itm, nsb;
  uint64_t fcert, bcert, ccert;
  uint64_t tc, reps, auts, fixm, fixst;
  uint32_t fixcap, reps_cap;
  uint64_t bytes;
  uint32_t nw, nsw;
  uint32_t stride;  // elements per representative array / ring entry
};

// 32-bit words of a bitmap over n positions that is read four words at a time
__host__ __device__ inline uint32_t sp_pad_words(uint32_t n) {
  return ((n + 31) / 32 + 3) & ~3u;
}

__host__ __device__ inline SpLayout sp_layout(uint32_t n, uint64_t m2, uint32_t pool,
                                              uint32_t cap, uint32_t fixcap = 0) {
  SpLayout L{};
  uint64_t o = 0;
  auto take = [&](uint64_t bytes) {
    const uint64_t at = o;
    o = (o + bytes + 255u) & ~255ull;
    return at;
  };
  const uint64_t N1 = (uint64_t)n + 2;
  L.stride = (uint32_t)N1;
  // (256 entries at least: the colour sort's histogram)
  for (int i = 0; i < 13; ++i) L.u32n[i] = take(4 * (N1 < 256 ? 256 : N1));
  L.elem = take(2 * N1);
  L.pos = take(2 * N1);
  L.cnt = take(2 * N1);
  L.fcode = take(4 * (N1 + 1));
  L.ccode = take(4 * (N1 + 1));
  L.pool_owner = take(4 * N1);
  L.nw = (n + 63) / 64 + 1;
  L.nsw = (L.nw + 63) / 64 + 1;
  L.stb = take(8ull * L.nw);
  L.sts = take(8ull * L.nsw);
  const uint64_t wp = sp_pad_words(n);
  L.act = take(4 * wp);
  L.itm = take(4 * wp);
  L.nsb = take(4 * wp);
  L.fcert = take(4 * (m2 + 1));
  L.bcert = take(4 * (m2 + 1));
  L.ccert = take(4 * (m2 + 1));
  L.tc = take(sizeof(SpTc) * N1);
  // the target cells of a path, each a part of the one before or of the rest,
  // have at most n + (n - 1) + ... vertices
  const uint64_t all = N1 * (N1 + 1) / 2;
  L.reps_cap = (uint32_t)(pool * N1 < all ? pool * N1 : all);
  L.reps = take(4ull * L.reps_cap);
  L.auts = take(2ull * cap * N1);
  L.fixm = take(4ull * ((cap + 31) / 32) * N1);
  L.fixcap = fixcap;
  L.fixst = take(8ull * fixcap);
  L.bytes = o;
  return L;
}

// Shared-memory staging: the arrays every refinement step touches (elem, pos,
// neighbour counts by position, the start bitmap with its summary, the active
// cells, the marks of the hash) live in the warp's shared-memory region
// when they fit.  elem lies at offset 0.
struct SpStage {
  uint32_t pos, cnt, stb, sts, act, itm, nsb, bytes;
};
__host__ __device__ inline SpStage sp_stage(uint32_t n) {
  const uint32_t nw = (n + 63) / 64 + 1, nsw = (nw + 63) / 64 + 1;
  const uint32_t a = ((n + 2) * 2u + 15) & ~15u;
  SpStage G{};
  G.pos = a;
  G.cnt = 2 * a;
  G.stb = 3 * a;
  G.sts = G.stb + 8 * nw;
  G.act = (G.sts + 8 * nsw + 15) & ~15u;
  G.itm = G.act + 4 * sp_pad_words(n);
  G.nsb = G.itm + 4 * sp_pad_words(n);
  G.bytes = G.nsb + 4 * sp_pad_words(n);
  return G;
}
__host__ __device__ inline uint64_t sp_smem_bytes(uint32_t n) { return sp_stage(n).bytes; }
extern __shared__ __align__(16) uint8_t sp_dyn[];

struct SpWarp {
  uint16_t *elem, *pos;  // position -> vertex, vertex -> position (n <= 65536)
  uint16_t* cnt;         // position -> neighbours in the splitter, zero between steps
  // a block whose other warps count for this one (the first path): the
  // splitter's positions, equal to end them
  uint32_t helpers, job_s, job_e;
  uint32_t soff;         // the warp's shared-memory region (offset in sp_dyn), or kNone
  uint32_t *slog, *tmp, *lst1, *hist, *pre;
  uint32_t *seq, *fseq, *bseq, *flabel, *blabel, *dsu;
  int32_t *fcode, *ccode, *pool_owner, *pathcode;
  uint32_t *umark;  // per level: start-log size when the level's child was made
  uint2* fixst;     // per stored automorphism: {prefix of seq it fixes, first
                    // position of seq it moves or kNone}, valid for the path
  uint64_t *stb, *sts;         // cell starts (position n too) and their summary
  uint32_t *act, *itm, *nsb;   // active cells; marks of the hash: touched fragments,
                               // fragment starts (sp_pad_words words each)
  uint32_t *fcert, *bcert, *ccert;
  uint32_t* reps;   // stack of target cells' {vertex, representative << 16}
  uint32_t* fixm;   // per vertex: a bit per ring entry that fixes it
  uint32_t fixw;    // words of a vertex's row in fixm
  SpTc* tc;
  uint16_t* auts;
  const int32_t* rp;
  const int32_t* col;
  uint32_t n, nw, nsw, stride;  // stride: elements per pool / ring entry
  uint32_t ncells, nact;
  uint32_t pool_top, pool_frames, pool_cap, aut_cap, max_aut;
  uint32_t scr[32];  // a word per lane: the union-find of a small target cell
  alignas(16) uint16_t list[256];  // items of a hash
  uint32_t utop;  // entries of slog
  uint32_t fixcap;  // store entries whose fix state is kept (later ones are checked in full)
};

__shared__ SpWarp g_sp[kSpWarps];

// Loads of data that warps on other SMs write during the same launch (the
// shared automorphism store and best leaf of the many-warp search) go
// through L2 only; everything else uses ordinary loads.
template <bool kCg, typename T>
__device__ __forceinline__ T ldx(const T* p) {
  if constexpr (kCg) return __ldcg(p);
  else return *p;
}
__device__ __forceinline__ SpWarp& sp_w() { return g_sp[threadIdx.x >> 5]; }

// ---- bitmaps with a summary word per 64 words ----------------------------
// smallest set position >= p, or n
__device__ __noinline__ uint32_t bm_next(const uint64_t* B, const uint64_t* Sm, uint32_t p, uint32_t n,
                            uint32_t nw, uint32_t nsw) {
  if (p >= n) return n;
  uint32_t w = p >> 6;
  const uint64_t x = B[w] & ge_mask(p & 63);
  if (x) return min(n, w * 64 + ctz64(x));
  ++w;
  if (w >= nw) return n;
  uint32_t sw = w >> 6;
  uint64_t y = Sm[sw] & ge_mask(w & 63);
  while (!y) {
    if (++sw >= nsw) return n;
    y = Sm[sw];
  }
  const uint32_t w2 = sw * 64 + ctz64(y);
  if (w2 >= nw) return n;
  return min(n, w2 * 64 + ctz64(B[w2]));
}
// largest set position <= p, or kNone
__device__ __noinline__ uint32_t bm_prev(const uint64_t* B, const uint64_t* Sm, uint32_t p) {
  uint32_t w = p >> 6;
  const uint64_t x = B[w] & low_mask((p & 63) + 1);
  if (x) return w * 64 + msb64(x);
  if (w == 0) return kNone;
  --w;
  uint32_t sw = w >> 6;
  uint64_t y = Sm[sw] & low_mask((w & 63) + 1);
  while (!y) {
    if (sw == 0) return kNone;
    y = Sm[--sw];
  }
  const uint32_t w2 = sw * 64 + msb64(y);
  return w2 * 64 + msb64(B[w2]);
}
// single-writer set / clear (summary kept exact)
__device__ __forceinline__ void bm_set1(uint64_t* B, uint64_t* Sm, uint32_t p) {
  B[p >> 6] |= bit64(p & 63);
  Sm[p >> 12] |= bit64((p >> 6) & 63);
}
// warp: rebuild a summary from its bitmap
__device__ void bm_resummarize(const uint64_t* B, uint64_t* Sm, uint32_t nw, uint32_t nsw) {
  const uint32_t lane = lane_id();
  for (uint32_t sw = 0; sw < nsw; ++sw) {
    const uint32_t w0 = sw * 64 + lane, w1 = w0 + 32;
    const bool a = w0 < nw && B[w0] != 0, b = w1 < nw && B[w1] != 0;
    const uint64_t m = ballot2(a, b);
    if (lane == 0) Sm[sw] = m;
  }
  __syncwarp();
}

__device__ __forceinline__ uint32_t sp_cell_end(const SpWarp& W, uint32_t c) {
  const uint32_t* st = (const uint32_t*)W.stb;
  const uint32_t w = c >> 5, x = st[w] & (0xfffffffeu << (c & 31u));
  if (x) return w * 32 + (uint32_t)__ffs((int)x) - 1;
  return bm_next(W.stb, W.sts, (w + 1) * 32, W.n, W.nw, W.nsw);
}
__device__ __forceinline__ uint32_t lanemask_lt() {
  uint32_t m;
  asm("mov.u32 %0, %%lanemask_lt;" : "=r"(m));
  return m;
}

// ---- log of the cell starts --------------------------------------------------
// Every cell start made after the root refinement is logged in order of
// creation, and umark[L] is the log's size when the node of level L got its
// child, so a backtrack to level L clears exactly the starts logged from
// there on.  That is reconstruct_at_level (partition_refinement.cpp:541-604):
// it merges every maximal run of cells created below L with the cell that
// follows it, and a split gives every fragment but the last the new level, so
// the starts that survive are those made at or above L.  The in_level of a
// cell has no other use.  A cell start is made once between two backtracks
// past it, so the log holds at most n entries.  Vertex order inside cells is
// not restored: only cells as sets matter.

// lane 0: new cell start, logged
__device__ __forceinline__ void add_start(SpWarp& W, uint32_t p) {
  W.slog[W.utop++] = p;
  bm_set1(W.stb, W.sts, p);
}

// ---------------------------------------------------------------------------
// The refinement's view of the partition: the arrays and bitmaps every step
// touches, in the warp's shared memory (kS, so the compiler emits shared-memory
// loads and atomics) or in its device-memory slot.
// ---------------------------------------------------------------------------
template <bool kS>
struct SpRef {
  uint16_t *elem, *pos, *cnt;
  uint64_t *stb, *sts;
  uint32_t *st, *act, *itm, *nsb;  // st: stb as 32-bit words
  __device__ __forceinline__ explicit SpRef(const SpWarp& W) {
    if constexpr (kS) {
      const SpStage G = sp_stage(W.n);
      uint8_t* b = sp_dyn + W.soff;
      elem = (uint16_t*)b;
      pos = (uint16_t*)(b + G.pos);
      cnt = (uint16_t*)(b + G.cnt);
      stb = (uint64_t*)(b + G.stb);
      sts = (uint64_t*)(b + G.sts);
      act = (uint32_t*)(b + G.act);
      itm = (uint32_t*)(b + G.itm);
      nsb = (uint32_t*)(b + G.nsb);
    } else {
      elem = W.elem;
      pos = W.pos;
      cnt = W.cnt;
      stb = W.stb;
      sts = W.sts;
      act = W.act;
      itm = W.itm;
      nsb = W.nsb;
    }
    st = (uint32_t*)stb;
  }
  // whether the vertex at position p is alone in its cell: p and p + 1 are
  // starts (position n is marked as one)
  __device__ __forceinline__ bool alone(uint32_t p) const {
    const uint32_t w = p >> 5;
    return (__funnelshift_r(st[w], st[w + 1], p & 31u) & 3u) == 3u;
  }
  __device__ __forceinline__ bool active(uint32_t c) const {
    return (act[c >> 5] >> (c & 31u)) & 1u;
  }
  // the end of the cell of position p, and its start and length: in p's word of
  // 64 starts, else through the summary
  __device__ __forceinline__ uint32_t end_of(uint32_t p, uint32_t n) const {
    const uint32_t w = p >> 6;
    const uint64_t x = stb[w] & (~1ull << (p & 63u));
    if (x) return w * 64 + ctz64(x);
    const uint64_t y = sts[w >> 6] & (~1ull << (w & 63u));
    if (!y) return bm_next(stb, sts, (w + 1) * 64, n, (n + 63) / 64 + 1, ((n + 63) / 64 + 64) / 64 + 1);
    const uint32_t v = (w & ~63u) + ctz64(y);
    return v * 64 + ctz64(stb[v]);
  }
  __device__ __forceinline__ void cell_of(uint32_t p, uint32_t n, uint32_t* c, uint32_t* len) const {
    const uint32_t w = p >> 6;
    const uint64_t x = stb[w] & (~0ull >> (63u - (p & 63u)));
    uint32_t a;
    if (x) {
      a = w * 64 + msb64(x);
    } else {
      const uint64_t y = sts[w >> 6] & (bit64(w & 63u) - 1);
      if (y) {
        const uint32_t v = (w & ~63u) + msb64(y);
        a = v * 64 + msb64(stb[v]);
      } else {
        a = bm_prev(stb, sts, w * 64 - 1);  // position 0 is a start
      }
    }
    *c = a;
    *len = end_of(p, n) - a;
  }
  // the same for n <= 1,024 without a branch: `some` has a bit per word of 32
  // positions that holds a start (lanes of one step lie in cells of all sizes,
  // and the two-way choices above run one after the other)
  __device__ __forceinline__ void cell_of_1k(uint32_t p, uint32_t n, uint32_t some, uint32_t* c,
                                             uint32_t* len) const {
    const uint32_t w = p >> 5, sh = p & 31u, x = st[w];
    const uint32_t lo = x & (0xffffffffu >> (31u - sh)), hi = x & (0xfffffffeu << sh);
    const uint32_t below = some & ((1u << w) - 1u), above = some & (0xfffffffeu << w);
    // words that hold the cell's start (word 0 holds one) and the next one; with
    // none above, the cell ends at n and p's own word is read in its place
    const uint32_t wl = lo || !below ? w : 31u - (uint32_t)__clz((int)below);
    const uint32_t wh = hi || !above ? w : (uint32_t)__ffs((int)above) - 1u;
    const uint32_t y = lo ? lo : st[wl], z = hi ? hi : st[wh];
    const uint32_t a = wl * 32 + 31u - (uint32_t)__clz((int)y);
    const uint32_t e = hi || above ? min(n, wh * 32 + (uint32_t)__ffs((int)z) - 1u) : n;
    *c = a;
    *len = e - a;
  }
};

__device__ __forceinline__ void or_bit32(uint32_t* B, uint32_t p) {
  atomicOr(B + (p >> 5), 1u << (p & 31u));
}
// any lane: set a bit of a two-level bitmap
__device__ __forceinline__ void bm_or(uint64_t* B, uint64_t* Sm, uint32_t p) {
  or_bit32((uint32_t*)B, p);
  or_bit32((uint32_t*)Sm, p >> 6);
}
// starts of the non-singleton cells among positions 32 wi .. 32 wi + 31
__device__ __forceinline__ uint32_t sp_nonsingle_word(const uint64_t* stb, uint32_t n,
                                                      uint32_t wi) {
  const uint32_t* s = (const uint32_t*)stb;
  const uint32_t b = s[wi];
  const uint32_t ns = b & ~((b >> 1) | (s[wi + 1] << 31));
  const uint32_t left = n - wi * 32;  // position n is marked as a start
  return left >= 32 ? ns : ns & ((1u << left) - 1u);
}
// the j-th (from 0) set bit of x, found by clearing the lower ones: j is
// almost always 0 or 1 here, where __fns takes a long search
__device__ __forceinline__ uint32_t nth_bit(uint32_t x, uint32_t j) {
  for (; j; --j) x &= x - 1;
  return (uint32_t)(__ffs((int)x) - 1);
}

// ---------------------------------------------------------------------------
// The invariant hash of a non-singleton splitter (partition_refinement.cpp:
// 253-373): mash folded in position order over one item per fragment start,
// the start plus its vertices' neighbour count (zero unless the position is
// marked in `itm`).  The fragment starts are the old non-singleton cells' and
// the marked positions, or, when `listed`, the bits of `nsb`.
//
// A lane takes kW words of 32 positions.  Up to 256 items are compacted into a
// list and folded one after the other, two instructions each.  More are folded
// one bit of the running value at a time over all positions at once: bit j of
// the value before item i is bit j of the initial value xor the parity of the
// flips of the items before it (a prefix parity within the word, a ballot
// across the lanes), and that gives the carries into bit j + 1.  A position's
// own bits are constants of its word, so no list of cells is built.  Listing
// the cells and taking 15 ballots per 32 of them took 61,700 of a step's 67,600
// cycles on a 64 x 64 torus (about 1,200 cells); with the bit-wise fold the
// search of that torus took 71 ms instead of 270.
template <bool kS, int kW>
__device__ __noinline__ uint32_t sp_fold(uint32_t lc, bool listed) {
  constexpr uint32_t C = 065435u;
  // a list item takes about 14 cycles, the bit-wise fold 3,000 (one word per
  // lane) to 5,000 (four) in all: the line lies at the list's size
  constexpr uint32_t kList = 256;
  SpWarp& W = sp_w();
  const SpRef<kS> R(W);
  const uint32_t lane = lane_id(), n = W.n, nwd = (n + 31) / 32, lt = lanemask_lt();
  for (uint32_t base = 0; base < nwd; base += 32 * kW) {
    uint32_t vw[kW], mw[kW], K = 0;
    const uint32_t w0 = base + lane * kW;
#pragma unroll
    for (int w = 0; w < kW; ++w) {
      const uint32_t wi = w0 + w;
      vw[w] = mw[w] = 0;
      if (wi < nwd) {
        const uint32_t m = R.itm[wi];
        vw[w] = listed ? R.nsb[wi] : sp_nonsingle_word(R.stb, n, wi) | m;
        mw[w] = m & vw[w];
        K += (uint32_t)__popc(vw[w]);
      }
    }
    const uint32_t total = __reduce_add_sync(GCL_FULL, K);
    bool dense = total > kList;
    uint32_t kb[6][kW];
    if (dense) {  // the counts, one bit per word (larger counts take the other way)
      bool big = false;
#pragma unroll
      for (int w = 0; w < kW; ++w) {
#pragma unroll
        for (int j = 0; j < 6; ++j) kb[j][w] = 0;
        for (uint32_t m = mw[w]; m; m &= m - 1) {
          const uint32_t b = (uint32_t)__ffs((int)m) - 1, k = R.cnt[(w0 + w) * 32 + b];
          big |= k >= 64;
#pragma unroll
          for (int j = 0; j < 6; ++j) kb[j][w] |= ((k >> j) & 1u) << b;
        }
      }
      dense = !__any_sync(GCL_FULL, big);
    }
    if (!dense) {
      // the items in position order, 256 at a time (one round unless a large
      // count turned the bit-wise fold away)
      uint32_t at = K;
      const uint32_t used = (nwd - base + kW - 1) / kW;  // lanes that hold words
      for (uint32_t o = 1; o < 32 && o < used; o <<= 1) {
        const uint32_t y = __shfl_up_sync(GCL_FULL, at, o);
        if (lane >= o) at += y;
      }
      at -= K;
      for (uint32_t done = 0; done < total; done += kList) {
        const uint32_t m = min(kList, total - done);
        uint32_t i = at - done;  // index in this round's list (wraps below it)
#pragma unroll
        for (int w = 0; w < kW; ++w)
          for (uint32_t x = vw[w]; x; x &= x - 1, ++i) {
            if (i >= kList) continue;
            const uint32_t b = (uint32_t)__ffs((int)x) - 1, p = (w0 + w) * 32 + b;
            // the low 15 bits of an item are all that counts
            W.list[i] = (uint16_t)(p + ((mw[w] >> b) & 1u ? R.cnt[p] : 0u));
          }
        __syncwarp();
        const uint4* l4 = (const uint4*)W.list;
        auto two = [&](uint32_t x) {  // bits above 14 never come down
          lc = (lc ^ C) + x;
          lc = (lc ^ C) + (x >> 16);
        };
        for (uint32_t q = 0; q < m / 8; ++q) {
          const uint4 x = l4[q];
          two(x.x);
          two(x.y);
          two(x.z);
          two(x.w);
        }
        if (m & 7u) {
          const uint4 x = l4[m / 8];
          uint32_t a = x.x, b = x.y;
          if (m & 4u) {
            two(a);
            two(b);
            a = x.z;
            b = x.w;
          }
          if (m & 2u) {
            two(a);
            a = b;
          }
          if (m & 1u) lc = (lc ^ C) + a;
        }
        __syncwarp();
      }
      continue;
    }
    uint32_t carry[kW], cp[kW], out = 0;
#pragma unroll
    for (int w = 0; w < kW; ++w) carry[w] = cp[w] = 0;
#pragma unroll
    for (int j = 0; j < 15; ++j) {
      constexpr uint32_t kPat[5] = {0xaaaaaaaau, 0xccccccccu, 0xf0f0f0f0u, 0xff00ff00u,
                                    0xffff0000u};
      const uint32_t Cm = ((C >> j) & 1u) ? 0xffffffffu : 0u;
      uint32_t vj[kW], inc[kW], par = 0;
#pragma unroll
      for (int w = 0; w < kW; ++w) {
        // bit j of the item: position plus count
        const uint32_t pj = j < 5 ? kPat[j < 5 ? j : 0] : 0u - (((w0 + w) * 32 >> j) & 1u);
        const uint32_t kj = j < 6 ? kb[j < 6 ? j : 0][w] : 0u;
        vj[w] = pj ^ kj ^ cp[w];
        cp[w] = (pj & kj) | (cp[w] & (pj ^ kj));
        uint32_t f = vw[w] & (Cm ^ vj[w] ^ carry[w]);
        f ^= f << 1;
        f ^= f << 2;
        f ^= f << 4;
        f ^= f << 8;
        f ^= f << 16;
        inc[w] = f;
        par ^= f;
      }
      const uint32_t B = __ballot_sync(GCL_FULL, par >> 31);
      const uint32_t x0 = (lc >> j) & 1u;
      uint32_t run = x0 ^ ((uint32_t)__popc(B & lt) & 1u);
#pragma unroll
      for (int w = 0; w < kW; ++w) {
        const uint32_t y = (0u - run) ^ (inc[w] << 1) ^ Cm;  // the value before, xor 065435
        carry[w] = (y & vj[w]) | (carry[w] & (y ^ vj[w]));
        run ^= inc[w] >> 31;
      }
      out |= (x0 ^ ((uint32_t)__popc(B) & 1u)) << j;
    }
    lc = out;
  }
  return lc;
}

// The first path runs on one warp of a block whose other warps wait at named
// barrier 1 for a splitter to count, and meet it again at barrier 2.
constexpr uint32_t kSpHelpThreads = 256;
// members from which the two barriers (about 100 cycles) cost less than the
// 32-wide count they save (some 300 cycles per 32 members)
constexpr uint32_t kSpHelpMin = 96;
__device__ __forceinline__ void sp_block_sync(int id) {
  asm volatile("bar.sync %0, %1;" ::"r"(id), "n"(kSpHelpThreads) : "memory");
}

// Thread t of nt: the neighbours of the splitter's vertices [s, e), counted at
// their positions.
template <bool kS>
__device__ __forceinline__ void sp_count(const SpWarp& W, uint32_t s, uint32_t e, uint32_t t,
                                         uint32_t nt) {
  const SpRef<kS> R(W);
  auto add = [&](uint32_t u) {
    const uint32_t p = R.pos[u];
    atomicAdd((uint32_t*)R.cnt + (p >> 1), 1u << ((p & 1u) * 16u));
  };
  if (e - s <= 8) {  // the threads share each row
    for (uint32_t q = s; q < e; ++q) {
      const uint32_t w = R.elem[q];
      const int32_t f = W.rp[w + 1];
      for (int32_t i = W.rp[w] + (int32_t)t; i < f; i += (int32_t)nt) add((uint32_t)W.col[i]);
    }
    return;
  }
  for (uint32_t q = s + t; q < e; q += nt) {
    const uint32_t w = R.elem[q];
    const int32_t f = W.rp[w + 1];
    for (int32_t i = W.rp[w]; i < f; ++i) add((uint32_t)W.col[i]);
  }
}

// ---------------------------------------------------------------------------
// A step whose splitter has more than 32 edges.  Neighbour counts are kept by
// position, so a cell's counts are contiguous: a lane tests whole small cells
// for a common count, and each cell without one is sorted by count -- up to 32
// vertices by a radix pass over ballots, larger ones by a counting sort.  A
// singleton splitter's cells split into [neighbours, non-neighbours]
// (:296-309, 399-435), the others into ascending counts (:326-465).
// ---------------------------------------------------------------------------
struct SpStep {
  uint32_t lc, hint, made;  // made: new cell starts
};

template <bool kS>
__device__ __noinline__ SpStep sp_refine_general(uint32_t s, uint32_t e, uint32_t lc,
                                                 uint32_t hint, uint32_t utop) {
  SpWarp& W = sp_w();
  const SpRef<kS> R(W);
  const uint32_t lane = lane_id(), n = W.n, lt = lanemask_lt();
  const uint32_t nwd = (n + 31) / 32;
  const bool single = e - s == 1;
  const uint32_t flip = single ? 1u : 0u;  // a neighbour's key is 0, a non-neighbour's 1
  const uint32_t utop0 = utop;
  if (W.helpers && e - s >= kSpHelpMin) {
    if (lane == 0) {
      W.job_s = s;
      W.job_e = e;
    }
    __syncwarp();
    sp_block_sync(1);
    sp_count<kS>(W, s, e, lane, kSpHelpThreads);
    sp_block_sync(2);
  } else {
    sp_count<kS>(W, s, e, lane, 32);
  }
  for (uint32_t wi = lane; wi < nwd; wi += 32) R.nsb[wi] = sp_nonsingle_word(R.stb, n, wi);
  __syncwarp();
  // a fragment of a split cell: its start, hint and place in the active set
  // are those of partition_refinement.cpp:399-460; returns the new starts
  auto fragment = [&](bool frag, uint32_t c, uint32_t f, uint32_t size, uint32_t count,
                      bool active) {
    const bool fresh = frag && f != c;
    const uint32_t m = __ballot_sync(GCL_FULL, fresh);
    if (frag && count && !single) or_bit32(R.itm, f);
    if (fresh) {
      W.slog[utop + (uint32_t)__popc(m & lt)] = f;
      bm_or(R.stb, R.sts, f);
      or_bit32(R.nsb, f);
    }
    if (frag && active) or_bit32(R.act, f);
    utop += (uint32_t)__popc(m);
    if (!single) {
      const uint32_t h = __reduce_max_sync(GCL_FULL, fresh && size == 1 ? f + 1 : 0u);
      if (h) hint = h - 1;
    }
  };
  // the split of a singleton splitter: nb neighbours, nn others
  auto split_single = [&](uint32_t c, uint32_t nb, uint32_t nn, bool was) {
    const bool rest = was || nb >= nn;
    lc = (lc ^ 065435u) + (c + nb - 1);
    if (rest && nn == 1) hint = c + nb;
    if (!rest && nb == 1) hint = c;
    fragment(lane < 2, c, lane == 1 ? c + nb : c, 0, 0, lane == (rest ? 1u : 0u));
  };
  for (uint32_t base = 0; base < nwd; base += 32) {
    const uint32_t wi = base + lane;
    uint32_t pend = 0;
    for (uint32_t x = wi < nwd ? R.nsb[wi] : 0u; x; x &= x - 1) {
      const uint32_t b = (uint32_t)__ffs((int)x) - 1, c = wi * 32 + b;
      const uint32_t ce = R.end_of(c, n);
      bool differ = ce - c > 32;  // large cells are tested by the whole warp
      if (!differ) {
        const uint32_t a = R.cnt[c];
        for (uint32_t q = c + 1; q < ce; ++q) differ |= R.cnt[q] != a;
        if (!differ && a && !single) or_bit32(R.itm, c);
      }
      if (differ) pend |= 1u << b;
    }
    __syncwarp();
    for (uint32_t any = __ballot_sync(GCL_FULL, pend != 0); any; any &= any - 1) {
      const int src = __ffs((int)any) - 1;
      for (uint32_t m = __shfl_sync(GCL_FULL, pend, src); m; m &= m - 1) {
        const uint32_t c = (base + (uint32_t)src) * 32 + (uint32_t)__ffs((int)m) - 1;
        const uint32_t ce = R.end_of(c, n), L = ce - c;
        const bool was = R.active(c);
        if (L <= 32) {
          const bool in = lane < L;
          const uint32_t v = in ? R.elem[c + lane] : 0u, a = in ? R.cnt[c + lane] : 0u;
          const uint32_t key = in ? a ^ flip : 0u;
          uint32_t peers = L == 32 ? 0xffffffffu : (1u << L) - 1u, less = 0;
          const uint32_t top = __reduce_max_sync(GCL_FULL, key);
          for (int bit = 31 - __clz((int)top); bit >= 0; --bit) {
            const bool one = (key >> bit) & 1u;
            const uint32_t m1 = __ballot_sync(GCL_FULL, in && one);
            if (one) {
              less += (uint32_t)__popc(peers & ~m1);
              peers &= m1;
            } else {
              peers &= ~m1;
            }
          }
          const uint32_t eq = (uint32_t)__popc(peers & lt), size = (uint32_t)__popc(peers);
          const uint32_t f = c + less;
          __syncwarp();
          if (in) {
            R.elem[f + eq] = (uint16_t)v;
            R.pos[v] = (uint16_t)(f + eq);
            R.cnt[f + eq] = (uint16_t)a;
          }
          if (single) {
            const uint32_t nb = (uint32_t)__popc(__ballot_sync(GCL_FULL, in && key == 0));
            split_single(c, nb, L - nb, was);
          } else {
            const bool frag = in && eq == 0;
            const uint32_t rank = frag ? (size << 6) | (63u - less) : 0u;
            const uint32_t best = __reduce_max_sync(GCL_FULL, rank);
            fragment(frag, c, f, size, a, was ? f != c : rank != best);
          }
          __syncwarp();
          continue;
        }
        // a large cell: its touched positions, eight counts per lane at a time
        if (lane == 0) W.scr[0] = 0;
        __syncwarp();
        uint32_t mn = 0xffffffffu, mx = 0;
        for (uint32_t q0 = (c & ~7u) + lane * 8; q0 < ce; q0 += 256) {
          const uint4 x4 = *(const uint4*)(R.cnt + q0);
          if (!(x4.x | x4.y | x4.z | x4.w)) continue;
          const uint32_t xs[4] = {x4.x, x4.y, x4.z, x4.w};
#pragma unroll
          for (int j = 0; j < 8; ++j) {
            const uint32_t a = (xs[j / 2] >> (j % 2 * 16)) & 0xffffu, q = q0 + j;
            if (!a || q < c || q >= ce) continue;
            mn = min(mn, a);
            mx = max(mx, a);
            const uint32_t i = atomicAdd(&W.scr[0], 1u);
            if (i < 256) W.list[i] = (uint16_t)q;
          }
        }
        __syncwarp();
        const uint32_t touched = W.scr[0];
        mn = __reduce_min_sync(GCL_FULL, mn);
        mx = __reduce_max_sync(GCL_FULL, mx);
        if (touched < L) mn = 0;
        if (mn == mx) {
          if (mn && !single && lane == 0) or_bit32(R.itm, c);
          __syncwarp();
          continue;
        }
        if (touched <= 32 && touched < L && !single) {
          // few touched vertices: they go to the cell's last places, ranked by
          // count, and swap with the untouched ones found there -- the cost of
          // the touched ones, not of the cell (a counting sort of the whole
          // cell took some 100 cycles per 32 vertices)
          const bool on = lane < touched;
          const uint32_t p = on ? W.list[lane] : 0u, u = on ? R.elem[p] : 0u;
          const uint32_t a = on ? R.cnt[p] : 0u;
          const uint32_t all = touched == 32 ? 0xffffffffu : (1u << touched) - 1u;
          uint32_t peers = all, less = 0;
          for (int bit = 31 - __clz((int)mx); bit >= 0; --bit) {
            const bool one = (a >> bit) & 1u;
            const uint32_t m1 = __ballot_sync(GCL_FULL, on && one);
            if (one) {
              less += (uint32_t)__popc(peers & ~m1);
              peers &= m1;
            } else {
              peers &= ~m1;
            }
          }
          const uint32_t eq = (uint32_t)__popc(peers & lt), size = (uint32_t)__popc(peers);
          const uint32_t R0 = ce - touched, f = R0 + less;
          const bool in = on && p >= R0, mv = on && p < R0, frag = on && eq == 0;
          const uint32_t inner = __reduce_or_sync(GCL_FULL, in ? 1u << (p - R0) : 0u);
          const uint32_t outs = __ballot_sync(GCL_FULL, mv);
          const uint32_t h = mv ? R0 + nth_bit(~inner & all, (uint32_t)__popc(outs & lt)) : 0u;
          const uint32_t x = mv ? R.elem[h] : 0u;
          const uint32_t rank = frag ? (size << 6) | (63u - less) : 0u;
          const uint32_t best = __reduce_max_sync(GCL_FULL, rank);
          const bool rest = L - touched >= (best >> 6);  // the untouched fragment is the largest
          __syncwarp();
          if (mv) {
            R.elem[p] = (uint16_t)x;
            R.pos[x] = (uint16_t)p;
            R.cnt[p] = 0;
          }
          __syncwarp();
          if (on) {
            R.elem[f + eq] = (uint16_t)u;
            R.pos[u] = (uint16_t)(f + eq);
            R.cnt[f + eq] = (uint16_t)a;
          }
          if (lane == 0 && !was && !rest) or_bit32(R.act, c);
          fragment(frag, c, f, size, a, was || rest || rank != best);
          __syncwarp();
          continue;
        }
        const uint32_t range = mx - mn + 1;
        // counts and offsets by key: in shared memory for up to 64 keys
        uint32_t* const hist = range <= 64 ? (uint32_t*)W.list : W.hist;
        uint32_t* const pre = range <= 64 ? (uint32_t*)W.list + 64 : W.pre;
        for (uint32_t i = lane; i < range; i += 32) hist[i] = 0;
        __syncwarp();
        for (uint32_t i = lane; i < L; i += 32)
          atomicAdd(&hist[(uint32_t)(R.cnt[c + i] - mn) ^ flip], 1u);
        __syncwarp();
        // fragment starts (relative) and the first largest fragment
        uint32_t run = 0, best = 0, bestf = 0;
        for (uint32_t i0 = 0; i0 < range; i0 += 32) {
          const uint32_t i = i0 + lane, h = i < range ? hist[i] : 0u;
          uint32_t incl = h;
          for (int o = 1; o < 32; o <<= 1) {
            const uint32_t y = __shfl_up_sync(GCL_FULL, incl, o);
            if (lane >= (uint32_t)o) incl += y;
          }
          const uint32_t f = run + incl - h;
          if (i < range) pre[i] = f;
          const uint32_t mxh = __reduce_max_sync(GCL_FULL, h);
          if (mxh > best) {
            best = mxh;
            bestf = __shfl_sync(GCL_FULL, f, __ffs((int)__ballot_sync(GCL_FULL, h == mxh)) - 1);
          }
          run += __shfl_sync(GCL_FULL, incl, 31);
        }
        __syncwarp();
        if (single) {
          split_single(c, hist[0], hist[1], was);
        } else {
          for (uint32_t i0 = 0; i0 < range; i0 += 32) {
            const uint32_t i = i0 + lane, h = i < range ? hist[i] : 0u;
            const uint32_t f = i < range ? pre[i] : 0u;
            fragment(h != 0, c, c + f, h, mn + i, was ? f != 0 : f != bestf);
          }
        }
        __syncwarp();
        for (uint32_t i = lane; i < L; i += 32) {
          const uint32_t a = R.cnt[c + i];
          W.tmp[atomicAdd(&pre[(a - mn) ^ flip], 1u)] = (a << 16) | R.elem[c + i];
        }
        __syncwarp();
#pragma unroll 4
        for (uint32_t i = lane; i < L; i += 32) {
          const uint32_t x = W.tmp[i], v = x & 0xffffu;
          R.elem[c + i] = (uint16_t)v;
          R.pos[v] = (uint16_t)(c + i);
          R.cnt[c + i] = (uint16_t)(x >> 16);
        }
        __syncwarp();
      }
    }
  }
  __syncwarp();
  if (!single) lc = n <= 1024 ? sp_fold<kS, 1>(lc, true) : sp_fold<kS, 4>(lc, true);
  __syncwarp();
  uint4* z = (uint4*)R.cnt;
  for (uint32_t i = lane; i < (2 * (n + 2) + 15) / 16; i += 32) z[i] = make_uint4(0, 0, 0, 0);
  for (uint32_t wi = lane; wi < nwd; wi += 32) R.itm[wi] = 0;
  __syncwarp();
  return {lc, hint, utop - utop0};
}

// ---------------------------------------------------------------------------
// Partition_s_refinement (partition_refinement.cpp:150-485).  The active
// bitmap holds the initially active cells; returns the code (-1 on a failed
// consistency check).  The caller increments the level.
//
// Steps whose splitter has at most 32 edges -- nearly all -- are
// warp-synchronous: lane i takes the i-th edge, cells are grouped with
// match_any, and every split cell's start, log entry and active bits are
// written by its own lane with shared-memory atomics; only the hash follows
// position order.  A split makes as many active cells as cell starts: a cell
// that was active gets its new fragments, one that was not all but its first
// largest.  Singleton neighbours end a step early.  With one lane writing the
// splits one after the other a singleton step took 1,900-2,500 cycles and a
// non-singleton one 6,000 beside its hash; the change took a mixed batch up to 256
// vertices from 432 to 252 ms and four copies of a 4-regular graph on 64
// vertices from 219 to 133.
// ---------------------------------------------------------------------------
template <bool kS>
__device__ __noinline__ int sp_refine_t() {
  SpWarp& W = sp_w();
  const SpRef<kS> R(W);
  const uint32_t lane = lane_id(), lt = lanemask_lt();
  const uint32_t n = W.n, nwd = (n + 31) / 32;
  constexpr uint32_t C = 065435u;
  uint32_t ncells = W.ncells, nact = W.nact, utop = W.utop;
  uint32_t lc = ncells, hint = 0, iters = 0;
  int ok = 1;
  const int32_t* const rp = W.rp;
  const int32_t* const col = W.col;
  uint32_t* const slog = W.slog;
  // the splitter: the first active position from the hint on, else from 0
  auto next_active = [&]() -> uint32_t {
    const uint32_t near = R.act[hint >> 5] >> (hint & 31u);
    if (near) return hint + (uint32_t)__ffs((int)near) - 1;
    if (nwd <= 32) {  // a word per lane
      const uint32_t w = lane < nwd ? R.act[lane] : 0u, hw = hint >> 5;
      const uint32_t ge = lane > hw ? w : lane == hw ? w & (0xffffffffu << (hint & 31u)) : 0u;
      uint32_t m = __ballot_sync(GCL_FULL, ge != 0), x = ge;
      if (!m) {
        m = __ballot_sync(GCL_FULL, w != 0);
        x = w;
      }
      if (!m) return kNone;
      const uint32_t src = (uint32_t)__ffs((int)m) - 1;
      return src * 32 + (uint32_t)__ffs((int)__shfl_sync(GCL_FULL, x, (int)src)) - 1;
    }
    // four words per lane from the word after the hint's, then from word 0
    const uint32_t from = (hint >> 5) + 1, wp = sp_pad_words(n);
    for (int wrap = 0; wrap < 2; ++wrap)
      for (uint32_t base = wrap ? 0 : from & ~127u; base < wp; base += 128) {
        const uint32_t w0 = base + lane * 4;
        uint4 x = make_uint4(0, 0, 0, 0);
        if (w0 < wp) x = *(const uint4*)(R.act + w0);
        if (!wrap && base < from) {
          if (w0 < from) x.x = 0;
          if (w0 + 1 < from) x.y = 0;
          if (w0 + 2 < from) x.z = 0;
          if (w0 + 3 < from) x.w = 0;
        }
        const uint32_t m = __ballot_sync(GCL_FULL, (x.x | x.y | x.z | x.w) != 0);
        if (!m) continue;
        const uint32_t p = x.x   ? (uint32_t)__ffs((int)x.x)
                           : x.y ? 32 + (uint32_t)__ffs((int)x.y)
                           : x.z ? 64 + (uint32_t)__ffs((int)x.z)
                                 : 96 + (uint32_t)__ffs((int)x.w);
        return __shfl_sync(GCL_FULL, w0 * 32 + p - 1, __ffs((int)m) - 1);
      }
    return kNone;
  };
  while (ncells < n && nact > 0) {
    if (++iters > 4 * n + 64) {  // every step removes an active cell or splits one
      ok = 0;
      break;
    }
    const uint32_t s = next_active();
    if (s >= n) {
      ok = 0;
      break;
    }
    const uint32_t w = R.elem[s];
    const bool one = R.alone(s);
    const int32_t sb = rp[w], sd = rp[w + 1] - sb;
    __syncwarp();
    if (lane == 0) atomicAnd(R.act + (s >> 5), ~(1u << (s & 31u)));
    nact -= 1;
    if (one) {
      lc = (lc ^ C) + (2 * s);  // split1 + split2
      if (sd <= 32) {
        // Singleton splitter: a cell splits into [neighbours, non-neighbours]
        // when only some of its vertices are neighbours (:296-309, 399-435).
        uint32_t u = 0, p = 0, c = kNone, L = 0;
        bool on = false;
        if ((int32_t)lane < sd) {
          u = (uint32_t)col[sb + (int32_t)lane];
          p = R.pos[u];
          on = !R.alone(p);
        }
        __syncwarp();
        if (!__any_sync(GCL_FULL, on)) continue;
        if (nwd <= 32) {
          const uint32_t some = __ballot_sync(GCL_FULL, lane < nwd && R.st[lane] != 0);
          if (on) R.cell_of_1k(p, n, some, &c, &L);
        } else if (on) {
          R.cell_of(p, n, &c, &L);
        }
        const uint32_t grp = __match_any_sync(GCL_FULL, c);
        const uint32_t k = (uint32_t)__popc(grp);
        const bool spl = on && k < L;
        if (!__any_sync(GCL_FULL, spl)) continue;
        // misplaced neighbours swap with the non-neighbours inside the cell's
        // first k positions
        uint32_t h = c, x = 0;
        bool mv = false;
        if (__any_sync(GCL_FULL, spl && k > 1)) {
          // the places taken, collected at the cell's first lane
          const bool in = p < c + k;
          const uint32_t first = (uint32_t)__ffs((int)grp) - 1;
          W.scr[lane] = 0;
          __syncwarp();
          if (spl && in) atomicOr(&W.scr[first], 1u << (p - c));
          const uint32_t outs = __ballot_sync(GCL_FULL, spl && !in) & grp;
          __syncwarp();
          mv = spl && !in;
          if (mv)
            h = c + nth_bit(~W.scr[first] & (k >= 32 ? 0xffffffffu : (1u << k) - 1u),
                            (uint32_t)__popc(outs & lt));
        } else {
          mv = spl && p != c;
        }
        const bool lead = spl && (grp & lt) == 0;
        const bool was = R.active(lead ? c : 0);
        if (mv) x = R.elem[h];
        const uint32_t leaders = __ballot_sync(GCL_FULL, lead);
        const uint32_t made = (uint32_t)__popc(leaders);
        __syncwarp();
        if (mv) {
          R.elem[h] = (uint16_t)u;
          R.pos[u] = (uint16_t)h;
          R.elem[p] = (uint16_t)x;
          R.pos[x] = (uint16_t)p;
        }
        // key: start, neighbours and whether the split sets the hint to its
        // first (1) or second (2) fragment
        uint32_t key = kNone;
        if (lead) {
          const uint32_t pp = c + k, nn = L - k;
          const bool rest = was || k >= nn;
          key = (c << 8) | (k << 2) | (rest ? (nn == 1 ? 2u : 0u) : (k == 1 ? 1u : 0u));
          slog[utop + (uint32_t)__popc(leaders & lt)] = pp;
          bm_or(R.stb, R.sts, pp);
          or_bit32(R.act, rest ? pp : c);
        }
        utop += made;
        ncells += made;
        nact += made;
        // hash (cell.first + neighbors_size - 1) in position order; the hint
        // is the last split cell's that sets one
        auto fold = [&](uint32_t x) {
          const uint32_t cc = x >> 8, pp = cc + ((x >> 2) & 63u);
          lc = (lc ^ C) + (pp - 1);
          if (x & 2u) hint = pp;
          if (x & 1u) hint = cc;
        };
        if (made <= 2) {  // one or two cells: no reduction
          const uint32_t x = __shfl_sync(GCL_FULL, key, __ffs((int)leaders) - 1);
          const uint32_t y = __shfl_sync(GCL_FULL, key, 31 - __clz((int)leaders));
          fold(min(x, y));
          if (made == 2) fold(max(x, y));
        } else {
          for (uint32_t i = 0; i < made; ++i) {
            const uint32_t x = __reduce_min_sync(GCL_FULL, key);
            if (key == x) key = kNone;
            fold(x);
          }
        }
        __syncwarp();
        continue;
      }
    }
    const uint32_t e = one ? s + 1 : R.end_of(s, n), len = e - s;
    if (!one) {
      lc = (lc ^ C) + (s + e - 1);
      lc = (lc ^ C) + len;
    }
    if (len > 1 && len <= 32) {
      // the splitter's edges, lane by lane
      uint32_t d = 0;
      int32_t b = 0;
      if (lane < len) {
        const uint32_t w = R.elem[s + lane];
        b = rp[w];
        d = (uint32_t)(rp[w + 1] - b);
      }
      uint32_t incl = d;
      for (int o = 1; o < 32; o <<= 1) {
        const uint32_t y = __shfl_up_sync(GCL_FULL, incl, o);
        if (lane >= (uint32_t)o) incl += y;
      }
      const uint32_t D = __shfl_sync(GCL_FULL, incl, 31);
      if (D <= 32) {
        const uint32_t excl = incl - d;
        const uint32_t nonempty = __ballot_sync(GCL_FULL, d > 0);
        const uint32_t firsts = __reduce_or_sync(GCL_FULL, d > 0 ? 1u << excl : 0u);
        // lane i < D: member = the k-th non-empty one, k = firsts up to lane i
        const uint32_t kth = (uint32_t)__popc(firsts & (lt | (1u << lane)));
        int src = 0;
        if (lane < D)
          src = (nonempty & (nonempty + 1)) == 0 ? (int)kth - 1 : (int)nth_bit(nonempty, kth - 1);
        const int32_t bs = __shfl_sync(GCL_FULL, b, src);
        const uint32_t es = __shfl_sync(GCL_FULL, excl, src);
        uint32_t u = kNone, p = 0, c = kNone, L = 0;
        if (lane < D) {
          u = (uint32_t)col[bs + (int32_t)(lane - es)];
          p = R.pos[u];
          if (R.alone(p)) u = kNone;  // singleton cells never split (:257-259)
        }
        // lanes on the same neighbour: the group's size is its count
        const uint32_t gu = __match_any_sync(GCL_FULL, u);
        const uint32_t cnt = (uint32_t)__popc(gu);
        const bool lead = u != kNone && (gu & lt) == 0;
        if (nwd <= 32) {
          const uint32_t some = __ballot_sync(GCL_FULL, lane < nwd && R.st[lane] != 0);
          if (lead) R.cell_of_1k(p, n, some, &c, &L);
        } else if (lead) {
          R.cell_of(p, n, &c, &L);
        }
        const uint32_t gc = __match_any_sync(GCL_FULL, c);
        const uint32_t k = (uint32_t)__popc(gc);  // touched vertices of the cell
        // rank by count within the cell: a radix pass over ballots
        uint32_t peers = lead ? gc : 0u, less = 0;
        const uint32_t top = __reduce_max_sync(GCL_FULL, lead ? cnt : 0u);
        for (int bit = 31 - __clz((int)top); bit >= 0; --bit) {
          const bool one = (cnt >> bit) & 1u;
          const uint32_t m1 = __ballot_sync(GCL_FULL, lead && one);
          if (one) {
            less += (uint32_t)__popc(peers & ~m1);
            peers &= m1;
          } else {
            peers &= ~m1;
          }
        }
        const uint32_t eq = (uint32_t)__popc(peers & lt), size = (uint32_t)__popc(peers);
        const bool uniform = lead && k == L && size == k;  // one common count: no split
        const bool split = lead && !uniform;
        const bool cell_lead = lead && (gc & lt) == 0;
        const uint32_t R0 = c + (L - k), f = R0 + less;
        uint32_t h = 0, x = 0, made = 0;
        if (__any_sync(GCL_FULL, split)) {
          // untouched vertices first, then ascending count: touched vertices go
          // to R0 + rank, the untouched ones found in [R0, c + L) to the
          // positions the touched ones leave
          const bool in = p >= R0;
          const bool frag = split && eq == 0;
          const uint32_t rank = frag ? (size << 6) | (63u - less) : 0u;
          // per cell, at its first lane: the places taken in [R0, c + L) and the
          // first largest fragment (a reduction per cell, one after the other,
          // took 1,000 cycles of a step that splits five cells)
          const uint32_t first = (uint32_t)__ffs((int)gc) - 1;
          uint32_t* const top_of = (uint32_t*)W.list;
          W.scr[lane] = 0;
          top_of[lane] = 0;
          __syncwarp();
          if (split && in) atomicOr(&W.scr[first], 1u << (p - R0));
          if (frag) atomicMax(&top_of[first], rank);
          const uint32_t outs = __ballot_sync(GCL_FULL, split && !in) & gc;
          __syncwarp();
          const uint32_t best = top_of[first];
          const bool mv = split && !in;
          if (mv) {
            h = R0 + nth_bit(~W.scr[first] & (k >= 32 ? 0xffffffffu : (1u << k) - 1u),
                             (uint32_t)__popc(outs & lt));
            x = R.elem[h];
          }
          const bool was = split && R.active(c);
          // the first largest fragment is the untouched one (it comes first)
          const bool rest = L - k >= (best >> 6);
          const bool fresh = frag && f != c;
          const uint32_t fm = __ballot_sync(GCL_FULL, fresh);
          made = (uint32_t)__popc(fm);
          __syncwarp();
          if (mv) {
            R.elem[p] = (uint16_t)x;
            R.pos[x] = (uint16_t)p;
          }
          if (split) {
            R.elem[f + eq] = (uint16_t)u;
            R.pos[u] = (uint16_t)(f + eq);
          }
          if (frag && (was ? f != c : rest || rank != best)) or_bit32(R.act, f);
          if (cell_lead && split && L > k && !was && !rest) or_bit32(R.act, c);
          if (fresh) slog[utop + (uint32_t)__popc(fm & lt)] = f;
          const uint32_t hv = __reduce_max_sync(GCL_FULL, fresh && size == 1 ? f + 1 : 0u);
          if (hv) hint = hv - 1;
        }
        const bool item = (uniform && cell_lead) || (split && eq == 0);
        if (item) {
          R.cnt[f] = (uint16_t)cnt;
          or_bit32(R.itm, f);
        }
        __syncwarp();
        lc = n <= 1024 ? sp_fold<kS, 1>(lc, false) : sp_fold<kS, 4>(lc, false);
        __syncwarp();
        if (item) {
          R.cnt[f] = 0;
          R.itm[f >> 5] = 0;
          if (split && f != c) bm_or(R.stb, R.sts, f);
        }
        utop += made;
        ncells += made;
        nact += made;
        __syncwarp();
        continue;
      }
    }
    __syncwarp();
    const SpStep st = sp_refine_general<kS>(s, e, lc, hint, utop);
    lc = st.lc;
    hint = st.hint;
    utop += st.made;
    ncells += st.made;
    nact += st.made;
  }
  // clear what is left of the active set
  __syncwarp();
  if (nact)
    for (uint32_t w = lane; w < sp_pad_words(n); w += 32) R.act[w] = 0;
  if (lane == 0) {
    W.ncells = ncells;
    W.utop = utop;
    W.nact = 0;
  }
  __syncwarp();
  if (!ok) return -1;
  return cleanup(mash(lc & 077777u, ncells));
}

__device__ __forceinline__ int sp_refine() {
  return sp_w().soff != kNone ? sp_refine_t<true>() : sp_refine_t<false>();
}

// split_by_and_refine's split (partition_refinement.cpp:486-528)
__device__ __forceinline__ bool sp_individualize(uint32_t level, uint32_t v, uint32_t t) {
  SpWarp& W = sp_w();
  const uint32_t lane = lane_id();
  const uint32_t* st = (const uint32_t*)W.stb;
  if ((st[(t + 1) >> 5] >> ((t + 1) & 31u)) & 1u) return false;  // a singleton
  __syncwarp();
  if (lane == 0) {
    W.umark[level] = W.utop;  // backtracking to `level` undoes from here
    const uint32_t p = W.pos[v], x = W.elem[t];
    W.elem[p] = x;
    W.pos[x] = p;
    W.elem[t] = v;
    W.pos[v] = t;
    add_start(W, t + 1);
    W.ncells += 1;
    or_bit32(W.act, t);
    W.nact = 1;
  }
  __syncwarp();
  return true;
}

// Backtrack to node level Lv (reconstruct_at_level,
// partition_refinement.cpp:541-604): the starts logged since that node's child
// was made go.  False if the log is inconsistent.
__device__ __forceinline__ bool sp_backtrack(uint32_t Lv) {
  SpWarp& W = sp_w();
  const uint32_t lane = lane_id();
  const uint32_t lo = W.umark[Lv], hi = W.utop;
  if (lo > hi) return false;
  for (uint32_t i = lo + lane; i < hi; i += 32) {
    const uint32_t p = W.slog[i];
    atomicAnd((unsigned long long*)&W.stb[p >> 6], (unsigned long long)~bit64(p & 63));
  }
  __syncwarp();
  for (uint32_t i = lo + lane; i < hi; i += 32) {
    const uint32_t w = W.slog[i] >> 6;
    if (W.stb[w] == 0)
      atomicAnd((unsigned long long*)&W.sts[w >> 6], (unsigned long long)~bit64(w & 63));
  }
  __syncwarp();
  if (lane == 0) {
    W.ncells -= hi - lo;
    W.utop = lo;
  }
  __syncwarp();
  return true;
}

// ---- leaves ----------------------------------------------------------------
// A certificate row of at most kD entries by one lane, in registers.
template <int kD>
__device__ __forceinline__ void sp_cert_row(const SpWarp& W, uint32_t* cert, int32_t b, int32_t d) {
  uint32_t x[kD];
#pragma unroll
  for (int i = 0; i < kD; ++i) x[i] = i < d ? (uint32_t)W.col[b + i] : 0u;
#pragma unroll
  for (int i = 0; i < kD; ++i) x[i] = i < d ? W.pos[x[i]] : kNone;
#pragma unroll
  for (int i = 0; i < kD; ++i) {
    int32_t r = 0;
#pragma unroll
    for (int k = 0; k < kD; ++k) r += x[k] < x[i];
    if (i < d) cert[b + r] = x[i];
  }
}

// Certificate of a discrete partition: for every vertex, the canonical
// positions of its neighbours in ascending order, stored at its CSR offset --
// each written once, at its rank in the row (sorting the row in place read back
// every entry from device memory: 40,400 cycles for a tree of 1,000 vertices).
// Warp `warp` of `warps` takes every warps-th group of 32 rows.
__device__ __forceinline__ void sp_leaf_cert_part(const SpWarp& W, uint32_t* cert, uint32_t warp,
                                                  uint32_t warps) {
  const uint32_t lane = lane_id();
  for (uint32_t v0 = warp * 32; v0 < W.n; v0 += warps * 32) {
    const uint32_t v = v0 + lane;
    int32_t b = 0, d = 0;
    if (v < W.n) {
      b = W.rp[v];
      d = W.rp[v + 1] - b;
    }
    // a row per lane; what the widest row of up to 16 entries needs decides
    // how many compares every row takes
    const int32_t ds = d <= 16 ? d : 0, top = __reduce_max_sync(GCL_FULL, ds);
    if (top <= 4)
      sp_cert_row<4>(W, cert, b, ds);
    else if (top <= 8)
      sp_cert_row<8>(W, cert, b, ds);
    else
      sp_cert_row<16>(W, cert, b, ds);
    // longer rows: the warp takes a row at a time, an entry per lane
    for (uint32_t m = __ballot_sync(GCL_FULL, d > 16); m; m &= m - 1) {
      const int src = __ffs((int)m) - 1;
      const int32_t rb = __shfl_sync(GCL_FULL, b, src), rd = __shfl_sync(GCL_FULL, d, src);
      for (int32_t i0 = 0; i0 < rd; i0 += 32) {
        const int32_t i = i0 + (int32_t)lane;
        const uint32_t x = i < rd ? W.pos[W.col[rb + i]] : kNone;
        int32_t r = 0;
        for (int32_t k0 = 0; k0 < rd; k0 += 32) {
          const int32_t kk = k0 + (int32_t)lane;
          const uint32_t y = k0 == i0 ? x : kk < rd ? W.pos[W.col[rb + kk]] : kNone;
          const int32_t cnt = min(32, rd - k0);
          for (int32_t k = 0; k < cnt; ++k) r += __shfl_sync(GCL_FULL, y, k) < x;
        }
        if (i < rd) cert[rb + r] = x;
      }
    }
  }
}

__device__ __forceinline__ void sp_leaf_cert(uint32_t* cert) {
  sp_leaf_cert_part(sp_w(), cert, 0, 1);
  __syncwarp();
}

// Compare the certificate rows of the current leaf (vertex order elem[])
// with a stored leaf (vertex order label[], rows in cert2) in canonical
// row order.  upper: compare_adj_upper (entries right of the diagonal,
// sequential.cpp:114-124), -1/0/+1; otherwise 0 when every row is equal.
template <bool kCg = false>
__device__ __forceinline__ int sp_cmp_leaf(const uint32_t* cur, const uint32_t* label,
                                        const uint32_t* cert2, bool upper) {
  SpWarp& W = sp_w();
  const uint32_t lane = lane_id();
  const uint32_t n = W.n;
  if (!upper) {  // equal rows or not: every entry's load is independent
    for (uint32_t i0 = 0; i0 < n; i0 += 32) {
      const uint32_t i = i0 + lane;
      bool differ = false;
      if (i < n) {
        const uint32_t va = W.elem[i], vb = ldx<kCg>(label + i);
        const int32_t a = W.rp[va], b = W.rp[vb], d = W.rp[va + 1] - a;
        differ = W.rp[vb + 1] - b != d;
        if (!differ) {
#pragma unroll 4
          for (int32_t k = 0; k < d; ++k) differ |= cur[a + k] != ldx<kCg>(cert2 + b + k);
        }
      }
      if (__any_sync(GCL_FULL, differ)) return 1;
    }
    return 0;
  }
  for (uint32_t i0 = 0; i0 < n; i0 += 32) {
    const uint32_t i = i0 + lane;
    int r = 0;
    if (i < n) {
      const uint32_t va = W.elem[i], vb = ldx<kCg>(label + i);
      int32_t a = W.rp[va], ae = W.rp[va + 1], b = W.rp[vb], be = W.rp[vb + 1];
      while (a < ae && cur[a] <= i) ++a;
      while (b < be && ldx<kCg>(cert2 + b) <= i) ++b;
      while (true) {
        const bool ea = a >= ae, eb = b >= be;
        if (ea && eb) break;
        if (ea) {  // b has a 1 where a has 0
          r = -1;
          break;
        }
        if (eb) {
          r = 1;
          break;
        }
        const uint32_t x = cur[a], y = ldx<kCg>(cert2 + b);
        if (x != y) {
          r = x < y ? 1 : -1;
          break;
        }
        ++a;
        ++b;
      }
    }
    const uint32_t diff = __ballot_sync(GCL_FULL, r != 0);
    if (diff) {
      const int src = __ffs(diff) - 1;
      return __shfl_sync(GCL_FULL, r, src);
    }
  }
  return 0;
}

template <typename T>
__device__ __forceinline__ void sp_copy_u32(uint32_t* dst, const T* src, uint32_t k) {
  // eight loads in flight at a time
  for (uint32_t i0 = lane_id(); i0 < k; i0 += 256) {
    uint32_t x[8];
#pragma unroll
    for (int j = 0; j < 8; ++j) x[j] = i0 + 32 * j < k ? src[i0 + 32 * j] : 0u;
#pragma unroll
    for (int j = 0; j < 8; ++j)
      if (i0 + 32 * j < k) dst[i0 + 32 * j] = x[j];
  }
  __syncwarp();
}

// get_gca_level (sequential.cpp:183-213)
__device__ __forceinline__ int sp_gca(const uint32_t* a, uint32_t na, uint32_t seqlen) {
  SpWarp& W = sp_w();
  const uint32_t lane = lane_id();
  const uint32_t m = min(na, seqlen);
  for (uint32_t j0 = 0; j0 < m; j0 += 32) {
    const uint32_t j = j0 + lane;
    const uint32_t b = __ballot_sync(GCL_FULL, j < m && a[j] != W.seq[j]);
    if (b) return (int)(j0 + (uint32_t)(__ffs(b) - 1)) + 1;
  }
  return -1;
}

// first non-singleton cell (target_cell_selector, partition_refinement.cpp:607-655)
__device__ __forceinline__ uint32_t sp_first_nonsingleton() {
  SpWarp& W = sp_w();
  const uint32_t lane = lane_id();
  const uint32_t n = W.n, nwd = (n + 31) / 32;
  for (uint32_t w0 = 0; w0 < nwd; w0 += 32) {
    const uint32_t x = w0 + lane < nwd ? sp_nonsingle_word(W.stb, n, w0 + lane) : 0u;
    const uint32_t m = __ballot_sync(GCL_FULL, x != 0);
    if (!m) continue;
    const uint32_t src = (uint32_t)__ffs((int)m) - 1;
    return (w0 + src) * 32 + (uint32_t)__ffs((int)__shfl_sync(GCL_FULL, x, (int)src)) - 1;
  }
  return kNone;
}

// next representative of target cell idx: smallest vertex >= counter among
// its members whose representative is itself (sequential.cpp:359-361)
__device__ __forceinline__ uint32_t sp_next_rep(const SpTc& t) {
  SpWarp& W = sp_w();
  const uint32_t lane = lane_id();
  uint32_t best = kNone;
  if (t.rslot == kNone) {
    for (uint32_t q = t.first + lane; q < t.first + t.len; q += 32) {
      const uint32_t v = W.elem[q];
      if (v >= t.counter) best = min(best, v);
    }
  } else {
    for (uint32_t i = lane; i < t.len; i += 32) {
      const uint32_t x = W.reps[t.rslot + i], v = x & 0xffffu;
      if (v >= t.counter && (x >> 16) == v) best = min(best, v);
    }
  }
  return __reduce_min_sync(GCL_FULL, best);
}

// The representatives of levels Lv and deeper are dropped (after a backtrack
// to level Lv; their target-cell headers are still in place).
__device__ __forceinline__ void sp_pool_pop(uint32_t Lv) {
  SpWarp& W = sp_w();
  const uint32_t lane = lane_id(), f = W.pool_frames;
  uint32_t keep = 0;  // frames of levels above Lv (owners ascend)
  for (uint32_t i0 = 0; i0 < f; i0 += 32)
    keep += (uint32_t)__popc(
        __ballot_sync(GCL_FULL, i0 + lane < f && W.pool_owner[i0 + lane] < (int32_t)Lv));
  __syncwarp();
  if (lane == 0 && keep < f) {
    W.pool_top = W.tc[W.pool_owner[keep]].rslot;
    W.pool_frames = keep;
  }
  __syncwarp();
}

__device__ __forceinline__ uint32_t sp_find(volatile uint32_t* d, uint32_t x, uint32_t n) {
  uint32_t p = d[x];
  for (uint32_t step = 0; p < x && step <= n; ++step) {
    x = p;
    p = d[x];
  }
  return x;
}

// Merge the cycles of permutation pm on the `count` vertices members[] into
// the min-root union-find W.dsu: hook the larger root under the smaller
// one, then shortcut every member to its root, until a round changes
// nothing (compute_orbits_fast's DSU, perm_group.cpp:60-116).  pm must map
// the member set onto itself.  False if the rounds do not converge.
template <bool kCg, typename T>
__device__ __forceinline__ bool sp_dsu_apply(const uint16_t* pm, const T* members,
                                          uint32_t count, uint32_t n) {
  SpWarp& W = sp_w();
  const uint32_t lane = lane_id();
  volatile uint32_t* dsu = W.dsu;
  for (uint32_t round = 0;; ++round) {
    if (round > count + 1) return false;
    bool changed = false;
    for (uint32_t i = lane; i < count; i += 32) {
      const uint32_t v = members[i];
      const uint32_t img = ldx<kCg>(pm + v);
      if (img == v) continue;
      const uint32_t a = sp_find(dsu, v, n), b = sp_find(dsu, img, n);
      if (a != b) {
        atomicMin((uint32_t*)&dsu[max(a, b)], min(a, b));
        changed = true;
      }
    }
    __syncwarp();
    for (uint32_t i = lane; i < count; i += 32) {
      const uint32_t v = members[i];
      atomicMin((uint32_t*)&dsu[v], sp_find(dsu, v, n));
    }
    __syncwarp();
    if (!__any_sync(GCL_FULL, changed)) return true;
  }
}

// Join the trees of a and b in the min-root union-find d, which other lanes join
// trees of at the same time: the larger root is hooked only while it still is one,
// so nothing is lost and no second pass over the edges is needed.  A failed hook
// means that another lane's took a root away; false past n of them.  A walk
// points what it passes at its grandparent: only roots are hooked, so that store
// meets no hook.
__device__ __forceinline__ bool sp_unite(volatile uint32_t* d, uint32_t a, uint32_t b,
                                         uint32_t n) {
  auto root = [&](uint32_t x) {
    uint32_t p = d[x];
    for (uint32_t step = 0; p < x && step <= n; ++step) {
      const uint32_t g = d[p];
      if (g < p) d[x] = g;
      x = p;
      p = g;
    }
    return x;
  };
  for (uint32_t step = 0; step <= n; ++step) {
    a = root(a);
    b = root(b);
    if (a == b) return true;
    const uint32_t hi = max(a, b);
    if (atomicCAS((uint32_t*)d + hi, hi, min(a, b)) == hi) return true;
  }
  return false;
}

// The orbits of a target cell of at most 32 vertices, a lane per vertex: a
// component is named by its least lane.
struct SpCellOrbits {
  uint32_t v, comp;  // the lane's vertex (kNone past the cell) and its component
};

// Merge the orbits of up to four automorphisms, whose images of the lane's
// vertex lie at indexes j of the cell (j == lane where there is none).
__device__ __forceinline__ void sp_cell_merge(SpCellOrbits& o, const uint32_t (&j)[4]) {
  SpWarp& W = sp_w();
  const uint32_t lane = lane_id();
  while (true) {  // every round with an open edge removes a component
    uint32_t cj[4];
    bool d = false;
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      cj[k] = __shfl_sync(GCL_FULL, o.comp, (int)j[k]);
      d |= cj[k] != o.comp;
    }
    if (!__any_sync(GCL_FULL, d)) return;
    W.scr[lane] = lane;
    __syncwarp();
#pragma unroll
    for (int k = 0; k < 4; ++k)
      if (cj[k] != o.comp) atomicMin(&W.scr[max(o.comp, cj[k])], min(o.comp, cj[k]));
    __syncwarp();
    bool moved;
    do {  // to the root (links go to smaller lanes)
      const uint32_t r = W.scr[o.comp];
      moved = r != o.comp;
      o.comp = r;
    } while (__any_sync(GCL_FULL, moved));
    __syncwarp();
  }
}

// subgroup_fixing_sequence + compute_orbits_fast (perm_group.cpp:5-116).
// The reference unites v with aut[v] over all vertices; an automorphism that
// fixes the sequence maps the node's partition onto itself, cell by cell, so
// the orbits that meet the target cell lie inside it and are found by
// uniting over the cell's members alone (O(cell) per automorphism instead of
// O(n)); the least vertex of each orbit -- the representative -- is the same.
//
// The ring's search (kCg false) keeps a bit per vertex and entry that says
// whether the entry fixes the vertex, so the entries that fix the sequence and
// move a member of the cell are the and of the sequence's rows without the and
// of the cell's: a few independent loads, where testing every entry along the
// sequence took a chain of dependent ones (10,400 to 13,700 cycles a node, 40
// to 47% of the time, on trees of 65 to 1,000 vertices).  An entry that moves
// no member changes nothing.  Cells of up to 32 vertices -- all but the
// largest -- are merged in registers.
//
// The shared store's search (kCg true) tests an entry per lane along the
// sequence and then, for cells of up to 32 vertices, on the members: on a tree
// nearly every entry that fixes the sequence acts elsewhere.  Merging those too,
// four at a time, took 32,000 cycles a node on a tree of 2,100 vertices (255
// entries), 14,000 now: the search 790 ms then and 500 now with its state in
// device memory, that of a tree of 8,192 vertices 25.2 s and 11.4.
//
// Larger cells: the members that a word's entries move are listed and joined a
// lane each.  An entry of a symmetric group moves two or a few, so joining entry
// after entry kept two lanes busy: a star of 100 leaves took 400,000 cycles a node
// (965 ms in the wide search, 1,111 in the batched one), 69,000 now (185 and 194 ms).
//
// Returns kOk, kAutOverflow (no room for the representatives) or kInternal.
template <bool kCg = false>
__device__ __noinline__ int32_t sp_orbits(int idx, int num_aut, uint32_t seqlen) {
  SpWarp& W = sp_w();
  const uint32_t lane = lane_id();
  const uint32_t n = W.n;
  SpTc t = W.tc[idx];
  const int limit = num_aut < (int)W.max_aut ? num_aut : (int)W.max_aut;
  const int from = t.last == -1 ? 0 : t.last;
  const bool small = t.len <= 32;
  volatile uint32_t* dsu = W.dsu;
  const uint16_t* mem = W.elem + t.first;
  bool any = false, begun = false;
  SpCellOrbits o{kNone, lane};
  // the cell's orbits so far
  auto begin = [&] {
    if (small) {
      if (lane < t.len) o.v = mem[lane];
      if (t.rslot != kNone) {
        // the list is keyed by vertex: its order is that of its last writing
        uint32_t rep = kNone - lane;
        if (lane < t.len) {
          const uint32_t x = W.reps[t.rslot + lane];
          W.scr[W.pos[x & 0xffffu] - t.first] = x >> 16;
        }
        __syncwarp();
        if (lane < t.len) rep = W.scr[lane];
        o.comp = (uint32_t)__ffs((int)__match_any_sync(GCL_FULL, rep)) - 1;
        __syncwarp();
      }
      return;
    }
    for (uint32_t i = lane; i < t.len; i += 32) {
      const uint32_t x = t.rslot != kNone ? W.reps[t.rslot + i] : mem[i] * 0x10001u;
      dsu[x & 0xffffu] = x >> 16;
    }
    __syncwarp();
  };
  // the entries base + i, i a bit of m: kInternal if one does not map the cell
  // onto itself
  auto merge = [&](uint32_t base, uint32_t m) -> int32_t {
    if (t.len == 2) {  // an entry that takes part swaps the two
      any = true;
      return kOk;
    }
    if (small) {
      if (!any) begin();
      any = true;
      while (m) {
        // up to four entries' images at once, so their loads overlap
        uint32_t j[4];
#pragma unroll
        for (int k = 0; k < 4; ++k) {
          j[k] = lane < t.len ? o.v : kNone;
          if (!m) continue;
          const uint16_t* pm = W.auts + (uint64_t)(base + (uint32_t)__ffs((int)m) - 1) * W.stride;
          m &= m - 1;
          if (lane < t.len) j[k] = ldx<kCg>(pm + o.v);
        }
        bool out = false;
#pragma unroll
        for (int k = 0; k < 4; ++k) {
          j[k] = j[k] == kNone ? lane : j[k] == o.v ? lane : (uint32_t)W.pos[j[k]] - t.first;
          out |= lane < t.len && j[k] >= t.len;
        }
        if (__any_sync(GCL_FULL, out)) return kInternal;
        sp_cell_merge(o, j);
      }
      return kOk;
    }
    // larger cells: a lane takes every 32nd member through all the entries, and
    // the members they move are listed and joined 32 at a time
    if (!begun) begin();
    begun = true;
    uint32_t* const edge = (uint32_t*)W.list;  // 128 of {vertex, image << 16}
    uint32_t edges = 0;
    bool out = false, moves = false;
    auto join = [&] {
      __syncwarp();
      for (uint32_t x = lane; x < edges; x += 32)
        out |= !sp_unite(dsu, edge[x] & 0xffffu, edge[x] >> 16, n);
      __syncwarp();
      edges = 0;
    };
    for (uint32_t i0 = 0; i0 < t.len; i0 += 32) {
      const bool in = i0 + lane < t.len;
      const uint32_t v = in ? mem[i0 + lane] : 0u;
      for (uint32_t r = m; r;) {
        uint32_t img[4];
#pragma unroll
        for (int k = 0; k < 4; ++k) {
          img[k] = v;
          if (!r) continue;
          const uint16_t* pm = W.auts + (uint64_t)(base + (uint32_t)__ffs((int)r) - 1) * W.stride;
          r &= r - 1;
          if (in) img[k] = ldx<kCg>(pm + v);
        }
#pragma unroll
        for (int k = 0; k < 4; ++k) {
          bool mv = img[k] != v;
          if (mv && (uint32_t)W.pos[img[k]] - t.first >= t.len) {
            out = true;
            mv = false;
          }
          const uint32_t b = __ballot_sync(GCL_FULL, mv);
          if (!b) continue;
          moves = true;
          if (edges + (uint32_t)__popc(b) > 128) join();
          if (mv) edge[edges + (uint32_t)__popc(b & lanemask_lt())] = v | (img[k] << 16);
          edges += (uint32_t)__popc(b);
        }
      }
    }
    join();
    if (__any_sync(GCL_FULL, out)) return kInternal;
    if (!moves) return kOk;
    any = true;
    for (uint32_t i = lane; i < t.len; i += 32) {  // every member to its root
      const uint32_t v = mem[i];
      atomicMin(W.dsu + v, sp_find(dsu, v, n));
    }
    __syncwarp();
    return kOk;
  };
  if constexpr (kCg) {
    // the store entries that fix the sequence, one per lane at a time
    for (int base = from; base < limit; base += 32) {
      const int a = base + (int)lane;
      bool fix = a < limit;
      if (fix) {
        // extend what is known about entry a along the current sequence: the
        // prefix it fixes and the first position it moves stay valid until a
        // backtrack shortens the sequence below them (sp_fix_clamp)
        const bool kept = (uint32_t)a < W.fixcap;
        uint2 st = kept ? W.fixst[a] : make_uint2(0u, kNone);
        if (st.y != kNone && st.y < seqlen) {
          fix = false;
        } else {
          const uint16_t* pa = W.auts + (uint64_t)a * W.stride;
          uint32_t j = st.x;
          for (; j < seqlen; ++j) {
            const uint32_t sv = W.seq[j];
            if (ldx<kCg>(pa + sv) != sv) break;
          }
          fix = j >= seqlen;
          st.x = j;
          st.y = fix ? kNone : j;
          if (kept) W.fixst[a] = st;
        }
      }
      // ... and move a member (merge tests the members of larger cells)
      bool out = false;
      if (fix && small) {
        const uint16_t* pa = W.auts + (uint64_t)a * W.stride;
        uint32_t moved = 0, first = 0, last = 0;
#pragma unroll 4
        for (uint32_t i = 0; i < t.len; ++i) {
          last = ldx<kCg>(pa + mem[i]);
          if (i == 0) first = last;
          moved |= last ^ mem[i];
        }
        fix = moved != 0;
        out = fix && t.len == 2 && (first != mem[1] || last != mem[0]);
      }
      if (__any_sync(GCL_FULL, out)) return kInternal;
      const uint32_t fm = __ballot_sync(GCL_FULL, fix);
      if (!fm) continue;
      const int32_t st = merge((uint32_t)base, fm);
      if (st != kOk) return st;
    }
  } else if (from < limit) {
    // the entries' words [w0, w1], up to 32 at a time: `per` lanes (a power of
    // two) take a row's words, the other lanes further rows
    const uint32_t w0 = (uint32_t)from / 32, w1 = (uint32_t)(limit - 1) / 32;
    for (uint32_t wb = w0; wb <= w1; wb += 32) {
      const uint32_t nwd = min(32u, w1 - wb + 1);
      const uint32_t lg = nwd <= 1 ? 0u : 32u - (uint32_t)__clz((int)nwd - 1), per = 1u << lg;
      const uint32_t wl = lane & (per - 1), row = lane >> lg, rows = 32u >> lg;
      uint32_t fs = 0xffffffffu, fc = 0xffffffffu;
      if (wl < nwd) {
        const uint32_t* F = W.fixm + wb + wl;
        const uint64_t fw = W.fixw;
#pragma unroll 4
        for (uint32_t j = row; j < seqlen; j += rows) fs &= F[W.seq[j] * fw];
#pragma unroll 4
        for (uint32_t i = row; i < t.len; i += rows) fc &= F[mem[i] * fw];
      }
      for (uint32_t d = per; d < 32; d <<= 1) {
        fs &= __shfl_xor_sync(GCL_FULL, fs, (int)d);
        fc &= __shfl_xor_sync(GCL_FULL, fc, (int)d);
      }
      uint32_t sel = 0;
      if (lane < nwd) {
        const int b = (int)(wb + lane) * 32;  // entries b .. b + 31, those in [from, limit)
        sel = fs & ~fc;
        if (b < from) sel &= 0xffffffffu << (from - b);
        if (limit - b < 32) sel &= (1u << (limit - b)) - 1u;
      }
      for (uint32_t m = __ballot_sync(GCL_FULL, sel != 0); m; m &= m - 1) {
        const int src = __ffs((int)m) - 1;
        const int32_t st = merge((wb + (uint32_t)src) * 32, __shfl_sync(GCL_FULL, sel, src));
        if (st != kOk) return st;
      }
    }
  }
  if (!any) return kOk;
  if (t.rslot == kNone) {
    if (W.pool_top + t.len > W.pool_cap) return kAutOverflow;
    t.rslot = W.pool_top;
    __syncwarp();
    if (lane == 0) {
      W.pool_owner[W.pool_frames++] = idx;
      W.pool_top += t.len;
      W.tc[idx].rslot = t.rslot;
    }
    __syncwarp();
  }
  uint32_t* rw = W.reps + t.rslot;
  if (t.len == 2) {
    const uint32_t a = mem[0], b = mem[1], r = min(a, b);
    if (lane < 2) rw[lane] = (lane ? b : a) | (r << 16);
  } else if (small) {
    // the least vertex of each component (a reduction per component, one after
    // the other, took 3,200 of the 7,400 cycles of a call)
    W.scr[lane] = kNone;
    __syncwarp();
    if (lane < t.len) atomicMin(&W.scr[o.comp], o.v);
    __syncwarp();
    if (lane < t.len) rw[lane] = o.v | (W.scr[o.comp] << 16);
  } else {
    for (uint32_t i = lane; i < t.len; i += 32) {
      const uint32_t v = mem[i];
      rw[i] = v | (sp_find(dsu, v, n) << 16);
    }
  }
  __syncwarp();
  return kOk;
}

// After a backtrack to sequence length s: positions >= s of the sequence
// change, so what entries [0, count) knew about them is dropped.
__device__ __forceinline__ void sp_fix_clamp(uint32_t s, uint32_t count) {
  SpWarp& W = sp_w();
  count = min(count, W.fixcap);
  for (uint32_t a = lane_id(); a < count; a += 32) {
    uint2 st = W.fixst[a];
    if (st.x > s || (st.y != kNone && st.y >= s)) {
      st.x = min(st.x, s);
      if (st.y != kNone && st.y >= s) st.y = kNone;
      W.fixst[a] = st;
    }
  }
  __syncwarp();
}

// Ring entry si := aut[label[j]] = elem[j] (sequential.cpp:505-520, 544-555),
// with its bit of every vertex it fixes.
__device__ __forceinline__ void sp_store_aut(const uint32_t* label, uint32_t si) {
  SpWarp& W = sp_w();
  const uint32_t lane = lane_id();
  uint16_t* dst = W.auts + (uint64_t)si * W.stride;
  const uint32_t bit = 1u << (si & 31u);
  for (uint32_t j = lane; j < W.n; j += 32) {
    const uint32_t v = label[j], img = W.elem[j];
    dst[v] = (uint16_t)img;
    uint32_t* f = W.fixm + (uint64_t)v * W.fixw + si / 32;
    *f = v == img ? *f | bit : *f & ~bit;
  }
  __syncwarp();
}

// The refinement's scratch starts clear: no counts, marks or active cells.
__device__ __forceinline__ void sp_clear_scratch() {
  SpWarp& W = sp_w();
  const uint32_t lane = lane_id();
  for (uint32_t i = lane; i < W.n; i += 32) W.cnt[i] = 0;
  for (uint32_t w = lane; w < sp_pad_words(W.n); w += 32) W.itm[w] = W.act[w] = 0;
  __syncwarp();
}

// Colour partition (initializePartition_s, partition_refinement.cpp:28-68):
// a stable LSD radix sort of the identity order by colour.
__device__ __noinline__ void sp_init_partition(const int32_t* color) {
  SpWarp& W = sp_w();
  const uint32_t lane = lane_id();
  const uint32_t n = W.n;
  for (uint32_t i = lane; i < n; i += 32) {
    W.elem[i] = (uint16_t)i;
    W.lst1[i] = i;
  }
  __syncwarp();
  bool colored = false;
  if (color)
    for (uint32_t i = lane; i < n; i += 32) colored |= color[i] != 0;
  colored = __any_sync(GCL_FULL, colored);
  if (colored) {
    uint32_t* a = W.lst1;
    uint32_t* b = W.tmp;
    for (int pass = 0; pass < 4; ++pass) {
      const int sh = pass * 8;
      for (uint32_t i = lane; i < 256; i += 32) W.hist[i] = 0;
      __syncwarp();
      for (uint32_t i = lane; i < n; i += 32) {
        const uint32_t key = (uint32_t)color[a[i]] ^ 0x80000000u;
        atomicAdd(&W.hist[(key >> sh) & 255u], 1u);
      }
      __syncwarp();
      if (lane == 0) {
        uint32_t run = 0;
        for (int d = 0; d < 256; ++d) {
          W.pre[d] = run;
          run += W.hist[d];
        }
      }
      __syncwarp();
      // stable scatter: one lane walks the digits in order
      if (lane == 0)
        for (uint32_t i = 0; i < n; ++i) {
          const uint32_t key = (uint32_t)color[a[i]] ^ 0x80000000u;
          b[W.pre[(key >> sh) & 255u]++] = a[i];
        }
      __syncwarp();
      uint32_t* t = a;
      a = b;
      b = t;
    }
    // four passes: the result is back in lst1
    for (uint32_t i = lane; i < n; i += 32) W.elem[i] = (uint16_t)W.lst1[i];
    __syncwarp();
  }
  for (uint32_t i = lane; i < n; i += 32) W.pos[W.elem[i]] = i;
  for (uint32_t w = lane; w < W.nw; w += 32) W.stb[w] = 0;
  sp_clear_scratch();
  // cell starts where the colour changes
  for (uint32_t i = lane; i < n; i += 32) {
    const bool st = i == 0 || (color && color[W.elem[i]] != color[W.elem[i - 1]]);
    if (st) or_bit32((uint32_t*)W.stb, i);
  }
  __syncwarp();
  uint32_t cells = 0;
  for (uint32_t w = lane; w < W.nw; w += 32) cells += popc64(W.stb[w]);
  cells = __reduce_add_sync(GCL_FULL, cells);
  // every cell starts active (sequential.cpp:628, refinement with no subsequence)
  for (uint32_t w = lane; w < (n + 31) / 32; w += 32) W.act[w] = ((const uint32_t*)W.stb)[w];
  __syncwarp();
  if (lane == 0) or_bit32((uint32_t*)W.stb, n);
  __syncwarp();
  bm_resummarize(W.stb, W.sts, W.nw, W.nsw);
  if (lane == 0) {
    W.ncells = cells;
    W.nact = cells;
  }
  __syncwarp();
}

// Input checks, thread t of nt: offsets and indices in range, rows strictly
// ascending (so no duplicate edge), no loop ...
__device__ __forceinline__ bool sp_check_rows(const int32_t* rp, const int32_t* col, uint32_t n,
                                              int64_t m, uint32_t t, uint32_t nt) {
  if (rp[0] != 0 || (int64_t)rp[n] != m) return false;
  for (uint32_t v = t; v < n; v += nt) {
    const int32_t b = rp[v], e = rp[v + 1];
    if (b < 0 || e < b || (int64_t)e > m) return false;
    int32_t prev = -1;
    for (int32_t i = b; i < e; ++i) {
      const int32_t u = col[i];
      if (u <= prev || (uint32_t)u >= n || (uint32_t)u == v) return false;
      prev = u;
    }
  }
  return true;
}
// ... and, the rows being right, both directions of every edge stored.
__device__ __forceinline__ bool sp_check_mates(const int32_t* rp, const int32_t* col, uint32_t n,
                                               uint32_t t, uint32_t nt) {
  for (uint32_t v = t; v < n; v += nt) {
    const int32_t b = rp[v], e = rp[v + 1];
    for (int32_t i = b; i < e; ++i) {
      const uint32_t u = (uint32_t)col[i];
      int32_t lo = rp[u], hi = rp[u + 1] - 1;
      bool found = false;
      while (lo <= hi) {
        const int32_t mid = (lo + hi) >> 1;
        const uint32_t x = (uint32_t)col[mid];
        if (x == v) {
          found = true;
          break;
        }
        if (x < v)
          lo = mid + 1;
        else
          hi = mid - 1;
      }
      if (!found) return false;
    }
  }
  return true;
}

__device__ __noinline__ bool sp_check_input(int64_t m) {
  const SpWarp& W = sp_w();
  if (!__all_sync(GCL_FULL, sp_check_rows(W.rp, W.col, W.n, m, lane_id(), 32))) return false;
  return __all_sync(GCL_FULL, sp_check_mates(W.rp, W.col, W.n, lane_id(), 32));
}

struct SpResult {
  int32_t status;
  int num_aut;
  int64_t nodes;
};

// Point the warp's arrays into its slot (and its shared-memory region when
// the per-step arrays fit there).  Lane 0 writes; the caller syncs the warp.
__device__ __noinline__ void sp_bind(uint8_t* slot, const SpLayout& Lo, uint32_t n,
                                     const int32_t* rp, const int32_t* col, uint8_t* smem,
                                     uint64_t smem_bytes, uint32_t cap, uint32_t max_aut) {
  SpWarp& W = sp_w();
  if (lane_id() != 0) return;
  W.elem = (uint16_t*)(slot + Lo.elem);
  W.pos = (uint16_t*)(slot + Lo.pos);
  W.cnt = (uint16_t*)(slot + Lo.cnt);
  // the n-sized u32 arrays
  uint32_t* base[13];
  for (int i = 0; i < 13; ++i) base[i] = (uint32_t*)(slot + Lo.u32n[i]);
  W.slog = base[0];
  W.umark = base[1];
  W.tmp = base[2];
  W.lst1 = base[3];
  W.hist = base[4];
  W.pre = base[5];
  W.seq = base[6];
  W.fseq = base[7];
  W.bseq = base[8];
  W.flabel = base[9];
  W.blabel = base[10];
  W.dsu = base[11];
  W.pathcode = (int32_t*)base[12];
  W.fixm = (uint32_t*)(slot + Lo.fixm);
  W.fixw = (cap + 31) / 32;
  W.fixst = (uint2*)(slot + Lo.fixst);
  W.fixcap = Lo.fixcap;
  W.utop = 0;
  W.fcode = (int32_t*)(slot + Lo.fcode);
  W.ccode = (int32_t*)(slot + Lo.ccode);
  W.pool_owner = (int32_t*)(slot + Lo.pool_owner);
  W.stb = (uint64_t*)(slot + Lo.stb);
  W.sts = (uint64_t*)(slot + Lo.sts);
  W.act = (uint32_t*)(slot + Lo.act);
  W.itm = (uint32_t*)(slot + Lo.itm);
  W.nsb = (uint32_t*)(slot + Lo.nsb);
  W.fcert = (uint32_t*)(slot + Lo.fcert);
  W.bcert = (uint32_t*)(slot + Lo.bcert);
  W.ccert = (uint32_t*)(slot + Lo.ccert);
  W.tc = (SpTc*)(slot + Lo.tc);
  W.reps = (uint32_t*)(slot + Lo.reps);
  W.auts = (uint16_t*)(slot + Lo.auts);
  W.rp = rp;
  W.col = col;
  W.n = n;
  W.nw = (n + 63) / 64 + 1;
  W.nsw = (W.nw + 63) / 64 + 1;
  W.stride = Lo.stride;
  W.helpers = 0;
  W.soff = kNone;
  if (smem && sp_smem_bytes(n) <= smem_bytes) {
    // stage the per-step arrays in this warp's shared memory
    const SpStage G = sp_stage(n);
    W.soff = (uint32_t)(smem - sp_dyn);
    W.elem = (uint16_t*)smem;
    W.pos = (uint16_t*)(smem + G.pos);
    W.cnt = (uint16_t*)(smem + G.cnt);
    W.stb = (uint64_t*)(smem + G.stb);
    W.sts = (uint64_t*)(smem + G.sts);
    W.act = (uint32_t*)(smem + G.act);
    W.itm = (uint32_t*)(smem + G.itm);
    W.nsb = (uint32_t*)(smem + G.nsb);
  }
  W.pool_top = 0;
  W.pool_frames = 0;
  W.pool_cap = Lo.reps_cap;
  W.aut_cap = cap;
  W.max_aut = max_aut;
}

__device__ __noinline__ SpResult sp_search(const BatchArgs& A, int g, uint8_t* slot,
                                           const SpLayout& Lo, uint32_t cap, uint8_t* smem,
                                           uint64_t smem_bytes) {
  SpWarp& W = sp_w();
  const uint32_t lane = lane_id();
  const int64_t vo = A.voff[g];
  const uint32_t n = (uint32_t)(A.voff[g + 1] - vo);
  const int64_t eo = A.eoff[g];
  const int64_t m = A.eoff[g + 1] - eo;
  SpResult res{kOk, 0, 1};
  if (n == 0) return res;
  sp_bind(slot, Lo, n, A.rowptr + vo + g, A.col + eo, smem, smem_bytes, cap, A.max_aut);
  __syncwarp();
  if (!sp_check_input(m)) {
    res.status = kBadInput;
    return res;
  }
  uint64_t deadline = 0;
  if (A.budget_ns)
    deadline = __shfl_sync(GCL_FULL, lane == 0 ? global_ns() : 0ull, 0) + A.budget_ns;
  sp_init_partition(A.color ? A.color + vo : nullptr);

  uint32_t level = 0, seqlen = 0, eqlevfirst = 0, first_seqlen = 0, best_seqlen = 0;
  int code = 0, canon_level = 0, eqlevcanon = 0, comp_canon = 0, tcl = 0, num_aut = 0;
  bool first_found = false;
  int64_t nodes = 1;
  int32_t status = kOk;
  bool pending = true;  // root refinement with every cell active
  uint64_t iter = 0;
  while (true) {
    if (pending) {
      pending = false;
      code = sp_refine();
      if (code < 0) {
        status = kInternal;
        break;
      }
      ++level;
      __syncwarp();
      if (lane == 0) {
        W.fcode[level - 1] = code;
        if (level == 1) W.utop = 0;  // the root partition is never undone
      }
      __syncwarp();
      continue;
    }
    if (level == 0) break;
    if ((++iter & 15) == 0 && deadline &&
        __shfl_sync(GCL_FULL, lane == 0 ? global_ns() : 0ull, 0) > deadline) {
      status = kTimeout;
      break;
    }
    int bt = -1, descend = -1;
    bool classify = false;
    const bool disc = W.ncells == n;
    if (!first_found) {
      if (disc) {
        // first_terminal (sequential.cpp:259-303)
        sp_leaf_cert(W.fcert);
        sp_copy_u32(W.bcert, W.fcert, (uint32_t)m);
        sp_copy_u32(W.flabel, W.elem, n);
        sp_copy_u32(W.blabel, W.elem, n);
        sp_copy_u32(W.fseq, W.seq, seqlen);
        sp_copy_u32(W.bseq, W.seq, seqlen);
        sp_copy_u32((uint32_t*)W.ccode, (const uint32_t*)W.fcode, level);
        if (lane == 0) {
          W.fcode[level] = kSentinel;
          W.ccode[level] = kSentinel;
        }
        __syncwarp();
        eqlevfirst = level;
        first_seqlen = best_seqlen = seqlen;
        first_found = true;
        canon_level = eqlevcanon = (int)level;
        comp_canon = 0;
        bt = (int)level - 1;
      } else {
        const uint32_t t = sp_first_nonsingleton();
        if (t == kNone || tcl > (int)n) {
          status = kInternal;
          break;
        }
        if (lane == 0) {
          SpTc h;
          h.first = t;
          h.len = sp_cell_end(W, t) - t;
          h.counter = 0;
          h.last = 0;
          h.rslot = kNone;
          h.pad = 0;
          W.tc[tcl] = h;
        }
        __syncwarp();
        ++tcl;
        descend = tcl - 1;
      }
    } else {
      classify = true;
      if (!disc && (eqlevfirst == level || comp_canon >= 0)) {
        if (tcl < (int)level) {
          const uint32_t t = sp_first_nonsingleton();
          if (t == kNone || tcl > (int)n) {
            status = kInternal;
            break;
          }
          if (lane == 0) {
            SpTc h;
            h.first = t;
            h.len = sp_cell_end(W, t) - t;
            h.counter = 0;
            h.last = 0;
            h.rslot = kNone;
            h.pad = 0;
            W.tc[tcl] = h;
          }
          __syncwarp();
          ++tcl;
        }
        const int idx = (int)level - 1;
        if (W.tc[idx].counter >= n) {
          bt = (int)level - 1;
          classify = false;
        } else {
          if (num_aut > 0 && num_aut > W.tc[idx].last) {
            status = sp_orbits(idx, num_aut, seqlen);
            if (status != kOk) break;
            __syncwarp();
            if (lane == 0) W.tc[idx].last = num_aut;
            __syncwarp();
          }
          descend = idx;
        }
      }
    }
    if (descend >= 0) {
      const SpTc t = W.tc[descend];
      const uint32_t v = sp_next_rep(t);
      if (v == kNone) {
        __syncwarp();
        if (lane == 0) W.tc[descend].counter = n;
        __syncwarp();
        bt = (int)level - 1;
        classify = false;
      } else {
        __syncwarp();
        if (lane == 0) {
          W.tc[descend].counter = v + 1;
          W.seq[seqlen] = v;
        }
        __syncwarp();
        ++seqlen;
        ++nodes;
        if (sp_individualize(level, v, t.first)) {
          if (!first_found) {
            pending = true;
            continue;
          }
          code = sp_refine();
          if (code < 0) {
            status = kInternal;
            break;
          }
          ++level;
        } else if (!first_found) {
          __syncwarp();
          if (lane == 0) W.fcode[level - 1] = code;
          __syncwarp();
          continue;
        }
      }
    }
    if (classify) {
      // classify_node (sequential.cpp:396-624)
      const uint32_t Lv = level;
      if (eqlevfirst == Lv - 1 && code == W.fcode[Lv - 1]) eqlevfirst = Lv;
      if (eqlevcanon == (int)Lv - 1) {
        const int cc = W.ccode[Lv - 1];
        if (code < cc) {
          comp_canon = -1;
        } else if (code > cc) {
          comp_canon = 1;
        } else {
          comp_canon = 0;
          eqlevcanon = (int)Lv;
        }
      }
      if (comp_canon > 0) {
        __syncwarp();
        if (lane == 0) W.ccode[Lv - 1] = code;
        __syncwarp();
      }
      int dec = 0;
      if (eqlevfirst != Lv && comp_canon < 0) {
        dec = 4;
      } else if (W.ncells == n) {
        sp_leaf_cert(W.ccert);
        if (eqlevfirst == Lv && sp_cmp_leaf(W.ccert, W.flabel, W.fcert, false) == 0) dec = 1;
        if (dec == 0) {
          if (comp_canon == 0) {
            if ((int)Lv < canon_level)
              comp_canon = 1;
            else
              comp_canon = sp_cmp_leaf(W.ccert, W.blabel, W.bcert, true);
          }
          dec = comp_canon == 0 ? 2 : (comp_canon > 0 ? 3 : 4);
        }
      }
      if (dec == 1 || dec == 2) {
        const uint32_t si = (uint32_t)num_aut % W.max_aut;
        if (si >= W.aut_cap) {
          status = kAutOverflow;
          break;
        }
        sp_store_aut(dec == 1 ? W.flabel : W.blabel, si);
        ++num_aut;
        const int gg = dec == 1 ? sp_gca(W.fseq, first_seqlen, seqlen)
                                : sp_gca(W.bseq, best_seqlen, seqlen);
        bt = gg >= 0 ? gg : (int)Lv - 1;
      } else if (dec == 3) {
        canon_level = eqlevcanon = (int)Lv;
        comp_canon = 0;
        sp_copy_u32(W.bcert, W.ccert, (uint32_t)m);
        sp_copy_u32(W.blabel, W.elem, n);
        sp_copy_u32(W.bseq, W.seq, seqlen);
        if (lane == 0) W.ccode[Lv] = kSentinel;
        __syncwarp();
        best_seqlen = seqlen;
        bt = (int)Lv - 1;
      } else if (dec == 4) {
        bt = (int)Lv - 1;
      }
    }
    if (bt >= 0) {
      // backtrack_to (sequential.cpp:650-670)
      const uint32_t Lv = (uint32_t)bt;
      if (Lv == 0) {
        level = 0;
        continue;
      }
      if (!sp_backtrack(Lv)) {
        status = kInternal;
        break;
      }
      if (Lv < eqlevfirst) eqlevfirst = Lv;
      if ((int)Lv <= eqlevcanon) {
        eqlevcanon = (int)Lv;
        comp_canon = 0;
      }
      seqlen = Lv - 1;
      tcl = (int)Lv;
      level = Lv;
      sp_pool_pop(Lv);
    }
  }
  res.status = status;
  res.num_aut = num_aut;
  res.nodes = nodes;
  return res;
}

// Outputs from the best leaf: labeling and the dense canonical matrix.
__device__ __noinline__ void sp_write_outputs(const BatchArgs& A, int g) {
  SpWarp& W = sp_w();
  const uint32_t lane = lane_id();
  const uint32_t n = W.n;
  const int64_t vo = A.voff[g];
  if (A.out_label)
    for (uint32_t j = lane; j < n; j += 32) A.out_label[vo + j] = (int32_t)W.blabel[j];
  if (A.out_rows) {  // row i: bit j set iff canonical i ~ j, ceil(n/64) words
    const uint32_t words = (n + 63) / 64;
    uint64_t* o = A.out_rows + A.roff[g];
    for (uint32_t i = lane; i < n; i += 32) {
      uint64_t* row = o + (uint64_t)i * words;
      for (uint32_t w = 0; w < words; ++w) row[w] = 0;
      const uint32_t v = W.blabel[i];
      for (int32_t j = W.rp[v]; j < W.rp[v + 1]; ++j) {
        const uint32_t c = W.bcert[j];
        row[c >> 6] |= bit64(c & 63);
      }
    }
  }
  if (A.out_dense) {
    uint8_t* o = A.out_dense + A.ooff[g];
    const uint64_t nn = (uint64_t)n * n;
    for (uint64_t i = lane; i < nn; i += 32) o[i] = 0;
    __syncwarp();
    for (uint32_t i = 0; i < n; ++i) {
      const uint32_t v = W.blabel[i];
      const int32_t b = W.rp[v], e = W.rp[v + 1];
      for (int32_t j = b + (int32_t)lane; j < e; j += 32) o[(uint64_t)i * n + W.bcert[j]] = 1;
    }
  }
  __syncwarp();
}

}  // namespace gcl
