// Batched path: replica-bit-packed state, two kernels per step.
//
// Layout in HBM, node-major, 32 replicas per uint32 word; every node row is
// padded to a multiple of 4 words so that a lane moves 128 replicas with one
// 16-byte access:
//   sa, sb    state planes; replica bit (a, b): S (0,0), E (0,1), I (1,0),
//             R (1,1)
//   mask      infectious bits (a & ~b); k_infect reads it, then k_flow
//             rewrites the words whose state changed
//   evs       infection events of the step (items with events only)
//   bits      four bitmaps with one bit per item (item = node x 4-word column,
//             128 replicas): act (some replica may move: E, I, waning R), inf
//             (some may be infectious), sus (some may be susceptible), evb
//             (infection events of this step).  act, inf and sus are supersets
//             of the state; evb is exact.
// The window CSR holds {col, weight} pairs (int32 contact-seconds).
//
// k_infect (exposure SpMM + infection draws), per row with contacts, lanes
// over 4-word columns (the replacement of cusparseSpMM,
// tool/gpu_cpu_temporal_sim.cu:1062, and monte_carlo_simulation, :137-159):
//   0. one lane per row ORs the neighbours' inf bits, 4 B per contact for 32
//      columns: only items with an infectious neighbour and susceptible
//      replicas go on;
//   1. inf = OR over neighbours j of mask_t[j] (16 B per lane per entry);
//   2. exposed = inf & S; the exposed replicas of a word compare the top
//      byte of their infection uniforms (8 bit-sliced planes, two Philox
//      calls per word) with that of the word bound B = max bs_r * e_max
//      (e_max = the row's total contact-seconds, so every P <= B); only
//      replicas at or below it compute their exact int64 exposure and
//      P = 1 - exp(-beta_r s_i e) and finish the comparison against
//      floor(P 2^64) (infect_event; the uniform's low 56 bits are drawn
//      only on a tie of the top byte).  Rows of more than kHeavyPairs pairs
//      sum every replica's exposure bit-sliced instead;
//   3. events are OR-ed into evs and flag their item (evb).
// k_flow (transitions + count reduction), every item set in act or evb:
//   reads the planes and the item's infection events, draws the bit-sliced
//   flow uniforms of the E, I (and waning R) replicas, 32 replicas per random
//   plane (flow_top, flow_rest), applies all moves with bitwise operations, writes the
//   planes and mask_{t+1}, and adds every transition event to the step's event
//   row; k_finalize turns initial counts + events into per-step counts.
// Every decision uses the state at the start of the step: k_infect reads the
// planes before k_flow rewrites them.
#include "rp_device.cuh"
#include "rp_internal.h"
#include "unit_rows.h"

namespace rp {
namespace {

constexpr unsigned kFull = 0xFFFFFFFFu;
constexpr int kFieldBits = 21;  // global event fields: S->E | ->I | I->
constexpr int kThreads = 256;
constexpr int kWarps = kThreads / 32;

__device__ __forceinline__ uint32_t word_mask(const PackedLayout &L, int word) {
  return word < L.vwords - 1 ? kFull : (word == L.vwords - 1 ? L.last_mask : 0u);
}

__device__ __forceinline__ uint32_t get4(const uint4 &v, int w) {
  return w == 0 ? v.x : (w == 1 ? v.y : (w == 2 ? v.z : v.w));
}

__device__ __forceinline__ void or4(uint4 &a, const uint4 b) {
  a.x |= b.x;
  a.y |= b.y;
  a.z |= b.z;
  a.w |= b.w;
}

__device__ __forceinline__ int warp_excl_scan(int v, int lane, int &total) {
  int incl = v;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const int y = __shfl_up_sync(kFull, incl, o);
    if (lane >= o) incl += y;
  }
  total = __shfl_sync(kFull, incl, 31);
  return incl - v;
}

// Position of the k-th (from 0) set bit of t (k < popc(t)), by halving.
__device__ __forceinline__ int nth_set_bit(uint32_t t, int k) {
  int pos = 0;
#pragma unroll
  for (int w = 16; w > 0; w >>= 1) {
    const int c = __popc(t & ((1u << w) - 1u));
    if (k >= c) {
      k -= c;
      pos += w;
      t >>= w;
    }
  }
  return pos;
}

__device__ __forceinline__ int find_owner(const int32_t *off, int p) {
  int owner = 0;
#pragma unroll
  for (int st = 16; st > 0; st >>= 1)
    if (off[owner + st] <= p) owner += st;
  return owner;
}

// Bitmap word and bit of item (row, col): rows of at most 32 columns share a
// word (1 << lb bits per row), wider rows take one word per slice of 32
// columns.
__device__ __forceinline__ int64_t bit_word(int lb, int n_slices, int row, int col) {
  return (int64_t)(row >> (5 - lb)) * n_slices + (col >> 5);
}
__device__ __forceinline__ int bit_shift(int lb, int row, int col) {
  return ((row & ((32 >> lb) - 1)) << lb) + (col & 31);
}
__device__ __forceinline__ uint32_t bit_of(int lb, int row, int col) {
  return 1u << bit_shift(lb, row, col);
}

// ---- k_infect ---------------------------------------------------------------
// Every warp works alone on units of consecutive rows and one slice of 32
// columns: no block-wide step, so a warp that waits for memory or draws
// holds up nobody, and units interleave over the whole grid.  (One task of
// 226 rows per 256-thread block, staged by bulk copies behind mbarriers, took
// 51 us on a step of 256 sparse networks with 17% of the items active, and a
// network of 1,000 nodes used 32 of 148 SMs.)
constexpr int kInfectQueue = 160;  // 31 left over + 4 words x 32 lanes of one pass
// Items are listed by the lanes, each in a loop over its own bits, or by the
// warp, row by row (word by word): the first takes as many turns as the fullest
// lane has items, the second one a row.  With the lanes always listing where
// their items fit, a unit of one full word took 32 turns of one lane: 32.4 us a
// step for N = 20,011, M = 1,001, 28.2 with this line (1 and 4 turns a row:
// 28.2), N = 5,000 with hubs and M = 16,384 193 and 185, N = 1,000 12.2 and 11.3.
constexpr int kListTurns = 2;

// Per warp: the unit's rows and items, and a queue of exposed words that
// accumulates over units and is decided 32 words at a time.
template <bool kCountdown>
struct InfectWarp {
  uint4 pl[32][2];             // the 8 random planes of each word (round scratch)
  UnitRows<kCountdown> u;      // the unit's rows with pairs
  int32_t list[128];           // items of a batch of 32 rows: row in batch << 5 | column
  uint32_t rmask[32];          // column masks of the batch's rows
  uint4 q[kInfectQueue];       // row, word in the row, exposed replicas, ef(e_max) of the row
                               // (countdown rule: x_max, or kSure)
  int2 span[kInfectQueue];     // the row's first CSR pair and pairs
  uint16_t cl[1024];           // candidates after the bound test: lane << 5 | bit (round scratch)
  // candidates carried to the next round (fewer than 32), self-contained
  int32_t krow[32];
  int32_t kwb[32];             // word << 5 | replica bit
  int32_t kbeg[32];
  int32_t knpr[32];
  uint8_t ku8[32];             // top 8 bits of the replica's uniform
  int32_t nk;
};
// Per warp, for rows of more than kHeavyPairs pairs (before the queue is used).
struct HeavyWarp {
  uint32_t e[32][32];  // bit k of the exposures of lane o's 32 replicas: e[k][o]
  uint4 pl[32][2];
  uint32_t C[32];
  int32_t off[32];
};
template <bool kCountdown>
constexpr int kInfectWarpBytes =
    (int)((sizeof(InfectWarp<kCountdown>) > sizeof(HeavyWarp) ? sizeof(InfectWarp<kCountdown>)
                                                              : sizeof(HeavyWarp)) + 15) / 16 * 16;
template <bool kCountdown>
constexpr int kInfectDynSmem = kWarps * kInfectWarpBytes<kCountdown>;
static_assert(kHeavyPairs < 1 << 24, "a listed geometric row's pairs beside its row");
static_assert(3 * (kInfectDynSmem<true> + 1024 + 64) <= 228 * 1024, "three blocks per SM");

// Top 8 uniform bits of replica bit b from a queued word's planes.
__device__ __forceinline__ uint32_t queued_top8(const uint4 (&q)[2], uint32_t b) {
  const uint4 a = q[0], c = q[1];
  const uint32_t pl[8] = {a.x, a.y, a.z, a.w, c.x, c.y, c.z, c.w};
  return top8_of(pl, b);
}

// What the kernel reads and writes.
struct InfectArgs {
  const int32_t *row_ptr;
  const int2 *ent;
  const uint32_t *mask, *sa, *sb;
  uint32_t *evs;
  const uint32_t *infb, *susb;
  uint32_t *evb;
  const int32_t *heavy, *heavy_end;    // rows of more than kHeavyPairs / kHugePairs pairs (window.cu)
  const unsigned long long *n_heavy;  // [0] heavy, [2] huge rows
  RowList list;                        // sparse window: rows with pairs
  uint32_t step;
  float scale;
  int32_t unit_rows, n_units;          // sparse: units follow from the list's length
};

// Decides candidate replica b of (row, word) from its exact exposure e
// (contact-seconds) and its uniform's top byte u8.
__device__ __forceinline__ void decide(const InfectArgs &d, const StepConsts &c,
                                       const PackedLayout &L, int row, int word, int b,
                                       long long e, uint32_t u8) {
  const float br = c.beta_r ? __ldg(c.beta_r + word * 32 + b) : c.beta;
  const float bs = c.sus ? __fmul_rn(br, __ldg(c.sus + row)) : br;
  float ef = __ll2float_rn(e);
  if (d.scale != 1.0f) ef = __fmul_rn(ef, d.scale);
  const float xx = __fmul_rn(bs, ef);
  if (!(xx > 0.0f)) return;
  // P <= x: a uniform whose top byte is above x's cannot infect (no
  // exponential)
  if (xx < 1.0f && u8 > fixed8(xx)) return;
  const uint32_t gword = (uint32_t)word + (c.roff >> 5);
  if (infect_event(one_minus_exp_neg(xx), u8, c.rk, (uint32_t)row, d.step,
                   gword * 32u + (uint32_t)b)) {
    atomicOr(&d.evs[(int64_t)row * L.words + word], 1u << b);
    atomicOr(&d.evb[bit_word(L.lb, L.n_slices, row, word >> 2)], bit_of(L.lb, row, word >> 2));
  }
}

// max over the word's replicas of |beta_r s_i|: every x is at most this times
// ef(e)
__device__ __forceinline__ float word_bs(const StepConsts &c, int row, int word) {
  const float bs = c.beta_r ? __ldg(c.beta_word + word) : fabsf(c.beta);
  return c.sus ? __fmul_rn(bs, fabsf(__ldg(c.sus + row))) : bs;
}

// ---- countdown rule -----------------------------------------------------------
// The reference's rule on the same gather (countdown.cu holds the rest): the
// exposed replicas draw the plain path's uniforms (Philox counter (node, step,
// replica / 4, 3), output replica % 4, on the 24-bit grid) and are candidates
// when u < x_max = -log(1 - p) * (e_max / 3600), e_max the in-order FP32 sum
// of the row's weights (every in-order sum of a subset is at most the full
// one, and P <= x).  Candidates add their infectious neighbours' weights one
// by one in CSR order, as Eigen's row-major product does, and infect iff P > u.
// Where the row's smallest weight alone gives x >= 87, P is 1 whatever the
// exposure: those replicas infect iff u < 1, without a sum.
constexpr float kSure = -1.0f;
__device__ __forceinline__ float countdown_x(const StepConsts &c, float e) {
  return __fmul_rn(c.neg_log_base, __fdiv_rn(e, 3600.0f));
}
__device__ __forceinline__ void set_events(const InfectArgs &d, const PackedLayout &L, int row,
                                           int word, uint32_t ev) {
  atomicOr(&d.evs[(int64_t)row * L.words + word], ev);
  atomicOr(&d.evb[bit_word(L.lb, L.n_slices, row, word >> 2)], bit_of(L.lb, row, word >> 2));
}
__device__ __forceinline__ void countdown_decide(const InfectArgs &d, const StepConsts &c,
                                                 const PackedLayout &L, int row, int word, int b,
                                                 float e) {
  uint32_t x[4];
  philox4x32_10_rk((uint32_t)row, d.step, (uint32_t)(word * 8 + (b >> 2)) + (c.roff >> 2),
                   kStreamInfect, c.rk, x);
  const uint32_t xb = (b & 2) ? ((b & 1) ? x[3] : x[2]) : ((b & 1) ? x[1] : x[0]);
  if (one_minus_exp_neg(countdown_x(c, e)) > unit24(xb)) set_events(d, L, row, word, 1u << b);
}
// Candidates of the round's words into Q.cl; returns their number.  One lane
// takes one quad of replicas with an exposed member (a draw covers a quad), so
// that sparse words share the draws; the events of sure words are set here.
__device__ __forceinline__ int countdown_candidates(InfectWarp<true> &Q, int at0, int n, int lane,
                                                    const InfectArgs &d, const StepConsts &c,
                                                    const PackedLayout &L) {
  uint16_t *quads = reinterpret_cast<uint16_t *>(Q.pl[0]);  // lane << 3 | quad, at most 256
  uint32_t *events = reinterpret_cast<uint32_t *>(Q.pl[16]);  // of the sure words
  const uint32_t X = lane < n ? Q.q[at0 + lane].z : 0u;
  int nq = 0;
#pragma unroll
  for (int q = 0; q < 8; ++q) {
    const bool has = ((X >> (4 * q)) & 15u) != 0u;
    const unsigned hm = __ballot_sync(kFull, has);
    if (has) quads[nq + __popc(hm & ((1u << lane) - 1u))] = (uint16_t)(lane << 3 | q);
    nq += __popc(hm);
  }
  events[lane] = 0;
  __syncwarp();
  int total = 0;
  for (int p = lane; p - lane < nq; p += 32) {
    uint32_t m = 0;
    int o = 0, q = 0;
    if (p < nq) {
      o = quads[p] >> 3;
      q = quads[p] & 7;
      const uint4 w4 = Q.q[at0 + o];
      const int row = (int)w4.x, word = (int)w4.y;
      const bool sure = __uint_as_float(w4.w) == kSure;
      const float lim = sure ? 1.0f : __uint_as_float(w4.w);
      // u = k 2^-24 < lim with k = (x >> 8) + 1, as x <= (K << 8) - 1 for the
      // largest such k
      const uint32_t K = !(lim > 0.0f) ? 0u
                         : lim > 1.0f ? 1u << 24
                                      : (uint32_t)ceilf(__fmul_rn(lim, 0x1p24f)) - 1u;
      const uint32_t last = (K << 8) - 1u;
      uint32_t x[4];
      philox4x32_10_rk((uint32_t)row, d.step, (uint32_t)(word * 8 + q) + (c.roff >> 2),
                       kStreamInfect, c.rk, x);
#pragma unroll
      for (int k = 0; k < 4; ++k) m |= x[k] <= last ? 1u << k : 0u;
      m = K ? m & w4.z >> (4 * q) : 0u;
      if (sure) {
        if (m) atomicOr(&events[o], m << (4 * q));
        m = 0;
      }
    }
    int sum;
    int at = total + warp_excl_scan(__popc(m), lane, sum);
    for (; m; m &= m - 1) Q.cl[at++] = (uint16_t)(o << 5 | 4 * q + __ffs(m) - 1);
    total += sum;
  }
  __syncwarp();
  if (events[lane]) {
    const uint4 w4 = Q.q[at0 + lane];
    set_events(d, L, (int)w4.x, (int)w4.y, events[lane]);
  }
  return total;
}

// Decides the n <= 32 queued exposed words from at0: the bound test one word per lane,
// then the exact test of the surviving candidates, one replica per lane, in
// full batches of 32 together with the candidates carried from earlier
// rounds; fewer than 32 left over are carried to the next round unless
// `drain` is set.  Events are OR-ed into their words and flag their items.
template <bool kCountdown>
__device__ __forceinline__ void infect_round(InfectWarp<kCountdown> &Q, int at0, int n, bool drain, int lane,
                                             const PackedLayout &L, const InfectArgs &d,
                                             const StepConsts &c) {
  // ---- bound test, one word per lane ----
  int ctotal;
  if constexpr (kCountdown) {
    ctotal = countdown_candidates(Q, at0, n, lane, d, c, L);
  } else {
    uint32_t Cw = 0;
    if (lane < n) {
      const uint4 q = Q.q[at0 + lane];
      const int row = (int)q.x, word = (int)q.y;
      // every exposed replica has P <= x <= |bs_r| ef(e_max) =: B; replicas
      // whose uniform's top byte is above B's cannot infect
      const float B = __fmul_rn(word_bs(c, row, word), __uint_as_float(q.w));
      if (B > 0.0f) {
        uint32_t pl[8];
        infect_planes(c.rk, (uint32_t)row, d.step, (uint32_t)word + (c.roff >> 5), pl);
        Cw = B >= 1.0f ? q.z : top8_le(q.z, fixed8(B), pl);
        Q.pl[lane][0] = make_uint4(pl[0], pl[1], pl[2], pl[3]);
        Q.pl[lane][1] = make_uint4(pl[4], pl[5], pl[6], pl[7]);
      }
    }
    int pos = warp_excl_scan(__popc(Cw), lane, ctotal);
    for (; Cw; Cw &= Cw - 1) Q.cl[pos++] = (uint16_t)(lane << 5 | (__ffs(Cw) - 1));
  }
  __syncwarp();
  // ---- exact test of 32 candidates at a time: each lane sums its own row in
  // CSR order, four mask words in flight ----
  const int nk = Q.nk;
  const int total = nk + ctotal;
  int base = 0;
  for (; total - base >= 32 || (drain && base < total); base += 32) {
    const int p = base + lane;
    if (p < total) {
      int row, word, b, npairs;
      int32_t beg;
      uint32_t u8 = 0;
      if (p < nk) {
        const int wb = Q.kwb[p];
        row = Q.krow[p];
        word = wb >> 5;
        b = wb & 31;
        if (!kCountdown) u8 = Q.ku8[p];
        beg = Q.kbeg[p];
        npairs = Q.knpr[p];
      } else {
        const int ob = Q.cl[p - nk], o = ob >> 5;
        b = ob & 31;
        const uint2 rw = *reinterpret_cast<const uint2 *>(&Q.q[at0 + o]);
        const int2 sp = Q.span[at0 + o];
        row = (int)rw.x;
        word = (int)rw.y;
        npairs = sp.y;
        if (!kCountdown) u8 = queued_top8(Q.pl[o], (uint32_t)b);
        beg = sp.x;
      }
      long long e = 0;
      float ef = 0.0f;
      for (int32_t k = 0; k < npairs; k += 4) {
        uint32_t m[4];
        int32_t wt[4];
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          m[j] = 0;
          wt[j] = 0;
          if (k + j < npairs) {
            const int2 q = __ldg(d.ent + beg + k + j);
            m[j] = __ldg(d.mask + (int64_t)q.x * L.words + word);
            wt[j] = q.y;
          }
        }
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          if (kCountdown) {
            if ((m[j] >> b) & 1u) ef = __fadd_rn(ef, __int_as_float(wt[j]));
          } else {
            e += ((m[j] >> b) & 1u) ? wt[j] : 0;
          }
        }
      }
      if (kCountdown)
        countdown_decide(d, c, L, row, word, b, ef);
      else
        decide(d, c, L, row, word, b, e, u8);
    }
  }
  __syncwarp();
  // carry the rest: slots below nk keep their entries when no batch ran
  const int rest = total - base;
  if (rest > 0) {
    const int p = base + lane;
    if (p < total && p >= nk) {
      const int ob = Q.cl[p - nk], o = ob >> 5, b = ob & 31;
      const int2 sp = Q.span[at0 + o];
      Q.kwb[lane] = (int)Q.q[at0 + o].y << 5 | b;
      Q.krow[lane] = (int)Q.q[at0 + o].x;
      Q.kbeg[lane] = sp.x;
      Q.knpr[lane] = sp.y;
      if (!kCountdown) Q.ku8[lane] = (uint8_t)queued_top8(Q.pl[o], (uint32_t)b);
    }
  }
  __syncwarp();
  if (lane == 0) Q.nk = rest > 0 ? rest : 0;
  __syncwarp();
}

// ---- rows of more than kHeavyPairs pairs ------------------------------------
// Lane = one 32-replica word, 32 words (1,024 replicas) per warp.  The exact
// exposures of a word's replicas are kept bit-sliced: s[k] holds bit k of all
// 32 sums, and adding a pair's weight to the replicas of its mask word is a
// ripple-carry add, three logic operations per bit of the row's total
// whatever the number of replicas.  Afterwards a word's candidates are the
// replicas whose uniform's top byte is at most floor(256 x') with x' >= x the
// exposure times the next power of two above beta, compared bit-sliced; their
// exposures are read back from the planes, so no candidate walks its row
// again.  (Before, a word with candidates took one pass over its row with lane
// = replica and an e_max bound near 1 let nearly every exposed replica
// through: 7.5 ms on the first steps of the dense network, N = 5,000 and
// M = 16,384, 0.15-0.44 ms now.  The line at 48 pairs and the block-wide line
// at 256, chosen when a step took 216 us there (185 now): 48/128 222, 32/128
// 224, 63/192 222, 32/512 242, 16/512 261.)
__device__ __forceinline__ void sliced_add(uint32_t (&s)[32], uint32_t m, uint32_t w, int nb) {
  uint32_t cy = 0;
#pragma unroll
  for (int g = 0; g < 8; ++g) {
    if (4 * g >= nb) break;
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const int k = 4 * g + j;
      const uint32_t a = ((w >> k) & 1u) ? m : 0u, t = s[k];
      s[k] = t ^ a ^ cy;
      cy = (t & a) | (t & cy) | (a & cy);
    }
  }
}

struct HeavyUnit {
  int row, w0;          // first word
  int32_t beg, end;
  int nb;               // bits of the row's total weight
  uint32_t S;           // the lane's susceptible replicas
};

// Loads unit u of `rows` x nws words; false when no replica is susceptible.
__device__ __forceinline__ bool heavy_load(HeavyUnit &h, const int32_t *list, int dir, int u,
                                           int nws, int lane, const PackedLayout &L,
                                           const InfectArgs &d) {
  h.row = list[dir * (u / nws)];
  if (d.list.rows) {  // sparse window: an entry of its row list
    const int2 sp = __ldg(d.list.span + h.row);
    h.beg = sp.x;
    h.end = sp.x + sp.y;
    h.row = __ldg(d.list.rows + h.row);
  } else {
    h.beg = d.row_ptr[h.row];
    h.end = d.row_ptr[h.row + 1];
  }
  const int ws = u % nws;
  h.w0 = ws * 32;
  const int word = h.w0 + lane;
  const uint32_t sb8 = d.susb[bit_word(L.lb, L.n_slices, h.row, ws * 8)] >>
                       bit_shift(L.lb, h.row, ws * 8);
  if (!(sb8 & (L.lb >= 3 ? 0xFFu : (1u << (1 << L.lb)) - 1u))) return false;
  h.S = 0;
  if (word < L.vwords) {
    const int64_t wi = (int64_t)h.row * L.words + word;
    h.S = ~d.sa[wi] & ~d.sb[wi] & word_mask(L, word);
  }
  if (!__any_sync(kFull, h.S != 0u)) return false;
  long long emax = 0;
  for (int32_t k = h.beg + lane; k < h.end; k += 32) emax += __ldg(&d.ent[k].y);
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) emax += __shfl_xor_sync(kFull, emax, o);
  h.nb = 64 - __clzll(emax);
  return true;
}

// Adds the pairs first, first + stride, ... of the unit's row to H.e (planes
// of the 32 words) and returns the lane's exposed replicas.
__device__ __forceinline__ uint32_t heavy_sum(const HeavyUnit &h, HeavyWarp &H, int first,
                                              int stride, int lane, const PackedLayout &L,
                                              const InfectArgs &d) {
  uint32_t s[32];
#pragma unroll
  for (int k = 0; k < 32; ++k) s[k] = 0;
  uint32_t X = 0;
  const uint32_t *mw = d.mask + min(h.w0 + lane, L.words - 1);
  const int nb = min(h.nb, 32);
  for (int32_t k = h.beg + first; k < h.end; k += 2 * stride) {
    uint32_t m[2], w[2];
#pragma unroll
    for (int j = 0; j < 2; ++j) {
      m[j] = 0;
      w[j] = 0;
      if (k + j * stride < h.end) {
        const int2 q = __ldg(d.ent + k + j * stride);
        w[j] = (uint32_t)q.y;
        m[j] = __ldg(mw + (int64_t)q.x * L.words);
      }
    }
#pragma unroll
    for (int j = 0; j < 2; ++j) {
      m[j] &= h.S;
      X |= m[j];
      if (h.nb <= 32 && __any_sync(kFull, m[j] != 0u)) sliced_add(s, m[j], w[j], nb);
    }
  }
#pragma unroll
  for (int k = 0; k < 32; ++k)
    if (k < nb) H.e[k][lane] = s[k];
  return X;
}

// The candidates among the lane's exposed replicas X, their random planes and
// the scan offsets, for heavy_decide.
__device__ __forceinline__ void heavy_candidates(const HeavyUnit &h, HeavyWarp &H, uint32_t X,
                                                 int lane, const PackedLayout &L,
                                                 const InfectArgs &d, const StepConsts &c) {
  uint32_t cand = 0;
  if (X) {
    const int word = h.w0 + lane;
    uint32_t pl[8];
    infect_planes(c.rk, (uint32_t)h.row, d.step, (uint32_t)word + (c.roff >> 5), pl);
    H.pl[lane][0] = make_uint4(pl[0], pl[1], pl[2], pl[3]);
    H.pl[lane][1] = make_uint4(pl[4], pl[5], pl[6], pl[7]);
    // x <= e t (the 1.0001 covers the roundings of x), t < 2^ex
    const float t = __fmul_rn(__fmul_rn(word_bs(c, h.row, word), d.scale), 1.0001f);
    if (!(t < 0x1p-8f) || h.nb > 32) {
      cand = X;
    } else if (t > 0.0f) {
      const int ex = (int)((__float_as_uint(t) >> 23) & 0xFFu) - 126;
      const int p0 = -ex - 8;  // floor(256 e 2^ex) = e >> p0
      uint32_t hi = 0;
      for (int k = p0 + 8; k < h.nb; ++k) hi |= H.e[k][lane];
      uint32_t lt = 0, und = X & ~hi;
#pragma unroll
      for (int j = 0; j < 8; ++j) {
        const int k = p0 + 7 - j;
        const uint32_t v = k < h.nb ? H.e[k][lane] : 0u;
        lt |= und & v & ~pl[j];
        und &= ~(v ^ pl[j]);
      }
      cand = (X & hi) | lt | und;
    }
  }
  H.C[lane] = cand;
  int total;
  H.off[lane] = warp_excl_scan(__popc(cand), lane, total);
}

// Exact decisions of H's candidates in batches first, first + stride, ...
__device__ __forceinline__ void heavy_decide(const HeavyUnit &h, const HeavyWarp &H, int first,
                                             int stride, int lane, const PackedLayout &L,
                                             const InfectArgs &d, const StepConsts &c) {
  const int total = H.off[31] + __popc(H.C[31]);
  for (int p = 32 * first + lane; p < total; p += 32 * stride) {
    const int o = find_owner(H.off, p);
    const int b = nth_set_bit(H.C[o], p - H.off[o]);
    unsigned long long e = 0;
    if (h.nb <= 32) {
      for (int k = 0; k < h.nb; ++k) e |= (unsigned long long)((H.e[k][o] >> b) & 1u) << k;
    } else {  // totals beyond 2^32 contact-seconds: a plain sum
      for (int32_t k = h.beg; k < h.end; ++k) {
        const int2 q = __ldg(d.ent + k);
        if ((__ldg(d.mask + (int64_t)q.x * L.words + h.w0 + o) >> b) & 1u) e += (uint32_t)q.y;
      }
    }
    decide(d, c, L, h.row, h.w0 + o, b, (long long)e, queued_top8(H.pl[o], (uint32_t)b));
  }
}

template <bool kCountdown>
__global__ void __launch_bounds__(kThreads, 3)
    k_infect(PackedLayout L, const __grid_constant__ InfectArgs d,
             const __grid_constant__ StepConsts c) {
  extern __shared__ __align__(16) unsigned char s_dyn[];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  // warps of one block are gridDim.x apart: neighbouring units go to
  // different SMs
  const int gw = warp * gridDim.x + blockIdx.x, tw = kWarps * gridDim.x;
  __shared__ unsigned s_next;  // the block's units handed out so far
  if (threadIdx.x == 0) s_next = 0;
  __syncthreads();
  int n_heavy = 0, n_huge = 0;
  if (!kCountdown) {  // the countdown rule's FP32 sums have an order
    n_heavy = (int)d.n_heavy[0];
    n_huge = (int)d.n_heavy[2];
  }
  if (!kCountdown && (n_heavy | n_huge)) {
    const int nws = (L.words + 31) / 32;
    HeavyWarp &H = *reinterpret_cast<HeavyWarp *>(s_dyn + warp * kInfectWarpBytes<kCountdown>);
    HeavyUnit h;
    // Rows of more than kHugePairs pairs first: the block's warps share the
    // pairs, warp 0 adds their planes, and the decisions are shared again.
    // Then one warp per unit.  (One loop for both: a second copy of the
    // unrolled sums costs more in instruction fetches than the tests here.)
    bool huge = n_huge > 0;
    for (int u = huge ? (int)blockIdx.x : gw;; u += huge ? (int)gridDim.x : tw) {
      if (huge && u >= n_huge * nws) {  // the same for all warps of the block
        huge = false;
        u = gw;
      }
      if (!huge && u >= n_heavy * nws) break;
      if (!heavy_load(h, huge ? d.heavy_end - 1 : d.heavy, huge ? -1 : 1, u, nws, lane, L, d))
        continue;
      uint32_t X = heavy_sum(h, H, huge ? warp : 0, huge ? kWarps : 1, lane, L, d);
      HeavyWarp &Hd = huge ? *reinterpret_cast<HeavyWarp *>(s_dyn) : H;
      if (huge) {
        H.C[lane] = X;
        __syncthreads();
        for (int v = 1; v < kWarps && warp == 0; ++v) {
          const HeavyWarp &Hv = *reinterpret_cast<const HeavyWarp *>(s_dyn + v * kInfectWarpBytes<kCountdown>);
          X |= Hv.C[lane];
          uint32_t cy = 0;
          for (int k = 0; k < min(h.nb, 32); ++k) {
            const uint32_t a = H.e[k][lane], t = Hv.e[k][lane];
            H.e[k][lane] = a ^ t ^ cy;
            cy = (a & t) | (a & cy) | (t & cy);
          }
        }
      }
      if (!huge || warp == 0) heavy_candidates(h, Hd, X, lane, L, d, c);
      if (huge) __syncthreads(); else __syncwarp();
      heavy_decide(h, Hd, huge ? warp : 0, huge ? kWarps : 1, lane, L, d, c);
      if (huge) __syncthreads(); else __syncwarp();
    }
  }

  InfectWarp<kCountdown> &Q = *reinterpret_cast<InfectWarp<kCountdown> *>(s_dyn + warp * kInfectWarpBytes<kCountdown>);
  if (lane == 0) Q.nk = 0;
  __syncwarp();
  int nq = 0;  // queued words
  const int n_rows = d.list.rows ? (int)d.list.counts[1] : L.n_nodes;
  const int n_units =
      d.list.rows ? (n_rows + d.unit_rows - 1) / d.unit_rows * L.n_slices : d.n_units;
  // the block's units, blockIdx.x + k gridDim.x, go to its warps as they ask;
  // warps that arrive together (no rows taken above) start with one each
  const bool own_first = !(n_heavy | n_huge);
  auto next_unit = [&]() {
    int k = 0;
    if (lane == 0) k = (int)atomicAdd(&s_next, 1u) + (own_first ? kWarps : 0);
    return (int)blockIdx.x + __shfl_sync(kFull, k, 0) * (int)gridDim.x;
  };
  int unit = -1;
  const uint4 *mask4 = reinterpret_cast<const uint4 *>(d.mask);
  const uint4 *sa4 = reinterpret_cast<const uint4 *>(d.sa);
  const uint4 *sb4 = reinterpret_cast<const uint4 *>(d.sb);
  bool more = true;
  int cbase = 0, cnt = 0;    // the current unit's first column; items listed
  int r0 = 0;                // the unit's first row
  int nrows = 0, ub = 0;     // the unit's rows with pairs; the first row not yet taken
  int lrow = 0, n = 0;       // the lane's row of the batch: pairs beg .. beg + n
  int32_t beg = 0;
  unsigned nz = 0;           // rows of the batch with items not yet listed
  for (;;) {
    if (cnt == 0 && !nz) {
      if (ub >= nrows) {
        unit = unit < 0 && own_first ? gw : next_unit();
        if (unit >= n_units) {
          more = false;
        } else {
          // the next unit's rows that have pairs (longer rows were taken above)
          const int rb = L.n_slices == 1 ? unit : unit / L.n_slices;
          cbase = L.n_slices == 1 ? 0 : (unit - rb * L.n_slices) * 32;
          r0 = rb * d.unit_rows;
          const int r1 = min(r0 + d.unit_rows, n_rows);
          nrows = ub = 0;
          __syncwarp();
          for (int r = r0; r < r1; r += 128) {
            int32_t b[4], len[4];
#pragma unroll
            for (int j = 0; j < 4; ++j) {
              const int row = r + 32 * j + lane;
              b[j] = len[j] = 0;
              if (row < r1) {
                if (d.list.rows) {
                  const int2 sp = __ldg(d.list.span + row);
                  b[j] = sp.x;
                  len[j] = sp.y;
                } else {
                  b[j] = __ldg(d.row_ptr + row);
                  len[j] = __ldg(d.row_ptr + row + 1) - b[j];
                }
              }
            }
#pragma unroll
            for (int j = 0; j < 4; ++j) {
              if (r + 32 * j >= r1) break;
              const bool has = len[j] > 0 && (kCountdown || len[j] <= kHeavyPairs);
              const unsigned hm = __ballot_sync(kFull, has);
              if (has) {
                Q.u.put(nrows + __popc(hm & ((1u << lane) - 1u)), r - r0 + 32 * j + lane, b[j],
                        len[j]);
              }
              nrows += __popc(hm);
            }
          }
          __syncwarp();
          if (nrows == 0) continue;
        }
      }
      // ---- phase 0: items of the next 32 rows with an infectious neighbour and
      // susceptible replicas.  Lane = row: the OR of the neighbours' inf bits
      // gives the row's columns at 4 B per contact, where the mask words of 32
      // columns cost 512 B ----
      if (more) {
        n = 0;
        if (ub + lane < nrows) {
          Q.u.get(ub + lane, lrow, beg, n);
          lrow += r0;
          if (d.list.rows) lrow = __ldg(d.list.rows + lrow);
        }
        ub += 32;
        auto row_bits = [&](const uint32_t *bits, int r) {
          return __ldg(bits + bit_word(L.lb, L.n_slices, r, cbase)) >> bit_shift(L.lb, r, 0);
        };
        const int ncols = min(32, L.q4 - cbase);
        uint32_t sus = n ? row_bits(d.susb, lrow) : 0u, m = 0;
        sus &= ncols == 32 ? kFull : (1u << ncols) - 1u;
        for (int k = 0; k < n && (!kCountdown || n <= 32); k += 4) {  // four words in flight
          uint32_t v[4];
#pragma unroll
          for (int j = 0; j < 4; ++j)
            v[j] = k + j < n ? row_bits(d.infb, __ldg(&d.ent[beg + k + j].x)) : 0u;
          m |= v[0] | v[1] | v[2] | v[3];
        }
        if (kCountdown)  // longer rows are shared by the warp
          for (unsigned big = __ballot_sync(kFull, n > 32); big; big &= big - 1) {
            const int o = __ffs(big) - 1;
            const int32_t ob = __shfl_sync(kFull, beg, o), on = __shfl_sync(kFull, n, o);
            uint32_t om = 0;
            for (int k = lane; k < on; k += 32) om |= row_bits(d.infb, __ldg(&d.ent[ob + k].x));
            om = __reduce_or_sync(kFull, om);
            if (lane == o) m = om;
          }
        m &= sus;
        // few items on many rows: every lane lists its own row's; else row by
        // row below, which takes about as long for a row as two turns of the
        // lanes' loop
        nz = __ballot_sync(kFull, m != 0u);
        if (!nz) continue;
        if (__reduce_max_sync(kFull, __popc(m)) <= kListTurns * __popc(nz)) {
          int tot;
          int pos = warp_excl_scan(__popc(m), lane, tot);
          if (tot <= 128) {
            for (; m; m &= m - 1) Q.list[pos++] = lane << 5 | (__ffs(m) - 1);
            cnt = tot;
            nz = 0;
          }
        }
        if (nz) Q.rmask[lane] = m;
        __syncwarp();
      }
    }
    while (cnt < 32 && nz) {
      const int o = __ffs(nz) - 1;
      nz &= nz - 1;
      const uint32_t m = Q.rmask[o];
      if ((m >> lane) & 1u) Q.list[cnt + __popc(m & ((1u << lane) - 1u))] = o << 5 | lane;
      cnt += __popc(m);
    }
    __syncwarp();
    // ---- phase 1: gather, one item per lane ----
    const int got = min(cnt, 32);
    cnt -= got;
    const bool ok = lane < got;
    const int it = ok ? Q.list[cnt + lane] : 0;
    __syncwarp();
    const int row = __shfl_sync(kFull, lrow, it >> 5), col = cbase + (it & 31);
    const int32_t rbeg = __shfl_sync(kFull, beg, it >> 5);
    const int rn = __shfl_sync(kFull, n, it >> 5);
    uint32_t X[4] = {0, 0, 0, 0};
    float efmax = 0.0f;
    if (ok) {
      const int64_t idx = (int64_t)row * L.q4 + col;
      // countdown rule: one plane, the replicas that are not susceptible
      const uint4 a4 = __ldg(sa4 + idx), b4 = kCountdown ? a4 : __ldg(sb4 + idx);
      uint4 inf = make_uint4(0, 0, 0, 0);
      long long emax = 0;
      float fmax = 0.0f, wmin = 3e38f;  // countdown rule: in-order sum, smallest weight
      for (int k = 0; k < rn; k += 4) {  // four mask items in flight
        uint4 m[4];
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          m[j] = make_uint4(0, 0, 0, 0);
          if (k + j < rn) {
            const int2 q = __ldg(d.ent + rbeg + k + j);
            m[j] = __ldg(mask4 + (int64_t)q.x * L.q4 + col);
            if (kCountdown) {
              const float wt = __int_as_float(q.y);
              fmax = __fadd_rn(fmax, wt);
              if (wt > 0.0f) wmin = fminf(wmin, wt);  // duplicates merged away weigh 0
            } else {
              emax += q.y;
            }
          }
        }
#pragma unroll
        for (int j = 0; j < 4; ++j) or4(inf, m[j]);
      }
#pragma unroll
      for (int w = 0; w < 4; ++w)
        X[w] = get4(inf, w) & ~get4(a4, w) & ~get4(b4, w) & word_mask(L, 4 * col + w);
      if (kCountdown) {
        efmax = countdown_x(c, wmin) >= 87.0f ? kSure : countdown_x(c, fmax);
      } else {
        efmax = __ll2float_rn(emax);
        if (d.scale != 1.0f) efmax = __fmul_rn(efmax, d.scale);
      }
    }
    // ---- queue the exposed words ----
#pragma unroll
    for (int w = 0; w < 4; ++w) {
      const unsigned qm = __ballot_sync(kFull, X[w] != 0u);
      if (X[w]) {
        const int pos = nq + __popc(qm & ((1u << lane) - 1u));
        Q.q[pos] = make_uint4((uint32_t)row, (uint32_t)(4 * col + w), X[w], __float_as_uint(efmax));
        Q.span[pos] = make_int2(rbeg, rn);
      }
      nq += __popc(qm);
    }
    __syncwarp();
    // ---- decide full rounds, the last queued words first, and what is left
    // past the last unit ----
    while (nq >= 32 || (!more && (nq > 0 || Q.nk > 0))) {
      const int take = min(nq, 32);
      nq -= take;
      infect_round<kCountdown>(Q, nq, take, !more && nq == 0, lane, L, d, c);
    }
    if (!more) break;
  }
}

// ---- k_flow -------------------------------------------------------------------
// Transition events go straight to the step's event row with one 64-bit
// reduction each: about 1% of the active replicas move in a step, and warps
// that share no counters need no barrier.  (Counters in shared memory cost
// every block a clear, a flush and two barriers per task, and tied a block's
// warps to one network and slice.)
__device__ __forceinline__ void count_bits(unsigned long long *s_ev, int wl, uint32_t t,
                                           unsigned long long inc) {
  while (t) {
    const int r = __ffs(t) - 1;
    atomicAdd(&s_ev[wl * 32 + r], inc);
    t &= t - 1;
  }
}

struct FlowArgs {
  uint32_t *evs, *mask, *sa, *sb;
  uint32_t *actb, *infb, *susb, *evb;
  unsigned long long *ev_row, *rs_row;
  const int32_t *net_first;  // several networks: their first rows
  int32_t n_nets;
  uint32_t step;
  int32_t split;             // a unit is 1 / (1 << split) of a bitmap word
  int32_t take;              // units a warp takes at a time (at most 32)
  int64_t n_units;
};

// Applies one word's infection events and flows (disjoint state bits) to the
// start-of-step planes, writes what changed and counts the events.
__device__ __forceinline__ void apply_word(const PackedLayout &L, const FlowArgs &d,
                                           const StepConsts &c, bool waning, int row, int word,
                                           uint32_t A, uint32_t B, uint32_t evS, uint32_t f) {
  const uint32_t E = ~A & B, I = A & ~B, Rw = waning ? (A & B) : 0u;
  const uint32_t evE = f & E, evI = f & I, evR = f & Rw;
  uint32_t all = evS | evE | evI | evR;
  if (!all) return;
  uint32_t na = A, nb = B;
  if (c.has_exposed)
    nb |= evS;
  else
    na |= evS;
  na |= evE;
  nb &= ~evE;
  if (c.ir_to_s)
    na &= ~evI;
  else
    nb |= evI;
  na &= ~evR;
  nb &= ~evR;
  const int64_t wi = (int64_t)row * L.words + word;
  d.sa[wi] = na;
  d.sb[wi] = nb;
  const uint32_t mk = na & ~nb;
  if (mk != I) {
    d.mask[wi] = mk;
    if (!I) atomicOr(&d.infb[bit_word(L.lb, L.n_slices, row, word >> 2)], bit_of(L.lb, row, word >> 2));
  }
  int net = 0;
  if (d.n_nets > 1) {  // the row's network: last first row <= row
    int hi = d.n_nets;
    while (hi - net > 1) {
      const int mid = (net + hi) >> 1;
      if (__ldg(d.net_first + mid) <= row) net = mid; else hi = mid;
    }
  }
  const int64_t base = (int64_t)net * L.m + word * 32;
  for (; all; all &= all - 1) {
    const uint32_t bit = all & (0u - all);
    const int64_t rep = base + __ffs(all) - 1;
    if (evR & bit) {
      atomicAdd(&d.rs_row[rep], 1ull);
    } else {
      const int field = (evI & bit) ? 2 * kFieldBits
                                    : (((evE & bit) || !c.has_exposed) ? kFieldBits : 0);
      atomicAdd(&d.ev_row[rep], 1ull << field);
    }
  }
}

// Per-warp queue of words with flow candidates or infection events (dynamic
// shared memory): words are queued while the warp streams its items and drawn
// in full 32-lane rounds, so sparse candidates do not leave lanes idle.  An
// entry carries its planes: read again from global memory they miss the
// L1 that the passes of 24 warps stream through.
constexpr int kFlowIPL = 2;      // items per lane per pass (loads in flight)
constexpr int kFlowQueue = 31 + 4 * kFlowIPL * 32 + 1;  // left over + one pass
struct FlowQueue {
  uint4 q[kFlowQueue];           // row, word (kWordEvent: infection events), planes a and b
  uint4 q2[64];                  // words that the first draw left with candidates or events
  uint32_t cand2[64];
  uint32_t list[32 * kFlowIPL];  // items of the next pass (see k_flow)
};
constexpr int kFlowDynSmem = kWarps * (int)sizeof(FlowQueue);
constexpr uint32_t kWordEvent = 1u << 30;

// Streams the active items (act | evb, 32 items per bitmap word), units of
// the bitmap interleaved over all blocks and handed to a block's warps as they
// ask; words with flow candidates or infection events are queued.
// Loading an item also brings its act, inf and sus bits up to date with the
// planes it found; moves made afterwards only set bits (inf, on a word's first
// infectious replica), so a bit may stay set one step too long and is never
// missing.
__global__ void __launch_bounds__(kThreads, 3)
    k_flow(PackedLayout L, const __grid_constant__ FlowArgs d, const __grid_constant__ StepConsts c) {
  extern __shared__ __align__(16) unsigned char s_dynf[];
  FlowQueue &Q = reinterpret_cast<FlowQueue *>(s_dynf)[threadIdx.x >> 5];
  const int lane = threadIdx.x & 31;
  const bool waning = c.th.tr_all || c.th.tr != 0;
  __shared__ unsigned s_next;  // the block's units, blockIdx.x + k gridDim.x, taken so far
  const int warp = threadIdx.x >> 5;
  if (threadIdx.x == 0) s_next = kWarps * d.take;
  __syncthreads();
  const uint4 *sa4 = reinterpret_cast<const uint4 *>(d.sa);
  const uint4 *sb4 = reinterpret_cast<const uint4 *>(d.sb);
  const uint4 *evs4 = reinterpret_cast<const uint4 *>(d.evs);
  // the lane's unit of the current block: its bitmap word and bits
  int64_t wi = 0;
  bool more = true, first = true;  // a warp's first block of units is its own
  int wrow = 0, wcol = 0;     // first row and column of the lane's word
  uint32_t aw = 0, ew = 0, iw = 0, sw = 0;
  unsigned nz = 0;            // lanes with items not yet listed
  int got = 0, n1 = 0, n2 = 0;  // items listed; words queued; words left by the first draw
  const bool certain = c.th.te_all || c.th.ti_all || c.th.tr_all;
  // warp-uniform passes of kFlowIPL items per lane, all loads issued first;
  // candidate words are queued, and full rounds of 32 decided after the pass
  // (one pass past the items decides the rest; one call site of the draws
  // keeps the kernel small)
  for (;;) {
    while (!nz && !got && more) {
      unsigned k = (unsigned)(warp * d.take);
      if (!first) {
        if (lane == 0) k = atomicAdd(&s_next, (unsigned)d.take);
        k = __shfl_sync(kFull, k, 0);
      }
      first = false;
      more = blockIdx.x + (int64_t)(k + d.take) * gridDim.x < d.n_units;
      const int64_t u = blockIdx.x + (int64_t)(k + lane) * gridDim.x;
      aw = ew = 0;
      if (lane < d.take && u < d.n_units) {
        wi = u >> d.split;
        const int len = 32 >> d.split;
        const uint32_t own = (kFull >> (32 - len)) << (len * (int)(u & ((1 << d.split) - 1)));
        aw = d.actb[wi] & own;
        ew = d.evb[wi] & own;
        iw = d.infb[wi];
        sw = d.susb[wi];
        if (aw | ew) {
          const int64_t wr = L.n_slices == 1 ? wi : wi / L.n_slices;
          wrow = (int)wr << (5 - L.lb);
          wcol = (int)(wi - wr * L.n_slices) * 32;
        }
        if (ew) atomicAnd(&d.evb[wi], ~own);
      }
      // few items in many words: every lane lists its own word's; else word by
      // word below (one word of 32 items is one turn there, 32 here)
      nz = __ballot_sync(kFull, (aw | ew) != 0u);
      if (nz && __reduce_max_sync(kFull, __popc(aw | ew)) <= kListTurns * __popc(nz)) {
        int tot;
        int pos = warp_excl_scan(__popc(aw | ew), lane, tot);
        if (tot <= 32 * kFlowIPL) {
          for (uint32_t t = aw | ew; t; t &= t - 1) {
            const int b = __ffs(t) - 1;
            Q.list[pos++] = (uint32_t)(lane << 5 | b) | ((aw >> b) & 1u) << 31 |
                            ((ew >> b) & 1u) << 30 | ((iw >> b) & 1u) << 29 |
                            ((sw >> b) & 1u) << 28;
          }
          got = tot;
          nz = 0;
        }
      }
    }
    while (nz && got <= 32 * (kFlowIPL - 1)) {
      const int o = __ffs(nz) - 1;
      nz &= nz - 1;
      const uint32_t a = __shfl_sync(kFull, aw, o), e = __shfl_sync(kFull, ew, o);
      const uint32_t i1 = __shfl_sync(kFull, iw, o), s1 = __shfl_sync(kFull, sw, o);
      const uint32_t w = a | e;
      if ((w >> lane) & 1u)
        Q.list[got + __popc(w & ((1u << lane) - 1u))] =
            (uint32_t)(o << 5 | lane) | ((a >> lane) & 1u) << 31 | ((e >> lane) & 1u) << 30 |
            ((i1 >> lane) & 1u) << 29 | ((s1 >> lane) & 1u) << 28;
      got += __popc(w);
    }
    __syncwarp();
    const bool flushing = got == 0;
    if (flushing && n1 == 0 && n2 == 0) break;
    int rl[kFlowIPL], cl[kFlowIPL];
    uint32_t st[kFlowIPL];
    uint4 a4[kFlowIPL], b4[kFlowIPL], e4[kFlowIPL];
#pragma unroll
    for (int h = 0; h < kFlowIPL; ++h) {
      st[h] = 0;
      rl[h] = cl[h] = 0;
      a4[h] = b4[h] = e4[h] = make_uint4(0, 0, 0, 0);
      if (32 * h >= got) continue;  // warp-uniform, as below
      const bool in = 32 * h + lane < got;
      if (in) st[h] = Q.list[32 * h + lane];
      const int o = (st[h] >> 5) & 31, bit = st[h] & 31;
      rl[h] = __shfl_sync(kFull, wrow, o) + (bit >> L.lb);
      cl[h] = __shfl_sync(kFull, wcol, o) + (bit & ((1 << L.lb) - 1));
      if (in) {
        const int64_t idx = (int64_t)rl[h] * L.q4 + cl[h];
        a4[h] = sa4[idx];
        b4[h] = sb4[idx];
        if ((st[h] >> 30) & 1u) e4[h] = evs4[idx];
      }
    }
#pragma unroll
    for (int h = 0; h < kFlowIPL; ++h) {
      if (32 * h >= got) continue;
      uint32_t cm = 0, evm = 0, s4 = 0, i4 = 0, r4 = 0;
#pragma unroll
      for (int w = 0; w < 4; ++w) {  // padding replicas are S: no replica mask needed
        const uint32_t A = get4(a4[h], w), B = get4(b4[h], w);
        if ((waning ? (A | B) : (A ^ B)) != 0u) cm |= 1u << w;
        i4 |= A & ~B;
        r4 |= A & B;
        // padding replicas are S, so only a row's last item needs the mask
        const uint32_t S = ~(A | B);
        s4 |= 4 * cl[h] + 4 > L.vwords ? S & word_mask(L, 4 * cl[h] + w) : S;
      }
      // S now, or back to S this step (waning R, or I -> S)
      if (waning) s4 |= r4;
      if (c.ir_to_s) s4 |= i4;
      // words with infection events join the queue (they need no draw)
#pragma unroll
      for (int w = 0; w < 4; ++w)
        if (get4(e4[h], w)) evm |= 1u << w;
      cm |= evm;
#pragma unroll
      for (int w = 0; w < 4; ++w) {
        const unsigned qm = __ballot_sync(kFull, (cm >> w) & 1u);
        if (!qm) continue;
        if ((cm >> w) & 1u)
          Q.q[n1 + __popc(qm & ((1u << lane) - 1u))] =
              make_uint4((uint32_t)rl[h],
                         (uint32_t)(4 * cl[h] + w) | ((evm >> w) & 1u ? kWordEvent : 0u),
                         get4(a4[h], w), get4(b4[h], w));
        n1 += __popc(qm);
      }
      const uint32_t now = (cm ? 8u : 0u) | ((st[h] >> 28) & 4u) |
                           (i4 ? 2u : 0u) | (s4 ? 1u : 0u);
      const uint32_t diff = st[h] >> 28 ? now ^ (st[h] >> 28) : 0u;  // the list entry is in use
      if (diff) {
        const int64_t bw = bit_word(L.lb, L.n_slices, rl[h], cl[h]);
        const uint32_t bit = bit_of(L.lb, rl[h], cl[h]);
        if (diff & 8u) atomicXor(&d.actb[bw], bit);
        if (diff & 2u) atomicXor(&d.infb[bw], bit);
        if (diff & 1u) atomicXor(&d.susb[bw], bit);
      }
    }
    got = 0;
    __syncwarp();  // bits are cleared before a round of this warp may set them
    // Two rounds of draws, 32 words each.  With every rate below 1/16 (1/256)
    // the first round (planes 0-3, or 0-7) leaves one candidate in 16 (256),
    // and a word without any and without infection events is done: no second
    // draw, no write.  The words left are collected again, so that the second
    // round's lanes are full too.
    for (;;) {
      const bool draw = n1 >= 32 || (flushing && n1 > 0);
      if (draw) {
        const int take = min(n1, 32);
        n1 -= take;
        uint4 q = make_uint4(0, 0, 0, 0);
        bool keep = false;
        uint32_t cand = 0;
        if (lane < take) {
          q = Q.q[n1 + lane];
          cand = flow_candidates(~q.z & q.w, q.z & ~q.w, waning ? (q.z & q.w) : 0u, c.th);
          if (c.th.lead && cand)
            cand = flow_top(cand, c.th, c.rk, q.x, d.step, (q.y & ~kWordEvent) + (c.roff >> 5));
          keep = cand || q.y >= kWordEvent || certain;
        }
        const unsigned km = __ballot_sync(kFull, keep);
        if (keep) {
          const int at = n2 + __popc(km & ((1u << lane) - 1u));
          Q.q2[at] = q;
          Q.cand2[at] = cand;
        }
        n2 += __popc(km);
        __syncwarp();
      }
      if (n2 >= 32 || (flushing && !draw && n2 > 0)) {
        const int take = min(n2, 32);
        n2 -= take;
        if (lane < take) {
          const uint4 q = Q.q2[n2 + lane];
          const uint32_t cand = Q.cand2[n2 + lane], A = q.z, B = q.w;
          const int row = (int)q.x, word = (int)(q.y & ~kWordEvent);
          uint32_t ev = 0;
          if (q.y >= kWordEvent) {
            // one exchange: a load and a store of a sector that k_infect's
            // atomics left cost 21 us a step on the replica sweep
            ev = atomicExch(&d.evs[(int64_t)row * L.words + word], 0u);
          }
          const uint32_t E = ~A & B, I = A & ~B, R = waning ? (A & B) : 0u;
          uint32_t f = certain ? flow_sure(E, I, R, c.th) : 0u;
          if (cand)
            f |= flow_rest(cand, E, I, R, c.th, c.rk, (uint32_t)row, d.step,
                           (uint32_t)word + (c.roff >> 5));
          apply_word(L, d, c, waning, row, word, A, B, ev, f);
        }
        __syncwarp();
      } else if (!draw) {
        break;
      }
    }
    if (flushing) break;
  }
}

// Full E/I/R counts of the planes (initial state): one shared atomic per
// set bit, E | I << 21 | R << 42 per replica.
__global__ void __launch_bounds__(kThreads)
    k_packed_count(PackedLayout L, const PackedTask *__restrict__ tasks,
                   const uint32_t *__restrict__ sa, const uint32_t *__restrict__ sb,
                   unsigned long long *__restrict__ out) {
  __shared__ unsigned long long s_ev[128 * 32];
  for (int ti = blockIdx.x; ti < L.n_tasks; ti += gridDim.x) {
    const PackedTask T = tasks[ti];
    const int wbase = T.slice * 128;
    const int nw = min(128, L.words - wbase);
    for (int j = threadIdx.x; j < nw * 32; j += blockDim.x) s_ev[j] = 0;
    __syncthreads();
    const int64_t items = (int64_t)(T.row_end - T.row_begin) * nw;
    for (int64_t it = threadIdx.x; it < items; it += blockDim.x) {
      const int row = T.row_begin + (int)(it / nw);
      const int wl = (int)(it % nw);
      const int word = wbase + wl;
      const uint32_t vm = word_mask(L, word);
      const int64_t idx = (int64_t)row * L.words + word;
      const uint32_t a = sa[idx] & vm, b = sb[idx] & vm;
      count_bits(s_ev, wl, ~a & b, 1ull);
      count_bits(s_ev, wl, a & ~b, 1ull << kFieldBits);
      count_bits(s_ev, wl, a & b, 1ull << (2 * kFieldBits));
    }
    __syncthreads();
    for (int j = threadIdx.x; j < nw * 32; j += blockDim.x) {
      const int rep = wbase * 32 + j;
      if (rep < L.m && s_ev[j]) atomicAdd(&out[T.count_base + rep], s_ev[j]);
    }
    __syncthreads();
  }
}

// Bernoulli(p0) initial infection per (node, replica), stream 1, the plain
// path's uniforms.  Writes planes and the step-0 mask.
__global__ void __launch_bounds__(256)
    k_packed_init(PackedLayout L, uint32_t *__restrict__ sa, uint32_t *__restrict__ sb,
                  uint32_t *__restrict__ mask, float p0, StepConsts c) {
  const int64_t total = (int64_t)L.n_nodes * L.words;
  for (int64_t idx = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; idx < total;
       idx += (int64_t)gridDim.x * blockDim.x) {
    const int32_t row = (int32_t)(idx / L.words);
    const int32_t word = (int32_t)(idx % L.words);
    const uint32_t vmask = word_mask(L, word);
    uint32_t inf = 0;
    if (p0 > 0.0f && vmask) {
#pragma unroll
      for (int q = 0; q < 8; ++q) {
        uint32_t x[4];
        philox4x32_10((uint32_t)row, kStepInit, (uint32_t)((word + (c.roff >> 5)) * 8 + q), kStreamInit, c.key0,
                      c.key1, x);
#pragma unroll
        for (int cc = 0; cc < 4; ++cc)
          if (unit24(x[cc]) < p0) inf |= 1u << (4 * q + cc);
      }
    }
    inf &= vmask;
    sa[idx] = inf;
    sb[idx] = 0;
    mask[idx] = inf;
  }
}

// Exactly k infected per (network, replica) by Floyd's sampling, stream 2,
// node = index within the network.
__global__ void k_packed_pick(PackedLayout L, uint32_t *__restrict__ sa,
                              const int32_t *__restrict__ net_first_row,
                              const int32_t *__restrict__ net_rows, int32_t n_nets, int32_t k,
                              StepConsts c) {
  const int64_t gid = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (gid >= (int64_t)n_nets * L.m) return;
  const int32_t net = (int32_t)(gid / L.m), r = (int32_t)(gid % L.m);
  const int32_t n = net_rows[net], first = net_first_row[net];
  const uint32_t bit = 1u << (r & 31);
  const int32_t word = r >> 5;
  const int32_t kk = k < n ? k : n;
  for (int32_t j = n - kk; j < n; ++j) {
    uint32_t x[4];
    philox4x32_10((uint32_t)j, kStepPick, (uint32_t)r + c.roff, kStreamPick + 4u * (uint32_t)net, c.key0,
                  c.key1, x);
    const uint64_t r64 = (uint64_t)x[0] | ((uint64_t)x[1] << 32);
    const int32_t t = (int32_t)__umul64hi(r64, (uint64_t)(j + 1));
    const uint32_t old = atomicOr(&sa[(int64_t)(first + t) * L.words + word], bit);
    if (old & bit) atomicOr(&sa[(int64_t)(first + j) * L.words + word], bit);
  }
}

__global__ void k_mask_from_planes(int64_t total, const uint32_t *__restrict__ sa,
                                   const uint32_t *__restrict__ sb, uint32_t *__restrict__ mask) {
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < total;
       i += (int64_t)gridDim.x * blockDim.x)
    mask[i] = sa[i] & ~sb[i];
}

// Bit of every item whose words hold a set bit (one thread per bit).
__global__ void __launch_bounds__(256)
    k_bits_of(PackedLayout L, const uint4 *__restrict__ plane, uint32_t *__restrict__ bits) {
  const int64_t total = L.bit_words * 32;
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < total;
       i += (int64_t)gridDim.x * blockDim.x) {
    const int64_t wi = i >> 5;
    const int bit = (int)(i & 31), slice = (int)(wi % L.n_slices);
    const int64_t row = ((wi / L.n_slices) << (5 - L.lb)) + (bit >> L.lb);
    const int col = slice * 32 + (bit & ((1 << L.lb) - 1));
    bool set = false;
    if (row < L.n_nodes && col < L.q4) {
      const uint4 v = plane[row * L.q4 + col];
      set = (v.x | v.y | v.z | v.w) != 0u;
    }
    const uint32_t m = __ballot_sync(kFull, set);
    if ((i & 31) == 0) bits[wi] = m;
  }
}

// The bitmaps from the initial planes: one thread per bit.
__global__ void __launch_bounds__(256)
    k_bits_from_planes(PackedLayout L, const uint4 *__restrict__ sa, const uint4 *__restrict__ sb,
                       uint32_t *__restrict__ actb, uint32_t *__restrict__ infb,
                       uint32_t *__restrict__ susb, uint32_t *__restrict__ evb, bool waning) {
  const int64_t total = L.bit_words * 32;
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < total;
       i += (int64_t)gridDim.x * blockDim.x) {
    const int64_t wi = i >> 5;
    const int bit = (int)(i & 31), slice = (int)(wi % L.n_slices);
    const int64_t row = ((wi / L.n_slices) << (5 - L.lb)) + (bit >> L.lb);
    const int col = slice * 32 + (bit & ((1 << L.lb) - 1));
    bool act = false, inf = false, sus = false;
    if (row < L.n_nodes && col < L.q4) {
      const uint4 a4 = sa[row * L.q4 + col], b4 = sb[row * L.q4 + col];
#pragma unroll
      for (int w = 0; w < 4; ++w) {
        const uint32_t A = get4(a4, w), B = get4(b4, w), vm = word_mask(L, 4 * col + w);
        act |= (((A ^ B) | (waning ? (A & B) : 0u)) & vm) != 0u;
        inf |= (A & ~B & vm) != 0u;
        sus |= ((~A & ~B) & vm) != 0u;
      }
    }
    const uint32_t a = __ballot_sync(kFull, act), f = __ballot_sync(kFull, inf),
                   s = __ballot_sync(kFull, sus);
    if ((i & 31) == 0) {
      actb[wi] = a;
      infb[wi] = f;
      susb[wi] = s;
      evb[wi] = 0u;
    }
  }
}

// counts[t][net][r][4] from the initial counts and the per-step events.
__global__ void k_finalize(const unsigned long long *__restrict__ init,
                           const unsigned long long *__restrict__ ev,
                           const unsigned long long *__restrict__ rs, int32_t steps,
                           int32_t per_row, const int32_t *__restrict__ net_size, int32_t m,
                           int32_t has_exposed, int32_t ir_to_s, int32_t *__restrict__ counts) {
  const int32_t j = blockIdx.x * blockDim.x + threadIdx.x;
  if (j >= per_row) return;
  const unsigned long long fm = (1ull << kFieldBits) - 1;
  const int64_t N = net_size[j / m];
  const unsigned long long p = init[j];
  int64_t E = (int64_t)(p & fm), I = (int64_t)((p >> kFieldBits) & fm),
          R = (int64_t)((p >> (2 * kFieldBits)) & fm);
  int32_t *o = counts + (int64_t)j * 4;
  o[0] = (int32_t)E;
  o[1] = (int32_t)I;
  o[2] = (int32_t)R;
  o[3] = (int32_t)(N - E - I - R);
  for (int32_t t = 0; t < steps; ++t) {
    const unsigned long long e = ev[(int64_t)t * per_row + j];
    const int64_t se = (int64_t)(e & fm), xi = (int64_t)((e >> kFieldBits) & fm),
                  ix = (int64_t)((e >> (2 * kFieldBits)) & fm);
    const int64_t rsv = rs ? (int64_t)rs[(int64_t)t * per_row + j] : 0;
    E += se - (has_exposed ? xi : 0);
    I += xi - ix;
    R += (ir_to_s ? 0 : ix) - rsv;
    o = counts + ((int64_t)(t + 1) * per_row + j) * 4;
    o[0] = (int32_t)E;
    o[1] = (int32_t)I;
    o[2] = (int32_t)R;
    o[3] = (int32_t)(N - E - I - R);
  }
}

__global__ void k_packed_classify(PackedLayout L, const uint32_t *__restrict__ sa,
                                  const uint32_t *__restrict__ sb, uint8_t *__restrict__ out) {
  const int64_t total = (int64_t)L.n_nodes * L.m;
  for (int64_t g = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; g < total;
       g += (int64_t)gridDim.x * blockDim.x) {
    const int32_t r = (int32_t)(g / L.n_nodes), i = (int32_t)(g % L.n_nodes);
    const int64_t idx = (int64_t)i * L.words + (r >> 5);
    const uint32_t a = (sa[idx] >> (r & 31)) & 1u, b = (sb[idx] >> (r & 31)) & 1u;
    out[g] = (uint8_t)(a ? (b ? 3 : 2) : (b ? 1 : 0));
  }
}

// Exposure only (test hook): exposure[i * m + r] exact int64, masks with
// `W` words per node.
__global__ void __launch_bounds__(256)
    k_packed_exposure(const int32_t *__restrict__ row_ptr, const int2 *__restrict__ ent,
                      int32_t n, const uint32_t *__restrict__ masks, int32_t W, int32_t m,
                      int64_t *__restrict__ exposure) {
  const int64_t total = (int64_t)n * m;
  for (int64_t g = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; g < total;
       g += (int64_t)gridDim.x * blockDim.x) {
    const int32_t i = (int32_t)(g / m), r = (int32_t)(g % m);
    int64_t acc = 0;
    for (int32_t k = row_ptr[i]; k < row_ptr[i + 1]; ++k) {
      const int2 en = ent[k];
      if ((masks[(int64_t)en.x * W + (r >> 5)] >> (r & 31)) & 1u) acc += en.y;
    }
    exposure[g] = acc;
  }
}

int task_grid(int n_tasks, int per_sm) {
  int g = n_tasks < 148 * per_sm ? n_tasks : 148 * per_sm;
  return g < 1 ? 1 : g;
}

}  // namespace

rp_status packed_prepare() {
  cudaError_t e = cudaFuncSetAttribute(
      k_infect<false>, cudaFuncAttributeMaxDynamicSharedMemorySize, kInfectDynSmem<false>);
  if (e == cudaSuccess)
    e = cudaFuncSetAttribute(k_infect<true>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                             kInfectDynSmem<true>);
  if (e != cudaSuccess) return cuda_fail(e, "cudaFuncSetAttribute(k_infect)");
  e = cudaFuncSetAttribute(k_flow, cudaFuncAttributeMaxDynamicSharedMemorySize, kFlowDynSmem);
  if (e != cudaSuccess) return cuda_fail(e, "cudaFuncSetAttribute(k_flow)");
  return RP_OK;
}

int packed_init(const PackedLayout &L, uint32_t *sa, uint32_t *sb, uint32_t *mask,
                uint32_t *bits, float p0, int32_t k_exact, const int32_t *net_first_row,
                const int32_t *net_rows, int32_t n_nets, const StepConsts &c,
                cudaStream_t st) {
  const int64_t total = (int64_t)L.n_nodes * L.words;
  k_packed_init<<<1184, 256, 0, st>>>(L, sa, sb, mask, k_exact > 0 ? 0.0f : p0, c);
  if (k_exact > 0) {
    const int64_t nt = (int64_t)n_nets * L.m;
    k_packed_pick<<<(unsigned)((nt + 127) / 128), 128, 0, st>>>(L, sa, net_first_row, net_rows,
                                                                n_nets, k_exact, c);
    k_mask_from_planes<<<1184, 256, 0, st>>>(total, sa, sb, mask);
  }
  if (bits)
    k_bits_from_planes<<<1184, 256, 0, st>>>(
        L, reinterpret_cast<const uint4 *>(sa), reinterpret_cast<const uint4 *>(sb), bits,
        bits + L.bit_words, bits + 2 * L.bit_words, bits + 3 * L.bit_words,
        c.th.tr_all || c.th.tr != 0);
  return 1 + (k_exact > 0 ? 2 : 0) + (bits ? 1 : 0);
}

void cd_bits(const PackedLayout &L, const uint32_t *plane, uint32_t *bits, cudaStream_t st) {
  k_bits_of<<<1184, 256, 0, st>>>(L, reinterpret_cast<const uint4 *>(plane), bits);
}

// Blocks for `units` warp-sized units: one warp each over all SMs first, then
// up to the three resident blocks of each SM.
static int unit_grid(int64_t units) {
  return (int)(units < 1 ? 1 : (units < 148 * 3 ? units : 148 * 3));
}

// 8 rows per unit, so that a block's warps end together; fewer (down to 8
// items, one round of words) where blocks would have none, more where every
// warp has many: a unit's row pointers are loaded together, and sparse rows
// fold into batches of 32.
static void set_infect_units(const PackedLayout &L, int64_t n_rows, InfectArgs &d) {
  d.unit_rows = 8;
  const int64_t warps = 148 * 3 * kWarps;
  auto units = [&](int rows) { return (n_rows + rows - 1) / rows * L.n_slices; };
  while (d.unit_rows > 1 && units(d.unit_rows) * 2 < warps && (int64_t)d.unit_rows * L.q4 > 8)
    d.unit_rows >>= 1;
  while (d.unit_rows < kUnitRows &&
         (units(2 * d.unit_rows) >= 4 * warps || (int64_t)d.unit_rows * L.q4 < 8 ||
          ((int64_t)d.unit_rows * L.q4 < 32 && units(2 * d.unit_rows) >= warps)))
    d.unit_rows *= 2;
  d.n_units = (int32_t)units(d.unit_rows);
}

void packed_infect(const PackedLayout &L, const int32_t *row_ptr, const int2 *entries,
                   const RowList &list, const HeavyRows &heavy, const uint32_t *mask,
                   const uint32_t *sa, const uint32_t *sb, uint32_t *evs, uint32_t *bits,
                   uint32_t step, float scale, const StepConsts &c, cudaStream_t st) {
  InfectArgs d{};
  d.row_ptr = row_ptr;
  d.ent = entries;
  d.mask = mask;
  d.sa = sa;
  d.sb = sb;
  d.evs = evs;
  d.infb = bits + L.bit_words;
  d.susb = bits + 2 * L.bit_words;
  d.evb = bits + 3 * L.bit_words;
  d.heavy = heavy.rows;
  d.heavy_end = heavy.end;
  d.n_heavy = heavy.counts;
  d.list = list;
  d.step = step;
  d.scale = scale;
  set_infect_units(L, list.rows ? list.bound : L.n_nodes, d);
  k_infect<false><<<unit_grid(d.n_units), kThreads, kInfectDynSmem<false>, st>>>(L, d, c);
}

void cd_infect(const PackedLayout &L, const int32_t *row_ptr, const int2 *entries,
               const uint32_t *mask, const uint32_t *busy, uint32_t *evs, const uint32_t *infb,
               const uint32_t *susb, uint32_t *evb, uint32_t step, const StepConsts &c,
               cudaStream_t st) {
  InfectArgs d{};
  d.row_ptr = row_ptr;
  d.ent = entries;
  d.mask = mask;
  d.sa = busy;
  d.evs = evs;
  d.infb = infb;
  d.susb = susb;
  d.evb = evb;
  d.step = step;
  set_infect_units(L, L.n_nodes, d);
  k_infect<true><<<unit_grid(d.n_units), kThreads, kInfectDynSmem<true>, st>>>(L, d, c);
}

void packed_flow(const PackedLayout &L, uint32_t *mask, uint32_t *sa, uint32_t *sb, uint32_t *evs,
                 uint32_t *bits, unsigned long long *ev_row, unsigned long long *rs_row,
                 const int32_t *net_first, int32_t n_nets, uint32_t step, const StepConsts &c,
                 cudaStream_t st) {
  FlowArgs d{};
  d.evs = evs;
  d.mask = mask;
  d.sa = sa;
  d.sb = sb;
  d.actb = bits;
  d.infb = bits + L.bit_words;
  d.susb = bits + 2 * L.bit_words;
  d.evb = bits + 3 * L.bit_words;
  d.ev_row = ev_row;
  d.rs_row = rs_row;
  d.net_first = net_first;
  d.n_nets = n_nets;
  d.step = step;
  // a small bitmap is cut finer: 8 items of 128 replicas are one full round
  d.split = 0;
  while (d.split < 2 && (L.bit_words << (d.split + 1)) <= 148 * 3 * kWarps) ++d.split;
  d.n_units = L.bit_words << d.split;
  // units of a warp's block: up to 32, fewer so that a block's warps end together
  d.take = 1;
  while (d.take < 32 && d.n_units > (int64_t)148 * 3 * kWarps * 4 * d.take) d.take *= 2;
  k_flow<<<unit_grid(d.n_units), kThreads, kFlowDynSmem, st>>>(L, d, c);
}

void packed_count(const PackedLayout &L, const PackedTask *tasks, const uint32_t *sa,
                  const uint32_t *sb, unsigned long long *counts_row, cudaStream_t st) {
  k_packed_count<<<task_grid(L.n_tasks, 2), kThreads, 0, st>>>(L, tasks, sa, sb, counts_row);
}

void packed_finalize_events(const unsigned long long *init, const unsigned long long *ev,
                            const unsigned long long *rs, int32_t steps, int32_t per_row,
                            const int32_t *net_size, int32_t m, int32_t has_exposed,
                            int32_t ir_to_s, int32_t *counts, cudaStream_t st) {
  k_finalize<<<(per_row + 127) / 128, 128, 0, st>>>(init, ev, rs, steps, per_row, net_size, m,
                                                   has_exposed, ir_to_s, counts);
}

void packed_classify(const PackedLayout &L, const uint32_t *sa, const uint32_t *sb,
                     uint8_t *out, cudaStream_t st) {
  k_packed_classify<<<1184, 256, 0, st>>>(L, sa, sb, out);
}

void packed_exposure(const int32_t *row_ptr, const int2 *entries, int32_t n,
                     const uint32_t *masks, int32_t words, int32_t m, int64_t *exposure,
                     cudaStream_t st) {
  k_packed_exposure<<<1184, 256, 0, st>>>(row_ptr, entries, n, masks, words, m, exposure);
}

}  // namespace rp
