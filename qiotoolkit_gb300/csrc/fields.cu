// fields.cu -- the block-decided Metropolis sweep (sm_103a).
//
// One warp, the DECIDER, runs a walker's ordered sweep (markov/walker.h:
// 143-153,209-229) 32 variables at a time, a variable per lane.  At a block's
// start every lane gathers its field -- the cost difference of its flip in
// fixed point (model_host.cc, build_fields) -- from the walker's state in
// shared memory: a byte per literal of the terms' other members (Ising models of
// one- and two-member terms: per spin), or one per wide term.
//
// The block is then decided as a whole.  Lane v's decision depends on the
// decisions of the lanes before it in two ways: through the terms it shares
// with them (in-block entries list these with their members' lanes) and, on
// replayed streams, through the draw it gets (the uphill lanes before it each
// take one).  Both only look back, so the lanes iterate: decide with the accept
// mask of the last round, vote, and decide again where a member of a lane's
// in-block terms changed; a mask that no longer changes any lane's terms is the
// ordered sweep's, lane by lane from the first.  A field within its rounding
// margin of zero or a comparison inside the FP32 screen's margin
// ends the block early: the lanes before it are
// committed, the lane itself is tried alone with the reference's FP64 sum and
// ln-table expression, and the rest of the block is decided after it.
//
// A second warp, the FEEDER, runs ahead of the decider: it fills a ring with
// the walker's random draws as intervals of their ln-table values and brings
// each block's chunk of the model (records, in-block entries) into one of two to
// four shared-memory buffers by one TMA bulk copy.  Walkers of a block whose
// chunks are large have the same buffers, filled by the first one's feeder.
//
// FP64 models: a third warp, the ACCOUNTANT, consumes a log of the flips in
// batches of up to 32: every lane recomputes one flip's exact FP64 cost
// difference (the reference's order and rounding, model/ising.h:108-117,
// model/pubo.h:335-367) from the spins (pair-only Ising, rows of more than 32
// terms) or from the masks of the contributing terms that the decider gathered
// beside the field, then the
// running cost is accumulated in flip order exactly as cost_ += diff
// (markov/walker.h:225) and the lowest state is taken at the first strict
// improvement (markov/walker.h:269-280) from the accountant's own copy of the
// spins.  Neither the decisions nor the draws depend on the running cost.
// Integer models keep cost and lowest in the decider (exact in any order).
//
// What bounds it: the decider's chain of dependent votes, shared-memory loads
// and integer instructions, about five cycles each, and its branches, ten to
// twenty: 1300 cycles a block on a sparse Ising model (N = 1000, 64 walkers), 3500
// on a PUBO of 11.7 terms a variable, four walkers an SM, 2400 on 3-SAT, a third
// of it the gather, a fifth the decisions.  Measured on the way (ms: 1000 sweeps
// of the first / 100 of 512 tempering walkers of the second / 200 of 64 of the
// third): the windowed kernel 63 / 190 / 45; fields kept up to date by
// shared-memory atomics, 26 to 44 cycles of the warp's memory queue each where a
// load takes 5, 40 / 93 / -; gathered from a byte per term, which every flip has
// to write, 24.6 / 43.7 / 17.6; from literals, where a flip writes two bytes, 24.9
// / 35.6 / 13.1; the same with the accountant finding the contributing terms
// itself, a row a lane, 25.6 / 59 / 15.8 (its scattered loads take the memory
// pipe from the deciders), or a row a warp, 39 / 147 / 32; here 20.7 / 36.0 / 10.8.
//
// Waits between the warps poll shared-memory counters (acquire/release) with a
// time limit on lack of progress; on expiry the kernel raises the device error
// flag and all of the walker's warps return.
#include <algorithm>
#include <climits>
#include <cmath>
#include <type_traits>

#include "block_turns.h"
#include "metropolis.cuh"
#include "ordered_sum.cuh"
#include "qio_internal.h"

namespace qio
{
namespace fc
{
using namespace qio::mc;
static const unsigned kFull = 0xffffffffu;
static const int kIn = 4;         // in-block entries per lane of a staged block
static const int kLogBytes = 1024;  // flip log per walker: 64 entries of 16 bytes, pair models 256 of 4
static const int kRing = 128;     // draw intervals per walker (power of 2)
static const int kCtrl = 32;      // per-walker counters
static const int kBars = 48;      // mbarriers and the abort flag, before chunk buffers
static const int kTable = 4096;   // per block: screen row 0
static const uint32_t kWideMask = 0x0003FFFFu;  // wide term of a record or entry
static const uint32_t kNoWide = 0x40000000u;    // wide record: padding
static const uint32_t kSharedWide = 0x20000000u;  // an entry holds its value
static const unsigned kExactF = 0x80000000u;   // log entry: exact FP64 difference
static const int kMaxSmem = 227 * 1024;
static const int kSms = 152;
static const long long kPatience = 8000000000LL;  // cycles without progress, about 4 s

// the three forms of a field (build_fields)
enum Form
{
  PAIR = 0,     // Ising, terms of one or two members: spins alone
  COUNTER = 1,  // PUBO, MaxSat: a term counts when no other literal is true
  PARITY = 2    // Ising with larger terms: the parity of the other spins
};

// A block's chunk of the model's table (DevModel::fc_desc), in 8-byte words
template <int FM>
struct Chunk
{
  static const int kLane = 4;
  static const int kEnt = FM == PAIR ? 36 : 68;
  static const int kRec = kEnt + kIn * 32 * (FM == PAIR ? 1 : 2);
};
static const int kBufs = 4;  // chunk buffers per walker, at most (Shape::bufs)

__constant__ double c_ln[1024];
// screen of the ln-table comparison per (row, bucket): y0, dy, error margin;
// bucket 1 (log(0), never accepted) holds y0 = +inf
__device__ float4 g_scr[1024];
__constant__ ulonglong2 c_jump[33];
static const unsigned long long kMult = 6364136223846793005ULL;
static const unsigned long long kInc = 1442695040888963407ULL;

// ---- shared-memory synchronisation between a walker's warps -------------
__device__ __forceinline__ unsigned ld_acquire(const unsigned* p)
{
  unsigned v;
  asm volatile("ld.acquire.cta.shared::cta.u32 %0, [%1];"
               : "=r"(v)
               : "r"((unsigned)__cvta_generic_to_shared(p))
               : "memory");
  return v;
}
__device__ __forceinline__ void st_release(unsigned* p, unsigned v)
{
  asm volatile("st.release.cta.shared::cta.u32 [%0], %1;" ::"r"((unsigned)__cvta_generic_to_shared(p)),
               "r"(v)
               : "memory");
}
// A limit on waiting without progress: SM cycles from the first look (the
// nanosecond timer takes about a thousand cycles to read).
struct Patience
{
  long long t0 = 0;
  __device__ __forceinline__ void renew() { t0 = 0; }
  __device__ __forceinline__ bool over()
  {
    const long long t = clock64();
    if (t0 == 0) t0 = t;
    return t - t0 > kPatience;
  }
};
// all warps of a walker (integer models have no accountant)
template <bool INT>
__device__ __forceinline__ void walker_sync(int id)
{
  if (INT) asm volatile("bar.sync %0, 64;" ::"r"(id) : "memory");
  else asm volatile("bar.sync %0, 96;" ::"r"(id) : "memory");
}

// ---- TMA bulk copy of a tile of records, completion on an mbarrier --------
__device__ __forceinline__ unsigned smem_u32(const void* p)
{
  return (unsigned)__cvta_generic_to_shared(p);
}
__device__ __forceinline__ void mbar_init(unsigned long long* bar)
{
  asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(smem_u32(bar)) : "memory");
  asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
}
// (the buffer's reader is done: it has published that)
__device__ __forceinline__ void tile_issue(void* dst, const void* src, unsigned bytes, unsigned long long* bar)
{
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_u32(bar)), "r"(bytes)
               : "memory");
  asm volatile(
      "cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(
          smem_u32(dst)),
      "l"(src), "r"(bytes), "r"(smem_u32(bar))
      : "memory");
}
__device__ __forceinline__ bool mbar_try(unsigned long long* bar, unsigned parity)
{
  unsigned ok;
  asm volatile(
      "{\n .reg .pred p;\n mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n selp.u32 %0, 1, 0, p;\n}"
      : "=r"(ok)
      : "r"(smem_u32(bar)), "r"(parity)
      : "memory");
  return ok != 0;
}
__device__ __forceinline__ bool mbar_wait(unsigned long long* bar, unsigned parity)
{
  for (int it = 0; it < (1 << 22); it++)
    if (mbar_try(bar, parity)) return true;
  return false;
}
// The same for a chunk that may not have been issued yet, or never is once
// `abort` is raised.  Out of line: inside the decider it took sparse Ising from
// 21.2 to 21.7 ms and the PUBO tempering from 37.6 to 37.9.
__device__ __noinline__ bool chunk_wait(unsigned long long* bar, unsigned parity, const unsigned* abort)
{
  for (int it = 0; it < (1 << 22); it++)
  {
    if (mbar_try(bar, parity)) return true;
    if ((it & 255) == 255 && *(const volatile unsigned*)abort) return false;
  }
  return false;
}

__device__ __forceinline__ uint32_t spin_of(const uint32_t* spins, int v)
{
  return (spins[v >> 5] >> (v & 31)) & 1u;
}

// PCG state after k further draws
__device__ __noinline__ uint64_t jump_to(uint64_t st, uint32_t k)
{
  uint64_t A = kMult, C = kInc;
  for (; k; k >>= 1)
  {
    if (k & 1u) st = A * st + C;
    C = A * C + C;
    A = A * A;
  }
  return st;
}

// The redraw chain of an uphill attempt (markov/metropolis.h:93-103) on the
// stream's next draws.  Returns 1 accept / 0 reject.
__device__ __noinline__ int draw_chain(uint64_t rs, bool beta_inf, double dE, double beta)
{
  int row = -1, b = 0;
  uint32_t cur = 0;
  while (b == 0 && row < 3)
  {
    cur = pcg_out(rs);
    rs = rs * kMult + kInc;
    b = (int)(cur & 255u);
    row++;
  }
  if (b == 0) return 1;  // four zero buckets
  if (beta_inf) return 0;
  return lut_less_exact(c_ln, cur, row, __dmul_rn(dE, -beta)) ? 1 : 0;
}

// the same on the two 64-bit words of a counter stream's attempt
__device__ __noinline__ int counter_chain(uint64_t key, unsigned long long ctr, bool beta_inf, double dE, double beta)
{
  uint64_t w = counter_draw(key, 2ULL * ctr);
  int row = 0;
  uint32_t cur = (uint32_t)w;
  while ((cur & 255u) == 0u && row < 3)
  {
    row++;
    if (row == 2) w = counter_draw(key, 2ULL * ctr + 1ULL);
    cur = (row & 1) ? (uint32_t)(w >> 32) : (uint32_t)w;
  }
  if ((cur & 255u) == 0u) return 1;
  if (beta_inf) return 0;
  return lut_less_exact(c_ln, cur, row, __dmul_rn(dE, -beta)) ? 1 : 0;
}

// Exact cost difference of flipping v (FP64 models), row entries q .. qe - 1: the
// reference's sum over the row in ascending term id (model/ising.h:108-117, model/pubo.h:335-367).
// Members below v have their spins in `after`, the others in `before`.
template <int FM>
__device__ __forceinline__ double exact_dE(const DevModel& m, int v, int q, int qe, const uint32_t* before,
                                           const uint32_t* after)
{
  const uint32_t sv = spin_of(before, v);
  auto spin = [&](int u) -> uint32_t { return spin_of(u < v ? after : before, u); };
  auto lit = [&](uint32_t x) -> uint32_t {
    x &= 0xFFFFu;
    return x == 0xFFFFu ? 0u : spin((int)(x >> 1)) ^ (x & 1u);
  };
  constexpr int U = 4;  // loads in flight ahead of the dependent adds
  double d = 0.0;
  for (; q < qe; q += U)
  {
    double c[U];
    uint2 o[U];
    uint32_t on[U];
#pragma unroll
    for (int i = 0; i < U; i++)
    {
      const bool in = q + i < qe;
      if (FM == PAIR) o[i] = make_uint2(in ? (uint32_t)__ldg(m.other + q + i) : 0xffffffffu, 0u);
      else o[i] = in ? __ldg(m.fc_oth + q + i) : make_uint2(0xffffffffu, 0xffffu);
      c[i] = in ? __ldg(m.coef + q + i) : 0.0;
    }
#pragma unroll
    for (int i = 0; i < U; i++)
    {
      if (FM == PAIR)
      {
        on[i] = (int)o[i].x < 0 ? 0u : spin((int)o[i].x);
        continue;
      }
      const uint32_t a = lit(o[i].x), b = lit(o[i].x >> 16), e = lit(o[i].y);
      on[i] = FM == COUNTER ? (a | b | e) : (a ^ b ^ e);
      if (o[i].y & (1u << 17))
      {
        // a wide term: its members
        const int t = (int)(__ldg(m.inc + q + i) & ~kNegBit);
        for (int k = __ldg(m.trow + t), e1 = __ldg(m.trow + t + 1); k < e1; k++)
        {
          const uint32_t x = __ldg(m.tvar + k);
          const int u = (int)(x & ~kNegBit);
          if (u == v) continue;
          if (FM == COUNTER) on[i] |= spin(u) ^ (x >> 31);
          else on[i] ^= spin(u);
        }
      }
    }
#pragma unroll
    for (int i = 0; i < U; i++)
    {
      if (q + i >= qe) continue;
      if (FM != COUNTER) d = __dadd_rn(d, (sv ^ on[i]) ? -c[i] : c[i]);
      else if (!on[i]) d = (sv ^ (o[i].y >> 16)) & 1u ? __dadd_rn(d, c[i]) : __dsub_rn(d, c[i]);
    }
  }
  return FM == COUNTER ? d : neg2x(d);
}

// The accountant's batch of n flips where some rows are too wide for masks (this
// lane's: `wide`): those are summed from the spins, in index order as pair models'
// (account).  The differences, and the flips that are one sweep's.  (The decider
// summing them itself, an accepted flip at a time: QUBO of 128 variables, complete,
// 64 walkers, 200 sweeps 264 ms, here 16.5; 1000 variables of 40 terms, 100 sweeps
// 301 and 31; the windowed sweep 212 and 177.)
struct Summed
{
  double d;
  int n;
};
template <int FM>
__device__ __noinline__ Summed sum_rows(const DevModel& m, uint32_t* spins, int nw, int v, int q0, int q1, bool wide,
                                        int n, double d)
{
  const int lane = threadIdx.x & 31;
  if (__any_sync(kFull, wide))
  {
    const int prev = __shfl_up_sync(kFull, v, 1);
    const unsigned wrap = __ballot_sync(kFull, lane > 0 && lane < n && v <= prev);
    if (wrap) n = __ffs(wrap) - 1;
    uint32_t* after = spins + nw + 4;
    for (int q = lane; q < nw; q += 32) after[q] = spins[q];
    __syncwarp();
    if (lane < n) atomicXor(after + (v >> 5), 1u << (v & 31));
    __syncwarp();
    if (wide && lane < n) d = exact_dE<FM>(m, v, q0, q1, spins, after);
  }
  return {d, n};
}

// Exact cost difference from a log entry's masks (accountant): COUNTER: qm = the
// contributing incidences, sm = their signs; PARITY: all contribute.
template <int FM>
__device__ __forceinline__ double dE_from_masks(const double* pc, int deg, uint32_t qm, uint32_t sm)
{
  uint32_t q = (FM != COUNTER) ? ((deg >= 32) ? kFull : ((1u << deg) - 1u)) : qm;
  double d = 0.0;
  while (q)
  {
    // four loads in flight ahead of the dependent adds
    double c[4];
    int k[4];
#pragma unroll
    for (int i = 0; i < 4; i++)
    {
      k[i] = q ? __ffs(q) - 1 : -1;
      q &= q - 1;
      c[i] = k[i] >= 0 ? __ldg(pc + k[i]) : 0.0;
    }
#pragma unroll
    for (int i = 0; i < 4; i++)
      if (k[i] >= 0)
      {
        const bool s = ((sm >> k[i]) & 1u) != 0u;
        if (FM != COUNTER) d = __dadd_rn(d, s ? -c[i] : c[i]);
        else d = s ? __dadd_rn(d, c[i]) : __dsub_rn(d, c[i]);
      }
  }
  return (FM == COUNTER) ? d : neg2x(d);
}

__device__ __forceinline__ int warp_scan32(int x, int lane)
{
#pragma unroll
  for (int d = 1; d < 32; d <<= 1)
  {
    int y = __shfl_up_sync(kFull, x, d);
    if (lane >= d) x += y;
  }
  return x;
}
__device__ __forceinline__ long long warp_scan64(long long x, int lane)
{
#pragma unroll
  for (int d = 1; d < 32; d <<= 1)
  {
    long long y = __shfl_up_sync(kFull, x, d);
    if (lane >= d) x += y;
  }
  return x;
}

// Per-walker shared-memory region, sized for the launch's largest model.
struct Shape
{
  int nw;     // spin words of the population
  int zb;     // literal bytes and wide terms' bytes; pair models: a byte per variable
  int words;  // 8-byte words of a staged chunk (larger blocks read their records from HBM)
  int bufs;   // chunk buffers, kBufs at most
  int share;  // walkers that use the same ones (a block's, or 1)
  bool pair;
  bool second;  // FP64: a second copy of the accountant's spins
};
struct Region
{
  unsigned long long* bars;  // kBufs mbarriers, before the buffers
  unsigned* head;            // log entries published by the decider (with `used`, 8 bytes)
  unsigned* tail;            // log entries consumed by the accountant
  unsigned* done;            // the decider finished the walker
  unsigned* abort;           // a wait gave up: all warps leave (beside the mbarriers)
  unsigned* next;            // the walker taken from the queue
  unsigned* made;            // draws in the ring
  unsigned* used;            // draws taken by the decider
  unsigned* blocks;          // blocks the decider has finished (before `head`, `used`)
  float2* ring;              // kRing screen intervals
  uint32_t* raw;             // kRing: stream position after the draw (replay)
  uint4* log;                // kLogBytes (FP64 models)
  uint2* tiles;              // the block chunks
  uint8_t* z;                // literals, a byte each, then the wide terms'; pair models: spins
  uint32_t* spins;           // nw + 4 words (words of zeros after the last)
  uint32_t* aspins;          // the accountant's spins (FP64 models), two copies (Shape::second)
};

// a walker's own part, and the chunk buffers', which a block's walkers may share
__host__ __device__ inline int own_bytes(const Shape& s, bool integer)
{
  return kCtrl + kRing * 12 + (integer ? 0 : kLogBytes) + s.zb + 4 * (s.nw + 4) +
         (integer ? 0 : 4 * (s.nw + 4) * (s.second ? 2 : 1));
}
__host__ __device__ inline int chunk_bytes(const Shape& s) { return kBars + s.bufs * s.words * 8; }
__host__ __device__ inline int region_bytes(const Shape& s, bool integer)
{
  return own_bytes(s, integer) + (s.share > 1 ? 0 : chunk_bytes(s));
}
__host__ __device__ inline int common_bytes(const Shape& s) { return s.share > 1 ? chunk_bytes(s) : 0; }

// Every pointer is one of two bases and little more: with a choice for each of
// them an integer kernel, at its 128 registers, took 10 to 40 % longer.
template <bool INT>
__device__ __forceinline__ Region carve(unsigned char* smem, int walker, const Shape& s)
{
  Region R;
  const int at = kTable + common_bytes(s) + walker * region_bytes(s, INT);
  unsigned char* base = smem + at;
  unsigned char* chunks = smem + (s.share > 1 ? kTable : at + own_bytes(s, INT));
  R.bars = (unsigned long long*)chunks;
  R.abort = (unsigned*)(chunks + 32);
  R.tiles = (uint2*)(chunks + kBars);
  unsigned* c = (unsigned*)base;
  R.head = c;
  R.used = c + 1;
  R.tail = c + 2;  // (tail, made: one 8-byte word)
  R.made = c + 3;
  R.done = c + 4;
  R.next = c + 6;
  R.blocks = c + 7;
  R.ring = (float2*)(base + kCtrl);
  R.raw = (uint32_t*)(R.ring + kRing);
  R.log = (uint4*)(R.raw + kRing);
  R.z = (uint8_t*)(R.log + (INT ? 0 : kLogBytes / 16));
  R.spins = (uint32_t*)(R.z + s.zb);
  R.aspins = R.spins + s.nw + 4;
  return R;
}

__device__ __forceinline__ void raise_abort(const Region& R, int* err)
{
  if (err) atomicExch(err, 1);
  st_release(R.abort, 1u);
}

// The bytes that the gather reads, from the spins, by thread `me` of `n`: pair
// models the spins; else the literals (one more is false) and the wide terms'
template <int FM>
__device__ __noinline__ void make_bytes(const DevModel& m, uint8_t* z, const uint32_t* spins, int nw, int me, int n)
{
  for (int v = me; v < 32 * nw; v += n)
  {
    const uint32_t s = spin_of(spins, v);
    if (FM == PAIR) z[v] = (uint8_t)s;
    else ((uint16_t*)z)[v] = (uint16_t)(s | (s ^ 1u) << 8);
  }
  if (FM == PAIR) return;
  if (me < 16) z[64 * nw + me] = (uint8_t)(me & 1);
  for (int i = me; i < m.fc_wide; i += n)
  {
    const int t = __ldg(m.fc_wterm + i);
    uint32_t c = 0;
    for (int k = __ldg(m.trow + t), e = __ldg(m.trow + t + 1); k < e; k++)
    {
      const uint32_t x = __ldg(m.tvar + k);
      c += spin_of(spins, (int)(x & ~kNegBit)) ^ (FM == COUNTER ? x >> 31 : 0u);
    }
    z[64 * nw + 16 + i] = (uint8_t)(FM == PARITY ? c & 1u : c);
  }
}

// Mutable state of one walker's decider.
struct Walk
{
  uint64_t rs;          // replay: the stream's state at position raw0
  uint32_t raw0;
  uint64_t key;         // counter streams
  unsigned taken;       // draws taken
  unsigned long long natt, nacc, nwin;
  long long icost, ilow;  // integer models
};

// replay: the stream's state after the draws taken
__device__ __forceinline__ uint64_t stream_state(const Region& R, const Walk& W)
{
  const uint32_t at = W.taken ? R.raw[(W.taken - 1u) & (unsigned)(kRing - 1)] : 0u;
  return jump_to(W.rs, at - W.raw0);
}

// ---------------------------------------------------------------------------
// The feeder.
//
// Draws: the ring holds the walker's draws as screen intervals [lo, hi] of
// their ln-table values, kRing ahead of the decider at most.  Replay: the
// stream's draws in order; a zero bucket is skipped by the attempt that meets
// it (markov/metropolis.h:93-103: the next draw counts, one ln-table row
// further down) and four of them accept, so an entry is what one uphill attempt
// takes.  Counter streams: the entry of every attempt in turn.  An entry that
// always accepts is (-inf, -inf).
//
// Chunks: a block's goes to the next buffer in turn (T, kept over the warp's
// walkers) once the decider is done with the block `bufs` before.  Where walkers
// share the buffers, the first one's feeder brings the chunks, once all of them
// are done with that block (`live` of them, 0 for the others' feeders; their
// counters `stride` words apart).
// ---------------------------------------------------------------------------
template <int FM, bool REPLAY>
__device__ __noinline__ void feed(const Region R, const float4* s_scr, const int4* desc, const uint2* table, int tile_w,
                                  int cap, Turns& turns, int n_sweeps, uint64_t rs, uint64_t key, unsigned long long ctr,
                                  int n_vars, int live, int stride, int* err)
{
  const int lane = threadIdx.x & 31;
  const unsigned lt = (1u << lane) - 1u;
  uint64_t st = REPLAY ? c_jump[lane].x * rs + c_jump[lane].y : 0;
  const uint64_t jA = c_jump[32].x, jC = c_jump[32].y;
  unsigned made = 0;
  uint32_t raw = (uint32_t)lane + 1u;  // stream position after this lane's draw
  int carry = 0;                       // zeros at the end of the last 32 draws that await the next
  int first = 0;                       // counter: the first variable of the coming attempts
  Turns T = turns;                     // the next chunk's place
  unsigned issued = 0;                 // chunks
  int4 d = __ldg(desc);                // ... and its descriptor
  Patience limit;
  unsigned last_u = 0, last_b = 0;
  while (true)
  {
    // what the decider has done
    const unsigned used = ld_acquire(R.used);
    const unsigned blocks = *(volatile unsigned*)R.blocks;
    unsigned held = in_flight(issued, blocks);  // chunks that the slowest walker needs yet
    for (int k = 1; k < live; k++) held = max(held, in_flight(issued, ld_acquire(R.blocks + k * stride)));
    for (; live > 0 && T.sweep < n_sweeps && held < (unsigned)T.bufs; held++)
    {
      if (lane == 0)
        tile_issue(R.tiles + T.buf * tile_w, table + d.x, (unsigned)min(d.y, cap) * 8u, &R.bars[T.buf]);
      issued++;
      T.next();
      d = __ldg(desc + T.block);
    }
    if (made + 32u - used >= (unsigned)kRing)
    {
      // no room for draws (the last one taken stays: its stream position)
      bool leave = ld_acquire(R.done) != 0u || ld_acquire(R.abort) != 0u;
      if (!leave)
      {
        if (used != last_u || blocks != last_b)
        {
          last_u = used;
          last_b = blocks;
          limit.renew();
        }
        else if (limit.over())
        {
          raise_abort(R, err);
          leave = true;
        }
      }
      leave = __shfl_sync(kFull, (int)leave, 0) != 0;
      if (!leave)
      {
        __nanosleep(100);  // (its polls would take the decider's turns at shared memory)
        continue;
      }
      // the copies in flight land before the region is given up
      if (lane == 0 && live > 0)
      {
        Turns U = T;
        unsigned n = 0;
        for (int k = 0; k < live; k++) n = max(n, in_flight(issued, *(volatile unsigned*)(R.blocks + k * stride)));
        U.back(n);
        for (unsigned x = 0; x < n; x++, U.next_buffer()) mbar_wait(&R.bars[U.buf], U.phase);
      }
      turns = T;
      return;
    }
    uint32_t pd;
    int row = 0, n = 32, at = lane;
    bool put = true, always = false;
    if (REPLAY)
    {
      pd = pcg_out(st);
      st = jA * st + jC;
      const bool zero = (pd & 255u) == 0u;
      const unsigned Z = __ballot_sync(kFull, zero);
      if (Z || carry)
      {
        int run = lane ? __clz(~(Z << (32 - lane))) : 0;  // zeros just before this draw
        if (run == lane) run += carry;
        row = run & 3;
        always = zero && row == 3;
        put = !zero || always;
        const unsigned P = __ballot_sync(kFull, put);
        at = __popc(P & lt);
        n = __popc(P);
        carry = __shfl_sync(kFull, zero ? (run + 1) & 3 : 0, 31);
      }
    }
    else
    {
      const unsigned long long c = ctr + (unsigned long long)(first + lane);
      const uint64_t w = counter_draw(key, 2ULL * c);
      pd = (uint32_t)w;
      if ((pd & 255u) == 0u)
      {
        row = 1;
        pd = (uint32_t)(w >> 32);
        if ((pd & 255u) == 0u)
        {
          const uint64_t x = counter_draw(key, 2ULL * c + 1ULL);
          row = 2;
          pd = (uint32_t)x;
          if ((pd & 255u) == 0u)
          {
            row = 3;
            pd = (uint32_t)(x >> 32);
            always = (pd & 255u) == 0u;
          }
        }
      }
      first += 32;
      if (first >= n_vars)
      {
        first = 0;
        ctr += (unsigned long long)n_vars;
      }
    }
    const float4 e = row ? g_scr[row * 256 + (int)(pd & 255u)] : s_scr[pd & 255u];
    const float val = __fmaf_rn(__fmul_rn((float)(pd >> 8), 5.96046483e-08f), e.y, e.x);
    if (put)
    {
      const unsigned i = (made + (unsigned)at) & (unsigned)(kRing - 1);
      R.ring[i] = always ? make_float2(-INFINITY, -INFINITY) : make_float2(__fsub_rn(val, e.z), __fadd_rn(val, e.z));
      if (REPLAY) R.raw[i] = raw;
    }
    raw += 32u;
    made += (unsigned)n;
    __syncwarp();
    if (lane == 0) st_release(R.made, made);
  }
}

// Waits until *p (another warp's counter; counters wrap) reaches `want`; the
// value seen, or want - 1 when the walker is given up (abort raised, or no
// progress within the time limit).  Lane 0 polls for the warp.
__device__ __noinline__ unsigned wait_count(const unsigned* p, unsigned want, unsigned* abort, int* err)
{
  unsigned seen = want - 1u;
  if ((threadIdx.x & 31) == 0)
  {
    Patience limit;
    unsigned last = 0;
    bool any = false;
    while (true)
    {
      seen = ld_acquire(p);
      if ((int)(seen - want) >= 0) break;
      if (!any || seen != last)
      {
        any = true;
        last = seen;
        limit.renew();
      }
      if (ld_acquire(abort))
      {
        seen = want - 1u;
        break;
      }
      if (limit.over())
      {
        if (err) atomicExch(err, 1);
        st_release(abort, 1u);
        seen = want - 1u;
        break;
      }
    }
  }
  return __shfl_sync(kFull, seen, 0);
}

// ---------------------------------------------------------------------------
// The decider: one walker's sweeps.  Returns false when a wait gave up.
//
// What it keeps per sweep and per block, in the order of use.  A block's
// counters (flips logged, draws taken) are published, and the other warps'
// looked at, where no global load is outstanding: a shared-memory release or
// acquire waits for those (336 cycles measured against 30).
// ---------------------------------------------------------------------------
struct Sweep
{
  double beta, beta_next;
  const double* betas;
  bool beta_inf;
  float nbeta_f, fscale, fsa;
  unsigned long long ctr0;
};

// the constants of the sweep that starts, and the next one's beta
template <int FM, bool INT>
__device__ __forceinline__ void next_sweep(Sweep& S, const SweepArgs& a, double inv, int N, int k)
{
  const long long swp = a.sweep_base + k;
  S.beta = S.beta_next;
  S.beta_inf = ((unsigned long long)__double_as_longlong(S.beta) & 0x7FFFFFFFFFFFFFFFULL) == 0x7FF0000000000000ULL;
  // thr = field * fscale approximates dE * (-beta); an infinite beta accepts
  // nothing uphill: thr = -3e38 with no margin, from a zero scale
  S.nbeta_f = S.beta_inf ? 0.f : -approx_float(S.beta);
  S.fscale = INT ? S.nbeta_f : (S.beta_inf ? 0.f : (float)(S.beta * inv * (FM == COUNTER ? -1.0 : 2.0)));
  S.fsa = INT ? 0.f : fabsf(S.fscale) * 1.0001f;
  S.ctr0 = (unsigned long long)swp * (unsigned long long)N;
  if (k + 1 < a.n_sweeps) S.beta_next = S.betas[(swp + 1) * a.bs_s];
}

// publishes the blocks finished, the flips logged and the draws taken (head,
// used: one 8-byte word)
__device__ __forceinline__ void publish(const Region& R, unsigned blocks, unsigned head, unsigned taken)
{
  *(volatile unsigned*)R.blocks = blocks;
  const unsigned long long x = (unsigned long long)head | ((unsigned long long)taken << 32);
  asm volatile("st.release.cta.shared::cta.b64 [%0], %1;" ::"r"(smem_u32(R.head)), "l"(x) : "memory");
}

// the other warps' counters: flips accounted, draws in the ring
__device__ __forceinline__ void look(const Region& R, unsigned& tail, unsigned& made)
{
  unsigned long long x;
  asm volatile("ld.acquire.cta.shared::cta.b64 %0, [%1];" : "=l"(x) : "r"(smem_u32(R.tail)) : "memory");
  tail = __shfl_sync(kFull, (unsigned)x, 0);
  made = __shfl_sync(kFull, (unsigned)(x >> 32), 0);
}

// waits for room for 32 flips in the log and 32 draws in the ring
template <bool INT, int LOG>
__device__ __noinline__ void wait_room(unsigned* tail, unsigned* made, unsigned* abort, int* err, unsigned head,
                                      unsigned taken)
{
  if (!INT) wait_count(tail, head + 32u - (unsigned)LOG, abort, err);
  wait_count(made, taken + 32u, abort, err);
}

// Running cost and first lowest of integer models over a round's flips F
// (this lane's difference g), in lane order; `word`: the block's spins after.
__device__ __forceinline__ void account_int(const Region& R, Walk& W, bool scan32, int g, unsigned F, int bi,
                                            int nblocks, uint32_t* g_lsp)
{
  const int lane = threadIdx.x & 31;
  const bool mine = ((F >> lane) & 1u) != 0u;
  const int de = mine ? g : 0;
  int low = -1;
  if (scan32)
  {
    const int sum = __reduce_add_sync(kFull, de);
    const int neg = __reduce_add_sync(kFull, min(de, 0));
    if ((long long)neg < W.ilow - W.icost)  // the lowest prefix is at least icost + neg
    {
      const int pre = warp_scan32(de, lane);
      const int mn = __reduce_min_sync(kFull, mine ? pre : INT_MAX);
      if ((long long)mn < W.ilow - W.icost)
      {
        low = __ffs(__ballot_sync(kFull, mine && pre == mn)) - 1;
        W.ilow = W.icost + mn;
      }
    }
    W.icost += sum;
  }
  else
  {
    const long long pre = warp_scan64((long long)de, lane);
    const long long ci = W.icost + pre;
    long long mn = mine ? ci : LLONG_MAX;
#pragma unroll
    for (int s = 16; s; s >>= 1) mn = min(mn, __shfl_xor_sync(kFull, mn, s));
    if (mn < W.ilow)
    {
      low = __ffs(__ballot_sync(kFull, mine && ci == mn)) - 1;
      W.ilow = mn;
    }
    W.icost += __shfl_sync(kFull, pre, 31);
  }
  if (low >= 0)
  {
    // the state at the improvement: the round's later flips undone
    const unsigned undo = F & ~((2u << low) - 1u);
    for (int q = lane; q < nblocks; q += 32) g_lsp[q] = R.spins[q] ^ (q == bi ? undo : 0u);
  }
}

// a flip's change of a wide term's byte, v's literal `lit` before it (several
// lanes may hold the term, or its word's other bytes)
template <int FM>
__device__ __forceinline__ void flip_wide(uint8_t* zw, unsigned t, uint32_t lit)
{
  const unsigned sh = (t & 3u) * 8u;
  unsigned* word = (unsigned*)(zw + (t & ~3u));
  if (FM == PARITY) atomicXor(word, 1u << sh);
  else if (lit) atomicSub(word, 1u << sh);
  else atomicAdd(word, 1u << sh);
}

// Lane f's attempt alone: the reference's sum, draws and comparison.  Bit 0:
// accepted; bit 1: it drew.
template <int FM, bool REPLAY, bool INT>
__device__ __noinline__ unsigned exact_attempt(const DevModel& m, int v, int g, const uint32_t* spins, uint64_t rs,
                                              uint64_t key, unsigned long long ctr, double beta, double* dE_out)
{
  const double dE = INT ? (double)g : exact_dE<FM>(m, v, __ldg(m.row + v), __ldg(m.row + v + 1), spins, spins);
  const bool inf = ((unsigned long long)__double_as_longlong(beta) & 0x7FFFFFFFFFFFFFFFULL) == 0x7FF0000000000000ULL;
  *dE_out = dE;
  if (le_zero(dE)) return 1u;
  if (REPLAY) return 2u | (unsigned)draw_chain(rs, inf, dE, beta);
  return 2u | (unsigned)counter_chain(key, ctr, inf, dE, beta);
}

template <int FM, bool REPLAY, bool INT>
__device__ __forceinline__ bool decide_sweeps(const SweepArgs& a, const DevModel& m, const Region R, const Shape& sh, int r,
                                              Turns& turns, Walk& W, uint32_t* g_lsp)
{
  constexpr int KI = kIn;  // in-block entries held in registers
  constexpr int kLog = FM == PAIR ? kLogBytes / 4 : kLogBytes / 16;  // entries, a power of two
  constexpr bool MASKS = !INT && FM != PAIR;  // the log needs the row's masks, and weights carry row positions
  using C = Chunk<FM>;
  const int lane = threadIdx.x & 31;
  const unsigned lt = (1u << lane) - 1u;
  const int N = m.n_vars;
  Turns T = turns;  // the coming block
  const int nblocks = T.nblocks;
  if (a.n_sweeps <= 0) return true;
  const bool scan32 = m.scan32 != 0;
  const double inv = m.fc_inv;
  // (read once: `m` may be the launch's parameter or lie in device memory)
  const uint2* table = m.fc_tab;
  const int4* descs = m.fc_desc;
  const int cap = sh.words;
  uint8_t* zw = R.z + 64 * sh.nw + 16;  // the wide terms' bytes

  unsigned head = 0;                // log entries written
  unsigned moved = 0;               // draws taken when the stream's origin last moved
  unsigned acc_tail = 0, fed = 0;   // the other warps' counters when last looked at
  Sweep S;
  S.betas = a.beta + (long long)r * a.bs_w;
  S.beta_next = S.betas[a.sweep_base * a.bs_s];

  unsigned finished = 0;  // blocks
  while (true)
  {
    const int bi = T.block;
    if (bi == 0)
    {
      if (T.sweep == a.n_sweeps) break;
      if (REPLAY && W.taken - moved > (1u << 28))
      {
        // stream positions are 32-bit: move their origin along
        W.rs = stream_state(R, W);
        W.raw0 = R.raw[(W.taken - 1u) & (unsigned)(kRing - 1)];
        moved = W.taken;
      }
      next_sweep<FM, INT>(S, a, inv, N, T.sweep);
    }
    const int nvalid = min(32, N - (bi << 5));
    const int v = (bi << 5) + lane;
    // this block's chunk
    if (!__all_sync(kFull, mbar_try(&R.bars[T.buf], T.phase)))
    {
      const bool landed = chunk_wait(&R.bars[T.buf], T.phase, R.abort);
      if (!__all_sync(kFull, landed))
      {
        raise_abort(R, a.err);
        return false;
      }
    }
    const uint2* chunk = R.tiles + T.buf * cap;
    T.next();
    // the header through shuffles, so that what depends on it is known not to
    // divide the warp: rows, entry rows and further entry rows
    const uint2 head0 = *chunk;
    const unsigned h0 = __shfl_sync(kFull, head0.x, 0);
    const unsigned h1 = __shfl_sync(kFull, head0.y, 0);
    const int n0 = (int)(h0 & 127u) * 4, n1 = FM == PAIR ? 0 : (int)((h0 >> 7) & 255u) * 2;
    const int n2 = FM == PAIR ? 0 : (int)((h0 >> 15) & 255u) * 2, n3 = FM == PAIR ? 0 : (int)(h1 & 255u);
    const int ents = (int)((h0 >> 23) & 7u), xn = (int)(h1 >> 8);
    const int recs = C::kRec + 32 * (n0 + n1 + n2 + n3) + 16 * n2;  // words before the further entries
    const bool special = h1 != 0u || recs > cap;
    // The block itself.  SP: it has records or entries beyond its chunk, or wide
    // terms; the other form, most blocks', has a branch less for each of these
    // (a branch costs ten to twenty cycles of its warp): sparse Ising 23.6 and
    // 20.7 ms with the stream's positions looked after once a sweep, 3-SAT 11.9
    // and 10.8.
    auto block = [&](auto sp) __attribute__((always_inline)) -> bool {
      constexpr bool SP = decltype(sp)::value;
      const bool staged = !SP || recs + (FM == PAIR ? (xn ? 512 : 0) : 64 * xn) <= cap;
      const uint2* tile = chunk + lane;
      int4 own;  // field, degree, negated literals, terms of v alone
      if (FM == PAIR)
      {
        const int2 x = *(const int2*)(tile + C::kLane);
        own = make_int4(x.x, x.y, 0, 0);
      }
      else own = *((const int4*)(chunk + C::kLane) + lane);
      const uint4* tent = (const uint4*)(chunk + C::kEnt) + lane;

      const uint32_t word = R.spins[bi];  // the block's spins before its flips
      const uint32_t sv = (word >> lane) & 1u;
      const int deg = own.y;
      const int bnd = deg + 1;  // |field - exact| < bnd units
      const float xmargin = INT ? 0.f : S.fsa * (float)(bnd + 1);

      // ---- the field: the lane's value less the weights of the records whose
      // op is 1.  Rows come in fours (one literal) and twos and are taken four or
      // eight at a time, a load's latency being six rows' work (3-SAT, 18 rows of
      // two: 1120 cycles a block in twos; 200 sweeps 13.1 and 12.5 ms; sparse Ising
      // in fours and eights 24.5 and 23.4 ms).
      int base = own.x;
      unsigned qm = (unsigned)own.w;  // COUNTER: the incidences that contribute; PARITY: those of odd parity
      auto op = [](uint32_t x, uint32_t y) -> uint32_t { return FM == COUNTER ? (x | y) : (x ^ y); };
      // a record's op (0 or 1) and weight into field and mask
      auto put = [&](uint32_t on, uint32_t w) {
        if (MASKS)
        {
          base -= (int)on * (int)(w & ~255u);
          if ((FM == COUNTER) != (on != 0u)) qm |= __funnelshift_l(0u, 1u, w);
        }
        else base -= (int)on * (int)w;
      };
      auto gather = [&](const uint2* t0) {
        if constexpr (FM == PAIR)
        {
          uint2 e[8];
          for (int i = 0; i + 8 <= n0; i += 8)
          {
#pragma unroll
            for (int x = 0; x < 8; x++) e[x] = t0[32 * (i + x)];
#pragma unroll
            for (int x = 0; x < 8; x++) put(R.z[e[x].x], e[x].y);
          }
          if (n0 & 4)
          {
#pragma unroll
            for (int x = 0; x < 4; x++) e[x] = t0[32 * (n0 - 4 + x)];
#pragma unroll
            for (int x = 0; x < 4; x++) put(R.z[e[x].x], e[x].y);
          }
        }
        else
        {
          {
            uint2 e[4];
#pragma unroll
            for (int x = 0; x < 4; x++) e[x] = n0 ? t0[32 * x] : make_uint2(0u, 0u);
            for (int i = 4; i <= n0; i += 4)
            {
              uint2 f[4];
              const uint2* t1 = t0 + 32 * (i < n0 ? i : 0);
#pragma unroll
              for (int x = 0; x < 4; x++) f[x] = t1[32 * x];
#pragma unroll
              for (int x = 0; x < 4; x++) put(R.z[e[x].x], e[x].y);
#pragma unroll
              for (int x = 0; x < 4; x++) e[x] = f[x];
            }
          }
          t0 += 32 * n0;
          if (n1)
          {
            auto two = [&](const uint2& e) { put(op(R.z[e.x & 0xFFFFu], R.z[e.x >> 16]), e.y); };
            uint2 e[4];
#pragma unroll
            for (int x = 0; x < 4; x++) e[x] = t0[32 * min(x, n1 - 1)];
            int i = 4;
            for (; i <= n1; i += 4)
            {
              uint2 f[4];
#pragma unroll
              for (int x = 0; x < 4; x++) f[x] = t0[32 * min(i + x, n1 - 1)];
#pragma unroll
              for (int x = 0; x < 4; x++) two(e[x]);
#pragma unroll
              for (int x = 0; x < 4; x++) e[x] = f[x];
            }
            if (i - 4 < n1)
            {
              two(e[0]);
              two(e[1]);
            }
            t0 += 32 * n1;
          }
          if (n2)
          {
            const uint32_t* c0 = (const uint32_t*)(t0 - lane + 32 * n2) + lane;  // the third literals
            uint2 e0 = t0[0], e1 = t0[32];
            uint32_t k0 = c0[0], k1 = c0[32];
            for (int i = 2; i <= n2; i += 2)
            {
              const int nx = i < n2 ? i : 0;
              const uint2 f0 = t0[32 * nx], f1 = t0[32 * nx + 32];
              const uint32_t g0 = c0[32 * nx], g1 = c0[32 * nx + 32];
              const uint32_t a0 = R.z[e0.x & 0xFFFFu], b0 = R.z[e0.x >> 16], d0 = R.z[k0];
              const uint32_t a1 = R.z[e1.x & 0xFFFFu], b1 = R.z[e1.x >> 16], d1 = R.z[k1];
              put(op(op(a0, b0), d0), e0.y);
              put(op(op(a1, b1), d1), e1.y);
              e0 = f0;
              e1 = f1;
              k0 = g0;
              k1 = g1;
            }
            t0 += 48 * n2;
          }
          // wide terms: the true literals but for the own, or the others' parity
          for (int i = 0; SP && i < n3; i++)
          {
            const uint2 e = t0[32 * i];
            const uint32_t zz = zw[e.x & kWideMask];
            const uint32_t on = FM == COUNTER ? (zz != ((sv ^ (e.x >> 31)) & 1u) ? 1u : 0u) : ((zz ^ sv) & 1u);
            if (!(e.x & (kNoWide | kSharedWide))) put(on, e.y);
          }
        }
      };
      const uint2* far = table;  // (not staged) the records
      if (!SP || staged) gather(tile + C::kRec);
      else
      {
        far = table + __ldg(descs + bi).x + C::kRec + lane;
        gather(far);
      }

      // ---- the in-block terms under a given accept mask, all against the state
      // at the block's start.  Pair models: the member's flip changes the field
      // by c0.  Counter models: the other literals are all false when those of
      // the members before this lane (em) are -- the flipped ones are exactly the
      // true ones (et) -- and those after it or elsewhere were (else em = 0, et =
      // 1: never).  Parities: c0 of the others, and of the flips in em.
      unsigned watch = 0;  // lanes whose flips change this lane's field
      int val[KI];
      unsigned bit[KI];  // its place in the mask
      unsigned em[KI], et[KI];
      // further entries, xn rows of them, or a pair block's matrix
      const uint2* more = (!SP || staged ? chunk : far - lane - C::kRec) + recs;
      const uint4* xterm = (const uint4*)more + lane;
      const int* mat = (const int*)more + lane;
      unsigned done = 0;  // the block's flips so far
      // an entry's em and et; D: flips whose bytes are written already
      auto entry = [&](const uint4& e, unsigned D, unsigned& mm, unsigned& mt) {
        const uint32_t M = e.x, L = (word ^ e.y) & M;  // members before this lane, their true literals
        const bool wide = FM != PAIR && (e.z >> 18) == 0x3FFFu;
        uint32_t o;  // the other members: whether a literal is true, or their parity
        if (!wide) o = op(R.z[e.z & 0xFFFFu], R.z[e.z >> 16]);
        else
        {
          const uint32_t zz = zw[e.z & kWideMask], lit = (sv ^ (e.y >> lane)) & 1u;
          if (FM == COUNTER) o = (int)zz - (int)lit != __popc((L ^ D) & M) ? 1u : 0u;
          else o = (zz ^ sv ^ (uint32_t)__popc((word ^ D) & M)) & 1u;
        }
        mm = M;
        mt = FM == COUNTER ? L : (o ^ (uint32_t)__popc(word & M)) & 1u;
        if (FM == COUNTER && o)
        {
          mm = 0u;
          mt = 1u;
        }
      };
      auto holds = [&](unsigned A, unsigned mm, unsigned mt) -> bool {
        return FM == COUNTER ? (A & mm) == mt : ((mt ^ (unsigned)__popc(A & mm)) & 1u) != 0u;
      };
#pragma unroll
      for (int i = 0; i < KI; i++)
      {
        em[i] = bit[i] = 0u;
        et[i] = 1u;
        val[i] = 0;
      }
      auto take = [&](int i) {
        if (FM == PAIR)
        {
          const uint2 e = tile[C::kEnt + 32 * i];
          em[i] = e.x;
          val[i] = (word & e.x) ? (int)e.y : -(int)e.y;
          watch |= e.x;
        }
        else
        {
          const uint4 e = tent[32 * i];
          entry(e, 0u, em[i], et[i]);
          val[i] = MASKS ? (int)(e.w & ~255u) : (int)e.w;
          bit[i] = MASKS && e.x ? __funnelshift_l(0u, 1u, e.w) : 0u;
          watch |= e.x;
        }
      };
      take(0);
      take(1);
      if (FM == PAIR || ents > 2)  // (most blocks have two at most; one branch for both: 3-SAT 10.6 and 10.3 ms)
      {
        take(2);
        take(3);
      }
      if (SP && FM != PAIR)
        for (int i = 0; i < xn; i++) watch |= xterm[32 * i].x;

      // ---- the other warps: room for this block's flips and draws
      auto room = [&]() -> bool {
        return (INT || (int)(head + 32u - (unsigned)kLog - acc_tail) <= 0) && (int)(fed - (W.taken + 32u)) >= 0;
      };
      if (!room())
      {
        look(R, acc_tail, fed);
        if (!room())
        {
          wait_room<INT, kLog>(R.tail, R.made, R.abort, a.err, head, W.taken);
          look(R, acc_tail, fed);
          if (!room()) return false;
        }
      }

      // ---- rounds: one, unless a lane has to be tried alone
      float2 iv0 = make_float2(0.f, 0.f);
      if (!REPLAY) iv0 = R.ring[(W.taken + (unsigned)lane) & (unsigned)(kRing - 1)];
      int cursor = 0;
      // Dense pair blocks: the flips in `mA` change the field by hm, kept up from
      // the matrix as decisions change.  Complete +-1 graphs of 64, 128 and 200
      // spins, 8 walkers, 400 sweeps (ms): 1.25, 2.72 and 5.68; every entry beyond
      // the fourth read again in each iteration: 2.00, 4.07 and 10.8.
      unsigned mA = 0;
      int hm = 0;
      while (true)
      {
        const bool active = lane >= cursor && lane < nvalid;
        const unsigned before = lt & ~((1u << cursor) - 1u);
        // ---- decisions: iterate until no lane's in-block members change
        unsigned A = done, U = 0, lm = 0;
        int g = 0;
        bool rare = false;
        while (true)
        {
          int h = base;
          lm = qm;
          auto apply = [&](int i) {
            if (FM == PAIR)
            {
              h += (A & em[i]) ? val[i] : 0;
              return;
            }
            const bool on = holds(A, em[i], et[i]);
            if (FM == COUNTER) h += on ? val[i] : 0;
            else h += on ? -val[i] : val[i];
            if (MASKS && on) lm |= bit[i];
          };
          apply(0);
          apply(1);
          if (FM == PAIR || ents > 2)
          {
            apply(2);
            apply(3);
          }
          if (FM == PAIR && SP && xn)
          {
            // the lanes whose decisions changed, from their rows of the matrix
            for (unsigned d = A ^ mA; d;)
            {
              int w[4];
              bool minus[4];
#pragma unroll
              for (int x = 0; x < 4; x++)
              {
                const int b = d ? __ffs(d) - 1 : 0;
                w[x] = d ? mat[32 * b] : 0;
                minus[x] = (((A ^ word) >> b) & 1u) != 0u;
                d &= d - 1u;
              }
#pragma unroll
              for (int x = 0; x < 4; x++) hm += minus[x] ? -w[x] : w[x];
            }
            mA = A;
            h += hm;
          }
          for (int i = 0; FM != PAIR && SP && i < xn; i++)
          {
            const uint4 e = xterm[32 * i];
            unsigned mm, mt;
            entry(e, done, mm, mt);
            const bool on = e.x && holds(A, mm, mt);
            const int w = MASKS ? (int)(e.w & ~255u) : (int)e.w;
            if (FM == COUNTER) h += on ? w : 0;
            else h += on ? -w : w;
            if (MASKS && on) lm |= __funnelshift_l(0u, 1u, e.w);
          }
          // the field in the variable's own direction, its sign and threshold
          bool up;
          float x;
          if (INT)
          {
            g = FM == COUNTER ? (sv ? h : -h) : (sv ? 2 * h : -2 * h);  // the cost difference
            up = active && g > 0;
            x = (float)g;
            rare = false;
          }
          else if (FM == COUNTER)
          {
            const int fd = sv ? (h >> 8) : -(h >> 8);
            const bool zero = lm == 0u;  // nothing contributes: +0.0
            up = active && !zero && fd > bnd;
            rare = active && !zero && (unsigned)(fd + bnd) <= (unsigned)(2 * bnd);
            x = (float)fd;
          }
          else
          {
            if (FM == PARITY) h >>= 8;
            g = sv ? -h : h;
            up = active && g < -bnd;
            rare = active && (unsigned)(g + bnd) <= (unsigned)(2 * bnd);
            x = (float)g;
          }
          // (an infinite beta: below every draw but an always accepting one)
          const float thr = S.beta_inf ? -3e38f : __fmul_rn(x, S.fscale);
          const float et = S.beta_inf ? 0.f : __fmaf_rn(fabsf(thr), 1.9073486328125e-06f, 1e-30f) + xmargin;  // 2^-19
          float2 iv = iv0;
          if (REPLAY)
          {
            U = __ballot_sync(kFull, up);
            iv = R.ring[(W.taken + (unsigned)__popc(U & before)) & (unsigned)(kRing - 1)];
          }
          const bool yes = iv.y < __fsub_rn(thr, et);
          const bool no = iv.x > __fadd_rn(thr, et);
          rare = rare || (up && !yes && !no);
          const bool acc = active && !rare && (!up || yes);
          const unsigned An = __ballot_sync(kFull, acc) | done;
          const unsigned diff = An ^ A;
          A = An;
          if (!__any_sync(kFull, (diff & watch) != 0u)) break;
        }

        // ---- what is committed: all, or the lanes before the first rare one, or
        // that one alone
        const unsigned Rm = __ballot_sync(kFull, rare);
        unsigned F = A & ~done;
        bool exact = false, last = true;
        double dE = 0.0;
        if (Rm == 0u)
        {
          if (REPLAY) W.taken += (unsigned)__popc(U);
        }
        else
        {
          const int f = __ffs(Rm) - 1;
          if (f > cursor)
          {
            F &= (1u << f) - 1u;
            if (REPLAY) W.taken += (unsigned)__popc(U & ((1u << f) - 1u));
            cursor = f;
          }
          else
          {
            const uint64_t rs = REPLAY ? stream_state(R, W) : 0;
            unsigned res = 0;
            if (lane == f)
              res = exact_attempt<FM, REPLAY, INT>(m, v, g, R.spins, rs, W.key, S.ctr0 + (unsigned long long)v, S.beta,
                                                   &dE);
            res = __shfl_sync(kFull, res, f);
            F = (res & 1u) << f;
            if (REPLAY) W.taken += res >> 1;
            exact = true;
            cursor = f + 1;
          }
          last = cursor >= nvalid;
        }
        const bool mine = ((F >> lane) & 1u) != 0u;
        const unsigned at = (head + (unsigned)__popc(F & lt)) & (unsigned)(kLog - 1);
        const unsigned all = done | F;
        if (!INT && mine)
        {
          if (FM == PAIR) ((uint32_t*)R.log)[at] = (uint32_t)v;
          else
          {
            const unsigned long long bits = (unsigned long long)__double_as_longlong(dE);
            const unsigned negs = (unsigned)own.z;
            uint4 ent;
            ent.x = (unsigned)v | ((unsigned)deg << 16) | (exact ? kExactF : 0u);
            // COUNTER: the sign is the literal; PARITY: the term's, the other
            // members' parity and the own spin
            ent.y = exact ? (unsigned)bits : lm;
            ent.z = exact ? (unsigned)(bits >> 32) : (FM == COUNTER ? (sv ? ~negs : negs) : (sv ? ~lm : lm));
            ent.w = 0u;
            R.log[at] = ent;
          }
        }
        if (FM == PAIR)
        {
          if (mine) R.z[v] = (uint8_t)(sv ^ 1u);
        }
        else if (F)
        {
          if (SP && !INT && xn) __syncwarp();  // (entries have been read)
          if (mine) ((uint16_t*)R.z)[v] = (uint16_t)((sv ^ 1u) | sv << 8);
          if (SP && n3 && mine)
          {
            const uint2* t3 = (staged ? tile + C::kRec : far) + 32 * (n0 + n1) + 48 * n2;
            for (int i = 0; i < n3; i++)
            {
              const uint32_t x = t3[32 * i].x;
              if (!(x & kNoWide)) flip_wide<FM>(zw, x & kWideMask, (sv ^ (x >> 31)) & 1u);
            }
          }
        }
        __syncwarp();
        R.spins[bi] = word ^ all;  // (every lane the same word)
        __syncwarp();
        if (INT && F) account_int(R, W, scan32, g, F, bi, nblocks, g_lsp);
        const unsigned nfl = (unsigned)__popc(F);
        head += nfl;
        W.nacc += nfl;
        W.nwin++;
        done = all;
        if (last) break;
      }
      return true;
    };
    if (special)
    {
      if (!block(std::true_type{})) return false;
    }
    else if (!block(std::false_type{})) return false;
    if (!REPLAY) W.taken += 32u;
    W.natt += (unsigned)nvalid;
    publish(R, ++finished, head, W.taken);
  }
  turns = T;
  return true;
}

// The running cost over n flips (lane i < n: the i-th difference d), in order, as
// prefix sums of whole numbers (ordered_sum.cuh) between the flips that need an
// add of their own; the first lowest (lane lowpos) below klow.
__device__ __forceinline__ void accumulate(double d, int n, double& cost, long long& klow, double& low, int& lowpos)
{
  const int lane = threadIdx.x & 31;
  int start = 0;
  // four prefixes at most (a cost near zero changes its binade often)
  for (int round = 0; round < 4 && n - start > 4; round++)
  {
    int ce;
    const long long C = osum::scaled(cost, ce);
    const bool in = lane >= start && lane < n, normal = ce != 0 && ce != 0x7FF;
    long long D = 0;
    bool ok = normal, tie = false;
    if (normal && in) ok = osum::step_of(d, ce, D, tie);
    const long long P = osum::prefix(C, D, tie);
    const unsigned bad = __ballot_sync(kFull, in && !(ok && osum::inside(C, P)));
    const int f = bad ? __ffs(bad) - 1 : n;
    if (f > start)
    {
      const bool taken = in && lane < f;
      long long mn = taken ? P : LLONG_MAX;
#pragma unroll
      for (int s = 16; s; s >>= 1) mn = min(mn, __shfl_xor_sync(kFull, mn, s));
      const double vmin = osum::unscaled(mn, ce);
      const long long km = order_key(vmin);
      if (km < klow)
      {
        klow = km;
        low = vmin;
        lowpos = __ffs(__ballot_sync(kFull, taken && P == mn)) - 1;
      }
      cost = osum::unscaled(__shfl_sync(kFull, P, f - 1), ce);
      start = f;
    }
    if (f < n)
    {
      cost = __dadd_rn(cost, __shfl_sync(kFull, d, f));
      const long long kc = order_key(cost);
      if (kc < klow)
      {
        klow = kc;
        low = cost;
        lowpos = f;
      }
      start = f + 1;
    }
  }
  double dn = __shfl_sync(kFull, d, start & 31);
  for (int i = start; i < n; i++)
  {
    const double di = dn;
    dn = __shfl_sync(kFull, d, (i + 1) & 31);  // ahead of the dependent add
    cost = __dadd_rn(cost, di);
    const long long kc = order_key(cost);
    if (kc < klow)
    {
      klow = kc;
      low = cost;
      lowpos = i;
    }
  }
}

// ---------------------------------------------------------------------------
// The accountant (FP64 models): running cost, lowest cost and lowest state
// from the log.  WIDE: a term model with rows of more than 32 terms.
// ---------------------------------------------------------------------------
template <int FM, bool WIDE>
__device__ __noinline__ bool account(const SweepArgs& a, const DevModel& m, const Region R, double& cost,
                                        double& low, uint32_t* g_lsp)
{
  const int lane = threadIdx.x & 31;
  const int nw = a.p.nw;
  constexpr int kLog = FM == PAIR ? kLogBytes / 4 : kLogBytes / 16;
  unsigned tail = 0;
  long long klow = order_key(low);
  // the coming batch's entries and row bounds, in the lanes below `ready`: their
  // loads run beside the sum over the batch before
  int v = 0, q0 = 0, q1 = 0, ready = 0;
  uint4 ent = make_uint4(0u, 0u, 0u, 0u);
  auto fetch = [&](unsigned at) {
    if (FM == PAIR) v = (int)((const uint32_t*)R.log)[at & (unsigned)(kLog - 1)];
    else
    {
      ent = R.log[at & (unsigned)(kLog - 1)];
      v = (int)(ent.x & 0x7FFFu);
    }
    q0 = __ldg(m.row + v);
    q1 = __ldg(m.row + v + 1);
  };
  while (true)
  {
    // wait for a batch (16 entries, or whatever is left once the decider is done)
    unsigned h = 0;
    int fin = 0;
    if (lane == 0)
    {
      Patience limit;
      unsigned last_h = tail, last_u = ld_acquire(R.used);
      while (true)
      {
        h = ld_acquire(R.head);
        if (h - tail >= 16u) break;
        if (ld_acquire(R.done))
        {
          h = ld_acquire(R.head);
          fin = 1;
          break;
        }
        if (ld_acquire(R.abort))
        {
          fin = 2;
          break;
        }
        const unsigned u = ld_acquire(R.used);
        if (h != last_h || u != last_u)
        {
          last_h = h;
          last_u = u;
          limit.renew();
        }
        if (limit.over())
        {
          raise_abort(R, a.err);
          fin = 2;
          break;
        }
        __nanosleep(20);
      }
    }
    h = __shfl_sync(kFull, h, 0);
    fin = __shfl_sync(kFull, fin, 0);
    if (fin == 2) return false;
    while (h != tail)
    {
      int n = (int)min(32u, h - tail);
      double d = 0.0;
      if (lane < n && lane >= ready) fetch(tail + (unsigned)lane);
      if (FM == PAIR)
      {
        // Flips of one sweep, in index order: a member below the flip has its
        // spin after the batch, one above it its spin before.
        uint32_t* after = R.aspins + nw + 4;
        const int prev = __shfl_up_sync(kFull, v, 1);
        const unsigned wrap = __ballot_sync(kFull, lane > 0 && lane < n && v <= prev);
        if (wrap) n = __ffs(wrap) - 1;
        if (lane < n) atomicXor(after + (v >> 5), 1u << (v & 31));
        __syncwarp();
        if (lane < n) d = exact_dE<FM>(m, v, q0, q1, R.aspins, after);
      }
      else
      {
        const int deg = (int)((ent.x >> 16) & 255u);
        const bool exact = (ent.x & kExactF) != 0u;
        if (lane < n && exact)
          d = __longlong_as_double((long long)((unsigned long long)ent.y | ((unsigned long long)ent.z << 32)));
        else if (lane < n && (!WIDE || deg <= 32)) d = dE_from_masks<FM>(m.coef + q0, deg, ent.y, ent.z);
        if constexpr (WIDE)
        {
          const Summed x = sum_rows<FM>(m, R.aspins, nw, v, q0, q1, lane < n && !exact && deg > 32, n, d);
          d = x.d;
          n = x.n;
        }
      }
      __syncwarp();
      tail += (unsigned)n;
      if (lane == 0) st_release(R.tail, tail);
      const int fv = v;  // this batch's
      ready = (int)min(32u, h - tail);
      if (lane < ready) fetch(tail + (unsigned)lane);
      // running cost in flip order (markov/walker.h:225) and the first
      // strict improvement of the lowest (markov/walker.h:269-280)
      int lowpos = -1;
      accumulate(d, n, cost, klow, low, lowpos);
      // the accountant's spins, and the lowest state at lowpos
      if (lane < n && lane <= lowpos) atomicXor(R.aspins + (fv >> 5), 1u << (fv & 31));
      __syncwarp();
      if (lowpos >= 0)
      {
        for (int q = lane; q < nw; q += 32) g_lsp[q] = R.aspins[q];
        __syncwarp();
      }
      if (lane < n && lane > lowpos) atomicXor(R.aspins + (fv >> 5), 1u << (fv & 31));
      __syncwarp();
    }
    if (fin == 1) return true;
  }
}

// copy n 16-byte words, four in flight per thread
__device__ __noinline__ void copy16(uint4* dst, const uint4* src, int n, int t, int nt)
{
  int q = t;
  for (; q + 3 * nt < n; q += 4 * nt)
  {
    const uint4 x0 = src[q], x1 = src[q + nt], x2 = src[q + 2 * nt], x3 = src[q + 3 * nt];
    dst[q] = x0;
    dst[q + nt] = x1;
    dst[q + 2 * nt] = x2;
    dst[q + 3 * nt] = x3;
  }
  for (; q < n; q += nt) dst[q] = src[q];
}

// A walker's warps: decider, feeder and, for FP64 models, accountant (warp w of
// the block: role w / wpc of walker slot w % wpc, so that a block's deciders
// lie on different schedulers).  Walker slot s of block b takes stream s *
// gridDim + b: neighbouring streams (tempering: the hottest, which come first)
// lie on different SMs.
template <int FM, bool REPLAY, bool INT>
__global__ void __launch_bounds__(INT ? 512 : 384, 1) fc_sweep_kernel(const __grid_constant__ SweepArgs a, int wpc,
                                                                     Shape sh)
{
  extern __shared__ __align__(128) unsigned char smem[];
  float4* s_scr = (float4*)smem;
  for (int t = threadIdx.x; t < 256; t += blockDim.x) s_scr[t] = g_scr[t];
  if (sh.share > 1 && threadIdx.x == 0)
  {
    const Region R = carve<INT>(smem, 0, sh);
    for (int i = 0; i < kBufs; i++) mbar_init(&R.bars[i]);
    *R.abort = 0u;
  }
  const int stride = region_bytes(sh, INT);
  // (blocks that the walkers have finished, before the first one's feeder looks)
  if (sh.share > 1 && (int)threadIdx.x < wpc)
    *carve<INT>(smem, (int)threadIdx.x, sh).blocks = 0u;
  // A chained launch: the kernel before is done from here on (this one's launch
  // and table overlap with it), and the one behind may start to.  PT on 3-SAT,
  // 200 steps of a 50 us sweep and its swaps: 12.8 and 11.9 ms.
  asm volatile("griddepcontrol.wait;" ::: "memory");
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
  __syncthreads();

  constexpr int kRoles = INT ? 2 : 3;
  const int lane = threadIdx.x & 31;
  // the warp's index through a shuffle: the compiler then knows that the roles
  // below do not divide a warp, and puts no convergence check around every
  // vote and shuffle (those took more than half of the decider's time)
  const int wib = __shfl_sync(0xffffffffu, (int)threadIdx.x >> 5, 0);
  const int role = wib / wpc;  // 0 decider, 1 feeder, 2 accountant
  const int ws = wib - role * wpc;
  const bool decider = role == 0;
  const int ws0 = ws * (int)gridDim.x + (int)blockIdx.x;
  const bool queued = a.queue != nullptr;
  if (!queued && ws0 >= a.n_streams) return;
  const int w = queued ? 0 : (a.order ? a.order[ws0] : ws0);
  const Region R = carve<INT>(smem, ws, sh);
  // the walkers whose chunks this one's feeder brings
  const int live = sh.share <= 1 ? 1 : ws ? 0 : min(wpc, (a.n_streams - (int)blockIdx.x + (int)gridDim.x - 1) / (int)gridDim.x);
  const int bar_id = 1 + ws;
  const int me = role * 32 + lane, nme = kRoles * 32;  // thread of the walker
  // (the feeder's own barriers; the first walker_sync below shows them to the decider)
  if (sh.share <= 1 && role == 1 && lane == 0)
    for (int i = 0; i < kBufs; i++) mbar_init(&R.bars[i]);
  uint64_t rs = (REPLAY && !queued) ? a.rng[w] : 0;
  Turns turns(1, sh.bufs);

  int r = w;
  while (true)
  {
    if (queued)
    {
      if (decider && lane == 0) *R.next = (unsigned)atomicAdd(a.queue, 1);
      walker_sync<INT>(bar_id);
      r = __shfl_sync(kFull, (int)*(volatile unsigned*)R.next, 0);
    }
    if (r >= a.n_walkers) break;
    const DevModel& m = queued ? a.models[a.model_of[r]] : a.m;
    const int N = m.n_vars;
    turns.walker((N + 31) >> 5);
    const int slot = a.slot_of ? a.slot_of[r] : r;
    uint32_t* g_spins = a.p.spins + (size_t)slot * a.p.nw;
    if (queued && REPLAY) rs = a.rng[r];
    if (decider && lane == 0)
    {
      *R.head = 0u;
      *R.tail = 0u;
      *R.done = 0u;
      if (sh.share <= 1) *R.abort = 0u;
      *R.made = 0u;
      *R.used = 0u;
      *R.blocks = 0u;
    }
    copy16((uint4*)R.spins, (const uint4*)g_spins, a.p.nw >> 2, me, nme);
    if (me < 4) R.spins[a.p.nw + me] = 0u;
    if (!INT) copy16((uint4*)R.aspins, (const uint4*)g_spins, a.p.nw >> 2, me, nme);
    if (!INT && FM == PAIR) copy16((uint4*)(R.aspins + a.p.nw + 4), (const uint4*)g_spins, a.p.nw >> 2, me, nme);
    walker_sync<INT>(bar_id);
    make_bytes<FM>(m, R.z, R.spins, a.p.nw, me, nme);
    walker_sync<INT>(bar_id);

    uint64_t key = 0;
    if (!REPLAY)
    {
      const long long lr = queued ? a.local_of[r] : r;
      key = counter_key(a.seed + (uint32_t)(lr / a.key_div), a.key_base + (unsigned long long)(lr % a.key_div));
    }
    uint32_t* g_lsp = a.p.lspins + (size_t)r * a.p.nw;
    if (decider)
    {
      Walk W;
      W.natt = W.nacc = W.nwin = 0;
      W.icost = W.ilow = 0;
      W.rs = rs;
      W.raw0 = 0;
      W.key = key;
      W.taken = 0;
      if (INT)
      {
        W.icost = (long long)a.p.cost[slot];
        W.ilow = (long long)a.p.lowest[r];
      }
      const bool ok = decide_sweeps<FM, REPLAY, INT>(a, m, R, sh, r, turns, W, g_lsp);
      if (lane == 0) st_release(R.done, 1u);
      if (REPLAY) rs = stream_state(R, W);
      walker_sync<INT>(bar_id);
      if (ok && !*(volatile unsigned*)R.abort && lane == 0)
      {
        a.p.attempts[r] += W.natt;
        a.p.accepts[r] += W.nacc;
        a.p.step_att[r] += W.natt;
        a.p.step_acc[r] += W.nacc;
        if (a.p.windows) a.p.windows[r] += W.nwin;
        if (queued && REPLAY) a.rng[r] = rs;
        if (INT)
        {
          a.p.cost[slot] = (double)W.icost;
          const double nlow = (double)W.ilow;
          if (a.p.lowtag && nlow < a.p.lowest[r]) a.p.lowtag[r] = a.tag;
          a.p.lowest[r] = nlow;
        }
      }
    }
    else if (role == 1)
    {
      feed<FM, REPLAY>(R, s_scr, m.fc_desc, m.fc_tab, sh.words, sh.words, turns, a.n_sweeps, rs, key,
                       (unsigned long long)a.sweep_base * (unsigned long long)N, N, live, stride / 4, a.err);
      walker_sync<INT>(bar_id);
    }
    else
    {
      double cost = a.p.cost[slot], low = a.p.lowest[r];
      const bool ok = FM != PAIR && m.max_deg > 32 ? account<FM, FM != PAIR>(a, m, R, cost, low, g_lsp)
                                                   : account<FM, false>(a, m, R, cost, low, g_lsp);
      walker_sync<INT>(bar_id);
      if (ok && !*(volatile unsigned*)R.abort && lane == 0)
      {
        a.p.cost[slot] = cost;
        if (a.p.lowtag && low < a.p.lowest[r]) a.p.lowtag[r] = a.tag;
        a.p.lowest[r] = low;
      }
    }
    if (*(volatile unsigned*)R.abort) return;
    copy16((uint4*)g_spins, (const uint4*)R.spins, a.p.nw >> 2, me, nme);
    walker_sync<INT>(bar_id);  // the region is reused by the next walker
    if (!queued) break;
  }
  if (REPLAY && !queued && decider && lane == 0) a.rng[w] = rs;
}

template <int FM, bool R, bool I>
static cudaError_t go(const SweepArgs& a, cudaStream_t s, int wpc, const Shape& sh)
{
  auto k = fc_sweep_kernel<FM, R, I>;
  const int smem = kTable + common_bytes(sh) + wpc * region_bytes(sh, I);
  const int threads = (I ? 64 : 96) * wpc;
  const cudaError_t allowed = allow_shared((const void*)k, smem);
  if (allowed != cudaSuccess) return allowed;
  int blocks = (a.n_streams + wpc - 1) / wpc;
  if (a.queue)
  {
    // persistent: as many blocks as stay resident, the queue feeds them
    int per_sm = 0;
    cudaError_t e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k, threads, smem);
    if (e != cudaSuccess) return e;
    blocks = std::max(1, std::min((a.n_walkers + wpc - 1) / wpc, std::max(1, per_sm) * kSms));
  }
  if (blocks <= 0) return cudaGetLastError();
  if (!a.chained)
  {
    k<<<blocks, threads, smem, s>>>(a, wpc, sh);
    return cudaGetLastError();
  }
  cudaLaunchAttribute early{};
  early.id = cudaLaunchAttributeProgrammaticStreamSerialization;
  early.val.programmaticStreamSerializationAllowed = 1;
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = dim3((unsigned)blocks);
  cfg.blockDim = dim3((unsigned)threads);
  cfg.dynamicSmemBytes = (size_t)smem;
  cfg.stream = s;
  cfg.attrs = &early;
  cfg.numAttrs = 1;
  return cudaLaunchKernelEx(&cfg, k, a, wpc, sh);
}

template <int FM>
static cudaError_t go_fm(const SweepArgs& a, cudaStream_t s, int wpc, const Shape& sh)
{
  const bool I = a.m.int_mode != 0;
  if (a.replay) return I ? go<FM, true, true>(a, s, wpc, sh) : go<FM, true, false>(a, s, wpc, sh);
  return I ? go<FM, false, true>(a, s, wpc, sh) : go<FM, false, false>(a, s, wpc, sh);
}

// a walker's region for a model in a population of this stride
static Shape shape_of(const DevModel& m, int nw, int bufs, bool shared)
{
  Shape s;
  s.pair = m.flavor == F_PARITY && m.pair_only;
  s.second = s.pair || m.max_deg > 32;
  s.nw = nw;
  s.zb = s.pair ? nw * 32 : (64 * nw + 16 + m.fc_wide + 15) & ~15;
  s.words = m.fc_words;
  s.bufs = bufs;
  s.share = shared ? 2 : 1;
  // a state that leaves less room: smaller tiles (larger blocks read their
  // records from HBM)
  const int least = Chunk<COUNTER>::kRec;
  const int room = (kMaxSmem - kTable - common_bytes(s) - region_bytes(s, m.int_mode != 0)) / (8 * bufs);
  if (room < 0) s.words = std::max(least, (s.words + room - 1) & ~1);
  return s;
}
// walkers of a block, at most
static int walkers_of(const Shape& s, bool integer)
{
  return std::min(integer ? 8 : 4, (kMaxSmem - kTable - common_bytes(s)) / region_bytes(s, integer));
}
}  // namespace fc

bool fc_fits(const DevModel& m, int nw)
{
  if (!m.fc_desc || m.sweep_size != m.n_vars || m.n_vars <= 0) return false;
  if (!(m.flavor == F_PARITY || m.flavor == F_COUNTER)) return false;
  // (the line as it has been: a launch may do with two buffers, which saves more
  // than a second copy of a term model's spins takes)
  fc::Shape s = fc::shape_of(m, nw, fc::kBufs, false);
  s.words = std::min(s.words, fc::Chunk<fc::COUNTER>::kRec);
  s.second = s.pair;
  return fc::kTable + fc::region_bytes(s, m.int_mode != 0) - 16 <= fc::kMaxSmem;
}

cudaError_t launch_fc_sweep(const SweepArgs& a, cudaStream_t s, int wpb)
{
  if (!fc_fits(a.m, a.p.nw)) return cudaErrorInvalidValue;
  if (!a.queue && a.n_streams != a.n_walkers) return cudaErrorInvalidValue;  // (a stream to a walker)
  const bool I = a.m.int_mode != 0;
  // The first of these shapes with the fewest waves of blocks (twice as long where
  // the largest blocks do not fit a buffer): four chunk buffers each, which cover
  // the copy's latency best, three, or a block's walkers on the same ones, in
  // step.  512 tempering walkers of a 4096-variable PUBO, 100 sweeps: 61.3 ms at
  // three walkers a block with four buffers each, 43.7 at four with three.  608
  // walkers of a 1000-spin model with 8 hubs of 200 couplings, 40 sweeps: 6.15 with
  // buffers of their own, one walker a block, 1.99 with the same, four a block; of a
  // complete +-1 graph of 200 spins, 100 sweeps: 5.8 and 1.75.
  struct Choice { int bufs; bool shared; };
  const Choice choices[] = {{4, false}, {3, false}, {4, true}, {3, true}, {2, false}, {2, true}};
  fc::Shape sh{};
  int wmax = 0;
  long long least = LLONG_MAX;
  for (const Choice& c : choices)
  {
    if (c.shared && a.queue) continue;
    const fc::Shape x = fc::shape_of(a.m, a.p.nw, c.bufs, c.shared);
    const int w = fc::walkers_of(x, I);
    if (w < 1) continue;
    const long long waves = (a.n_streams + (long long)w * fc::kSms - 1) / ((long long)w * fc::kSms);
    const long long cost = waves * (x.words < a.m.fc_words ? 2 : 1);
    if (cost >= least) continue;
    least = cost;
    sh = x;
    wmax = w;
  }
  // spread the walkers over the SMs: as few per block as fills them
  int wpc = (a.n_streams + fc::kSms - 1) / fc::kSms;
  if (a.queue) wpc = std::min(wpc, wpb);
  wpc = std::max(1, std::min(wpc, wmax));
  if (a.m.flavor == F_COUNTER) return fc::go_fm<fc::COUNTER>(a, s, wpc, sh);
  return a.m.pair_only ? fc::go_fm<fc::PAIR>(a, s, wpc, sh) : fc::go_fm<fc::PARITY>(a, s, wpc, sh);
}

void fc_upload(const double* ln, const float* scr, const unsigned long long* jA,
               const unsigned long long* jC)
{
  cudaMemcpyToSymbol(fc::c_ln, ln, 1024 * sizeof(double));
  float4 t[1024];
  for (int i = 0; i < 1024; i++)
  {
    t[i] = make_float4(scr[3 * i], scr[3 * i + 1], scr[3 * i + 2], 0.f);
    if ((i & 255) == 1) t[i].x = INFINITY;  // log(0): never accepted
  }
  cudaMemcpyToSymbol(fc::g_scr, t, sizeof t);
  ulonglong2 j[33];
  for (int i = 0; i < 33; i++) j[i] = make_ulonglong2(jA[i], jC[i]);
  cudaMemcpyToSymbol(fc::c_jump, j, sizeof j);
}
}  // namespace qio
