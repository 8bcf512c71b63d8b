// fields.cu -- the block-decided Metropolis sweep (sm_103a).
//
// One warp, the DECIDER, runs a walker's ordered sweep (markov/walker.h:
// 143-153,209-229) 32 variables at a time, a variable per lane.  At a block's
// start every lane gathers its field -- the cost difference of its flip in
// fixed point (model_host.cc, build_fields) -- from the walker's state in
// shared memory: the neighbours' spins (Ising models of one- and two-member
// terms) or one byte per term that holds the literals of all its members.
//
// The block is then decided as a whole.  Lane v's decision depends on the
// decisions of the lanes before it in two ways: through the terms it shares
// with them (fc_in lists these with their members' lanes) and, on replayed
// streams, through the draw it gets (the uphill lanes before it each take
// one).  Both only look back, so the lanes iterate: decide with the accept
// mask of the last round, vote, and decide again where a member of a lane's
// in-block terms changed; a mask that no longer changes any lane's terms is the
// ordered sweep's, lane by lane from the first.  A field within its rounding
// margin of zero, a comparison inside the FP32 screen's margin or a row too
// wide for the log's masks ends the block early: the lanes before it are
// committed, the lane itself is tried alone with the reference's FP64 sum and
// ln-table expression, and the rest of the block is decided after it.
//
// A second warp, the FEEDER, runs ahead of the decider: it fills a ring with
// the walker's random draws as intervals of their ln-table values and brings
// each block's chunk of the model (records, in-block terms) into one of four
// shared-memory buffers by one TMA bulk copy.
//
// FP64 models: a third warp, the ACCOUNTANT, consumes a log of the flips in
// batches of up to 32: every lane recomputes one flip's exact FP64 cost
// difference (the reference's order and rounding, model/ising.h:108-117,
// model/pubo.h:335-367), then the running cost is accumulated in flip order
// exactly as cost_ += diff (markov/walker.h:225) and the lowest state is taken
// at the first strict improvement (markov/walker.h:269-280) from the
// accountant's own copy of the spins.  Neither the decisions nor the draws
// depend on the running cost.  Integer models keep cost and lowest in the
// decider (exact in any order).
//
// What bounds it: the decider's chain of dependent votes, shared-memory loads
// and integer instructions: 1600 cycles a block on a sparse Ising model (N =
// 1000, 64 walkers: gather 370, decisions 330, wait and publication 320, commit
// 160), 4200 on a PUBO of 11.7 terms a variable (gather 1040, decisions 600,
// commit 1600).  A thousand sweeps of the first take 24.7 ms, where fields kept
// up to date by atomics took 63; 100 sweeps of 512 tempering walkers of the
// second 62 ms, where the windowed kernel took 190.  Shared-memory atomics have no
// place in it: one costs 26 to 44 cycles of its warp's memory queue on this
// chip (a load 5), so a form that kept the fields up to date by atomics on
// the co-members took 2300 to 7900 cycles a block, and gathering them anew
// costs less than a few flips' scatter.
//
// Waits between the warps poll shared-memory counters (acquire/release) with a
// time limit on lack of progress; on expiry the kernel raises the device error
// flag and all of the walker's warps return.
#include <algorithm>
#include <atomic>
#include <climits>
#include <cmath>

#include "metropolis.cuh"
#include "ordered_sum.cuh"
#include "qio_internal.h"

namespace qio
{
namespace fc
{
using namespace qio::mc;
static const unsigned kFull = 0xffffffffu;
static const int kMaxRows = 64;   // records per lane of a staged block, at most
static const int kIn = 4;         // in-block entries per lane of a staged block
static const int kLogBytes = 1024;  // flip log per walker: 64 entries of 16 bytes, pair models 256 of 4
static const int kRing = 128;     // draw intervals per walker (power of 2)
static const int kCtrl = 64;      // per-walker control block: mbarriers, counters
static const int kTable = 4096;   // per block: screen row 0
static const unsigned kExactF = 0x80000000u;   // log entry: exact FP64 difference
// record and in-block entry flags (build_fields)
static const uint32_t kTermMask = 0x0003FFFFu;
static const uint32_t kShared = 0x00080000u;   // record: another member in the block
static const uint32_t kBigTerm = 0x00100000u;  // record: more than eight members
static const uint32_t kBigEntry = 0x40000000u; // in-block entry: the same
static const unsigned kNoEntry = 0xffffffffu;  // no in-block entry
static const int kMaxSmem = 227 * 1024;
static const int kSms = 152;
static const long long kPatience = 8000000000LL;  // cycles without progress, about 4 s

// the three forms of a field (build_fields)
enum Form
{
  PAIR = 0,     // Ising, terms of one or two members: spins alone
  COUNTER = 1,  // PUBO, MaxSat: term bytes count true literals
  PARITY = 2    // Ising with larger terms: term bytes are parities
};

// A block's chunk of the model's table (build_fields), in 8-byte words: header
// (4: record rows | in-block entry rows << 8 | further entry rows << 16, first
// further entry), lane data (32), in-block entries (kIn x 32 of 8 or 16 bytes), record
// rows (of 32; term models 33, a bank's shift, as one lane's records are read
// across too)
template <int FM>
struct Chunk
{
  static const int kLane = 4;
  static const int kEnt = 36;
  static const int kRec = 36 + kIn * 32 * (FM == PAIR ? 1 : 2);
  static const int kPitch = FM == PAIR ? 32 : 33;
};
__host__ __device__ inline int chunk_words(bool pair, int rows)
{
  return 36 + kIn * 32 * (pair ? 1 : 2) + rows * (pair ? 32 : 33);
}
static const int kBufs = 4;  // chunk buffers per walker, at most (Shape::bufs)

__constant__ double c_ln[1024];
// screen of the ln-table comparison per (row, bucket): y0, dy, error margin;
// bucket 1 (log(0), never accepted) holds y0 = +inf
__device__ float4 g_scr[1024];
__constant__ ulonglong2 c_jump[33];
static const unsigned long long kMult = 6364136223846793005ULL;
static const unsigned long long kInc = 1442695040888963407ULL;

// ---- shared-memory synchronisation between the two warps -----------------
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

// Term bytes (COUNTER, PARITY).  A term of up to eight members: bit i set when
// the literal of its i-th member by variable id is true (Ising: its spin).  A
// larger term: the count of true literals, or the parity.
__device__ __forceinline__ bool big_term(const DevModel& m, uint32_t t)
{
  return __ldg(m.trow + t + 1) - __ldg(m.trow + t) > 8;
}

// Exact cost difference of flipping v (FP64 models): the reference's sum
// over the row in ascending term id, from the spins (pair) or the term bytes.
template <int FM>
__device__ __noinline__ double exact_dE(const DevModel& m, int v, const uint32_t* spins, const uint8_t* z)
{
  const int rb = __ldg(m.row + v), re = __ldg(m.row + v + 1);
  const uint32_t sv = spin_of(spins, v);
  double d = 0.0;
  for (int k = rb; k < re; k++)
  {
    const double c = __ldg(m.coef + k);
    if (FM == PAIR)
    {
      const int u = __ldg(m.other + k);
      const uint32_t par = sv ^ (u >= 0 ? spin_of(spins, u) : 0u);
      d = __dadd_rn(d, par ? -c : c);
      continue;
    }
    const uint32_t e = __ldg(m.inc + k);
    uint32_t n = z[e & ~kNegBit];  // true literals, or the parity
    if (!big_term(m, e & ~kNegBit)) n = (uint32_t)__popc(n);
    if (FM == PARITY) d = __dadd_rn(d, (n & 1u) ? -c : c);
    else
    {
      const bool lit = ((sv ^ (e >> 31)) & 1u) != 0u;
      if (n == (lit ? 1u : 0u)) d = lit ? __dadd_rn(d, c) : __dsub_rn(d, c);
    }
  }
  return (FM == COUNTER) ? d : neg2x(d);
}

// Exact cost difference from a log entry's masks (accountant): qm = the
// contributing incidences, sm = their signs.
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
  int nw;    // spin words of the population
  int mp;    // term bytes; pair models: a byte per variable
  int rows;  // record rows of a staged block
  int bufs;  // chunk buffers: kBufs, or one less where another walker then fits
  bool pair;
};
struct Region
{
  unsigned long long* bars;  // kBufs mbarriers
  unsigned* head;            // log entries published by the decider (with `used`, 8 bytes)
  unsigned* tail;            // log entries consumed by the accountant
  unsigned* done;            // the decider finished the walker
  unsigned* abort;           // a wait gave up: all warps leave
  unsigned* next;            // the walker taken from the queue
  unsigned* made;            // draws in the ring
  unsigned* used;            // draws taken by the decider
  unsigned* blocks;          // blocks the decider has finished (before `head`, `used`)
  float2* ring;              // kRing screen intervals
  uint32_t* raw;             // kRing: stream position after the draw (replay)
  uint4* log;                // kLogBytes (FP64 models)
  uint2* tiles;              // the block chunks
  uint8_t* z;                // term bytes; pair models: the spins, a byte each
  uint32_t* spins;           // nw + 4 words (words of zeros after the last)
  uint32_t* aspins;          // the accountant's spins (FP64 models), two copies for pair models
};

__host__ __device__ inline int tile_words(const Shape& s) { return (chunk_words(s.pair, s.rows) + 1) & ~1; }
__host__ __device__ inline int region_bytes(const Shape& s, bool integer)
{
  return kCtrl + kRing * 12 + (integer ? 0 : kLogBytes) + s.bufs * tile_words(s) * 8 + s.mp + 4 * (s.nw + 4) +
         (integer ? 0 : 4 * (s.nw + 4) * (s.pair ? 2 : 1));
}

template <bool INT>
__device__ __forceinline__ Region carve(unsigned char* base, const Shape& s)
{
  Region R;
  R.bars = (unsigned long long*)base;
  unsigned* c = (unsigned*)(base + 32);
  R.head = c;
  R.used = c + 1;
  R.tail = c + 2;  // (tail, made: one 8-byte word)
  R.made = c + 3;
  R.done = c + 4;
  R.abort = c + 5;
  R.next = c + 6;
  R.blocks = c + 7;
  R.ring = (float2*)(base + kCtrl);
  R.raw = (uint32_t*)(R.ring + kRing);
  R.log = (uint4*)(R.raw + kRing);
  R.tiles = (uint2*)(R.log + (INT ? 0 : kLogBytes / 16));
  R.z = (uint8_t*)(R.tiles + s.bufs * tile_words(s));
  R.spins = (uint32_t*)(R.z + s.mp);
  R.aspins = R.spins + s.nw + 4;
  return R;
}

__device__ __forceinline__ void raise_abort(const Region& R, int* err)
{
  if (err) atomicExch(err, 1);
  st_release(R.abort, 1u);
}

// term t's byte from the spins
template <int FM>
__device__ __forceinline__ uint8_t term_byte(const DevModel& m, int t, const uint32_t* spins)
{
  const int b = __ldg(m.trow + t), e = __ldg(m.trow + t + 1);
  uint32_t mask = 0, n = 0;
  for (int k = b; k < e; k++)
  {
    const uint32_t x = __ldg(m.tvar + k);
    const uint32_t lit = spin_of(spins, (int)(x & ~kNegBit)) ^ (x >> 31);
    n += lit;
    if (e - b > 8) continue;
    int at = 0;
    for (int j = b; j < e; j++) at += (__ldg(m.tvar + j) & ~kNegBit) < (x & ~kNegBit);
    mask |= lit << at;
  }
  if (e - b <= 8) return (uint8_t)mask;
  return (uint8_t)(FM == PARITY ? n & 1u : n);
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
// Chunks: block t's goes to buffer t % bufs once the decider is done with
// block t - bufs (t counts over the warp's walkers, from `t0`).
// ---------------------------------------------------------------------------
template <int FM, bool REPLAY>
__device__ __noinline__ void feed(const Region R, const float4* s_scr, const int4* desc, const uint2* table, int tile_w,
                                  int cap, int bufs, int nblocks, int total, unsigned t0, uint64_t rs, uint64_t key,
                                  unsigned long long ctr, int n_vars, int* err)
{
  const int lane = threadIdx.x & 31;
  const unsigned lt = (1u << lane) - 1u;
  uint64_t st = REPLAY ? c_jump[lane].x * rs + c_jump[lane].y : 0;
  const uint64_t jA = c_jump[32].x, jC = c_jump[32].y;
  unsigned made = 0;
  uint32_t raw = (uint32_t)lane + 1u;  // stream position after this lane's draw
  int carry = 0;                       // zeros at the end of the last 32 draws that await the next
  int first = 0;                       // counter: the first variable of the coming attempts
  int t = 0, tb = 0;                   // chunks issued; the next one's block
  int4 d = __ldg(desc);                // ... and its descriptor
  Patience limit;
  unsigned last_u = 0, last_b = 0;
  while (true)
  {
    // what the decider has done
    const unsigned used = ld_acquire(R.used);
    const unsigned blocks = *(volatile unsigned*)R.blocks;
    while (t < total && t < (int)blocks + bufs)
    {
      if (lane == 0)
      {
        const unsigned at = (t0 + (unsigned)t) % (unsigned)bufs;
        tile_issue(R.tiles + at * tile_w, table + d.x, (unsigned)chunk_words(FM == PAIR, min(d.y, cap)) * 8u,
                   &R.bars[at]);
      }
      t++;
      tb = tb + 1 < nblocks ? tb + 1 : 0;
      d = __ldg(desc + tb);
    }
    if (made + 32u - used >= (unsigned)kRing)
    {
      // no room for draws (the last one taken stays: its stream position)
      int leave = 0;
      if (ld_acquire(R.done)) leave = 1;
      else if (ld_acquire(R.abort)) leave = 2;
      else if (used != last_u || blocks != last_b)
      {
        last_u = used;
        last_b = blocks;
        limit.renew();
      }
      else if (limit.over())
      {
        raise_abort(R, err);
        leave = 2;
      }
      leave = __shfl_sync(kFull, leave, 0);
      if (leave == 0) continue;
      // given up: the copies in flight land before the region is
      if (leave == 2 && lane == 0)
        for (int x = max(0, t - bufs); x < t; x++)
        {
          const unsigned n = t0 + (unsigned)x;
          mbar_wait(&R.bars[n % (unsigned)bufs], (n / (unsigned)bufs) & 1u);
        }
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

// a flip's change of a term that it shares within the block (x: in-block entry)
template <int FM>
__device__ __forceinline__ void flip_shared(uint8_t* z, unsigned x, uint32_t sv)
{
  const unsigned t = x & kTermMask, sh = (t & 3u) * 8u;
  unsigned* word = (unsigned*)(z + (t & ~3u));
  if (!(x & kBigEntry)) atomicXor(word, 1u << (sh + ((x >> 23) & 7u)));
  else if (FM == PARITY) atomicXor(word, 1u << sh);
  else if ((sv ^ (x >> 31)) & 1u) atomicSub(word, 1u << sh);
  else atomicAdd(word, 1u << sh);
}

// Lane f's attempt alone: the reference's sum, draws and comparison.  Bit 0:
// accepted; bit 1: it drew.
template <int FM, bool REPLAY, bool INT>
__device__ __noinline__ unsigned exact_attempt(const DevModel& m, int v, int g, const uint32_t* spins, const uint8_t* z,
                                              uint64_t rs, uint64_t key, unsigned long long ctr, double beta,
                                              double* dE_out)
{
  const double dE = INT ? (double)g : exact_dE<FM>(m, v, spins, z);
  const bool inf = ((unsigned long long)__double_as_longlong(beta) & 0x7FFFFFFFFFFFFFFFULL) == 0x7FF0000000000000ULL;
  *dE_out = dE;
  if (le_zero(dE)) return 1u;
  if (REPLAY) return 2u | (unsigned)draw_chain(rs, inf, dE, beta);
  return 2u | (unsigned)counter_chain(key, ctr, inf, dE, beta);
}

template <int FM, bool REPLAY, bool INT>
__device__ __forceinline__ bool decide_sweeps(const SweepArgs& a, const DevModel& m, const Region R, const Shape& sh, int r,
                                              unsigned t0, Walk& W, uint32_t* g_lsp)
{
  constexpr int KI = kIn;  // in-block entries held in registers
  constexpr int kLog = FM == PAIR ? kLogBytes / 4 : kLogBytes / 16;  // entries, a power of two
  using C = Chunk<FM>;
  const int lane = threadIdx.x & 31;
  const unsigned lt = (1u << lane) - 1u;
  const int N = m.n_vars;
  const int nblocks = (N + 31) >> 5;
  const int total = nblocks * a.n_sweeps;
  if (total <= 0) return true;
  const bool scan32 = m.scan32 != 0;
  const bool big = m.fc_big != 0;
  const double inv = m.fc_inv;
  // (read once: `m` may be the launch's parameter or lie in device memory)
  const uint2* table = m.fc_tab;
  const int4* descs = m.fc_desc;
  const void* further = m.fc_in;
  const int tile_w = tile_words(sh), cap = sh.rows;

  unsigned buf = t0 % (unsigned)sh.bufs, par = (t0 / (unsigned)sh.bufs) & 1u;  // the coming chunk's buffer and phase
  unsigned head = 0;                // log entries written
  unsigned acc_tail = 0, fed = 0;   // the other warps' counters when last looked at
  Sweep S;
  S.betas = a.beta + (long long)r * a.bs_w;
  S.beta_next = S.betas[a.sweep_base * a.bs_s];

  int k = 0, bi = -1;  // sweep and block of gb
  for (int gb = 0; gb < total; gb++)
  {
    bi++;
    if (bi == nblocks)
    {
      bi = 0;
      k++;
    }
    if (bi == 0) next_sweep<FM, INT>(S, a, inv, N, k);
    const int nvalid = min(32, N - (bi << 5));
    const int v = (bi << 5) + lane;
    // this block's chunk
    if (!__all_sync(kFull, mbar_try(&R.bars[buf], par)))
    {
      const bool landed = mbar_wait(&R.bars[buf], par);
      if (!__all_sync(kFull, landed))
      {
        raise_abort(R, a.err);
        return false;
      }
    }
    const uint2* chunk = R.tiles + buf * tile_w;
    buf++;
    if (buf == (unsigned)sh.bufs)
    {
      buf = 0;
      par ^= 1u;
    }
    // the header through shuffles, so that what depends on it is known not to
    // divide the warp: rows, entry rows and further entry rows
    const uint2 head0 = *chunk;
    const unsigned sizes = __shfl_sync(kFull, head0.x, 0);
    const int rows = (int)(sizes & 255u), ents = (int)((sizes >> 8) & 255u), xn = (int)(sizes >> 16);
    const uint2* tile = chunk + lane;
    const int2 own = *(const int2*)(tile + C::kLane);
    const uint4* tent = (const uint4*)(chunk + C::kEnt) + lane;

    const uint32_t word = R.spins[bi];  // the block's spins before its flips
    const uint32_t sv = (word >> lane) & 1u;
    const int deg = own.y;
    const int bnd = deg + 1;  // |field - exact| < bnd units
    const float xmargin = INT ? 0.f : S.fsa * (float)(bnd + 1);

    // ---- the field; term models: the row's contributing incidences (qm)
    int base = FM == PAIR ? own.x : 0;
    unsigned qm = 0;
    // one record of a term model: true when the other literals are all false
    // (COUNTER), or the parity of the other members is odd
    auto term = [&](const uint32_t x) -> bool {
      const uint32_t zz = R.z[x & kTermMask];
      if (big && (x & kBigTerm))
        return FM == COUNTER ? zz == ((sv ^ (x >> 18)) & 1u) : ((zz ^ sv) & 1u) != 0u;
      return FM == COUNTER ? (zz & (x >> 24)) == 0u : (__popc(zz & (x >> 24)) & 1) != 0;
    };
    // a flipped variable's unshared term: its byte after
    auto put = [&](uint32_t x, uint32_t zz, uint32_t spin) {
      uint32_t zn = zz ^ (~(x >> 24) & 255u);
      if (big && (x & kBigTerm)) zn = FM == PARITY ? zz ^ 1u : (((spin ^ (x >> 18)) & 1u) ? zz - 1u : zz + 1u);
      if (!(x & kShared)) R.z[x & kTermMask] = (uint8_t)zn;
    };
    // (rows come in fours; the next four's records are under way meanwhile)
    auto gather = [&](const uint2* t0) {
      unsigned bit = 1u;
      uint2 e[4];
#pragma unroll
      for (int x = 0; x < 4; x++) e[x] = rows ? t0[C::kPitch * x] : make_uint2(0u, 0u);
      for (int i = 4; i <= rows; i += 4)
      {
        uint2 f[4];
        const uint2* t1 = t0 + C::kPitch * (i < rows ? i : 0);
#pragma unroll
        for (int x = 0; x < 4; x++) f[x] = t1[C::kPitch * x];
        if (FM == PAIR)
        {
#pragma unroll
          for (int x = 0; x < 4; x++) base -= (int)R.z[e[x].x] * (int)e[x].y;
        }
        else
        {
          bool t[4];
#pragma unroll
          for (int x = 0; x < 4; x++) t[x] = term(e[x].x);
#pragma unroll
          for (int x = 0; x < 4; x++)
          {
            if (FM == COUNTER) base += t[x] ? (int)e[x].y : 0;
            else base += t[x] ? -(int)e[x].y : (int)e[x].y;
            if (!INT && t[x]) qm |= bit << x;
          }
          bit <<= 4;
        }
#pragma unroll
        for (int x = 0; x < 4; x++) e[x] = f[x];
      }
    };
    if (rows <= cap) gather(tile + C::kRec);
    else gather(table + __ldg(descs + bi).x + C::kRec + lane);
    if (!INT && FM != PAIR) qm &= deg >= 32 ? kFull : ((1u << deg) - 1u);  // (padding records)

    // ---- the in-block terms under a given accept mask, all against the state
    // at the block's start.  Pair models: the member's flip changes the field
    // by c0.  Counter models: the other literals are all false when those of
    // the members before this lane (em) are -- the flipped ones are exactly the
    // true ones (et) -- and those after it or elsewhere were (else em = 0, et =
    // 1: never).  Parities: c0 of the others, and of the flips in em.
    unsigned watch = 0;  // lanes whose flips change this lane's field
    int val[KI];
    unsigned em[KI], et[KI];
    unsigned elog[KI];  // term, position in the row (5 bits), position in the term (3), big
    // further entries (rare): xn of them, in HBM
    const size_t xat = xn ? (size_t)__shfl_sync(kFull, head0.y, 0) + lane : 0;
    const uint2* xpair = (const uint2*)further + xat;
    const uint4* xterm = (const uint4*)further + xat;
    unsigned done = 0;  // the block's flips so far
    // an entry's em and et; D: flips whose bytes are written already
    auto entry = [&](const uint4& e, unsigned D, unsigned& mm, unsigned& mt) {
      const uint32_t zz = R.z[e.x & kTermMask];
      const int n = (e.x & kBigEntry) ? (int)zz : __popc(zz);
      const uint32_t M = e.y & lt, L = (word ^ e.z) & M;  // members before this lane, their true literals
      // the other true literals, as of the block's start
      const int o = n - (int)(sv ^ (e.x >> 31)) - (__popc(M & D) - 2 * __popc(L & D));
      mm = M;
      mt = FM == COUNTER ? L : (unsigned)o & 1u;
      if (FM == COUNTER && o != __popc(L))
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
        val[i] = (int)e.w;
        elog[i] = e.x;
        watch |= e.y & lt;
        if (e.y == 0u) elog[i] = kNoEntry;
      }
    }
    for (int i = 0; i < xn; i++) watch |= FM == PAIR ? __ldg(xpair + 32 * i).x : (__ldg(&xterm[32 * i].y) & lt);

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
    const uint32_t negs = (uint32_t)own.x;  // term models: the row's negated literals

    // ---- rounds: one, unless a lane has to be tried alone
    float2 iv0 = make_float2(0.f, 0.f);
    if (!REPLAY) iv0 = R.ring[(W.taken + (unsigned)lane) & (unsigned)(kRing - 1)];
    int cursor = 0;
    while (true)
    {
      const bool active = lane >= cursor && lane < nvalid;
      const unsigned before = lt & ~((1u << cursor) - 1u);
      // ---- decisions: iterate until no lane's in-block members change
      unsigned A = done, U = 0;
      int g = 0;
      bool rare = false;
      while (true)
      {
        int h = base;
#pragma unroll
        for (int i = 0; i < KI; i++)
        {
          if (FM == PAIR) h += (A & em[i]) ? val[i] : 0;
          else if (FM == COUNTER) h += holds(A, em[i], et[i]) ? val[i] : 0;
          else h += holds(A, em[i], et[i]) ? -val[i] : val[i];
        }
        for (int i = 0; i < xn; i++)
        {
          if (FM == PAIR)
          {
            const uint2 e = __ldg(xpair + 32 * i);
            h += (A & e.x) ? ((word & e.x) ? (int)e.y : -(int)e.y) : 0;
          }
          else
          {
            const uint4 e = __ldg(xterm + 32 * i);
            unsigned mm, mt;
            entry(e, done, mm, mt);
            const bool on = holds(A, mm, mt);
            if (FM == COUNTER) h += on ? (int)e.w : 0;
            else h += on ? -(int)e.w : (int)e.w;
          }
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
          const bool zero = (h & 255) == 0;  // nothing contributes: +0.0
          up = active && !zero && fd > bnd;
          rare = active && !zero && (unsigned)(fd + bnd) <= (unsigned)(2 * bnd);
          x = (float)fd;
        }
        else
        {
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
        if (!INT && FM != PAIR) rare = rare || (acc && deg > 32);  // its masks do not fit the log
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
            res = exact_attempt<FM, REPLAY, INT>(m, v, g, R.spins, R.z, rs, W.key, S.ctr0 + (unsigned long long)v,
                                                 S.beta, &dE);
          res = __shfl_sync(kFull, res, f);
          exact = true;
          F = (res & 1u) << f;
          if (REPLAY) W.taken += res >> 1;
          cursor = f + 1;
        }
        last = cursor >= nvalid;
      }
      const bool mine = ((F >> lane) & 1u) != 0u;
      const unsigned at = (head + (unsigned)__popc(F & lt)) & (unsigned)(kLog - 1);
      const unsigned all = done | F;
      if (FM == PAIR)
      {
        if (!INT && mine) ((uint32_t*)R.log)[at] = (uint32_t)v;
        if (mine) R.z[v] = (uint8_t)(sv ^ 1u);
      }
      else if (F)
      {
        // ---- the flips' log masks and term bytes.  In-block terms: their bits
        // under the final mask (an exact attempt's entry has no masks).
        unsigned lm = qm;
        auto log_bit = [&](unsigned x, bool on) {
          if (x == kNoEntry) return;
          const uint32_t bit = 1u << ((x >> 18) & 31u);
          lm = on ? lm | bit : lm & ~bit;
        };
        if (!INT)
        {
#pragma unroll
          for (int i = 0; i < KI; i++) log_bit(elog[i], holds(A, em[i], et[i]));
          for (int i = 0; i < xn && !exact; i++)
          {
            const uint4 e = __ldg(xterm + 32 * i);
            unsigned mm, mt;
            entry(e, done, mm, mt);
            if (e.y) log_bit(e.x, holds(A, mm, mt));
          }
          __syncwarp();  // the bytes have been read
        }
        // Terms of one member in the block: plain stores, the byte is this
        // block's alone.  The warp over the flips' records, sixteen lanes to a
        // flip, eight flips' loads under way at a time.
        auto flips = [&](const uint2* t0) {
          const int half = lane >> 4, sub = lane & 15;
          unsigned fl = F;
          while (fl)
          {
            uint32_t x[4], zz[4];
            int jj[4];
#pragma unroll
            for (int i = 0; i < 4; i++)
            {
              const int j0 = fl ? __ffs(fl) - 1 : -1;
              fl &= fl - 1u;
              const int j1 = fl ? __ffs(fl) - 1 : -1;
              fl &= fl - 1u;
              jj[i] = half ? j1 : j0;
            }
#pragma unroll
            for (int i = 0; i < 4; i++) x[i] = jj[i] >= 0 && sub < rows ? t0[C::kPitch * sub + (jj[i] - lane)].x : kShared;
#pragma unroll
            for (int i = 0; i < 4; i++) zz[i] = R.z[x[i] & kTermMask];
#pragma unroll
            for (int i = 0; i < 4; i++) put(x[i], zz[i], (word >> (jj[i] & 31)) & 1u);
            for (int at = 16 + sub; at < rows; at += 16)
            {
#pragma unroll
              for (int i = 0; i < 4; i++) x[i] = jj[i] >= 0 ? t0[C::kPitch * at + (jj[i] - lane)].x : kShared;
#pragma unroll
              for (int i = 0; i < 4; i++) zz[i] = R.z[x[i] & kTermMask];
#pragma unroll
              for (int i = 0; i < 4; i++) put(x[i], zz[i], (word >> (jj[i] & 31)) & 1u);
            }
          }
        };
        if (rows <= cap) flips(tile + C::kRec);
        else flips(table + __ldg(descs + bi).x + C::kRec + lane);
        // Terms of several: every flip changes its own bit (or the count by
        // one), in any order.
#pragma unroll
        for (int i = 0; i < KI; i++)
          if (i < ents && mine && elog[i] != kNoEntry) flip_shared<FM>(R.z, elog[i], sv);
        for (int i = 0; i < xn; i++)
        {
          const uint4 e = __ldg(xterm + 32 * i);
          if (mine && e.y) flip_shared<FM>(R.z, e.x, sv);
        }
        if (!INT && mine)
        {
          uint4 ent;
          ent.x = (unsigned)v | ((unsigned)deg << 16) | (exact ? kExactF : 0u);
          const unsigned long long bits = (unsigned long long)__double_as_longlong(dE);
          // COUNTER: the sign is the literal; PARITY: the term's bit, the
          // other members' parity and the own spin
          ent.y = exact ? (unsigned)bits : lm;
          ent.z = exact ? (unsigned)(bits >> 32) : (FM == COUNTER ? (sv ? ~negs : negs) : (sv ? ~lm : lm));
          ent.w = 0u;
          R.log[at] = ent;
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
    if (!REPLAY) W.taken += 32u;
    W.natt += (unsigned)nvalid;
    publish(R, (unsigned)gb + 1u, head, W.taken);
    if (REPLAY && (gb & 0xFFFF) == 0xFFFF)
    {
      // stream positions are 32-bit: move their origin along
      W.rs = stream_state(R, W);
      W.raw0 = W.taken ? R.raw[(W.taken - 1u) & (unsigned)(kRing - 1)] : 0u;
    }
  }
  return true;
}

// The running cost over n flips (lane i < n: the i-th difference d) as a prefix
// sum of whole numbers (ordered_sum.cuh).  False (nothing changed): a difference
// for which that does not do -- the caller adds one by one.
__device__ __forceinline__ bool cost_prefix(double d, int n, double& cost, long long& klow, double& low, int& lowpos)
{
  const int lane = threadIdx.x & 31;
  int ce;
  const long long C = osum::scaled(cost, ce);
  long long D = 0;
  bool ok = ce != 0 && ce != 0x7FF;
  if (ok && lane < n) ok = osum::step_of(d, ce, D);
  const long long P = C + osum::prefix(D);
  if (!__all_sync(kFull, ok && osum::inside(C, P))) return false;
  long long mn = P;  // (lanes past n repeat the last prefix)
#pragma unroll
  for (int s = 16; s; s >>= 1) mn = min(mn, __shfl_xor_sync(kFull, mn, s));
  const double vmin = osum::unscaled(mn, ce);
  const long long km = order_key(vmin);
  if (km < klow)
  {
    klow = km;
    low = vmin;
    lowpos = __ffs(__ballot_sync(kFull, P == mn)) - 1;
  }
  cost = osum::unscaled(__shfl_sync(kFull, P, 31), ce);
  return true;
}

// ---------------------------------------------------------------------------
// The accountant (FP64 models): running cost, lowest cost and lowest state
// from the log.
// ---------------------------------------------------------------------------
template <int FM>
__device__ __noinline__ bool account(const SweepArgs& a, const DevModel& m, const Region R, double& cost,
                                        double& low, uint32_t* g_lsp)
{
  constexpr int kLog = FM == PAIR ? kLogBytes / 4 : kLogBytes / 16;
  const int lane = threadIdx.x & 31;
  const int nw = a.p.nw;
  const int* row = m.row;
  const double* coef = m.coef;
  const int* other = m.other;
  unsigned tail = 0;
  long long klow = order_key(low);
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
      int v = 0;
      double d = 0.0;
      if (FM == PAIR)
      {
        // Flips of one sweep, in index order: a neighbour below the flip has
        // its spin after the batch, one above it its spin before.
        uint32_t* after = R.aspins + nw + 4;
        if (lane < n) v = (int)((const uint32_t*)R.log)[(tail + (unsigned)lane) & (unsigned)(kLog - 1)];
        const int prev = __shfl_up_sync(kFull, v, 1);
        const unsigned wrap = __ballot_sync(kFull, lane > 0 && lane < n && v <= prev);
        if (wrap) n = __ffs(wrap) - 1;
        if (lane < n) atomicXor(after + (v >> 5), 1u << (v & 31));
        __syncwarp();
        if (lane < n)
        {
          const uint32_t sv = spin_of(R.aspins, v);
          const int q1 = __ldg(row + v + 1);
          for (int q = __ldg(row + v); q < q1; q += 8)
          {
            // eight loads in flight ahead of the dependent adds
            double c[8];
            int u[8];
#pragma unroll
            for (int i = 0; i < 8; i++)
            {
              u[i] = q + i < q1 ? __ldg(other + q + i) : -1;
              c[i] = q + i < q1 ? __ldg(coef + q + i) : 0.0;
            }
#pragma unroll
            for (int i = 0; i < 8; i++)
            {
              const uint32_t su = u[i] < 0 ? 0u : spin_of(u[i] < v ? after : R.aspins, u[i]);
              if (sv ^ su) c[i] = -c[i];
            }
#pragma unroll
            for (int i = 0; i < 8; i++)
              if (q + i < q1) d = __dadd_rn(d, c[i]);
          }
          d = neg2x(d);
        }
      }
      else if (lane < n)
      {
        const uint4 ent = R.log[(tail + (unsigned)lane) & (unsigned)(kLog - 1)];
        v = (int)(ent.x & 0x7FFFu);
        const int deg = (int)((ent.x >> 16) & 255u);
        if (ent.x & kExactF)
          d = __longlong_as_double((long long)((unsigned long long)ent.y | ((unsigned long long)ent.z << 32)));
        else d = dE_from_masks<FM>(coef + __ldg(row + v), deg, ent.y, ent.z);
      }
      __syncwarp();
      tail += (unsigned)n;
      if (lane == 0) st_release(R.tail, tail);
      // running cost in flip order (markov/walker.h:225) and the first
      // strict improvement of the lowest (markov/walker.h:269-280)
      int lowpos = -1;
      if (!cost_prefix(d, n, cost, klow, low, lowpos))
      {
        double dn = __shfl_sync(kFull, d, 0);
        for (int i = 0; i < n; i++)
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
      // the accountant's spins, and the lowest state at lowpos
      if (lane < n && lane <= lowpos) atomicXor(R.aspins + (v >> 5), 1u << (v & 31));
      __syncwarp();
      if (lowpos >= 0)
      {
        for (int q = lane; q < nw; q += 32) g_lsp[q] = R.aspins[q];
        __syncwarp();
      }
      if (lane < n && lane > lowpos) atomicXor(R.aspins + (v >> 5), 1u << (v & 31));
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
  unsigned char* base = smem + kTable + (size_t)ws * region_bytes(sh, INT);
  const Region R = carve<INT>(base, sh);
  const int bar_id = 1 + ws;
  const int me = role * 32 + lane, nme = kRoles * 32;  // thread of the walker
  // (the feeder's own barriers; the first walker_sync below shows them to the decider)
  if (role == 1 && lane == 0)
    for (int i = 0; i < kBufs; i++) mbar_init(&R.bars[i]);
  uint64_t rs = (REPLAY && !queued) ? a.rng[w] : 0;
  unsigned t0 = 0;  // chunks of the walkers before this one

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
    const int slot = a.slot_of ? a.slot_of[r] : r;
    uint32_t* g_spins = a.p.spins + (size_t)slot * a.p.nw;
    uint8_t* g_ts = a.p.tstate + (size_t)slot * a.p.mp;
    const int zwords = FM == PAIR ? 0 : (m.n_terms + 15) >> 4;  // 16-byte words
    if (queued && REPLAY) rs = a.rng[r];
    if (decider && lane == 0)
    {
      *R.head = 0u;
      *R.tail = 0u;
      *R.done = 0u;
      *R.abort = 0u;
      *R.made = 0u;
      *R.used = 0u;
      *R.blocks = 0u;
    }
    copy16((uint4*)R.spins, (const uint4*)g_spins, a.p.nw >> 2, me, nme);
    if (me < 4) R.spins[a.p.nw + me] = 0u;
    if (!INT) copy16((uint4*)R.aspins, (const uint4*)g_spins, a.p.nw >> 2, me, nme);
    if (!INT && FM == PAIR) copy16((uint4*)(R.aspins + a.p.nw + 4), (const uint4*)g_spins, a.p.nw >> 2, me, nme);
    // term bytes: as the last launch left them, or from the spins
    if (FM != PAIR && a.terms_valid) copy16((uint4*)R.z, (const uint4*)g_ts, zwords, me, nme);
    walker_sync<INT>(bar_id);
    if (FM != PAIR && !a.terms_valid)
    {
      for (int t = me; t < m.n_terms; t += nme) R.z[t] = term_byte<FM>(m, t, R.spins);
      walker_sync<INT>(bar_id);
    }
    if (FM == PAIR)
    {
      for (int v = me; v < ((N + 31) & ~31); v += nme) R.z[v] = (uint8_t)spin_of(R.spins, v);
      walker_sync<INT>(bar_id);
    }

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
      const bool ok = decide_sweeps<FM, REPLAY, INT>(a, m, R, sh, r, t0, W, g_lsp);
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
      feed<FM, REPLAY>(R, s_scr, m.fc_desc, m.fc_tab, tile_words(sh), sh.rows, sh.bufs, (N + 31) >> 5,
                       ((N + 31) >> 5) * a.n_sweeps, t0, rs, key,
                       (unsigned long long)a.sweep_base * (unsigned long long)N, N, a.err);
      walker_sync<INT>(bar_id);
    }
    else
    {
      double cost = a.p.cost[slot], low = a.p.lowest[r];
      const bool ok = account<FM>(a, m, R, cost, low, g_lsp);
      walker_sync<INT>(bar_id);
      if (ok && !*(volatile unsigned*)R.abort && lane == 0)
      {
        a.p.cost[slot] = cost;
        if (a.p.lowtag && low < a.p.lowest[r]) a.p.lowtag[r] = a.tag;
        a.p.lowest[r] = low;
      }
    }
    if (*(volatile unsigned*)R.abort) return;
    t0 = (t0 + (unsigned)(((N + 31) >> 5) * a.n_sweeps)) % (unsigned)(2 * sh.bufs);  // buffer and phase
    copy16((uint4*)g_spins, (const uint4*)R.spins, a.p.nw >> 2, me, nme);
    if (FM != PAIR && !queued) copy16((uint4*)g_ts, (const uint4*)R.z, zwords, me, nme);
    walker_sync<INT>(bar_id);  // the region is reused by the next walker
    if (!queued)
    {
      r += a.n_streams;
      // a stream that serves several walkers goes on where the last one ended
      if (REPLAY && r < a.n_walkers)
      {
        if (decider && lane == 0) a.rng[w] = rs;
        __threadfence_block();
        walker_sync<INT>(bar_id);
        rs = *(volatile uint64_t*)(a.rng + w);
      }
    }
  }
  if (REPLAY && !queued && decider && lane == 0) a.rng[w] = rs;
}

template <int FM, bool R, bool I>
static cudaError_t go(const SweepArgs& a, cudaStream_t s, int wpc, const Shape& sh)
{
  auto k = fc_sweep_kernel<FM, R, I>;
  const int smem = kTable + wpc * region_bytes(sh, I);
  const int threads = (I ? 64 : 96) * wpc;
  static std::atomic<int> configured{48 * 1024};
  if (smem > configured.load())
  {
    cudaError_t e = cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, kMaxSmem);
    if (e != cudaSuccess) return e;
    configured = kMaxSmem;
  }
  int blocks = (a.n_streams + wpc - 1) / wpc;
  if (a.queue)
  {
    // persistent: as many blocks as stay resident, the queue feeds them
    int per_sm = 0;
    cudaError_t e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k, threads, smem);
    if (e != cudaSuccess) return e;
    blocks = std::max(1, std::min((a.n_walkers + wpc - 1) / wpc, std::max(1, per_sm) * kSms));
  }
  if (blocks > 0) k<<<blocks, threads, smem, s>>>(a, wpc, sh);
  return cudaGetLastError();
}

template <int FM>
static cudaError_t go_fm(const SweepArgs& a, cudaStream_t s, int wpc, const Shape& sh)
{
  const bool I = a.m.int_mode != 0;
  if (a.replay) return I ? go<FM, true, true>(a, s, wpc, sh) : go<FM, true, false>(a, s, wpc, sh);
  return I ? go<FM, false, true>(a, s, wpc, sh) : go<FM, false, false>(a, s, wpc, sh);
}

// a walker's region for a model in a population of these strides
static Shape shape_of(const DevModel& m, int nw, int mp)
{
  Shape s;
  s.pair = m.flavor == F_PARITY && m.pair_only;
  s.nw = nw;
  s.mp = s.pair ? nw * 32 : mp;
  s.rows = std::min(kMaxRows, m.fc_rows);
  s.bufs = kBufs;
  // a state that leaves less room: smaller tiles (larger blocks read HBM)
  while (s.rows > 4 && kTable + region_bytes(s, m.int_mode != 0) > kMaxSmem) s.rows -= 4;
  return s;
}
}  // namespace fc

bool fc_fits(const DevModel& m, int nw, int mp)
{
  if (!m.fc_desc || m.sweep_size != m.n_vars || m.n_vars <= 0) return false;
  if (!(m.flavor == F_PARITY || m.flavor == F_COUNTER)) return false;
  return fc::kTable + fc::region_bytes(fc::shape_of(m, nw, mp), m.int_mode != 0) <= fc::kMaxSmem;
}

cudaError_t launch_fc_sweep(const SweepArgs& a, cudaStream_t s, int wpb)
{
  if (!fc_fits(a.m, a.p.nw, a.p.mp)) return cudaErrorInvalidValue;
  fc::Shape sh = fc::shape_of(a.m, a.p.nw, a.p.mp);
  const bool I = a.m.int_mode != 0;
  auto fit = [&](int bufs) {
    sh.bufs = bufs;
    return std::min(I ? 8 : 4, (fc::kMaxSmem - fc::kTable) / fc::region_bytes(sh, I));
  };
  // Three chunk buffers where four would cost a wave of blocks: 512 tempering
  // walkers of a 4096-variable PUBO, 100 sweeps: 61.3 ms at three walkers a block
  // with four buffers, 43.7 at four with three.  Otherwise four: the third covers
  // the copy's latency only just.
  const int w3 = fit(fc::kBufs - 1), w4 = fit(fc::kBufs);
  auto waves = [&](int w) { return (a.n_streams + w * fc::kSms - 1) / (w * fc::kSms); };
  const int wmax = waves(w3) < waves(w4) ? w3 : w4;
  if (wmax != w4) sh.bufs = fc::kBufs - 1;
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
