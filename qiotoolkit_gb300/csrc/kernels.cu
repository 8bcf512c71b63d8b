// kernels.cu -- sm_103a kernels of the Metropolis hot path.
//
// The ordered sweep of the reference (markov/walker.h:143-153) is a strictly
// sequential chain: attempt i reads the state left by attempt i-1.  One warp
// owns one walker and evaluates a WINDOW of 32 consecutive variables at once
// (lane l takes variable i+l), each lane summing its own cost difference in
// the reference's term order (bit-identical FP64).  Decisions are then
// committed in lane order up to the first lane whose terms intersect an
// earlier accepted flip in the window (its difference was computed on a
// stale state) or that needs the Metropolis redraw path; the next window
// starts there.  Replay streams are PCG32 positions: lane l's draw is the
// stream advanced by the number of uphill lanes before it (an LCG jump), so
// the committed prefix consumes exactly the draws the sequential chain would.
// The result is the reference's trajectory, evaluated up to 32-wide.
#include <cstdio>
#include <mutex>
#include <type_traits>

#include "exp_cr.cuh"
#include "ordered_sum.cuh"
#include "qio_internal.h"

namespace qio
{
static const unsigned kFull = 0xffffffffu;
static const unsigned long long kMult = 6364136223846793005ULL;
static const unsigned long long kInc = 1442695040888963407ULL;
static const unsigned long long kGamma = 0x9E3779B97F4A7C15ULL;
static const unsigned long long kInitCounterBase = 1ULL << 62;

// ln table (utils/utils.cc:12-32, computed on the host with the C library's
// log) and LCG jump tables: k steps (k = 0..64) and 2^k steps.
__constant__ double c_ln[1024];
__constant__ unsigned long long c_jA[65], c_jC[65];
__constant__ unsigned long long c_pA[64], c_pC[64];

__device__ __forceinline__ uint32_t pcg_out(uint64_t old)
{
  uint32_t xs = (uint32_t)(((old >> 18u) ^ old) >> 27u);
  uint32_t rot = (uint32_t)(old >> 59u);
  return __funnelshift_r(xs, xs, rot);
}

__device__ __forceinline__ uint64_t jump_any(uint64_t s, unsigned long long k)
{
  for (int b = 0; k; b++, k >>= 1)
    if (k & 1ULL) s = c_pA[b] * s + c_pC[b];
  return s;
}

__device__ __forceinline__ uint64_t mix64(uint64_t z)
{
  z = (z ^ (z >> 30)) * 0xBF58476D1CE4E5B9ULL;
  z = (z ^ (z >> 27)) * 0x94D049BB133111EBULL;
  return z ^ (z >> 31);
}
__device__ __forceinline__ uint64_t counter_key(uint32_t seed, uint64_t stream)
{
  return mix64(((uint64_t)seed << 32) ^ mix64(stream + kGamma));
}
__device__ __forceinline__ uint64_t counter_draw(uint64_t key, uint64_t ctr)
{
  return mix64(key + ctr * kGamma);
}

// libstdc++ generate_canonical<double,53> over a 32-bit engine: two draws,
// sum = a + b * 2^32 rounded once, divided by 2^64, clamped below 1.
__device__ __forceinline__ double canonical(uint32_t a, uint32_t b)
{
  double s = __dadd_rn((double)a, __dmul_rn((double)b, 4294967296.0));
  double u = __dmul_rn(s, 5.421010862427522170037e-20);  // 2^-64
  if (u >= 1.0) u = 0.99999999999999988898;              // nextafter(1, 0)
  return u;
}

// value < -dE * beta with value interpolated in ln[row] at bucket r & 255,
// distance (r >> 8) / 16777214 (markov/metropolis.h:96-103).  Explicit _rn
// intrinsics keep the reference's rounding (no fused multiply-add).
__device__ __forceinline__ bool lut_less(const double* ln, uint32_t r, int row,
                                         double thr)
{
  int b = (int)(r & 255u);
  double y0 = ln[row * 256 + b - 1];
  double y1 = ln[row * 256 + b];
  // (r >> 8) / 16777214 correctly rounded: reciprocal product corrected by
  // one fused residual step (Markstein); equal to the IEEE quotient for all
  // 2^24 inputs (checked exhaustively by the oracle's test).
  const double x = (double)(r >> 8);
  const double inv = 5.9604648328104515e-08;  // RN(1 / 16777214)
  const double d0 = __dmul_rn(x, inv);
  const double dist = __fma_rn(__fma_rn(-d0, 16777214.0, x), inv, d0);
  double value = __dadd_rn(y0, __dmul_rn(dist, __dsub_rn(y1, y0)));
  return value < thr;
}

// Metropolis::accept (markov/metropolis.h:64-104) for an uphill move with
// the draws supplied by `draw(k)`; `used` receives the draw count.
template <class F>
__device__ __forceinline__ bool metropolis_uphill(double thr, const double* ln,
                                                  F draw, int& used)
{
  int row = -1, b = 0;
  uint32_t cur = 0;
  used = 0;
  while (b == 0)
  {
    if (row < 3)
    {
      cur = draw(used);
      used++;
      b = (int)(cur & 255u);
      row++;
    }
    else
      return true;
  }
  return lut_less(ln, cur, row, thr);
}

__device__ __forceinline__ uint32_t spin_of(const uint32_t* spins, int v)
{
  return (spins[v >> 5] >> (v & 31)) & 1u;
}

// Four terms of a lane, t0 + 32 u + lane: their state bytes (written to ts unless
// it is null), and their values; the loads of the four overlap.
template <int FL, bool INT>
__device__ __forceinline__ void four_terms(const DevModel& m, const uint32_t* spins, uint8_t* ts, int t0, int lane,
                                           double (&v)[4], long long& isum, bool (&skip)[4])
{
  constexpr int U = 4;
  constexpr bool PAR = FL == F_PARITY || FL == F_PLAIN_ISING;
  const int M = m.n_terms;
  int b[U], e[U];
  uint32_t acc[U];
#pragma unroll
  for (int u = 0; u < U; u++)
  {
    const int t = t0 + u * 32 + lane;
    b[u] = t < M ? __ldg(m.trow + t) : 0;
    e[u] = t < M ? __ldg(m.trow + t + 1) : 0;
    acc[u] = 0;
  }
  // the members of the four terms, position by position
  for (int k = 0;; k++)
  {
    bool more = false;
#pragma unroll
    for (int u = 0; u < U; u++)
      if (b[u] + k < e[u])
      {
        const uint32_t x = __ldg(m.tvar + b[u] + k);
        const uint32_t sx = spin_of(spins, (int)(x & ~kNegBit));
        if (PAR) acc[u] ^= sx;
        else acc[u] += sx ^ (x >> 31);
        more = more || b[u] + k + 1 < e[u];
      }
    if (!more) break;
  }
#pragma unroll
  for (int u = 0; u < U; u++)
  {
    const int t = t0 + u * 32 + lane;
    v[u] = 0.0;
    skip[u] = true;
    if (t >= M) continue;
    if (ts && (FL == F_PARITY || FL == F_COUNTER)) ts[t] = (uint8_t)acc[u];
    // parity: the term's sign; counter: the term counts when no literal is true
    skip[u] = PAR ? false : acc[u] != 0;
    if (INT) isum += skip[u] ? 0 : (PAR && acc[u] ? -(long long)m.tcost_i[t] : (long long)m.tcost_i[t]);
    else v[u] = skip[u] ? 0.0 : (PAR && acc[u] ? -m.tcost[t] : m.tcost[t]);
  }
}

// Term state bytes (written to ts unless it is null) and the cost of a state
// by one warp.  FP64 values are added in term order (bit-identical to a loop),
// integers per lane and reduced.
template <int FL, bool INT>
__device__ void warp_terms_cost(const DevModel& m, const uint32_t* spins, uint8_t* ts, int lane,
                                double& cost, long long& icost)
{
  double c = 0.0;
  long long ic = 0;
  for (int t0 = 0; t0 < m.n_terms; t0 += 128)
  {
    double v[4];
    bool skip[4];
    four_terms<FL, INT>(m, spins, ts, t0, lane, v, ic, skip);
    if (!INT)
    {
#pragma unroll
      for (int u = 0; u < 4; u++) osum::add_lanes(v[u], __ballot_sync(kFull, !skip[u]), c);
    }
  }
  if (INT)
  {
#pragma unroll
    for (int d = 16; d; d >>= 1) ic += __shfl_xor_sync(kFull, ic, d);
  }
  cost = c;
  icost = ic;
}

// The same by a block of four warps; the result on thread 0.  A warp alone
// waits for three dependent loads a term (1.5 M cycles for 20000 terms), so
// integer models spread the terms over all warps, and FP64 models have three
// warps evaluate 384 terms into shared memory while the first adds up the 384
// before them.  Initialising 512 walkers of 20000 FP64 terms 794 to 531 us, 1024
// of 32768 integer terms 909 to 240 us.
struct CostBuf
{
  double v[2][384];
  unsigned keep[2][12];
};
template <int FL, bool INT>
__device__ void block_terms_cost(const DevModel& m, const uint32_t* spins, uint8_t* ts, CostBuf& buf, double& cost,
                                 long long& icost)
{
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  double c = 0.0;
  long long ic = 0;
  double v[4];
  bool skip[4];
  if (INT)
  {
    for (int t0 = warp * 128; t0 < m.n_terms; t0 += 512) four_terms<FL, INT>(m, spins, ts, t0, lane, v, ic, skip);
#pragma unroll
    for (int d = 16; d; d >>= 1) ic += __shfl_xor_sync(kFull, ic, d);
    if (lane == 0) buf.v[0][warp] = __longlong_as_double(ic);
    __syncthreads();
    ic = 0;
    for (int i = 0; i < 4; i++) ic += __double_as_longlong(buf.v[0][i]);
  }
  else
  {
    const int chunks = (m.n_terms + 383) / 384;
    for (int k = 0; k <= chunks; k++)
    {
      if (warp > 0 && k < chunks)
      {
        four_terms<FL, INT>(m, spins, ts, k * 384 + (warp - 1) * 128, lane, v, ic, skip);
#pragma unroll
        for (int u = 0; u < 4; u++)
        {
          const int b = (warp - 1) * 4 + u;
          buf.v[k & 1][b * 32 + lane] = v[u];
          const unsigned keep = __ballot_sync(kFull, !skip[u]);
          if (lane == 0) buf.keep[k & 1][b] = keep;
        }
      }
      if (warp == 0 && k > 0)
        for (int b = 0; b < 12; b++) osum::add_lanes(buf.v[(k - 1) & 1][b * 32 + lane], buf.keep[(k - 1) & 1][b], c);
      __syncthreads();
    }
  }
  cost = c;
  icost = ic;
}

// Term state byte from spins: parity (Ising) or true-literal count.
template <int FL>
__device__ __forceinline__ uint8_t term_state(const DevModel& m,
                                              const uint32_t* spins, int t)
{
  int b = m.trow[t], e = m.trow[t + 1];
  uint32_t acc = 0;
  for (int k = b; k < e; k++)
  {
    uint32_t x = m.tvar[k];
    uint32_t s = spin_of(spins, (int)(x & ~kNegBit));
    if (FL == F_PARITY) acc ^= s;
    else acc += s ^ (x >> 31);
  }
  return (uint8_t)acc;
}

// ---------------------------------------------------------------------------
// init: random (or given) state, term cache, cost, lowest = current.
// Walker::init (markov/walker.h:50-58) with get_random_spin_state /
// get_random_binary_state (model/ising.h:23-41, model/pubo.h:16-34) or the
// MaxSat per-variable uniform() < 0.5 (model/max_sat.h:144-150).
// ---------------------------------------------------------------------------
// WPW: warps per walker, 4 (a block) or 1 (four walkers a block).
template <int FL, bool INT, int WPW>
__global__ void __launch_bounds__(128) init_kernel(InitArgs a)
{
  const int lane = threadIdx.x & 31, tid = WPW == 1 ? lane : (int)threadIdx.x;  // thread of the walker
  constexpr int T = 32 * WPW;
  const int w = WPW == 1 ? (int)((blockIdx.x * blockDim.x + threadIdx.x) >> 5) : (int)blockIdx.x;
  if (w >= a.n_walkers) return;
  const DevModel& m = a.m;
  const int N = m.n_vars;
  const int nwd = (N + 31) >> 5;
  const int slot = a.slot_of ? a.slot_of[w] : w;
  uint32_t* spins = a.p.spins + (size_t)slot * a.p.nw;
  uint8_t* ts = a.p.tstate + (size_t)slot * a.p.mp;
  uint32_t* lsp = a.p.lspins + (size_t)w * a.p.nw;
  // a.replay: 0 counter, 1 PCG replay (one draw per 32 variables);
  // 2 PCG replay / 3 counter with one uniform() per variable (MaxSat)
  const bool var_uniform = (a.replay == 2 || a.replay == 3);
  const bool replay = (a.replay == 1 || a.replay == 2);
  uint64_t key = 0;
  if (!replay)
    key = counter_key(a.seed + (uint32_t)(w / a.key_div),
                      a.key_base + (unsigned long long)(w % a.key_div));
  uint64_t rs = replay ? a.rng[w] : 0;
  if (var_uniform && !a.given)
  {
    // MaxSat: a word per warp, a variable per lane
    for (int q = tid >> 5; q < nwd; q += WPW)
    {
      const int v = q * 32 + lane;
      bool bit = false;
      if (v < N)
      {
        if (replay)
        {
          uint64_t s0 = jump_any(rs, 2ULL * (unsigned long long)v);
          uint32_t d0 = pcg_out(s0);
          uint32_t d1 = pcg_out(s0 * kMult + kInc);
          bit = canonical(d0, d1) < 0.5;
        }
        else
          bit = (counter_draw(key, kInitCounterBase + (unsigned long long)v) >> 63) == 0;
      }
      const unsigned word = __ballot_sync(kFull, bit);
      if (lane == 0) spins[q] = word;
    }
  }
  else
    for (int q = tid; q < nwd; q += T)
    {
      uint32_t word = 0;
      if (a.given)
      {
        for (int b = 0; b < 32; b++)
        {
          int v = q * 32 + b;
          if (v < N && a.given[(size_t)w * N + v]) word |= 1u << b;
        }
      }
      else if (replay) word = pcg_out(jump_any(rs, (unsigned long long)q));
      else word = (uint32_t)counter_draw(key, kInitCounterBase + (unsigned long long)q);
      if (q == nwd - 1 && (N & 31)) word &= (1u << (N & 31)) - 1u;
      spins[q] = word;
    }
  for (int q = nwd + tid; q < a.p.nw; q += T) spins[q] = 0;
  // (and every thread has read the walker's stream)
  if (WPW == 1) __syncwarp();
  else __syncthreads();
  if (replay && tid == 0)
    a.rng[w] = jump_any(rs, var_uniform ? 2ULL * (unsigned long long)N
                                        : (unsigned long long)nwd);
  double cost;
  long long icost;
  if constexpr (WPW == 1) warp_terms_cost<FL, INT>(m, spins, a.skip_terms ? nullptr : ts, lane, cost, icost);
  else
  {
    __shared__ CostBuf buf;
    block_terms_cost<FL, INT>(m, spins, a.skip_terms ? nullptr : ts, buf, cost, icost);
  }
  if (INT) cost = (double)icost;
  for (int q = tid; q < a.p.nw; q += T) lsp[q] = spins[q];
  if (tid == 0)
  {
    a.p.cost[slot] = cost;
    a.p.lowest[w] = cost;
    if (a.p.lowtag) a.p.lowtag[w] = -1;
    if (!a.keep_counters)
    {
      a.p.attempts[w] = 0;
      a.p.accepts[w] = 0;
    }
    a.p.step_att[w] = 0;
    a.p.step_acc[w] = 0;
    if (a.p.windows) a.p.windows[w] = 0;
  }
}

// ---------------------------------------------------------------------------
// Evaluation kernels for the per-state contract.
// ---------------------------------------------------------------------------
template <int FL, bool INT>
__global__ void __launch_bounds__(128) eval_cost_kernel(DevModel m, int n, const uint32_t* spins,
                                 int nw, double* out)
{
  __shared__ CostBuf buf;
  const int w = blockIdx.x;  // a block per state
  double c;
  long long ic;
  block_terms_cost<FL, INT>(m, spins + (size_t)w * nw, nullptr, buf, c, ic);
  if (threadIdx.x == 0) out[w] = INT ? (double)ic : c;
}

// State bytes (nonzero: set) to spin words, a warp per four words: bounded by
// the bytes' way to the device.  1024 states of 4096 variables: the host's loop
// over them took 11 ms, the copy of the bytes and this kernel 0.2.
__global__ void __launch_bounds__(256) pack_states_kernel(const uint8_t* st, long long n, int n_vars, int nw,
                                                          uint32_t* words)
{
  const int lane = threadIdx.x & 31;
  const int groups = (nw + 3) >> 2;  // of four words
  const long long total = n * groups, stride = (long long)gridDim.x * (blockDim.x >> 5);
  for (long long g = (long long)blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5); g < total; g += stride)
  {
    const long long q = g / groups;
    const int w0 = (int)(g - q * groups) * 4;
    const uint8_t* s = st + q * n_vars;
    uint32_t mine = 0;
#pragma unroll
    for (int i = 0; i < 4; i++)
    {
      const int v = (w0 + i) * 32 + lane;
      const unsigned word = __ballot_sync(kFull, v < n_vars && s[v] != 0);
      if (lane == i) mine = word;
    }
    if (lane < 4 && w0 + lane < nw) words[q * nw + w0 + lane] = mine;
  }
}

// calculate_cost_difference for query q: incident terms evaluated in
// parallel, summed in order (model/ising.h:108-117, model/pubo.h:335-367,
// model/pubo.cc:50-73, model/max_sat.h:173-236).
template <int FL, bool INT>
__global__ void eval_diff_kernel(DevModel m, int n, const uint32_t* spins,
                                 int nw, const long long* vars, double* out)
{
  const int lane = threadIdx.x & 31;
  const int w = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  if (w >= n) return;
  const uint32_t* sp = spins + (size_t)w * nw;
  const int v = (int)vars[w];
  const uint32_t sv = spin_of(sp, v);
  const int rb = m.row[v], re = m.row[v + 1];
  double diff = 0.0;
  long long idiff = 0;
  for (int q0 = rb; q0 < re; q0 += 32)
  {
    int q = q0 + lane;
    double val = 0.0;
    long long ival = 0;
    bool skip = true;
    if (q < re)
    {
      uint32_t e = m.inc[q];
      int t = (int)(e & ~kNegBit);
      int tb = m.trow[t], te = m.trow[t + 1];
      if (FL == F_PARITY || FL == F_PLAIN_ISING)
      {
        uint32_t par = 0;
        for (int u = tb; u < te; u++) par ^= spin_of(sp, (int)(m.tvar[u] & ~kNegBit));
        skip = false;
        if (INT) ival = par ? -(long long)m.coef_i[q] : (long long)m.coef_i[q];
        else val = par ? -m.coef[q] : m.coef[q];
      }
      else
      {
        int cnt = 0;
        for (int u = tb; u < te; u++)
        {
          uint32_t x = m.tvar[u];
          cnt += (int)(spin_of(sp, (int)(x & ~kNegBit)) ^ (x >> 31));
        }
        const bool lit = (sv ^ (e >> 31)) != 0;
        if (lit && cnt == 1)
        {
          skip = false;
          if (INT) ival = m.coef_i[q]; else val = m.coef[q];
        }
        else if (!lit && cnt == 0)
        {
          skip = false;
          if (INT) ival = -(long long)m.coef_i[q]; else val = -m.coef[q];
        }
      }
    }
    unsigned keep = __ballot_sync(kFull, !skip);
    while (keep)
    {
      int j = __ffs(keep) - 1;
      keep &= keep - 1;
      if (INT) idiff += __shfl_sync(kFull, ival, j);
      else diff = __dadd_rn(diff, __shfl_sync(kFull, val, j));
    }
  }
  if (lane == 0)
  {
    if (FL == F_PARITY || FL == F_PLAIN_ISING)
      out[w] = INT ? (double)(-2 * idiff) : __dmul_rn(2.0, -diff);
    else
      out[w] = INT ? (double)idiff : diff;
  }
}

// ---------------------------------------------------------------------------
// Tabu search (solver/tabu.h:22-164, markov/tabu_walker.h:14-218), one warp
// per walker.  A tabu sweep prices every variable against the current state
// (lanes take 32 variables at a time, each difference summed in the
// reference's term order), takes the first move that puts the cost below the
// lowest -- then hill-climbs on a copy (accepting differences <= 0, one
// variable after the other) while that improves the lowest -- or else the
// lowest-difference move not on the tabu list.  No random numbers after the
// initial state.
// ---------------------------------------------------------------------------
// FP64 instructions occupy a GB300 sub-partition's FP64 unit for ~64 cycles
// each, so the tabu kernel orders, signs and scales differences with integer
// bit operations where that is exact.
// fkey: unsigned key ordered as the doubles (finite values; -0 keyed as +0,
// as -0 == +0 compares)
__device__ __forceinline__ unsigned long long fkey(double x)
{
  unsigned long long b = (unsigned long long)__double_as_longlong(x);
  if (b == 0x8000000000000000ull) b = 0;
  return (b >> 63) ? ~b : (b | 0x8000000000000000ull);
}
// -2 * x for a normal x by the exponent and sign bits (__dmul_rn otherwise)
__device__ __forceinline__ double times_minus2(double x)
{
  const unsigned long long b = (unsigned long long)__double_as_longlong(x);
  const unsigned e = (unsigned)(b >> 52) & 0x7FFu;
  if (e == 0 || e >= 0x7FEu) return __dmul_rn(2.0, -x);
  return __longlong_as_double((long long)((b + (1ull << 52)) ^ 0x8000000000000000ull));
}

// calculate_cost_difference of variable v by one thread, terms in row order
template <int FL, bool INT>
__device__ double lane_diff(const DevModel& m, const uint32_t* sp, int v)
{
  const uint32_t sv = spin_of(sp, v);
  double diff = 0.0;
  long long idiff = 0;
  if (FL == F_PARITY && m.pair_only)
  {
    // one- or two-member terms: the parity is the spin of v xor that of the
    // other member; four incidences' loads in flight, added in row order
    const int qe = m.row[v + 1];
    for (int q = m.row[v]; q < qe; q += 4)
    {
      int o[4];
      double c[4];
      int ci[4];
#pragma unroll
      for (int u = 0; u < 4; u++)
        if (q + u < qe)
        {
          o[u] = __ldg(m.other + q + u);
          if (INT) ci[u] = __ldg(m.coef_i + q + u);
          else c[u] = __ldg(m.coef + q + u);
        }
#pragma unroll
      for (int u = 0; u < 4; u++)
        if (q + u < qe)
        {
          const uint32_t par = sv ^ (o[u] >= 0 ? spin_of(sp, o[u]) : 0u);
          if (INT) idiff += par ? -(long long)ci[u] : (long long)ci[u];
          else diff = __dadd_rn(diff, par ? -c[u] : c[u]);
        }
    }
    return INT ? (double)(-2 * idiff) : times_minus2(diff);
  }
  for (int q = m.row[v], qe = m.row[v + 1]; q < qe; q++)
  {
    const uint32_t e = m.inc[q];
    const int t = (int)(e & ~kNegBit);
    const int tb = m.trow[t], te = m.trow[t + 1];
    if (FL == F_PARITY || FL == F_PLAIN_ISING)
    {
      uint32_t par = 0;
      for (int u = tb; u < te; u++) par ^= spin_of(sp, (int)(m.tvar[u] & ~kNegBit));
      if (INT) idiff += par ? -(long long)m.coef_i[q] : (long long)m.coef_i[q];
      else diff = __dadd_rn(diff, par ? -m.coef[q] : m.coef[q]);
    }
    else
    {
      int cnt = 0;
      for (int u = tb; u < te; u++)
      {
        const uint32_t x = m.tvar[u];
        cnt += (int)(spin_of(sp, (int)(x & ~kNegBit)) ^ (x >> 31));
      }
      const bool lit = (sv ^ (e >> 31)) != 0;
      if (lit && cnt == 1)
      {
        if (INT) idiff += m.coef_i[q];
        else diff = __dadd_rn(diff, m.coef[q]);
      }
      else if (!lit && cnt == 0)
      {
        if (INT) idiff -= m.coef_i[q];
        else diff = __dadd_rn(diff, -m.coef[q]);
      }
    }
  }
  if (FL == F_PARITY || FL == F_PLAIN_ISING) return INT ? (double)(-2 * idiff) : times_minus2(diff);
  return INT ? (double)idiff : diff;
}

__device__ __forceinline__ void warp_copy(uint32_t* dst, const uint32_t* src, int n, int lane)
{
  for (int q = lane; q < n; q += 32) dst[q] = src[q];
  __syncwarp();
}

// Every walker keeps the cost difference of each of its variables (and its
// hill climber those of the copy) in HBM.  A flip of variable i changes only
// the differences of i and of the members of i's terms; those are summed
// afresh from the spins (term order, as calculate_cost_difference), so a
// cached value always equals a fresh evaluation bit for bit.
template <int FL, bool INT>
__device__ void tabu_refresh(const DevModel& m, const uint32_t* sp, double* df, int i, int lane)
{
  const int rb = m.row[i], re = m.row[i + 1];
  // i itself on the first lane without an incidence of i's row, so its sum
  // runs beside the co-members' instead of after one of them
  if (lane == min(re - rb, 31)) df[i] = lane_diff<FL, INT>(m, sp, i);
  if (FL == F_PARITY && m.pair_only)
  {
    for (int q = rb + lane; q < re; q += 32)
    {
      const int x = __ldg(m.other + q);
      if (x >= 0) df[x] = lane_diff<FL, INT>(m, sp, x);
    }
    __syncwarp();
    return;
  }
  for (int q = rb + lane; q < re; q += 32)
  {
    const int t = (int)(m.inc[q] & ~kNegBit);
    for (int u = m.trow[t], ue = m.trow[t + 1]; u < ue; u++)
    {
      const int x = (int)(m.tvar[u] & ~kNegBit);
      if (x != i) df[x] = lane_diff<FL, INT>(m, sp, x);
    }
  }
  __syncwarp();
}

template <int FL, bool INT>
__global__ void __launch_bounds__(128) tabu_kernel(TabuArgs a)
{
  const int lane = threadIdx.x & 31;
  const int w = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  if (w >= a.n_walkers) return;  // whole warps leave together
  const DevModel& m = a.m;
  // N strides the per-walker arrays; SW variables are swept (get_sweep_size:
  // N, or 1 for MaxSat unless the full sweep is asked for)
  const int N = m.n_vars, SW = m.sweep_size, nw = a.p.nw;
  uint32_t* sp = a.p.spins + (size_t)w * nw;
  uint32_t* ls = a.p.lspins + (size_t)w * nw;
  uint32_t* hs = a.hc + (size_t)w * nw;
  uint32_t* hl = a.hc_low + (size_t)w * nw;
  unsigned long long* tb = a.tabu + (size_t)w * N;
  double* df = a.diff + (size_t)w * N;
  double* hd = a.hdiff + (size_t)w * N;
  TabuState S = a.st[w];
  double cost = a.p.cost[w], low = a.p.lowest[w];
  unsigned long long att = 0, acc = 0;
  const unsigned long long tenure = a.tenures ? a.tenures[w] : a.tenure;
  if (!S.ready)
  {
    for (int v = lane; v < N; v += 32) df[v] = lane_diff<FL, INT>(m, sp, v);
    S.ready = 1;
    __syncwarp();
  }

  // HillClimbingWalker::make_sweep on the copy, then local_search_sweep's
  // bookkeeping (markov/tabu_walker.h:183-207).  The ordered sweep runs in
  // windows of 32 variables read at once: the lanes before the first
  // accepted one (d <= 0) hold what the sequential sweep would have seen and
  // were rejected; the window restarts after each accepted flip.
  auto local_sweep = [&]() {
    const double prev = S.hc_low;
    int v0 = 0;
    while (v0 < SW)
    {
      const int v = v0 + lane;
      const bool ok = v < SW;
      const double d = ok ? hd[v] : 0.0;
      // d <= 0 for a non-NaN double: its bits as a signed integer are <= 0
      const unsigned take = __ballot_sync(kFull, ok && __double_as_longlong(d) <= 0);
      if (!take)
      {
        att += (unsigned long long)min(32, SW - v0);
        v0 += 32;
        continue;
      }
      const int j = __ffs(take) - 1;
      const double dj = __shfl_sync(kFull, d, j);
      const int i = v0 + j;
      att += (unsigned long long)(j + 1);
      if (lane == 0) hs[i >> 5] ^= 1u << (i & 31);
      __syncwarp();
      acc++;
      S.hc_cost = __dadd_rn(S.hc_cost, dj);
      if (S.hc_cost < S.hc_low)
      {
        S.hc_low = S.hc_cost;
        warp_copy(hl, hs, nw, lane);
      }
      tabu_refresh<FL, INT>(m, hs, hd, i, lane);
      v0 = i + 1;
    }
    if (S.hc_low < prev)
    {
      low = S.hc_low;
      warp_copy(ls, hl, nw, lane);
    }
    else
      S.local = 0;
  };

  for (int step = 0; step < a.n_steps; step++)
  {
    if (S.local)
    {
      local_sweep();
      continue;
    }
    // the scan, markov/tabu_walker.h:68-127: 128 variables per round (four
    // loads in flight per lane), each lane keeping its own first-lowest
    // candidate off the tabu list.  fl(cost + d) < low is monotone in d, so
    // with t = fl(low - cost) and e = 2^-48 max(|cost|, |low|, |t|) every
    // d < fl(t - e) is taken and every d > fl(t + e) is not (the rounding
    // errors are below e / 16); only differences in between are added in FP64.
    bool taken = false;
    double bd = 0.0;
    unsigned long long bk = ~0ull;
    int bv = INT_MAX;
    const unsigned long long it = S.iter;
    const double t = __dadd_rn(low, -cost);
    const double e = fmax(__dmul_rn(fmax(fmax(fabs(cost), fabs(low)), fabs(t)), 0x1p-48), 0x1p-1000);
    const unsigned long long klo = fkey(__dadd_rn(t, -e)), khi = fkey(__dadd_rn(t, e));
    for (int c0 = 0; c0 < SW && !taken; c0 += 128)
    {
      double d[4];
      unsigned long long x[4];
#pragma unroll
      for (int u = 0; u < 4; u++)
      {
        const int v = c0 + 32 * u + lane;
        d[u] = v < SW ? df[v] : 0.0;
        x[u] = v < SW ? tb[v] : 0ull;
      }
#pragma unroll
      for (int u = 0; u < 4; u++)
      {
        const int v = c0 + 32 * u + lane;
        const bool ok = v < SW;
        const unsigned long long k = fkey(d[u]);
        unsigned take = __ballot_sync(kFull, ok && k < klo);
        const unsigned near = __ballot_sync(kFull, ok && k >= klo && k <= khi);
        if (near) take |= __ballot_sync(kFull, ((near >> lane) & 1) && __dadd_rn(cost, d[u]) < low);
        if (take)
        {
          const int j = __ffs(take) - 1;
          const int i = c0 + 32 * u + j;
          const double di = __shfl_sync(kFull, d[u], j);
          taken = true;
          // attempt_transition accepted it: flip, cost, lowest
          if (lane == 0) sp[i >> 5] ^= 1u << (i & 31);
          __syncwarp();
          acc++;
          cost = __dadd_rn(cost, di);
          low = cost;
          warp_copy(ls, sp, nw, lane);
          if (lane == 0) tb[i] = it + tenure;
          tabu_refresh<FL, INT>(m, sp, df, i, lane);
          // local_search_init: a hill climber on a copy, its cost computed afresh
          warp_copy(hs, sp, nw, lane);
          warp_copy(hl, sp, nw, lane);
          for (int q = lane; q < N; q += 32) hd[q] = df[q];
          __syncwarp();
          double c;
          long long ic;
          warp_terms_cost<FL, INT>(m, hs, nullptr, lane, c, ic);
          S.hc_cost = INT ? (double)ic : c;
          S.hc_low = S.hc_cost;
          S.local = 1;
          S.incomplete += (unsigned long long)i;
          att += (unsigned long long)(i + 1);
          if (S.incomplete < (unsigned long long)SW)
            local_sweep();
          else
            S.incomplete -= (unsigned long long)SW;
          break;
        }
        if (ok && !(x[u] >= it) && k < bk)
        {
          bk = k;
          bd = d[u];
          bv = v;
        }
      }
    }
    if (!taken)
    {
      att += (unsigned long long)SW;
      // the lowest difference off the tabu list, the first on ties
#pragma unroll
      for (int sh = 16; sh; sh >>= 1)
      {
        const unsigned long long ok_ = __shfl_xor_sync(kFull, bk, sh);
        const double od = __shfl_xor_sync(kFull, bd, sh);
        const int ov = __shfl_xor_sync(kFull, bv, sh);
        if (ov != INT_MAX && (bv == INT_MAX || ok_ < bk || (ok_ == bk && ov < bv)))
        {
          bk = ok_;
          bd = od;
          bv = ov;
        }
      }
      if (bv != INT_MAX)
      {
        // Walker::apply_transition(transition, diff)
        if (lane == 0) sp[bv >> 5] ^= 1u << (bv & 31);
        __syncwarp();
        cost = __dadd_rn(cost, bd);
        if (cost < low)
        {
          low = cost;
          warp_copy(ls, sp, nw, lane);
        }
        if (lane == 0) tb[bv] = it + tenure;
        tabu_refresh<FL, INT>(m, sp, df, bv, lane);
      }
    }
    S.iter++;
    __syncwarp();
  }
  if (lane == 0)
  {
    a.st[w] = S;
    a.p.cost[w] = cost;
    a.p.lowest[w] = low;
    a.p.attempts[w] += att;
    a.p.accepts[w] += acc;
  }
}

// The same for pair-only Ising models that fit an SM's shared memory: the model
// once a block (rows, the other members, coefficients), and per walker (a warp)
// the differences as ordered keys, the list and both spin vectors; the hill
// climber's differences stay in HBM.
//
// What bounds it: a flip's refresh -- the rows of its neighbours, added in order
// -- and a scan's comparisons, a few instructions a variable with one vote per
// 128; from HBM the refresh waited for four dependent loads (5500 cycles) and the
// scan took 10500.  1216 walkers of a 1000-spin model, 200 steps: 3.78 ms from
// HBM, 2.27 here; 4096 of 1180 spins, 60 steps, in waves: 10.9 and 9.2; 8 of 1000:
// 2.86 and 1.88.  (With the differences and lists alone in shared memory the rows
// fell out of the L1 cache: 3.56, and 11.8 and 2.98 for the other two.)
struct TabuFit
{
  size_t model, walker;  // bytes
  int warps;             // walkers a block, at most; 0: does not fit
};
static TabuFit tabu_fit(const DevModel& m, int nw)
{
  TabuFit f;
  f.model = ((size_t)(m.n_vars + 1) * 4 + (size_t)m.n_inc * 4 + 15) / 16 * 16 + ((size_t)m.n_inc * (m.int_mode ? 4 : 8) + 15) / 16 * 16;
  f.walker = (16 * (size_t)m.n_vars + 8 * (size_t)nw + 15) / 16 * 16;
  const size_t room = 226 * 1024;
  f.warps = f.model + f.walker > room ? 0 : (int)std::min<size_t>(8, (room - f.model) / f.walker);
  return f;
}

template <bool INT>
__global__ void __launch_bounds__(256, 1) tabu_pair_kernel(TabuArgs a, size_t model_bytes, size_t walker_bytes)
{
  using CT = typename std::conditional<INT, int, double>::type;
  extern __shared__ __align__(16) unsigned char tmem[];
  const DevModel& m = a.m;
  const int N = m.n_vars, K = m.n_inc, nw = a.p.nw;
  const int lane = threadIdx.x & 31, wib = threadIdx.x >> 5;
  int* row = (int*)tmem;
  int* other = row + N + 1;
  CT* coef = (CT*)(tmem + ((size_t)(N + 1) * 4 + (size_t)K * 4 + 15) / 16 * 16);
  for (int q = threadIdx.x; q <= N; q += blockDim.x) row[q] = __ldg(m.row + q);
  for (int q = threadIdx.x; q < K; q += blockDim.x)
  {
    other[q] = __ldg(m.other + q);
    if constexpr (INT) coef[q] = __ldg(m.coef_i + q);
    else coef[q] = __ldg(m.coef + q);
  }
  __syncthreads();
  const int w = blockIdx.x * (blockDim.x >> 5) + wib;
  if (w >= a.n_walkers) return;  // whole warps leave together
  unsigned char* base = tmem + model_bytes + wib * walker_bytes;
  unsigned long long* key = (unsigned long long*)base;  // differences (raw_key)
  unsigned long long* tb = key + N;
  uint32_t* sp = (uint32_t*)(tb + N);
  uint32_t* hs = sp + nw;
  uint32_t* g_sp = a.p.spins + (size_t)w * nw;
  uint32_t* ls = a.p.lspins + (size_t)w * nw;
  uint32_t* g_hs = a.hc + (size_t)w * nw;
  uint32_t* hl = a.hc_low + (size_t)w * nw;
  unsigned long long* g_tb = a.tabu + (size_t)w * N;
  double* g_df = a.diff + (size_t)w * N;
  double* hd = a.hdiff + (size_t)w * N;
  TabuState S = a.st[w];
  double cost = a.p.cost[w], low = a.p.lowest[w];
  unsigned long long att = 0, acc = 0;
  const unsigned long long tenure = a.tenures ? a.tenures[w] : a.tenure;

  // invertible and ordered but for -0, which `as_key` makes +0 where it matters
  auto raw_key = [](double x) -> unsigned long long {
    const unsigned long long b = (unsigned long long)__double_as_longlong(x);
    return (b >> 63) ? ~b : (b | 0x8000000000000000ull);
  };
  auto of_key = [](unsigned long long k) -> double {
    return __longlong_as_double((long long)((k >> 63) ? (k ^ 0x8000000000000000ull) : ~k));
  };
  auto as_key = [](unsigned long long k) -> unsigned long long {
    return k == 0x7FFFFFFFFFFFFFFFull ? 0x8000000000000000ull : k;
  };
  // the difference of flipping v, terms in row order (lane_diff)
  auto diff_of = [&](const uint32_t* s, int v) -> double {
    const uint32_t sv = spin_of(s, v);
    const int qe = row[v + 1];
    double d = 0.0;
    int id = 0;
    for (int q = row[v]; q < qe; q += 4)
    {
      int o[4];
      CT c[4];
#pragma unroll
      for (int u = 0; u < 4; u++)
      {
        o[u] = other[min(q + u, qe - 1)];
        c[u] = coef[min(q + u, qe - 1)];
      }
#pragma unroll
      for (int u = 0; u < 4; u++)
      {
        const uint32_t par = sv ^ (o[u] >= 0 ? spin_of(s, o[u]) : 0u);
        if (q + u >= qe) continue;
        if constexpr (INT) id += par ? -c[u] : c[u];
        else d = __dadd_rn(d, par ? -c[u] : c[u]);
      }
    }
    return INT ? (double)(-2ll * id) : times_minus2(d);
  };
  // i's flip: its difference and its neighbours' afresh (tabu_refresh)
  auto refresh = [&](const uint32_t* s, int i, bool climber) {
    const int rb = row[i], re = row[i + 1];
    for (int q0 = rb; q0 < max(re, rb + 1); q0 += 32)
    {
      const int q = q0 + lane;
      int x = q < re ? other[q] : -1;
      // i itself on the first free lane of the first pass
      if (q0 == rb && lane == min(re - rb, 31))
      {
        if (x < 0) x = i;
        else
        {
          const double d = diff_of(s, i);
          if (climber) hd[i] = d;
          else key[i] = raw_key(d);
        }
      }
      if (x >= 0)
      {
        const double d = diff_of(s, x);
        if (climber) hd[x] = d;
        else key[x] = raw_key(d);
      }
    }
    __syncwarp();
  };

  warp_copy(sp, g_sp, nw, lane);
  warp_copy(hs, g_hs, nw, lane);
  for (int q = lane; q < N; q += 32)
  {
    key[q] = raw_key(S.ready ? g_df[q] : diff_of(sp, q));
    tb[q] = g_tb[q];
  }
  S.ready = 1;
  __syncwarp();

  // (tabu_kernel's)
  auto local_sweep = [&]() {
    const double prev = S.hc_low;
    int v0 = 0;
    while (v0 < N)
    {
      const int v = v0 + lane;
      const bool ok = v < N;
      const double d = ok ? hd[v] : 0.0;
      const unsigned take = __ballot_sync(kFull, ok && __double_as_longlong(d) <= 0);
      if (!take)
      {
        att += (unsigned long long)min(32, N - v0);
        v0 += 32;
        continue;
      }
      const int j = __ffs(take) - 1;
      const double dj = __shfl_sync(kFull, d, j);
      const int i = v0 + j;
      att += (unsigned long long)(j + 1);
      if (lane == 0) hs[i >> 5] ^= 1u << (i & 31);
      __syncwarp();
      acc++;
      S.hc_cost = __dadd_rn(S.hc_cost, dj);
      if (S.hc_cost < S.hc_low)
      {
        S.hc_low = S.hc_cost;
        warp_copy(hl, hs, nw, lane);
      }
      refresh(hs, i, true);
      v0 = i + 1;
    }
    if (S.hc_low < prev)
    {
      low = S.hc_low;
      warp_copy(ls, hl, nw, lane);
    }
    else
      S.local = 0;
  };

  for (int step = 0; step < a.n_steps; step++)
  {
    if (S.local)
    {
      local_sweep();
      continue;
    }
    // the scan (tabu_kernel): a difference surely below t is taken, one surely
    // above it is not
    const unsigned long long it = S.iter;
    const double t = __dadd_rn(low, -cost);
    const double e = fmax(__dmul_rn(fmax(fmax(fabs(cost), fabs(low)), fabs(t)), 0x1p-48), 0x1p-1000);
    const unsigned long long klo = fkey(__dadd_rn(t, -e)), khi = fkey(__dadd_rn(t, e));
    unsigned long long bk = ~0ull;
    int bv = INT_MAX;
    int found = -1;
    for (int c0 = 0; c0 < N && found < 0; c0 += 128)
    {
      unsigned long long k[4];
      bool may = false;
#pragma unroll
      for (int u = 0; u < 4; u++)
      {
        const int v = c0 + 32 * u + lane;
        const bool ok = v < N;
        k[u] = ok ? as_key(key[v]) : ~0ull;
        const unsigned long long x = ok ? tb[v] : ~0ull;
        may = may || (ok && k[u] <= khi);
        const bool better = ok && x < it && k[u] < bk;
        bk = better ? k[u] : bk;
        bv = better ? v : bv;
      }
      if (!__any_sync(kFull, may)) continue;
#pragma unroll
      for (int u = 0; u < 4; u++)
      {
        const int v = c0 + 32 * u + lane;
        const bool ok = v < N && found < 0;
        unsigned take = __ballot_sync(kFull, ok && k[u] < klo);
        const unsigned near = __ballot_sync(kFull, ok && k[u] >= klo && k[u] <= khi);
        if (near) take |= __ballot_sync(kFull, ((near >> lane) & 1) && __dadd_rn(cost, of_key(k[u])) < low);
        if (take && found < 0) found = c0 + 32 * u + __ffs(take) - 1;
      }
    }
    if (found >= 0)
    {
      const int i = found;
      const double di = of_key(key[i]);
      __syncwarp();
      // attempt_transition accepted it: flip, cost, lowest
      if (lane == 0) sp[i >> 5] ^= 1u << (i & 31);
      __syncwarp();
      acc++;
      cost = __dadd_rn(cost, di);
      low = cost;
      warp_copy(ls, sp, nw, lane);
      if (lane == 0) tb[i] = it + tenure;
      refresh(sp, i, false);
      // local_search_init: a hill climber on a copy, its cost computed afresh
      warp_copy(hs, sp, nw, lane);
      warp_copy(hl, sp, nw, lane);
      for (int q = lane; q < N; q += 32) hd[q] = of_key(key[q]);
      __syncwarp();
      double c;
      long long ic;
      warp_terms_cost<F_PARITY, INT>(m, hs, nullptr, lane, c, ic);
      S.hc_cost = INT ? (double)ic : c;
      S.hc_low = S.hc_cost;
      S.local = 1;
      S.incomplete += (unsigned long long)i;
      att += (unsigned long long)(i + 1);
      if (S.incomplete < (unsigned long long)N)
        local_sweep();
      else
        S.incomplete -= (unsigned long long)N;
    }
    else
    {
      att += (unsigned long long)N;
      // the lowest difference off the tabu list, the first on ties
      const unsigned hi = __reduce_min_sync(kFull, (unsigned)(bk >> 32));
      const bool h1 = (unsigned)(bk >> 32) == hi;
      const unsigned lo = __reduce_min_sync(kFull, h1 ? (unsigned)bk : ~0u);
      bv = __reduce_min_sync(kFull, h1 && (unsigned)bk == lo ? bv : INT_MAX);
      if (bv != INT_MAX)
      {
        // Walker::apply_transition(transition, diff)
        const double bd = of_key(key[bv]);
        __syncwarp();
        if (lane == 0) sp[bv >> 5] ^= 1u << (bv & 31);
        __syncwarp();
        cost = __dadd_rn(cost, bd);
        if (cost < low)
        {
          low = cost;
          warp_copy(ls, sp, nw, lane);
        }
        if (lane == 0) tb[bv] = it + tenure;
        refresh(sp, bv, false);
      }
    }
    S.iter++;
    __syncwarp();
  }
  warp_copy(g_sp, sp, nw, lane);
  warp_copy(g_hs, hs, nw, lane);
  for (int q = lane; q < N; q += 32)
  {
    g_df[q] = of_key(key[q]);
    g_tb[q] = tb[q];
  }
  if (lane == 0)
  {
    a.st[w] = S;
    a.p.cost[w] = cost;
    a.p.lowest[w] = low;
    a.p.attempts[w] += att;
    a.p.accepts[w] += acc;
  }
}

// ---------------------------------------------------------------------------
// Substochastic Monte Carlo walker steps.  Replay: one thread per emulated
// OpenMP thread t of the reference, serving walkers [b_t, e_t) (libgomp's
// schedule(static) blocks) in index order on its PCG stream: per attempt one
// uniform() against p_step, then, when taken, one uniform() for the variable
// (floor(u * N), model/ising.h:138-143, model/pubo.h:102-107).  Counter
// mode: one thread per walker slot j, its c-th attempt drawing
// counter_draw(counter_key(seed, j), 2c) and (.., 2c + 1) as 53-bit uniforms.
// Every flip is accepted: cost += the difference (term order), lowest kept.
// ---------------------------------------------------------------------------
template <int FL, bool INT>
__device__ __forceinline__ void ssmc_flip(const DevModel& m, const DevPop& p, int w, int v)
{
  uint32_t* sp = p.spins + (size_t)w * p.nw;
  const double d = lane_diff<FL, INT>(m, sp, v);
  sp[v >> 5] ^= 1u << (v & 31);
  const double c = __dadd_rn(p.cost[w], d);
  p.cost[w] = c;
  p.attempts[w] += 1;
  p.accepts[w] += 1;
  if (c < p.lowest[w])
  {
    p.lowest[w] = c;
    uint32_t* ls = p.lspins + (size_t)w * p.nw;
    for (int q = 0; q < p.nw; q++) ls[q] = sp[q];
  }
}

template <int FL, bool INT>
__global__ void __launch_bounds__(128) ssmc_walk_kernel(SsmcArgs a)
{
  const int t = blockIdx.x * blockDim.x + threadIdx.x;
  const int N = a.m.n_vars;
  const int spw = a.steps_per_walker;
  if (a.replay)
  {
    if (t >= a.n_chains) return;
    const int R = a.n_walkers, T = a.n_chains;
    const int q = R / T, r = R % T;
    const int b = t < r ? t * (q + 1) : t * q + r;
    const int e = b + (t < r ? q + 1 : q);
    uint64_t s = a.rng[t];
    auto uni = [&]() {
      const uint32_t d0 = pcg_out(s);
      s = s * kMult + kInc;
      const uint32_t d1 = pcg_out(s);
      s = s * kMult + kInc;
      return canonical(d0, d1);
    };
    for (int w = b; w < e; w++)
      for (int k = 0; k < spw; k++)
        if (uni() < a.p_step)
        {
          const int v = (int)__dmul_rn(uni(), (double)N);
          ssmc_flip<FL, INT>(a.m, a.p, w, v);
        }
    a.rng[t] = s;
  }
  else
  {
    if (t >= a.n_walkers) return;
    const uint64_t key = counter_key(a.seed, (uint64_t)t);
    for (int k = 0; k < spw; k++)
    {
      const unsigned long long c = (unsigned long long)a.step * (unsigned long long)spw + (unsigned long long)k;
      const double u = (double)(counter_draw(key, 2 * c) >> 11) * 0x1p-53;
      if (u < a.p_step)
      {
        const double u2 = (double)(counter_draw(key, 2 * c + 1) >> 11) * 0x1p-53;
        ssmc_flip<FL, INT>(a.m, a.p, t, (int)__dmul_rn(u2, (double)N));
      }
    }
  }
}

template <int FL, bool I>
static void ssmc_dispatch(const SsmcArgs& a, cudaStream_t s)
{
  const int n = a.replay ? a.n_chains : a.n_walkers;
  const int blocks = (n + 127) / 128;
  if (blocks > 0) ssmc_walk_kernel<FL, I><<<blocks, 128, 0, s>>>(a);
}

cudaError_t launch_ssmc_walk(const SsmcArgs& a, cudaStream_t s)
{
  if (a.n_walkers <= 0 || a.steps_per_walker <= 0) return cudaSuccess;
  const bool I = a.m.int_mode != 0;
  switch (a.m.flavor)
  {
    case F_PARITY: I ? ssmc_dispatch<F_PARITY, true>(a, s) : ssmc_dispatch<F_PARITY, false>(a, s); break;
    case F_COUNTER: I ? ssmc_dispatch<F_COUNTER, true>(a, s) : ssmc_dispatch<F_COUNTER, false>(a, s); break;
    case F_PLAIN_ISING: I ? ssmc_dispatch<F_PLAIN_ISING, true>(a, s) : ssmc_dispatch<F_PLAIN_ISING, false>(a, s); break;
    default: I ? ssmc_dispatch<F_PLAIN_PUBO, true>(a, s) : ssmc_dispatch<F_PLAIN_PUBO, false>(a, s); break;
  }
  return cudaGetLastError();
}

// ---------------------------------------------------------------------------
// Quantum Monte Carlo, any number of slices: one warp per restart, lanes over
// its slices (slice k on lane k % 32).  For each variable v of the ordered sweep: every slice
// computes its difference and, for k > 0 with the same value of v as slice
// k-1, its bond (a uniform() below bond_prob); each run of bonded slices
// (slice 0 and every unbonded slice start one) sums its differences in slice
// order, is accepted below 1e-11 or on a uniform() of its first slice below
// exp(-beta_eff * sum), and all its slices flip together.  The per-warp
// differences, bonds and acceptances sit in shared memory.  After each sweep
// the restart keeps the first lowest-cost slice if it beats its lowest.
// ---------------------------------------------------------------------------
// the 64 random bits of one uniform(): replay, the stream's next two
// outputs X = d0 + d1 2^32 (canonical(d0, d1) = fl(X) 2^-64, clamped below
// 1); counter, one counter draw (uniform = (draw >> 11) 2^-53)
__device__ __forceinline__ unsigned long long qmc_bits(const QmcArgs& a, int slot, unsigned long long ctr)
{
  if (a.replay)
  {
    uint64_t s = a.rng[slot];
    const uint32_t d0 = pcg_out(s);
    s = s * kMult + kInc;
    const uint32_t d1 = pcg_out(s);
    a.rng[slot] = s * kMult + kInc;
    return ((unsigned long long)d1 << 32) | d0;
  }
  return counter_draw(counter_key(a.seed, (uint64_t)slot), ctr);
}
__device__ __forceinline__ double qmc_uniform(const QmcArgs& a, unsigned long long x)
{
  if (a.replay) return canonical((uint32_t)x, (uint32_t)(x >> 32));
  return (double)(x >> 11) * 0x1p-53;
}

template <int FL, bool INT>
__global__ void __launch_bounds__(128) qmc_kernel(QmcArgs a)
{
  extern __shared__ unsigned char qsm[];
  const int lane = threadIdx.x & 31;
  const int wib = threadIdx.x >> 5;
  const int r = blockIdx.x * (blockDim.x >> 5) + wib;
  if (r >= a.restarts) return;  // whole warps leave together
  // SW variables are swept (1 for MaxSat unless the full sweep is asked
  // for); draw positions stay indexed by N
  const int P = a.trotter, N = a.m.n_vars, SW = a.m.sweep_size, nw = a.p.nw;
  const size_t per_warp = (size_t)P * 8 + (((size_t)P * 2 + 7) & ~(size_t)7);
  double* dif = (double*)(qsm + (size_t)wib * per_warp);
  uint8_t* bond = (uint8_t*)(dif + P);
  uint8_t* acc = bond + P;
  const int base = r * P;
  for (int st = 0; st < a.n_steps; st++)
  {
    const long long S = a.step_base + st;
    const double be = a.beta_eff[S];
    const float bef = (float)be;
    const unsigned long long blim = a.bond_lim[S];
    const bool ball = a.bond_all[S] != 0;
    for (int v = 0; v < SW; v++)
    {
      const unsigned long long c = 2ull * ((unsigned long long)S * (unsigned long long)N + (unsigned long long)v);
      for (int k = lane; k < P; k += 32)
      {
        const uint32_t* sp = a.p.spins + (size_t)(base + k) * nw;
        dif[k] = lane_diff<FL, INT>(a.m, sp, v);
        uint8_t b = 0;
        if (k > 0 && spin_of(sp - nw, v) == spin_of(sp, v))
        {
          const unsigned long long x = qmc_bits(a, base + k, c);
          b = a.replay ? (ball || x < blim) : ((x >> 11) < blim);
        }
        bond[k] = b;
      }
      __syncwarp();
      for (int k = lane; k < P; k += 32)
      {
        if (bond[k]) continue;
        double sum = dif[k];
        int e = k + 1;
        for (; e < P && bond[e]; e++) sum = __dadd_rn(sum, dif[e]);
        uint8_t ok = 1;
        if (!(sum < 10E-12))
        {
          const unsigned long long ub = qmc_bits(a, base + k, c + 1);
          // FP32 screen: the draw's top 24 bits are within 2^-23 of it;
          // x = -be sum rounded through float and expf's error stay below
          // ef (|xf| + 2) 2^-20; the FP64 exp decides only near the draw
          const float uf = (float)(uint32_t)(ub >> 40) * 0x1p-24f;
          const float xf = -bef * (float)sum, ef = expf(xf);
          const float te = ef * (fabsf(xf) + 2.0f) * 0x1p-20f;
          if (uf + 0x1p-23f < ef - te)
            ok = 1;
          else if (uf - 0x1p-23f > ef + te)
            ok = 0;
          else
          {
            const double u = qmc_uniform(a, ub);
            const double e = exp(__dmul_rn(-be, sum));
            if (fabs(u - e) <= 1e-15 * e) atomicAdd(a.near_ties, 1ULL);
            ok = u < e;
          }
        }
        for (int i = k; i < e; i++) acc[i] = ok;
      }
      __syncwarp();
      for (int k = lane; k < P; k += 32)
        if (acc[k])
        {
          uint32_t* sp = a.p.spins + (size_t)(base + k) * nw;
          sp[v >> 5] ^= 1u << (v & 31);
          a.p.cost[base + k] = __dadd_rn(a.p.cost[base + k], dif[k]);
          a.p.accepts[base + k] += 1;
        }
      __syncwarp();
    }
    // add_difference_evaluations + save_lowest (first lowest slice)
    double bc = 0.0;
    int bk = INT_MAX;
    for (int k = lane; k < P; k += 32)
    {
      a.p.attempts[base + k] += (unsigned long long)SW;
      const double ck = a.p.cost[base + k];
      if (bk == INT_MAX || ck < bc)
      {
        bc = ck;
        bk = k;
      }
    }
#pragma unroll
    for (int sh = 16; sh; sh >>= 1)
    {
      const double oc = __shfl_xor_sync(kFull, bc, sh);
      const int ok = __shfl_xor_sync(kFull, bk, sh);
      if (ok != INT_MAX && (bk == INT_MAX || oc < bc || (oc == bc && ok < bk)))
      {
        bc = oc;
        bk = ok;
      }
    }
    if (bc < a.low[r])
    {
      const uint32_t* src = a.p.spins + (size_t)(base + bk) * nw;
      for (int q = lane; q < nw; q += 32) a.low_spins[(size_t)r * nw + q] = src[q];
      __syncwarp();
      if (lane == 0) a.low[r] = bc;
    }
    __syncwarp();
  }
}

// Quantum Monte Carlo of up to 32 slices, two warps to a restart, a lane to a
// slice.  Variable v's values are one word w[v] (bit k: slice k) in shared
// memory, so that a term's parities, or whether any other literal is true, take
// one word operation a member for all slices, lane j taking the row's j-th
// incidence.  Rows do not depend on the state: their copies run up to three
// variables ahead.
//
// The first warp decides.  The differences' FP64 adds (68 cycles each, one after
// another) and those of a run's sum (up to 31 more) are not on its way: it sums
// in FP32, over the runs by one prefix sum, with a bound on its error, and only
// where sign or comparison lie inside that does it sum as the reference does
// (exact_run_sum).  Integer models sum exactly.  The second warp gets a word of
// flips a variable, keeps its own w, and takes the exact differences of the
// flipped slices into their costs and lowest.
//
// What bounds it: the decider's chain of loads, votes and shuffles, 1750 cycles a
// variable (differences 540, draws and bonds 270, runs 250, comparison 200, flips
// 190), the accountant close behind.  N = 1000, 3000 couplings, 16 restarts of 32
// slices, 50 sweeps: 145.4 ms with a lane per slice on spins, costs and streams in
// HBM, 94 with w, costs and streams on the chip and every sum in FP64, 47.7 with
// the exact sums off the way and the rows ahead in registers, 45.5 here,
// 45.9 with a sign of progress every 32 variables.
namespace qs
{
static const int kRing = 512;  // flip words, a power of two
static const long long kPatience = 8000000000LL;  // cycles without progress
struct Sync
{
  unsigned head, tail;  // variables decided, accounted for; published every 32
  unsigned abort;
};
__device__ __forceinline__ unsigned acquire(const unsigned* p)
{
  unsigned v;
  asm volatile("ld.acquire.cta.shared::cta.u32 %0, [%1];" : "=r"(v) : "r"((unsigned)__cvta_generic_to_shared(p)) : "memory");
  return v;
}
__device__ __forceinline__ void release(unsigned* p, unsigned v)
{
  asm volatile("st.release.cta.shared::cta.u32 [%0], %1;" ::"r"((unsigned)__cvta_generic_to_shared(p)), "r"(v) : "memory");
}
// waits until *p (counters wrap) reaches `want`; false: given up, as it stood still
__device__ __noinline__ bool wait_for(const unsigned* p, unsigned want, unsigned* abort, int* err, unsigned& seen)
{
  unsigned ok = 1;
  if ((threadIdx.x & 31) == 0)
  {
    long long t0 = clock64();
    unsigned last = acquire(p);
    while (true)
    {
      seen = acquire(p);
      if ((int)(seen - want) >= 0) break;
      if (seen != last)
      {
        last = seen;
        t0 = clock64();
      }
      if (acquire(abort) || clock64() - t0 > kPatience)
      {
        if (err) atomicExch(err, 1);
        release(abort, 1u);
        ok = 0;
        break;
      }
    }
  }
  seen = __shfl_sync(kFull, seen, 0);
  return __shfl_sync(kFull, ok, 0) != 0u;
}

// A variable's row, lane j having its j-th incidence (the first 32): incidence and
// coefficient come three variables ahead, the term's bounds two, its first four
// members one, by asynchronous copies into the lane's own slots of shared memory
// (held in registers, moving them up a place would wait for them).  CT: the
// coefficients' type.
struct Slots
{
  uint32_t x[4][32];     // incidence, or the pair's other member
  double c[4][32];
  int2 t[4][32];         // its term's bounds
  uint32_t m[2][32][4];  // members
};
template <int BYTES>
__device__ __forceinline__ void copy_async(void* dst, const void* src)
{
  asm volatile("cp.async.ca.shared.global [%0], [%1], %2;" ::"r"((unsigned)__cvta_generic_to_shared(dst)), "l"(src), "n"(BYTES)
               : "memory");
}
template <int FL, bool PAIR, class CT>
struct Rows
{
  static constexpr bool PAR = FL == F_PARITY || FL == F_PLAIN_ISING;
  struct Row { int b, e; };
  const int *row, *other, *trow;
  const uint32_t *inc, *tvar;
  const CT* coef;
  Slots* S;
  int SW, lane, ahead;
  unsigned turn;
  Row r0, r1, r2, r3;

  __device__ __forceinline__ Row load_row(int v) const { return {row[v], row[v + 1]}; }
  __device__ __forceinline__ int next(int v) const { return v + 1 < SW ? v + 1 : 0; }
  __device__ __forceinline__ CT& coef_slot(unsigned t) const { return *(CT*)&S->c[t & 3u][lane]; }
  __device__ __forceinline__ void get_inc(unsigned t, Row r) const
  {
    if (r.b + lane >= r.e) return;
    copy_async<4>(&S->x[t & 3u][lane], PAIR ? (const void*)(other + r.b + lane) : (const void*)(inc + r.b + lane));
    copy_async<sizeof(CT)>(&coef_slot(t), coef + r.b + lane);
  }
  __device__ __forceinline__ void get_term(unsigned t, Row r) const
  {
    if (PAIR || r.b + lane >= r.e) return;
    const int* p = trow + (int)(S->x[t & 3u][lane] & ~kNegBit);
    copy_async<4>(&S->t[t & 3u][lane].x, p);
    copy_async<4>(&S->t[t & 3u][lane].y, p + 1);
  }
  __device__ __forceinline__ void get_mem(unsigned t, Row r) const
  {
    if (PAIR || r.b + lane >= r.e) return;
    const int2 b = S->t[t & 3u][lane];
#pragma unroll
    for (int i = 0; i < 4; i++)
      if (b.x + i < b.y) copy_async<4>(&S->m[t & 1u][lane][i], tvar + b.x + i);
  }
  __device__ __forceinline__ void arrived() const
  {
    asm volatile("cp.async.wait_all;" ::: "memory");
  }
  // (rows: the row bounds in shared memory)
  __device__ __forceinline__ void start(const DevModel& m, const CT* c, const int* rows, Slots* slots, int l)
  {
    row = rows, other = m.other, trow = m.trow, inc = m.inc, tvar = m.tvar, coef = c, S = slots;
    SW = m.sweep_size, lane = l, turn = 0;
    const int v1 = next(0), v2 = next(v1), v3 = next(v2);
    ahead = next(v3);
    r0 = load_row(0), r1 = load_row(v1), r2 = load_row(v2), r3 = load_row(v3);
    get_inc(0, r0), get_inc(1, r1), get_inc(2, r2);
    arrived();
    get_term(0, r0), get_term(1, r1);
    arrived();
    get_mem(0, r0);
  }
  // what the last turn fetched has come; the next turns' is sent for
  __device__ __forceinline__ void issue() const
  {
    arrived();
    get_inc(turn + 3u, r3);
    get_term(turn + 2u, r2);
    get_mem(turn + 1u, r1);
  }
  __device__ __forceinline__ void shift()
  {
    r0 = r1, r1 = r2, r2 = r3, r3 = load_row(ahead);
    ahead = next(ahead);
    turn++;
  }
  __device__ __forceinline__ int degree() const { return __shfl_sync(kFull, r0.e - r0.b, 0); }
  // incidences j0 .. j0 + 31 of variable v, for all slices: the terms' parities,
  // or the slices in which another literal is true; the coefficients, negated
  // where v's literal is; nothing past the row
  __device__ __forceinline__ void take(int v, int deg, int j0, const uint32_t* w, uint32_t& on, CT& c) const
  {
    on = 0u;
    c = (CT)0;
    if (j0 + lane >= deg) return;
    uint32_t x;
    int2 t = make_int2(0, 0);
    if (j0 == 0)
    {
      x = S->x[turn & 3u][lane];
      c = coef_slot(turn);
      if (!PAIR) t = S->t[turn & 3u][lane];
    }
    else
    {
      const int q = r0.b + j0 + lane;
      x = PAIR ? (uint32_t)__ldg(other + q) : __ldg(inc + q);
      c = __ldg(coef + q);
      if (!PAIR) t = make_int2(__ldg(trow + (x & ~kNegBit)), __ldg(trow + (x & ~kNegBit) + 1));
    }
    if constexpr (PAIR) on = w[v] ^ ((int)x >= 0 ? w[x] : 0u);
    else
    {
      for (int i = 0; i < t.y - t.x; i++)
      {
        const uint32_t y = j0 == 0 && i < 4 ? S->m[turn & 1u][lane][i] : __ldg(tvar + t.x + i);
        const int u = (int)(y & ~kNegBit);
        if (PAR) on ^= w[u];
        else if (u != v) on |= w[u] ^ ((y & kNegBit) ? kFull : 0u);
      }
      if (x & kNegBit) c = -c;
    }
  }
};

// The slice's exact difference of flipping v, times_minus2 taken (Ising); the
// sum in row order
template <int FL, bool INT, bool PAIR, class CT>
__device__ __forceinline__ double exact_dif(const Rows<FL, PAIR, CT>& R, int v, const uint32_t* w)
{
  constexpr bool PAR = FL == F_PARITY || FL == F_PLAIN_ISING;
  const uint32_t sv = (w[v] >> R.lane) & 1u;
  const int deg = R.degree();
  double d = 0.0;
  int id = 0;
  for (int j0 = 0; j0 < deg; j0 += 32)
  {
    uint32_t on;
    CT c;
    R.take(v, deg, j0, w, on, c);
    const int n = min(32, deg - j0);
#pragma unroll 4
    for (int j = 0; j < n; j++)
    {
      const uint32_t b = (__shfl_sync(kFull, on, j) >> R.lane) & 1u;
      const CT x = __shfl_sync(kFull, c, j);
      if (INT)
      {
        if (PAR) id += b ? -(int)x : (int)x;
        else if (!b) id += sv ? (int)x : -(int)x;
      }
      else if (PAR) d = __dadd_rn(d, b ? -(double)x : (double)x);
      else if (!b) d = __dadd_rn(d, sv ? (double)x : -(double)x);
    }
  }
  if (INT) return (double)(PAR ? -2ll * id : (long long)id);
  return PAR ? times_minus2(d) : d;
}

// Rare: a run's sum (lanes first .. end - 1, on its first) as the reference adds
// it
template <int FL, bool PAIR>
__device__ __noinline__ double exact_run_sum(const DevModel& m, int v, const uint32_t* w, bool head, int end)
{
  const int lane = threadIdx.x & 31;
  const uint32_t sv = (w[v] >> lane) & 1u;
  constexpr bool PAR = FL == F_PARITY || FL == F_PLAIN_ISING;
  double dif = 0.0;
  for (int q = __ldg(m.row + v), qe = __ldg(m.row + v + 1); q < qe; q++)
  {
    const double c = __ldg(m.coef + q);
    uint32_t on = 0;
    bool neg = false;
    if (PAIR)
    {
      const int u = __ldg(m.other + q);
      on = w[v] ^ (u >= 0 ? w[u] : 0u);
    }
    else
    {
      const uint32_t e = __ldg(m.inc + q);
      neg = !PAR && (e & kNegBit) != 0u;
      for (int k = __ldg(m.trow + (e & ~kNegBit)), ke = __ldg(m.trow + (e & ~kNegBit) + 1); k < ke; k++)
      {
        const uint32_t y = __ldg(m.tvar + k);
        const int u = (int)(y & ~kNegBit);
        if (PAR) on ^= w[u];
        else if (u != v) on |= w[u] ^ ((y & kNegBit) ? kFull : 0u);
      }
    }
    const uint32_t b = (on >> lane) & 1u;
    if (PAR) dif = __dadd_rn(dif, b ? -c : c);
    else if (!b) dif = __dadd_rn(dif, ((sv != 0u) != neg) ? c : -c);
  }
  if (PAR) dif = times_minus2(dif);
  double sum = dif;
  for (int i = 1; __any_sync(kFull, head && lane + i < end); i++)
  {
    const double d = __shfl_down_sync(kFull, dif, i);
    if (head && lane + i < end) sum = __dadd_rn(sum, d);
  }
  return sum;
}
}  // namespace qs

template <int FL, bool INT, bool PAIR>
__global__ void __launch_bounds__(64) qmc_sliced_kernel(const __grid_constant__ QmcArgs a)
{
  using namespace qs;
  constexpr bool PAR = FL == F_PARITY || FL == F_PLAIN_ISING;
  extern __shared__ uint32_t qmem[];
  __shared__ Sync sync;
  __shared__ uint32_t ring[kRing];
  __shared__ __align__(16) Slots slots[2];
  __shared__ __align__(16) uint2 pair[32];  // the decider's row: words and coefficients
  const DevModel& m = a.m;
  // (through a shuffle: known to be the same on all lanes)
  const int role = __shfl_sync(kFull, (int)threadIdx.x >> 5, 0);
  const int lane = threadIdx.x & 31, r = blockIdx.x;
  const int P = a.trotter, N = m.n_vars, SW = m.sweep_size, nw = a.p.nw, nwd = (N + 31) >> 5;
  uint32_t* w = qmem + (role ? N : 0);  // each warp's own
  int* rows = (int*)qmem + 2 * N;
  for (int v = threadIdx.x; v <= N; v += 64) rows[v] = __ldg(m.row + v);
  const bool mine = lane < P;
  const int slot = r * P + (mine ? lane : 0);
  uint32_t* g_spins = a.p.spins + (size_t)slot * nw;
  if (threadIdx.x == 0) sync.head = sync.tail = sync.abort = 0u;
  for (int q = 0; q < nwd; q++)
  {
    const uint32_t x = mine ? g_spins[q] : 0u;
    uint32_t out = 0;
#pragma unroll
    for (int b = 0; b < 32; b++)
    {
      const unsigned y = __ballot_sync(kFull, (x >> b) & 1u);
      if (lane == b) out = y;
    }
    if (q * 32 + lane < N) w[q * 32 + lane] = out;
  }
  __syncthreads();

  if (role == 1)
  {
    // ---- the accountant
    double cost = a.p.cost[slot], low = a.low[r];
    unsigned long long acc_n = 0;
    unsigned tail = 0, seen = 0;
    using CT = typename std::conditional<INT, int, double>::type;
    Rows<FL, PAIR, CT> R;
    if constexpr (INT) R.start(m, m.coef_i, rows, &slots[1], lane);
    else R.start(m, m.coef, rows, &slots[1], lane);
    for (int st = 0; st < a.n_steps; st++)
    {
      for (int v = 0; v < SW; v++)
      {
        if (seen == tail)
        {
          if (lane == 0) release(&sync.tail, tail);
          if (!wait_for(&sync.head, tail + 1u, &sync.abort, a.err, seen))
          {
            R.arrived();
            return;
          }
        }
        R.issue();
        const uint32_t F = __shfl_sync(kFull, ring[tail & (kRing - 1u)], 0);
        if (F)
        {
          const double d = exact_dif<FL, INT, PAIR, CT>(R, v, w);
          if ((F >> lane) & 1u)
          {
            cost = __dadd_rn(cost, d);
            acc_n++;
          }
          __syncwarp();
          if (lane == 0) w[v] ^= F;
          __syncwarp();
        }
        tail++;
        if ((tail & 31u) == 0u && lane == 0) release(&sync.tail, tail);
        R.shift();
      }
      // save_lowest: the first lowest slice
      double bc = cost;
      int bk = mine ? lane : INT_MAX;
#pragma unroll
      for (int sh = 16; sh; sh >>= 1)
      {
        const double oc = __shfl_xor_sync(kFull, bc, sh);
        const int ok = __shfl_xor_sync(kFull, bk, sh);
        if (ok != INT_MAX && (bk == INT_MAX || oc < bc || (oc == bc && ok < bk)))
        {
          bc = oc;
          bk = ok;
        }
      }
      if (__any_sync(kFull, bc < low))
      {
        low = bc;
        for (int q = 0; q < nwd; q++)
        {
          const int v = q * 32 + lane;
          const unsigned y = __ballot_sync(kFull, v < N && ((w[min(v, N - 1)] >> bk) & 1u));
          if (lane == 0) a.low_spins[(size_t)r * nw + q] = y;
        }
      }
    }
    for (int q = 0; q < nwd; q++)
    {
      uint32_t x = 0;
      for (int b = 0; b < 32 && q * 32 + b < N; b++) x |= ((w[q * 32 + b] >> lane) & 1u) << b;
      if (mine) g_spins[q] = x;
    }
    if (mine)
    {
      a.p.cost[slot] = cost;
      a.p.accepts[slot] += acc_n;
      a.p.attempts[slot] += (unsigned long long)SW * (unsigned long long)a.n_steps;
    }
    if (lane == 0) a.low[r] = low;
    R.arrived();
    return;
  }

  // ---- the decider
  uint64_t rs = a.replay ? a.rng[slot] : 0;
  const uint64_t key = a.replay ? 0 : counter_key(a.seed, (uint64_t)slot);
  // Replay: a slice's next two uniforms take its stream's next four outputs; both
  // are made before it is known whether it takes none, one or two.
  const unsigned long long A2 = kMult * kMult, C2 = kMult * kInc + kInc;
  const unsigned long long A4 = A2 * A2, C4 = A2 * C2 + C2;
  using CT = typename std::conditional<INT, int, float>::type;
  Rows<FL, PAIR, CT> R;
  if constexpr (INT) R.start(m, m.coef_i, rows, &slots[0], lane);
  else R.start(m, m.coef_f, rows, &slots[0], lane);
  unsigned head = 0, tail = 0;
  for (int st = 0; st < a.n_steps; st++)
  {
    const long long S = a.step_base + st;
    const double be = a.beta_eff[S];
    const float bef = (float)be;
    const unsigned long long blim = a.bond_lim[S];
    const bool ball = a.bond_all[S] != 0;
    for (int v = 0; v < SW; v++)
    {
      R.issue();
      const unsigned long long c = 2ull * ((unsigned long long)S * (unsigned long long)N + (unsigned long long)v);
      const uint32_t word = w[v];
      const uint32_t sv = (word >> lane) & 1u;
      // ---- the slices' differences; `mag`: the sum of their terms' magnitudes
      float fd = 0.f, mag = 0.f;
      int id = 0;
      const int deg = R.degree();
      for (int j0 = 0; j0 < deg; j0 += 32)
      {
        uint32_t on;
        CT cj;
        R.take(v, deg, j0, w, on, cj);
        // through shared memory to all lanes, four at a time (nothing pads)
        uint2 p;
        p.x = on;
        if (INT) p.y = (uint32_t)(int)cj;
        else p.y = __float_as_uint((float)cj);
        pair[lane] = p;
        __syncwarp();
        const int n = min(32, deg - j0);
        for (int j = 0; j < n; j += 4)
        {
          uint2 q[4];
#pragma unroll
          for (int i = 0; i < 4; i++) q[i] = pair[j + i];
#pragma unroll
          for (int i = 0; i < 4; i++)
          {
            const uint32_t b = (q[i].x >> lane) & 1u;
            if (INT)
            {
              const int x = (int)q[i].y;
              if (PAR) id += b ? -x : x;
              else id += b ? 0 : (sv ? x : -x);
            }
            else
            {
              const float x = __uint_as_float(q[i].y);
              if (PAR) fd += b ? -x : x;
              else fd += b ? 0.f : (sv ? x : -x);
              mag += fabsf(x);
            }
          }
        }
        __syncwarp();
      }
      if (PAR)
      {
        fd *= -2.f;
        mag *= 2.f;
      }
      // ---- the draws that may be taken (qmc_bits)
      unsigned long long x1, x2;
      uint64_t s2 = 0, s4 = 0;
      if (a.replay)
      {
        s2 = A2 * rs + C2;
        s4 = A4 * rs + C4;
        x1 = ((unsigned long long)pcg_out(rs * kMult + kInc) << 32) | pcg_out(rs);
        x2 = ((unsigned long long)pcg_out(s2 * kMult + kInc) << 32) | pcg_out(s2);
      }
      else
      {
        x1 = counter_draw(key, c);
        x2 = counter_draw(key, c + 1);
      }
      // ---- bonds to the slice before, on equal values
      const bool equal = mine && lane > 0 && !(((word ^ (word << 1)) >> lane) & 1u);
      const bool bonded = equal && (a.replay ? (ball || x1 < blim) : ((x1 >> 11) < blim));
      const unsigned B = __ballot_sync(kFull, bonded);
      const bool first = mine && !bonded;
      const unsigned long long ub = a.replay && !equal ? x1 : x2;
      // ---- every run's sum, on its first slice
      const unsigned above = ~B & ~((2u << lane) - 1u);
      const int end = min(P, above ? __ffs(above) - 1 : 32);
      float s, e;
      bool up, amb = false;
      double sum = 0.0;
      bool have = false;  // `sum` is the reference's
      if (INT)
      {
        long long x = PAR ? -2ll * id : (long long)id;
        const long long own = x;
#pragma unroll
        for (int d = 1; d < 32; d <<= 1)
        {
          const long long y = __shfl_up_sync(kFull, x, d);
          if (lane >= d) x += y;
        }
        const long long t = __shfl_sync(kFull, x, end - 1) - x + own;
        sum = (double)t;
        s = (float)sum;
        e = 0.f;
        up = first && t > 0;
        have = true;
      }
      else
      {
        float x = fd;
#pragma unroll
        for (int d = 1; d < 32; d <<= 1)
        {
          const float y = __shfl_up_sync(kFull, x, d);
          if (lane >= d) x += y;
        }
        s = __shfl_sync(kFull, x, end - 1) - x + fd;
        // A difference is off by (deg + 2) 2^-24 of mag, a prefix of 32 of them
        // by that and six more roundings of 32 mag, their difference by twice
        // the latter.
        e = mag * (float)(512 + 40 * (deg + 2)) * 0x1p-24f + 1e-30f;
        const bool dn = s + e < 0.99e-11f;
        up = first && s - e > 1.01e-11f;
        amb = first && !dn && !up;
        if (__any_sync(kFull, amb))
        {
          sum = exact_run_sum<FL, PAIR>(m, v, w, first, end);
          have = true;
          if (amb) up = !(sum < 10E-12);
        }
      }
      bool ok = first;
      amb = false;
      if (up)
      {
        // (the screen of qmc_kernel, with the sum's error)
        const float uf = (float)(uint32_t)(ub >> 40) * 0x1p-24f;
        const float xf = -bef * s, ef = expf(xf), de = bef * e;
        const float te = ef * ((fabsf(xf) + 2.0f) * 0x1p-20f + 1.1f * de);
        amb = !(de < 0.03f);
        ok = uf + 0x1p-23f < ef - te;
        amb = amb || !(ok || uf - 0x1p-23f > ef + te);
      }
      if (__any_sync(kFull, amb))
      {
        if (!INT && !have) sum = exact_run_sum<FL, PAIR>(m, v, w, first, end);
        if (amb)
        {
          const double u = qmc_uniform(a, ub);
          const double x = exp(__dmul_rn(-be, sum));
          if (fabs(u - x) <= 1e-15 * x) atomicAdd(a.near_ties, 1ULL);
          ok = u < x;
        }
      }
      rs = equal && up ? s4 : (equal || up ? s2 : rs);
      // ---- a run flips as its first slice decides
      const unsigned H = ~B, A = __ballot_sync(kFull, ok);
      const unsigned at = H & ((2u << lane) - 1u);
      const unsigned F = __ballot_sync(kFull, mine && ((A >> (31 - __clz(at))) & 1u));
      if (lane == 0)
      {
        w[v] = word ^ F;
        ring[head & (kRing - 1u)] = F;
      }
      __syncwarp();
      head++;
      R.shift();
      if ((head & 31u) == 0u)
      {
        if (lane == 0) release(&sync.head, head);
        if (head - tail > (unsigned)kRing - 32u &&
            !wait_for(&sync.tail, head - (unsigned)kRing + 32u, &sync.abort, a.err, tail))
        {
          R.arrived();
          return;
        }
      }
    }
  }
  if (lane == 0) release(&sync.head, head);
  R.arrived();
  if (mine && a.replay) a.rng[slot] = rs;
}

// Level-parallel QMC sweeps for counter streams (positional draws): one
// block per restart, its slices' spins in shared memory, the warps taking the
// variables of one level at a time (no two share a term, and every
// lower-index neighbour sits in an earlier level, so each variable sees the
// spins the ordered sweep would).  Flips are logged per slice; after the
// sweep each slice adds its flips' differences to its cost in variable order,
// as the ordered sweep's cost += diff does.
size_t qmc_level_smem(int trotter, int nw)
{
  if (trotter < 2 || trotter > 256) return 0;
  const size_t per_warp = (size_t)trotter * 8 + (((size_t)trotter * 2 + 7) & ~(size_t)7);
  const size_t b = 2 * (size_t)trotter * nw * 4 + kQmcLevelWarps * per_warp;
  return b <= 200 * 1024 ? b : 0;
}

template <int FL, bool INT>
__global__ void __launch_bounds__(kQmcLevelWarps * 32) qmc_level_kernel(QmcArgs a)
{
  extern __shared__ __align__(16) unsigned char qls[];
  const int lane = threadIdx.x & 31, wib = threadIdx.x >> 5, nwarps = blockDim.x >> 5;
  const int r = blockIdx.x;
  const int P = a.trotter, N = a.m.n_vars, nw = a.p.nw;
  uint32_t* sps = (uint32_t*)qls;
  uint32_t* flp = sps + (size_t)P * nw;
  const size_t per_warp = (size_t)P * 8 + (((size_t)P * 2 + 7) & ~(size_t)7);
  double* dif = (double*)((unsigned char*)(flp + (size_t)P * nw) + (size_t)wib * per_warp);
  uint8_t* bond = (uint8_t*)(dif + P);
  uint8_t* acc = bond + P;
  const int base = r * P;
  double* dl = a.dlog + (size_t)base * N;
  for (int i = threadIdx.x; i < P * nw; i += blockDim.x) sps[i] = a.p.spins[(size_t)base * nw + i];
  __syncthreads();
  for (int st = 0; st < a.n_steps; st++)
  {
    const long long S = a.step_base + st;
    const double be = a.beta_eff[S];
    const float bef = (float)be;
    const unsigned long long blim = a.bond_lim[S];
    for (int i = threadIdx.x; i < P * nw; i += blockDim.x) flp[i] = 0;
    __syncthreads();
    for (int L = 0; L < a.n_levels; L++)
    {
      const int e1 = a.lv_off[L + 1];
      for (int e = a.lv_off[L] + wib; e < e1; e += nwarps)
      {
        const int v = a.lv_var[e];
        const unsigned long long c =
            2ull * ((unsigned long long)S * (unsigned long long)N + (unsigned long long)v);
        for (int k = lane; k < P; k += 32)
        {
          const uint32_t* sp = sps + (size_t)k * nw;
          dif[k] = lane_diff<FL, INT>(a.m, sp, v);
          uint8_t b = 0;
          if (k > 0 && spin_of(sp - nw, v) == spin_of(sp, v))
            b = (counter_draw(counter_key(a.seed, (uint64_t)(base + k)), c) >> 11) < blim;
          bond[k] = b;
        }
        __syncwarp();
        for (int k = lane; k < P; k += 32)
        {
          if (bond[k]) continue;
          double sum = dif[k];
          int q = k + 1;
          for (; q < P && bond[q]; q++) sum = __dadd_rn(sum, dif[q]);
          uint8_t ok = 1;
          if (!(sum < 10E-12))
          {
            const unsigned long long ub = counter_draw(counter_key(a.seed, (uint64_t)(base + k)), c + 1);
            const float uf = (float)(uint32_t)(ub >> 40) * 0x1p-24f;
            const float xf = -bef * (float)sum, ef = expf(xf);
            const float te = ef * (fabsf(xf) + 2.0f) * 0x1p-20f;
            if (uf + 0x1p-23f < ef - te)
              ok = 1;
            else if (uf - 0x1p-23f > ef + te)
              ok = 0;
            else
            {
              const double u = (double)(ub >> 11) * 0x1p-53;
              const double x = exp(__dmul_rn(-be, sum));
              if (fabs(u - x) <= 1e-15 * x) atomicAdd(a.near_ties, 1ULL);
              ok = u < x;
            }
          }
          for (int i = k; i < q; i++) acc[i] = ok;
        }
        __syncwarp();
        for (int k = lane; k < P; k += 32)
          if (acc[k])
          {
            atomicXor(&sps[(size_t)k * nw + (v >> 5)], 1u << (v & 31));
            atomicOr(&flp[(size_t)k * nw + (v >> 5)], 1u << (v & 31));
            dl[(size_t)k * N + v] = dif[k];
          }
        __syncwarp();
      }
      __syncthreads();
    }
    // cost += diff over the sweep's flips in variable order, per slice
    for (int k = threadIdx.x; k < P; k += blockDim.x)
    {
      double cst = a.p.cost[base + k];
      unsigned long long nf = 0;
      for (int q = 0; q < nw; q++)
      {
        uint32_t f = flp[(size_t)k * nw + q];
        while (f)
        {
          const int b = __ffs(f) - 1;
          f &= f - 1;
          cst = __dadd_rn(cst, dl[(size_t)k * N + q * 32 + b]);
          nf++;
        }
      }
      a.p.cost[base + k] = cst;
      a.p.accepts[base + k] += nf;
      a.p.attempts[base + k] += (unsigned long long)N;
    }
    __syncthreads();
    if (wib == 0)
    {
      double bc = 0.0;
      int bk = INT_MAX;
      for (int k = lane; k < P; k += 32)
      {
        const double ck = a.p.cost[base + k];
        if (bk == INT_MAX || ck < bc)
        {
          bc = ck;
          bk = k;
        }
      }
#pragma unroll
      for (int sh = 16; sh; sh >>= 1)
      {
        const double oc = __shfl_xor_sync(kFull, bc, sh);
        const int ok = __shfl_xor_sync(kFull, bk, sh);
        if (ok != INT_MAX && (bk == INT_MAX || oc < bc || (oc == bc && ok < bk)))
        {
          bc = oc;
          bk = ok;
        }
      }
      if (bc < a.low[r])
      {
        for (int q = lane; q < nw; q += 32) a.low_spins[(size_t)r * nw + q] = sps[(size_t)bk * nw + q];
        __syncwarp();
        if (lane == 0) a.low[r] = bc;
      }
    }
    __syncthreads();
  }
  for (int i = threadIdx.x; i < P * nw; i += blockDim.x) a.p.spins[(size_t)base * nw + i] = sps[i];
}

template <int FL, bool I>
static cudaError_t qmc_level_dispatch(const QmcArgs& a, cudaStream_t s)
{
  const size_t smem = qmc_level_smem(a.trotter, a.p.nw);
  const cudaError_t allowed = allow_shared((const void*)qmc_level_kernel<FL, I>, (int)smem);
  if (allowed != cudaSuccess) return allowed;
  qmc_level_kernel<FL, I><<<a.restarts, kQmcLevelWarps * 32, smem, s>>>(a);
  return cudaGetLastError();
}

cudaError_t launch_qmc_levels(const QmcArgs& a, cudaStream_t s)
{
  if (a.restarts <= 0 || a.n_steps <= 0) return cudaSuccess;
  if (a.replay || !qmc_level_smem(a.trotter, a.p.nw) || !a.lv_off || !a.lv_var || !a.dlog)
    return cudaErrorInvalidValue;
  const bool I = a.m.int_mode != 0;
  switch (a.m.flavor)
  {
    case F_PARITY: return I ? qmc_level_dispatch<F_PARITY, true>(a, s) : qmc_level_dispatch<F_PARITY, false>(a, s);
    case F_COUNTER: return I ? qmc_level_dispatch<F_COUNTER, true>(a, s) : qmc_level_dispatch<F_COUNTER, false>(a, s);
    case F_PLAIN_ISING:
      return I ? qmc_level_dispatch<F_PLAIN_ISING, true>(a, s) : qmc_level_dispatch<F_PLAIN_ISING, false>(a, s);
    default: return I ? qmc_level_dispatch<F_PLAIN_PUBO, true>(a, s) : qmc_level_dispatch<F_PLAIN_PUBO, false>(a, s);
  }
}

template <int FL, bool I>
static cudaError_t qmc_dispatch(const QmcArgs& a, cudaStream_t s)
{
  // A slice per lane where there are lanes and the variables' words fit.  Rows of
  // more than 1024 incidences stay out: the screen's error bound grows with the
  // row until it decides nothing (complete graphs of 500 variables, N(0, 1)
  // couplings 118 ms here and there, of 1000, couplings of variance 1 / N, 332 here
  // and 495 there, PUBO rows of 2400 102 and 93), and the work of the 32 variables
  // between two signs of progress stays below what the warps' waits allow.  Nor do
  // launches of few decisions (partial MaxSat sweeps), as every variable's word is
  // made and put back: 8000 variables, a decision a sweep, 30 sweeps 0.49 ms against
  // 0.28, 100 0.63 against 0.79; 1000 variables 0.23 and 0.24, 0.45 and 0.68.  (The
  // restarts are at most the host's threads or 16, so each has its SM, or nearly:
  // 16000 variables, 16 restarts of 32 slices, 3 sweeps 49.9 ms against 165.)
  const size_t words = ((size_t)a.m.n_vars * 3 + 1) * 4;  // two copies, the row bounds
  const bool few = (long long)a.n_steps * a.m.sweep_size < a.m.n_vars / 64;
  if (a.trotter <= 32 && words <= 200 * 1024 && a.m.max_deg <= 1024 && !few)
  {
    auto k = FL == F_PARITY && a.m.pair_only ? qmc_sliced_kernel<FL, I, FL == F_PARITY> : qmc_sliced_kernel<FL, I, false>;
    const cudaError_t allowed = allow_shared((const void*)k, (int)words);
    if (allowed != cudaSuccess) return allowed;
    k<<<a.restarts, 64, words, s>>>(a);
    return cudaGetLastError();
  }
  const size_t per_warp = (size_t)a.trotter * 8 + (((size_t)a.trotter * 2 + 7) & ~(size_t)7);
  const int blocks = (a.restarts + 3) / 4;
  const size_t smem = 4 * per_warp;
  const cudaError_t allowed = allow_shared((const void*)qmc_kernel<FL, I>, (int)smem);
  if (allowed != cudaSuccess) return allowed;
  if (blocks > 0) qmc_kernel<FL, I><<<blocks, 128, smem, s>>>(a);
  return cudaGetLastError();
}

cudaError_t launch_qmc(const QmcArgs& a, cudaStream_t s)
{
  if (a.restarts <= 0 || a.n_steps <= 0) return cudaSuccess;
  if (a.trotter < 2 || a.trotter > kQmcMaxTrotter) return cudaErrorInvalidValue;
  const bool I = a.m.int_mode != 0;
  switch (a.m.flavor)
  {
    case F_PARITY: return I ? qmc_dispatch<F_PARITY, true>(a, s) : qmc_dispatch<F_PARITY, false>(a, s);
    case F_COUNTER: return I ? qmc_dispatch<F_COUNTER, true>(a, s) : qmc_dispatch<F_COUNTER, false>(a, s);
    case F_PLAIN_ISING: return I ? qmc_dispatch<F_PLAIN_ISING, true>(a, s) : qmc_dispatch<F_PLAIN_ISING, false>(a, s);
    default: return I ? qmc_dispatch<F_PLAIN_PUBO, true>(a, s) : qmc_dispatch<F_PLAIN_PUBO, false>(a, s);
  }
}

// ---------------------------------------------------------------------------
// PT: observations then alternating-parity neighbour swaps of the slot
// labels (solver/parallel_tempering.h:134-189); one thread per restart.
// ---------------------------------------------------------------------------
__global__ void pt_swap_kernel(SwapArgs a)
{
  // Launched while the sweep before it runs; the next one's blocks come in once
  // that is done.  (Let in before the wait, they held shared memory for the whole
  // sweep that other solves had use for: 64 tempering requests of 128 walkers
  // through a server 410 ms, so 339, 96 of 384 walkers 1433 and 1252; one solve
  // alone, 3-SAT of 64 walkers, 200 steps, 10.55 and 10.39.)
  asm volatile("griddepcontrol.wait;" ::: "memory");
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
  // one warp per restart: lanes over the ladder's walkers, then over the
  // step's pairs (pairs of one parity share no walker)
  const int lane = threadIdx.x & 31;
  const int k = (int)((blockIdx.x * blockDim.x + threadIdx.x) >> 5);
  if (k >= a.restarts) return;
  const int T = a.n_temps;
  const int base = k * T;
  for (int p = lane; p < T; p += 32)
  {
    const int w = base + p;
    const double att = (double)a.step_att_reset[w];
    const double acc = (double)a.step_acc_reset[w];
    a.obs_acc[w] = __dadd_rn(a.obs_acc[w], __ddiv_rn(acc, att));
    a.obs_cost[w] = __dadd_rn(a.obs_cost[w], a.cost[a.slot_of[w]]);
    a.obs_dir[w] = __dadd_rn(a.obs_dir[w], (double)a.dir[w]);
    a.step_att_reset[w] = 0;
    a.step_acc_reset[w] = 0;
  }
  __syncwarp();
  // pair j of the step is (i, i + 1), i = (step & 1) + 2j; replayed, it
  // takes draws 2j and 2j + 1 of the master stream (the reference's loop
  // draws them in pair order)
  const int first = (int)(a.step & 1);
  const int npairs = T - 1 > first ? (T - first) / 2 : 0;
  uint64_t ms = a.replay ? a.master[k] : 0;
  for (int j0 = 0; j0 < npairs; j0 += 32)
  {
    const int j = j0 + lane;
    if (j < npairs)
    {
      const int i = first + 2 * j;
      double u;
      if (a.replay)
      {
        uint64_t sj = c_jA[2 * lane] * ms + c_jC[2 * lane];
        const uint32_t d0 = pcg_out(sj);
        sj = sj * kMult + kInc;
        const uint32_t d1 = pcg_out(sj);
        u = canonical(d0, d1);
      }
      else
      {
        const uint64_t wd = counter_draw(a.swap_key[k], (unsigned long long)a.step * (unsigned long long)T +
                                                            (unsigned long long)i);
        u = __dmul_rn((double)(wd >> 11), 1.0 / 9007199254740992.0);
      }
      const int wa = base + i, wb = base + i + 1;
      const double x = __dmul_rn(__dsub_rn(a.cost[a.slot_of[wa]], a.cost[a.slot_of[wb]]),
                                 __dsub_rn(a.beta[wa], a.beta[wb]));
      double e = exp(x);
      if (fabs(u - e) <= 1e-15 * e)
      {
        // near tie: the correctly rounded exp, which the C library's exp
        // (the reference's) returns except for its rare misroundings
        e = dd::exp_cr(x);
        atomicAdd(a.near_ties, 1ULL);
      }
      if (u < e)
      {
        const int t = a.slot_of[wa];
        a.slot_of[wa] = a.slot_of[wb];
        a.slot_of[wb] = t;
        const int d = a.dir[wa];
        a.dir[wa] = a.dir[wb];
        a.dir[wb] = d;
        a.swap_acc[wa] += 1;
      }
      a.swap_cnt[wa] += 1;
    }
    // the master stream moves past this chunk's draws (at most 64)
    const int nin = min(32, npairs - j0);
    if (a.replay) ms = c_jA[2 * nin] * ms + c_jC[2 * nin];
  }
  __syncwarp();
  if (lane == 0)
  {
    a.dir[base] = 0;
    a.dir[base + T - 1] = 1;
    if (a.replay) a.master[k] = ms;
  }
}

// ---------------------------------------------------------------------------
// PA resampling copies (Population::resample, solver/population.h:171-218):
// every destination walker is an integer copy of its source walker.
// ---------------------------------------------------------------------------
__global__ void pa_copy_kernel(DevPop src, DevPop dst, const int* src_of, int n_dst)
{
  const int lane = threadIdx.x & 31;
  const int j = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  if (j >= n_dst) return;
  const int i = src_of[j];
  const uint4* a = (const uint4*)(src.spins + (size_t)i * src.nw);
  uint4* b = (uint4*)(dst.spins + (size_t)j * dst.nw);
  for (int q = lane; q < src.nw / 4; q += 32) b[q] = a[q];
  a = (const uint4*)(src.lspins + (size_t)i * src.nw);
  b = (uint4*)(dst.lspins + (size_t)j * dst.nw);
  for (int q = lane; q < src.nw / 4; q += 32) b[q] = a[q];
  a = (const uint4*)(src.tstate + (size_t)i * src.mp);
  b = (uint4*)(dst.tstate + (size_t)j * dst.mp);
  for (int q = lane; q < src.mp / 16; q += 32) b[q] = a[q];
  if (lane == 0)
  {
    dst.cost[j] = src.cost[i];
    dst.lowest[j] = src.lowest[i];
    dst.attempts[j] = src.attempts[i];
    dst.accepts[j] = src.accepts[i];
    dst.step_att[j] = 0;
    dst.step_acc[j] = 0;
    if (dst.windows) dst.windows[j] = src.windows ? src.windows[i] : 0;
  }
}

cudaError_t launch_pa_copy(const DevPop& src, const DevPop& dst, const int* src_of,
                           int n_dst, cudaStream_t s)
{
  int blocks = (n_dst + 7) / 8;
  if (blocks > 0) pa_copy_kernel<<<blocks, 256, 0, s>>>(src, dst, src_of, n_dst);
  return cudaGetLastError();
}

// ---------------------------------------------------------------------------
// launchers
// ---------------------------------------------------------------------------
void sw_upload(const double* ln, const float* scr, const unsigned long long* jA,
               const unsigned long long* jC);
void fc_upload(const double* ln, const float* scr, const unsigned long long* jA,
               const unsigned long long* jC);

void upload_tables(int)
{
  double ln[1024];
  for (int row = 0; row < 4; row++)
    for (int i = 0; i < 256; i++)
      ln[row * 256 + i] = log((i) / pow((double)256, (double)(row + 1)));
  unsigned long long jA[65], jC[65], pA[64], pC[64];
  jA[0] = 1;
  jC[0] = 0;
  for (int k = 1; k < 65; k++)
  {
    jA[k] = jA[k - 1] * kMult;
    jC[k] = jC[k - 1] * kMult + kInc;
  }
  pA[0] = kMult;
  pC[0] = kInc;
  for (int k = 1; k < 64; k++)
  {
    pA[k] = pA[k - 1] * pA[k - 1];
    pC[k] = pA[k - 1] * pC[k - 1] + pC[k - 1];
  }
  cudaMemcpyToSymbol(c_ln, ln, sizeof ln);
  cudaMemcpyToSymbol(c_jA, jA, sizeof jA);
  cudaMemcpyToSymbol(c_jC, jC, sizeof jC);
  cudaMemcpyToSymbol(c_pA, pA, sizeof pA);
  cudaMemcpyToSymbol(c_pC, pC, sizeof pC);
  // FP32 screen of the ln-table comparison: per (row, bucket) the double
  // y0 and RN(y1 - y0) rounded to float, and an error margin 2^-19 (|y0| +
  // |dy|) that covers the float rounding of y0, dy, the distance and the
  // multiply-add against the double expression
  float scr[3072];
  for (int row = 0; row < 4; row++)
    for (int b = 0; b < 256; b++)
    {
      float* e = scr + (row * 256 + b) * 3;
      if (b < 2)
      {
        e[0] = e[1] = e[2] = 0.f;
        continue;
      }
      double y0 = ln[row * 256 + b - 1], dy = ln[row * 256 + b] - y0;
      e[0] = (float)y0;
      e[1] = (float)dy;
      e[2] = (float)(ldexp(fabs(y0) + fabs(dy), -19));
    }
  sw_upload(ln, scr, jA, jC);
  fc_upload(ln, scr, jA, jC);
  lw_upload(ln, scr);
  lv_upload(ln, scr);
}

template <int FL, bool INT>
static void init_dispatch(const InitArgs& a, cudaStream_t s)
{
  if (a.n_walkers <= 0) return;
  // A block shortens one walker's chain of loads and sums; with few terms, or warps
  // enough on the chip, its idle lanes and waits cost more.  Initialising by block
  // and by warp (us): integer Ising of 4096 terms, 256 walkers 58 and 100, 4096 92
  // and 114, 65536 810 and 772, of 512 terms, 4096 walkers 66 and 62; FP64 PUBO of
  // 128 terms, 65536 walkers 472 and 356, of 4096, 256 walkers 180 and 217, 4096
  // 364 and 341.
  if (a.m.n_terms > 512 && a.n_walkers < (INT ? 8192 : 2048)) init_kernel<FL, INT, 4><<<a.n_walkers, 128, 0, s>>>(a);
  else init_kernel<FL, INT, 1><<<(a.n_walkers + 3) / 4, 128, 0, s>>>(a);
}

cudaError_t launch_init(const InitArgs& a, cudaStream_t s)
{
  const bool I = a.m.int_mode != 0;
  switch (a.m.flavor)
  {
    case F_PARITY: I ? init_dispatch<F_PARITY, true>(a, s) : init_dispatch<F_PARITY, false>(a, s); break;
    case F_COUNTER: I ? init_dispatch<F_COUNTER, true>(a, s) : init_dispatch<F_COUNTER, false>(a, s); break;
    case F_PLAIN_ISING: I ? init_dispatch<F_PLAIN_ISING, true>(a, s) : init_dispatch<F_PLAIN_ISING, false>(a, s); break;
    default: I ? init_dispatch<F_PLAIN_PUBO, true>(a, s) : init_dispatch<F_PLAIN_PUBO, false>(a, s); break;
  }
  return cudaGetLastError();
}

cudaError_t launch_pack_states(const uint8_t* states, long long n, int n_vars, int nw, uint32_t* words, cudaStream_t s)
{
  const long long warps = n * ((nw + 3) / 4);
  const long long blocks = std::min<long long>((warps + 7) / 8, 152 * 8);
  if (blocks > 0) pack_states_kernel<<<(unsigned)blocks, 256, 0, s>>>(states, n, n_vars, nw, words);
  return cudaGetLastError();
}

template <int FL, bool I>
static void cost_dispatch(const DevModel& m, int n, const uint32_t* sp, int nw,
                          double* out, cudaStream_t s)
{
  if (n > 0) eval_cost_kernel<FL, I><<<n, 128, 0, s>>>(m, n, sp, nw, out);
}

cudaError_t launch_eval_cost(const DevModel& m, int n, const uint32_t* sp,
                             int nw, double* out, cudaStream_t s)
{
  const bool I = m.int_mode != 0;
  switch (m.flavor)
  {
    case F_PARITY: I ? cost_dispatch<F_PARITY, true>(m, n, sp, nw, out, s) : cost_dispatch<F_PARITY, false>(m, n, sp, nw, out, s); break;
    case F_COUNTER: I ? cost_dispatch<F_COUNTER, true>(m, n, sp, nw, out, s) : cost_dispatch<F_COUNTER, false>(m, n, sp, nw, out, s); break;
    case F_PLAIN_ISING: I ? cost_dispatch<F_PLAIN_ISING, true>(m, n, sp, nw, out, s) : cost_dispatch<F_PLAIN_ISING, false>(m, n, sp, nw, out, s); break;
    default: I ? cost_dispatch<F_PLAIN_PUBO, true>(m, n, sp, nw, out, s) : cost_dispatch<F_PLAIN_PUBO, false>(m, n, sp, nw, out, s); break;
  }
  return cudaGetLastError();
}

template <int FL, bool I>
static void diff_dispatch(const DevModel& m, int n, const uint32_t* sp, int nw,
                          const long long* vars, double* out, cudaStream_t s)
{
  int blocks = (n + 3) / 4;
  if (blocks > 0) eval_diff_kernel<FL, I><<<blocks, 128, 0, s>>>(m, n, sp, nw, vars, out);
}

cudaError_t launch_eval_diff(const DevModel& m, int n, const uint32_t* sp,
                             int nw, const long long* vars, double* out,
                             cudaStream_t s)
{
  const bool I = m.int_mode != 0;
  switch (m.flavor)
  {
    case F_PARITY: I ? diff_dispatch<F_PARITY, true>(m, n, sp, nw, vars, out, s) : diff_dispatch<F_PARITY, false>(m, n, sp, nw, vars, out, s); break;
    case F_COUNTER: I ? diff_dispatch<F_COUNTER, true>(m, n, sp, nw, vars, out, s) : diff_dispatch<F_COUNTER, false>(m, n, sp, nw, vars, out, s); break;
    case F_PLAIN_ISING: I ? diff_dispatch<F_PLAIN_ISING, true>(m, n, sp, nw, vars, out, s) : diff_dispatch<F_PLAIN_ISING, false>(m, n, sp, nw, vars, out, s); break;
    default: I ? diff_dispatch<F_PLAIN_PUBO, true>(m, n, sp, nw, vars, out, s) : diff_dispatch<F_PLAIN_PUBO, false>(m, n, sp, nw, vars, out, s); break;
  }
  return cudaGetLastError();
}

cudaError_t launch_pt_swap(const SwapArgs& a, cudaStream_t s)
{
  const int threads = 128;  // four restarts per block, a warp each
  const int blocks = (a.restarts * 32 + threads - 1) / threads;
  if (blocks <= 0) return cudaGetLastError();
  cudaLaunchAttribute early{};
  early.id = cudaLaunchAttributeProgrammaticStreamSerialization;
  early.val.programmaticStreamSerializationAllowed = 1;
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = dim3((unsigned)blocks);
  cfg.blockDim = dim3((unsigned)threads);
  cfg.stream = s;
  cfg.attrs = &early;
  cfg.numAttrs = 1;
  return cudaLaunchKernelEx(&cfg, pt_swap_kernel, a);
}

// ---------------------------------------------------------------------------
// Allocation-free cost evaluation.  Callers that must not allocate device
// memory while they run -- a serving loop that has handed the free HBM to
// resident solves, or a host thread that cannot afford the device-wide
// synchronisation cudaMalloc / cudaFree bring -- evaluate the cost of states
// that already sit on the device here.  The packed spin words, the only
// scratch the cost kernel needs, go to the fixed file-scope array below
// instead of a buffer allocated per call.
//
// Limits and sharing: the array holds kNoAllocScratchWords 32-bit words
// (1 MiB); a call needs n_states * ceil(n_vars / 32) words, and the entry
// point rejects larger requests before launching.  Every word a call uses
// is written before it is read, so nothing in the array has to start at
// zero.  All calls on one device share the array: calls that overlap in
// time (different streams or host threads) race on it and must be
// serialised by the caller.  The first call on each device looks up the
// array's device address (cudaGetSymbolAddress) with that device current and
// loads the kernel of every model flavour (cudaFuncGetAttributes), so later
// calls load nothing; make that first call before any stream capture.
// ---------------------------------------------------------------------------
static __device__ __align__(256) uint32_t g_noalloc_scratch[kNoAllocScratchWords];

template <int FL, bool INT>
__global__ void eval_cost_noalloc_kernel(DevModel m, int n, const uint8_t* states, int n_vars,
                                         int nw, uint32_t* scratch, double* out)
{
  const int lane = threadIdx.x & 31;
  const int w = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  if (w >= n) return;
  // pack this state's bytes into its own scratch words (coalesced reads)
  const uint8_t* st = states + (size_t)w * n_vars;
  uint32_t* sp = scratch + (size_t)w * nw;
  for (int q = 0; q < nw; q++)
  {
    const int v = q * 32 + lane;
    const unsigned word = __ballot_sync(kFull, v < n_vars && st[v] != 0);
    if (lane == 0) sp[q] = word;
  }
  __syncwarp();
  double c;
  long long ic;
  warp_terms_cost<FL, INT>(m, sp, nullptr, lane, c, ic);
  if (lane == 0) out[w] = INT ? (double)ic : c;
}

template <int FL, bool I>
static void cost_noalloc_dispatch(const DevModel& m, int n, const uint8_t* st, int n_vars, int nw,
                                  uint32_t* scratch, double* out, cudaStream_t s)
{
  int blocks = (n + 3) / 4;
  if (blocks > 0) eval_cost_noalloc_kernel<FL, I><<<blocks, 128, 0, s>>>(m, n, st, n_vars, nw, scratch, out);
}

cudaError_t launch_eval_cost_noalloc(const DevModel& m, int n, const uint8_t* states, int n_vars,
                                     int nw, double* out, cudaStream_t s)
{
  if ((long long)n * (long long)nw > (long long)kNoAllocScratchWords) return cudaErrorInvalidValue;
  // set-up once per device, with that device current: the array's address
  static std::mutex mu;
  static uint32_t* addr[kMaxDevices] = {};
  int dev = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e != cudaSuccess) return e;
  if (dev < 0 || dev >= kMaxDevices) return cudaErrorInvalidDevice;
  uint32_t* scratch = nullptr;
  {
    std::lock_guard<std::mutex> g(mu);
    if (!addr[dev])
    {
      void* p = nullptr;
      e = cudaGetSymbolAddress(&p, g_noalloc_scratch);
      if (e != cudaSuccess) return e;
      // load every flavour's kernel now, so that no later call (another model
      // flavour) loads a module lazily inside a capture
      cudaFuncAttributes fa;
      const void* fns[] = {
          (const void*)eval_cost_noalloc_kernel<F_PARITY, true>,
          (const void*)eval_cost_noalloc_kernel<F_PARITY, false>,
          (const void*)eval_cost_noalloc_kernel<F_COUNTER, true>,
          (const void*)eval_cost_noalloc_kernel<F_COUNTER, false>,
          (const void*)eval_cost_noalloc_kernel<F_PLAIN_ISING, true>,
          (const void*)eval_cost_noalloc_kernel<F_PLAIN_ISING, false>,
          (const void*)eval_cost_noalloc_kernel<F_PLAIN_PUBO, true>,
          (const void*)eval_cost_noalloc_kernel<F_PLAIN_PUBO, false>};
      for (const void* f : fns)
      {
        e = cudaFuncGetAttributes(&fa, f);
        if (e != cudaSuccess) return e;
      }
      addr[dev] = (uint32_t*)p;
    }
    scratch = addr[dev];
  }
  const bool I = m.int_mode != 0;
  switch (m.flavor)
  {
    case F_PARITY: I ? cost_noalloc_dispatch<F_PARITY, true>(m, n, states, n_vars, nw, scratch, out, s) : cost_noalloc_dispatch<F_PARITY, false>(m, n, states, n_vars, nw, scratch, out, s); break;
    case F_COUNTER: I ? cost_noalloc_dispatch<F_COUNTER, true>(m, n, states, n_vars, nw, scratch, out, s) : cost_noalloc_dispatch<F_COUNTER, false>(m, n, states, n_vars, nw, scratch, out, s); break;
    case F_PLAIN_ISING: I ? cost_noalloc_dispatch<F_PLAIN_ISING, true>(m, n, states, n_vars, nw, scratch, out, s) : cost_noalloc_dispatch<F_PLAIN_ISING, false>(m, n, states, n_vars, nw, scratch, out, s); break;
    default: I ? cost_noalloc_dispatch<F_PLAIN_PUBO, true>(m, n, states, n_vars, nw, scratch, out, s) : cost_noalloc_dispatch<F_PLAIN_PUBO, false>(m, n, states, n_vars, nw, scratch, out, s); break;
  }
  return cudaGetLastError();
}
template <int FL, bool I>
static void tabu_dispatch(const TabuArgs& a, cudaStream_t s)
{
  const int blocks = (a.n_walkers + 3) / 4;
  if (blocks > 0) tabu_kernel<FL, I><<<blocks, 128, 0, s>>>(a);
}

cudaError_t launch_tabu(const TabuArgs& a, cudaStream_t s)
{
  if (a.n_walkers <= 0 || a.n_steps <= 0) return cudaSuccess;
  const bool I = a.m.int_mode != 0;
  if (a.m.flavor == F_PARITY && a.m.pair_only && a.m.sweep_size == a.m.n_vars)
  {
    const TabuFit f = tabu_fit(a.m, a.p.nw);
    // as few walkers a block as the SMs need
    const int wpb = std::min(f.warps, std::max(1, (a.n_walkers + 151) / 152));
    // A wave of walkers takes the pair kernel 0.69 of a wave's time on the other one
    // (integers 0.45), but that one's waves are 1216 walkers whatever the model (1.2
    // of a small wave's time when full, in proportion from there on), this one's
    // what fits beside the model.  Other / pair, 60 steps (ms): 1000 spins of 8000
    // couplings, 152 walkers 4.9 / 2.9, 608 5.0 / 11.0; of 5000, 608 3.3 / 2.2, 912 4.0 /
    // 4.2, 2432 10.0 / 8.2; 3000 spins, integers, 456 9.3 / 8.6, 912 11.4 / 13.0, 4096
    // 30 / 57; 1000 spins of 3000, 4096 9.7 / 6.7.
    const int waves = wpb > 0 ? (a.n_walkers + 152 * wpb - 1) / (152 * wpb) : 0;
    if (wpb > 0 && waves * (I ? 0.45 : 0.69) <= (a.n_walkers <= 1216 ? 1.2 : a.n_walkers / 800.0))
    {
      const size_t smem = f.model + wpb * f.walker;
      auto k = I ? tabu_pair_kernel<true> : tabu_pair_kernel<false>;
      const cudaError_t allowed = allow_shared((const void*)k, (int)smem);
      if (allowed != cudaSuccess) return allowed;
      k<<<(a.n_walkers + wpb - 1) / wpb, 32 * wpb, smem, s>>>(a, f.model, f.walker);
      return cudaGetLastError();
    }
  }
  switch (a.m.flavor)
  {
    case F_PARITY: I ? tabu_dispatch<F_PARITY, true>(a, s) : tabu_dispatch<F_PARITY, false>(a, s); break;
    case F_COUNTER: I ? tabu_dispatch<F_COUNTER, true>(a, s) : tabu_dispatch<F_COUNTER, false>(a, s); break;
    case F_PLAIN_ISING: I ? tabu_dispatch<F_PLAIN_ISING, true>(a, s) : tabu_dispatch<F_PLAIN_ISING, false>(a, s); break;
    default: I ? tabu_dispatch<F_PLAIN_PUBO, true>(a, s) : tabu_dispatch<F_PLAIN_PUBO, false>(a, s); break;
  }
  return cudaGetLastError();
}
}  // namespace qio
