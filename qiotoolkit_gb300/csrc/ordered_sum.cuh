// ordered_sum.cuh -- FP64 sums in the reference's order without its chain of
// adds.
//
// An FP64 add takes 64 cycles of a scheduler's unit on this chip and waits for
// the one before it, so 32 values added in order take a warp 2100 cycles (and
// warps on one scheduler share the unit).  While the running sum c stays inside
// one binade it is a whole number C of its last place u, and fl(c + d) = (C +
// rint(d / u)) u unless d / u lies halfway between whole numbers: so its
// roundings are a prefix sum of integers, 500 cycles.  A halfway step takes its
// floor there, and one more where the sum's floor is odd (ties go to even), which
// moves the sums after it by one: about 35 cycles each, in order.  Every prefix
// has to stay strictly between 2^52 and 2^53 in magnitude, where the sum before
// rounding lies in the binade too.  Where one does not -- a step out of the
// binade, a sum or value that is subnormal or not finite -- the values before it
// are taken and that one is added as it is.
#pragma once
#include <cstdint>

namespace qio
{
namespace osum
{
static const unsigned long long kOne = 1ULL << 52;

// the sum c as a whole number of its last place, and its exponent field
__device__ __forceinline__ long long scaled(double c, int& ce)
{
  const unsigned long long b = (unsigned long long)__double_as_longlong(c);
  ce = (int)((b >> 52) & 0x7FFu);
  const long long m = (long long)((b & (kOne - 1)) | kOne);
  return (long long)b < 0 ? -m : m;
}
__device__ __forceinline__ double unscaled(long long x, int ce)
{
  const unsigned long long a = (unsigned long long)(x < 0 ? -x : x) & (kOne - 1);
  return __longlong_as_double((long long)(((x < 0 ? 1ULL : 0ULL) << 63) | ((unsigned long long)ce << 52) | a));
}
// rint(d / u) for a sum of exponent field ce (`tie`: halfway, its floor); false:
// not to be had this way
__device__ __forceinline__ bool step_of(double d, int ce, long long& D, bool& tie)
{
  const unsigned long long b = (unsigned long long)__double_as_longlong(d);
  D = 0;
  tie = false;
  if ((b << 1) == 0ULL) return true;
  const int de = (int)((b >> 52) & 0x7FFu), sh = ce - de;
  if (de == 0 || de == 0x7FF || sh < 0) return false;  // (|D| < 2^53: no sum of 32 overflows)
  if (sh > 53) return true;
  const unsigned long long m = (b & (kOne - 1)) | kOne;
  if (sh > 0)
  {
    const unsigned long long rem = m & ((1ULL << sh) - 1ULL), half = 1ULL << (sh - 1);
    tie = rem == half;
    D = (long long)((m >> sh) + (rem > half || (tie && (long long)b < 0) ? 1ULL : 0ULL));
  }
  else D = (long long)m;
  if ((long long)b < 0) D = -D;
  return true;
}
// P, of the sign of C, is a prefix inside C's binade
__device__ __forceinline__ bool inside(long long C, long long P)
{
  const long long mag = C < 0 ? -P : P;
  return mag > (long long)kOne && mag < (long long)(kOne << 1);
}
// the sums' prefixes over all lanes, from C and the lanes' steps
__device__ __forceinline__ long long prefix(long long C, long long x, bool tie)
{
  const int lane = threadIdx.x & 31;
#pragma unroll
  for (int d = 1; d < 32; d <<= 1)
  {
    const long long y = __shfl_up_sync(0xffffffffu, x, d);
    if (lane >= d) x += y;
  }
  x += C;
  for (unsigned T = __ballot_sync(0xffffffffu, tie); T; T &= T - 1u)
  {
    const int f = __ffs(T) - 1;
    if ((__shfl_sync(0xffffffffu, (int)x, f) & 1) != 0 && lane >= f) x++;
  }
  return x;
}

// c plus the values of the lanes in `keep`, lane by lane; the same c on all
// lanes
__device__ __forceinline__ void add_lanes(double v, unsigned keep, double& c)
{
  const unsigned kAll = 0xffffffffu;
  const int lane = threadIdx.x & 31;
  // Three prefixes at most, and none after one that took eight values or fewer: a
  // sum near zero changes its binade often, and a prefix costs as much as eight
  // adds.  Initial costs of 8 walkers, terms of both signs (us): 256 Ising terms 65
  // and 62, 1024 PUBO terms 91 and 71, 4096 147 and 120.
  bool worth = true;
  for (int round = 0; round < 3 && worth && __popc(keep) > 4; round++)
  {
    int ce;
    const long long C = scaled(c, ce);
    const bool mine = ((keep >> lane) & 1u) != 0u;
    long long D = 0;
    bool ok = true, tie = false;
    if (ce == 0 || ce == 0x7FF) ok = false;
    else if (mine) ok = step_of(v, ce, D, tie);
    const long long P = prefix(C, D, tie);
    const unsigned bad = __ballot_sync(kAll, mine && !(ok && inside(C, P)));
    if (bad == 0u)
    {
      c = unscaled(__shfl_sync(kAll, P, 31), ce);
      return;
    }
    const int f = __ffs(bad) - 1;
    if (f > 0 && ce != 0 && ce != 0x7FF) c = unscaled(__shfl_sync(kAll, P, f - 1), ce);
    c = __dadd_rn(c, __shfl_sync(kAll, v, f));
    worth = __popc(keep & ((2u << f) - 1u)) > 8;
    keep &= ~((2u << f) - 1u);
  }
  while (keep)
  {
    const int j = __ffs(keep) - 1;
    keep &= keep - 1;
    c = __dadd_rn(c, __shfl_sync(kAll, v, j));
  }
}
}  // namespace osum
}  // namespace qio
