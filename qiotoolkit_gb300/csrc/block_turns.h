// block_turns.h -- counters that the warps of a block-decided sweep share
// (fields.cu), apart from the kernel so that a host program can check them.
#pragma once

#ifdef __CUDACC__
#define QIO_HD __host__ __device__ __forceinline__
#else
#define QIO_HD inline
#endif

namespace qio
{
namespace fc
{
// Chunks whose copies the feeder may not leave behind: those issued that the
// decider has not finished with.  None once a walker is done; a decider that
// gave up raises `abort` and `done` both, with up to all buffers' copies in
// flight.  Counters wrap.
QIO_HD unsigned in_flight(unsigned issued, unsigned finished) { return issued - finished; }
}  // namespace fc
}  // namespace qio
