// block_turns.h -- how the sweep kernels count a walker's blocks (fields.cu,
// sweep.cu), apart from the kernels so that a host program can check it.
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

// A warp's place among a walker's blocks, sweep by sweep, and the buffer and
// mbarrier phase of its chunk, which go on from walker to walker.  There is no
// product of blocks and sweeps: the sweeps of one launch may have more than
// 2^31 blocks.
struct Turns
{
  int nblocks, bufs;
  int block = 0;       // the coming block
  int sweep = 0;       // ... of the launch's sweeps
  unsigned buf = 0;    // its buffer
  unsigned phase = 0;  // ... and that buffer's phase

  QIO_HD Turns(int blocks_, int bufs_) : nblocks(blocks_), bufs(bufs_) {}
  // the next walker's first block
  QIO_HD void walker(int blocks_)
  {
    nblocks = blocks_;
    block = sweep = 0;
  }
  QIO_HD void next_block()
  {
    const bool end = ++block == nblocks;
    block = end ? 0 : block;
    sweep += end ? 1 : 0;
  }
  QIO_HD void next_buffer()
  {
    const bool end = ++buf == (unsigned)bufs;
    buf = end ? 0u : buf;
    phase ^= end ? 1u : 0u;
  }
  QIO_HD void next()
  {
    next_block();
    next_buffer();
  }
  // the buffer and phase of n chunks before, n <= bufs
  QIO_HD void back(unsigned n)
  {
    phase ^= buf < n ? 1u : 0u;
    buf = buf < n ? buf + (unsigned)bufs - n : buf - n;
  }
};
}  // namespace fc
}  // namespace qio
