// Host check of the block-decided sweep's shared counters
// (qiotoolkit_gb300/csrc/block_turns.h).  Compiled and run by
// tests/test_block_turns_cpu.py; prints one line a check that fails.
#include "../../qiotoolkit_gb300/csrc/block_turns.h"

#include <cstdio>
#include <initializer_list>

using namespace qio::fc;

static int bad = 0;
static void expect(bool ok, const char* what)
{
  if (!ok)
  {
    std::printf("%s\n", what);
    bad = 1;
  }
}

// A feeder with `bufs` buffers runs `total` blocks ahead of a decider that gives
// up in block `stop` (total: never): copies that it may not leave behind
static void leave(unsigned total, unsigned bufs, unsigned stop)
{
  unsigned issued = 0, finished = 0;
  while (true)
  {
    while (issued < total && in_flight(issued, finished) < bufs) issued++;
    if (finished == stop || finished == total) break;
    finished++;
  }
  const unsigned left = in_flight(issued, finished);
  expect(left == (stop < total ? (total - stop < bufs ? total - stop : bufs) : 0u), "chunks in flight at the end");
}

// A launch's blocks, sweep by sweep: as many as there are, in order, with the
// buffers in turn and a phase that changes each time round
static void walk(int nblocks, int sweeps, int bufs)
{
  Turns T(nblocks, bufs);
  long long n = 0;
  for (; T.sweep < sweeps; T.next()) n++;
  const long long want = (long long)nblocks * sweeps;
  expect(n == want, "blocks of a launch");
  expect(T.block == 0 && T.sweep == sweeps, "place after a launch");
  expect(T.buf == (unsigned)(want % bufs) && T.phase == (unsigned)(want / bufs % 2), "buffer and phase after a launch");
}

// Buffers and phases go on from walker to walker, and back by up to `bufs`
static void walkers(int bufs)
{
  Turns T(1, bufs);
  long long at = 0;
  for (int blocks : {1, 3, 2, 7, 1})
  {
    T.walker(blocks);
    for (; T.sweep < 3; T.next(), at++)
    {
      expect(T.buf == (unsigned)(at % bufs) && T.phase == (unsigned)(at / bufs % 2), "buffer and phase of a chunk");
      for (int n = 0; n <= bufs && n <= at; n++)
      {
        Turns U = T;
        U.back((unsigned)n);
        expect(U.buf == (unsigned)((at - n) % bufs) && U.phase == (unsigned)((at - n) / bufs % 2), "chunks before");
      }
    }
  }
}

int main()
{
  // 8000 variables, 9 million sweeps: 2250 million blocks; 1024 blocks, 4.2 million
  // sweeps: 2^32 and some more
  walk(250, 9000000, 4);
  walk(1024, 4200000, 3);
  walk(1, 5, 2);
  for (int bufs = 2; bufs <= 4; bufs++) walkers(bufs);

  for (unsigned bufs = 2; bufs <= 4; bufs++)
    for (unsigned stop = 0; stop <= 9; stop++) leave(9, bufs, stop);
  expect(in_flight(2u, 0xFFFFFFFFu) == 3u, "counters that wrap");
  return bad;
}
