// Host check of the block-decided sweep's shared counters
// (qiotoolkit_gb300/csrc/block_turns.h).  Compiled and run by
// tests/test_block_turns_cpu.py; prints one line a check that fails.
#include "../../qiotoolkit_gb300/csrc/block_turns.h"

#include <cstdio>

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

int main()
{
  for (unsigned bufs = 2; bufs <= 4; bufs++)
    for (unsigned stop = 0; stop <= 9; stop++) leave(9, bufs, stop);
  expect(in_flight(2u, 0xFFFFFFFFu) == 3u, "counters that wrap");
  return bad;
}
