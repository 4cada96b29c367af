// Whether work that later calls of a handle rely on has been done.
#pragma once

namespace mpm {

// Work submitted to a stream is done for every later call.  Work recorded in a stream
// capture is done for the calls of the same capture only: the graph may be discarded,
// or replayed at any later time.  Captures are told apart by CUDA's capture id (0: no
// capture).
struct Done {
  bool run = false;
  unsigned long long recorded = 0;
  bool holds(unsigned long long capture) const { return run || (capture != 0 && capture == recorded); }
  void mark(unsigned long long capture) {
    if (capture != 0)
      recorded = capture;
    else
      run = true;
  }
};

// A state that each call needs and leaves behind it (the p2g grid and the block flags
// are zero).  begin() says whether the state holds for a call in this capture, else the
// call makes it first; until end() it is unknown, as it stays after a call that failed.
struct Restored {
  Done now, before;
  bool begin(unsigned long long capture) {
    before = now;
    now = Done{};
    return before.holds(capture);
  }
  void end(unsigned long long capture) {
    now = before;
    now.mark(capture);
  }
};

}  // namespace mpm
