// waits.cuh - kernels whose bounded waits ran out (they never should).  Each such kernel counts on the device and stores the count to a word
// of host memory, which the host reads without a copy or a synchronisation: the entry points, and the engine behind each step's own
// synchronisation, answer with an error when it has moved, since what the launch left behind is not a result.
#pragma once

namespace b2 {

enum { WAITS_GROUPED = 0, WAITS_PORTIONS = 1, WAITS_KINDS = 2 };

int* wait_word(int kind);                          // for a launch; null when there is no host memory for it
int wait_count(int kind);                          // allocates nothing
int wait_check(int kind, const char* what);        // an error, once, when the count has moved

}  // namespace b2
