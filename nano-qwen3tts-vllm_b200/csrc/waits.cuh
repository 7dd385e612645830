// waits.cuh - kernels whose bounded waits ran out (they never should).  Each such kernel counts on the device and stores the count to a word
// of host memory, which the host reads without a copy or a synchronisation: the entry points, and the engines behind each step's own
// synchronisation, answer with an error when it has moved, since what the launch left behind is not a result.
#pragma once

namespace b2 {

enum { WAITS_GROUPED = 0, WAITS_PORTIONS = 1, WAITS_ROWS = 2, WAITS_KINDS = 3 };
constexpr int WAIT_DEVICES = 64;                   // as many as sm_count() knows; later ones share the last word

// Words lie [device][kind]: every device counts for itself, so two of them must not store to the same word (the second one's first
// lost wait would store the number that is there already).
inline int wait_slot(int device, int kind) { return (device < 0 ? 0 : device < WAIT_DEVICES ? device : WAIT_DEVICES - 1) * WAITS_KINDS + kind; }
inline int wait_total(const volatile int* words, int kind) {
  int n = 0;
  for (int d = 0; d < WAIT_DEVICES; ++d) n += words[wait_slot(d, kind)];
  return n;
}
// whether the count differs from the one that was told last; it is told by this call
inline bool wait_moved(const volatile int* words, int kind, int* told) {
  const int n = wait_total(words, kind);
  return __atomic_exchange_n(told, n, __ATOMIC_RELAXED) != n;
}

int* wait_word(int kind);                          // the current device's, for a launch; null when there is no host memory for it
int wait_count(int kind);                          // of all devices; allocates nothing
int wait_check(int kind, const char* what);        // an error, once, when the count has moved

}  // namespace b2
