// Model of a loader that gives up: `issued` chunks went through a ring of N
// slots, the copies of all but each slot's last use have landed (the MMAs have
// read them), the others land in any order while the drain waits.  An mbarrier
// parity wait passes when the phase in progress has the other parity.
#include <cstdio>
#include <functional>

#include "device/stage_ring.hpp"

using ostc::tc::StageRing;

template <int N>
struct Ring {
  int landed[N] = {}, started[N] = {};
  Ring(int issued, unsigned arrived) {
    for (int c = 0; c < issued; ++c) ++started[StageRing<N>::slot(c)];
    for (int s = 0; s < N; ++s) landed[s] = started[s] - (started[s] > 0 && !(arrived >> s & 1) ? 1 : 0);
  }
  // the wait of the drain: a copy in flight lands if that lets it pass
  void wait(int s, unsigned parity) {
    if ((landed[s] & 1u) == parity && landed[s] < started[s]) ++landed[s];
  }
  bool in_flight() const {
    for (int s = 0; s < N; ++s)
      if (landed[s] < started[s]) return true;
    return false;
  }
};

// cases in which a drain leaves a copy in flight
template <int N>
int left(int chunks, const std::function<void(Ring<N> &, int)> &drain) {
  int bad = 0;
  for (int issued = 0; issued <= chunks; ++issued)
    for (unsigned arrived = 0; arrived < (1u << N); ++arrived) {
      Ring<N> r(issued, arrived);
      drain(r, issued);
      bad += r.in_flight();
    }
  return bad;
}

template <int N>
int drained(int chunks) {
  return left<N>(chunks, [](Ring<N> &r, int issued) {
    for (int c = StageRing<N>::first_open(issued); c < issued; ++c)
      r.wait(StageRing<N>::slot(c), StageRing<N>::parity(c));
  });
}

int main() {
  // the layer kernels (2 slots, 1 or 4 chunks) and the weight gradients (3 slots)
  int bad = drained<2>(1) + drained<2>(4) + drained<2>(9);
  for (int n = 0; n < 40; ++n) bad += drained<3>(n);
  // mistakes the model has to see: the first phase of each slot, and the last
  // chunks of the whole range instead of the last ones that were started
  const int first = left<2>(4, [](Ring<2> &r, int) {
    for (int s = 0; s < 2; ++s) r.wait(s, 0);
  });
  const int range = left<3>(10, [](Ring<3> &r, int) {
    for (int c = 7; c < 10; ++c) r.wait(c % 3, static_cast<unsigned>(c / 3) & 1u);
  });
  std::printf("left in flight %d, planted mistakes seen %d %d\n", bad, first > 0, range > 0);
  return bad == 0 && first > 0 && range > 0 ? 0 : 1;
}
