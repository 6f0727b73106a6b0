// The ring of shared-memory stages that an operand loader fills with bulk
// copies: chunk c goes to slot c % N, and its arrival completes the phase of
// the slot's mbarrier with parity (c / N) & 1.  A loader that gives a chunk's
// slot away only after the MMAs on it are done has at most one copy in flight
// per slot, the slot's last one: chunks [first_open(issued), issued).
#pragma once

namespace ostc {
namespace tc {

template <int N>
struct StageRing {
  static constexpr int slot(int c) { return c % N; }
  static constexpr unsigned parity(int c) { return static_cast<unsigned>(c / N) & 1u; }
  static constexpr int first_open(int issued) { return issued > N ? issued - N : 0; }
};

}  // namespace tc
}  // namespace ostc
