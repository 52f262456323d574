// Bookkeeping of the exchanges between the CTAs of a cluster (lnt_cluster.cu), shared with the host
// model that checks it (tests/native/cluster_exchange_selftest.cpp).
//
// A squaring makes three exchanges, so exchange e of a launch belongs to squaring e / 3 and counts
// towards barrier e mod 3: blocks, segments, boundary carries.  A CTA sends exchange e completely or
// not at all, and goes on to e + 1 only when its own part of e has arrived.  When a wait gives up the
// CTA sends nothing more and re-arms nothing, but words may still be on their way to it, and shared
// memory may not go while they are.  From what each CTA sent it follows which words will never come:
// they are taken off the barriers' counts by hand, and the phases then complete when the last word
// that is on its way has landed.
#pragma once
#include <stdint.h>

#include "goldilocks.cuh"

namespace lnt {
namespace cluster {

// exchanges of barrier b among the first `count` ones
GL_HD uint64_t rounds(uint64_t count, int b) { return (count + 2 - (uint64_t)b) / 3; }

// phases of barrier b that a CTA has armed after `passed` exchanges: one ahead of what has arrived
GL_HD uint64_t armed(uint64_t passed, int b) { return rounds(passed, b) + 1; }

// bytes that CTA `from` sends to CTA `to` towards barrier b in one squaring; C CTAs of m words
GL_HD uint32_t bytes_sent(int b, uint32_t from, uint32_t to, uint32_t C, uint32_t m) {
  if (b < 2) return 8 * m / C;
  return (from + 1) % C == to ? 8 * C : 0;  // a segment's last carry goes to the next CTA
}

// Bytes of the armed phase of barrier b that never come to CTA `to`: those of the CTAs that left
// before sending them.  sent[c]: exchanges that CTA c sent.  No CTA sends a round of b later than
// the armed one: it would need words that `to` sends only after arming that round.
GL_HD uint32_t bytes_missing(int b, uint64_t passed, const uint64_t* sent, uint32_t to, uint32_t C, uint32_t m) {
  uint32_t bytes = 0;
  for (uint32_t c = 0; c < C; ++c)
    if (rounds(sent[c], b) < armed(passed, b)) bytes += bytes_sent(b, c, to, C, m);
  return bytes;
}

}  // namespace cluster
}  // namespace lnt
