/*
 * decode_tags.h — the tags of the words through which the CTAs of decode_stack.cuh exchange
 * logits and chains, and when those words are cleared.  Plain C++, so that a test without a GPU
 * can take the counter through its whole range.
 *
 * A layer's tag is what the round counter has to reach at the layer's first barrier.  The counter
 * has 32 bits and a round is worth DF_ROUND of it, so tags come again after 2^24 rounds: some
 * 215 000 steps of 40 layers, minutes of decoding.  A word that was written then and not since
 * (rows of tokens that have not been in use, far places of a token's list of chains) would pass as
 * this layer's.  So every launch that begins in the last CLEAR_ROUNDS rounds of the counter's
 * range clears all words first, behind a barrier of its own.
 *
 * That is enough.  A launch takes at most 2 * DS_LAYERS rounds, so of the launches that begin
 * in those rounds (there are several, as CLEAR_ROUNDS is eight times that) one comes after any
 * launch that began before them, and after any that ended within the first seven eighths of
 * them.  A word written by one of those is cleared before its tag comes again.  A word written
 * later has a tag of the last eighth, and whoever uses that tag again begins in the same rounds
 * and clears first; or it has a tag from behind the wrap, and is one of the next turn's.
 */
#pragma once
#include "exact_codes.h"

namespace apus {

constexpr unsigned DF_ROUND = 256;      /* >= the number of CTAs, a power of two */
constexpr int DS_LAYERS = 32;           /* layers of a launch, at most (parameter space) */
constexpr unsigned CLEAR_ROUNDS = 512;
static_assert(CLEAR_ROUNDS >= 8 * 2 * DS_LAYERS, "see above");

/* target: the counter at the end of a round, a multiple of DF_ROUND.  Never zero, which is what
 * words hold that nobody has written. */
APUS_HD unsigned stack_tag(unsigned target) { return target | 1u; }
/* ... at the end of a launch's first round */
APUS_HD bool stack_clears(unsigned target) { return target >= 0u - CLEAR_ROUNDS * DF_ROUND; }

}  // namespace apus
