// How the two softmax warps that share rows agree on what a tile needs (attention_prefill.cu, attention_wide.cu).
//
// A tile is taken in one round, or in two where its sum of P shows that the reference maximum is far too low; a round that
// searches the maximum has a barrier of the pair in it, and every round ends with a vote of the pair.  Those barriers have no limit,
// so the two warps have to meet at the same ones whatever their waits for mbarriers give: one warp may find a phase complete where
// the other has just been told that the block gives up.  A warp whose wait gave up therefore goes on to the votes, and the pair
// leaves the walk over the tiles together.
//
// The vote behind a search looks at the block's flag, which a wait that gives up has raised or seen raised, instead of a word of the
// warp's own: such a word, held through the softmax, cost attention_prefill.cu 7 % (32 heads of 2,048 tokens 43.3 -> 46.3 us; with
// the flag 43.8).
#pragma once

#ifdef __CUDACC__
#define ERB_PAIR_FN __host__ __device__ __forceinline__
#else
#define ERB_PAIR_FN inline
#endif

namespace erb {

class PairRounds {
 public:
  ERB_PAIR_FN explicit PairRounds(bool has_no_reference) : search_(has_no_reference) {}
  // Whether this round searches the tile's maximum (with the barrier that takes).
  ERB_PAIR_FN bool search() const { return search_; }
  // What a warp votes at the end of a round; low: its sum asks for a higher reference (not asked behind a search).  A warp whose
  // wait for the scores gave up votes true in every round.
  ERB_PAIR_FN bool vote(bool low, volatile const int* block_gave_up) const { return search_ ? *block_gave_up != 0 : low; }
  // Behind a vote that said yes: whether there is another round, with a search.  No: the pair leaves the walk (behind a search only
  // a warp that gave up can have said yes).
  ERB_PAIR_FN bool again() {
    const bool more = !search_;
    search_ = true;
    return more;
  }

 private:
  bool search_;
};

}  // namespace erb
