// Waits of a block that end, whatever happens, and are reported. Plain C++ around the question "has it happened?", so that a host
// compiler takes it too (the tests run it there, with copies that never land).
//
// The first wait of a block that runs out raises ``gave_up`` and is counted where the host looks, by the thread whose wait it was: nobody
// has to be there afterwards to report it. From then on no wait of the block lasts: every warp stays in step to the end, and what is
// computed is not valid. A thread that has copies under way sees them land (wait_landed) before it leaves, given up or not.
#pragma once

#ifdef __CUDACC__
#define SB_WAIT_FN __device__ __forceinline__
#else
#define SB_WAIT_FN inline
#endif

namespace sb {

// Notes: raise() sets the block's flag and says whether it was the first to do so, raised() reads it, count() tells the host.
template <typename Notes>
SB_WAIT_FN void give_up(Notes& notes) {
  if (notes.raise()) notes.count();
}

template <typename Happened, typename Notes>
SB_WAIT_FN void wait_in_step(Happened happened, Notes& notes, unsigned limit) {
  for (unsigned i = 0; i < limit; ++i) {
    if (happened()) return;
    if ((i & 1023u) == 1023u && notes.raised()) return;
  }
  give_up(notes);
}

template <typename Happened, typename Notes>
SB_WAIT_FN void wait_landed(Happened happened, Notes& notes, unsigned limit) {
  for (unsigned i = 0; i < limit; ++i)
    if (happened()) return;
  give_up(notes);
}

}  // namespace sb
