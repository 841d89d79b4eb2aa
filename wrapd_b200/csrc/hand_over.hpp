// Host side of the scalars' hand-over (SolverGPU::await_publish): words in pinned
// memory that a launch fills one by one, in any order.
#pragma once

namespace wrapd {

// Copies n words to out, looking at each until it is no longer `unset`.  Every 4096
// looks asks ended(), which says whether the work that writes the words has ended
// (it may wait for that, or throw): a word still unset after that never comes, and
// the result is false; out then holds nothing of use.
template <typename Ended>
bool take_words(const volatile unsigned long long* words, int n, unsigned long long unset, unsigned long long* out,
                Ended&& ended) {
    for (int k = 0; k < n; ++k) {
        unsigned long long w = words[k];
        for (int i = 1; w == unset; ++i) {
            const bool over = i % 4096 == 0 && ended();
            w = words[k];
            if (over && w == unset) return false;
        }
        out[k] = w;
    }
    return true;
}

}  // namespace wrapd
