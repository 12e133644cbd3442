// How the keys of the Llama's split attention are dealt over the CTAs of a cluster (host code without CUDA).
#pragma once
#include <cstddef>

namespace bpdq {

constexpr int kSplitThreads = 256, kSplitWarps = kSplitThreads / 32, kMaxCluster = 16;
constexpr size_t kSplitMaxSmem = 96 * 1024;

struct GqaSplit {
    int ranks, stretch;     // CTAs of a cluster, keys of a CTA
    size_t smem;
    bool fits;              // a CTA's scores in its shared memory: not beyond some number of keys, which the largest cluster sets
};
// clusters: key heads x groups of R query heads x queries; sees: the most keys of a query; D: size of a head; largest: CTAs that a cluster may have.
inline GqaSplit gqa_split(long clusters, int sees, int R, int D, int largest, int sms)
{
    // as many CTAs per cluster as bring a CTA to every SM, while each keeps 64 keys; more where the scores would not fit
    const size_t fixed = (size_t)(kSplitWarps + 1) * R * D * sizeof(float);
    GqaSplit s = {1, 0, 0, false};
    while (s.ranks < largest && clusters * s.ranks < sms && sees > 64 * s.ranks) s.ranks *= 2;
    auto smem_of = [&](int ranks) { return fixed + (size_t)((sees + ranks - 1) / ranks) * R * sizeof(float); };
    while (s.ranks < largest && smem_of(s.ranks) > kSplitMaxSmem) s.ranks *= 2;
    s.stretch = (sees + s.ranks - 1) / s.ranks;
    s.smem = smem_of(s.ranks);
    s.fits = s.smem <= kSplitMaxSmem;
    return s;
}

}  // namespace bpdq
