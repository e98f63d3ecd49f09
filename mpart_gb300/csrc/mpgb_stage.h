// Shared-memory staging of phase A: how many doubles a launch takes.
#pragma once
#include <algorithm>
#include <cstddef>

namespace mpgb {

// Largest phase-A staging (coefficient doubles plus table words) a fused
// launch keeps in shared memory.
constexpr int kStageCap = 2048;
// Smallest staging the fixed-point phase A works with (its chunks of nodes).
constexpr int kStageMin = 256;
constexpr size_t kSmemPerBlock = 227 * 1024;

// The doubles the components of a map ask for.  FP64 (phaseAStaged): the whole
// component's coefficients and two words a node, or nothing.  Limbs
// (phaseALimbs): 16 bytes a node and two nodes of look-ahead, in chunks of any
// size from kStageMin.
struct StageNeed {
    int fp64 = 0, limbs = 0;
    void add(int nSlots, int nNodes) {
        if (nSlots + nNodes <= kStageCap) fp64 = std::max(fp64, nSlots + nNodes);
        limbs = std::max(limbs, std::max(kStageMin, std::min(kStageCap, nSlots + 2 * (nNodes + 2))));
    }
};

// The largest staging that does not lower the number of blocks an SM holds (at
// most maxBlocks; `base` bytes a block without it).  A launch with limbs takes
// halves of its need down to kStageMin, and kStageMin in any case: it has no
// other form.  One without takes all or nothing: sized for limbs, an 8-D order-4
// map of Hermite functions did not stage its largest component (825 doubles of
// room asked for and 579 given), and a 12-D order-3 one ran three blocks an SM
// instead of four for 256 doubles that none of its larger components can use.
inline int stageRoom(const StageNeed& need, bool limbs, size_t base, size_t smemPerSM, size_t maxBlocks) {
    const int want = limbs ? need.limbs : need.fp64;
    if (want == 0 || smemPerSM == 0) return 0;
    auto blocks = [&](size_t b) { return std::min(maxBlocks, smemPerSM / b); };
    auto fits = [&](int n) {
        const size_t with = base + (size_t)n * sizeof(double);
        return with <= kSmemPerBlock && blocks(with) == blocks(base);
    };
    if (!limbs) return fits(want) ? want : 0;
    for (int n = want; n >= kStageMin; n /= 2)
        if (fits(n)) return n;
    return base + kStageMin * sizeof(double) <= kSmemPerBlock ? kStageMin : 0;
}

}  // namespace mpgb
