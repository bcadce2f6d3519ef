// k_ssw16's rules of use, and its launches for many tasks.
#include "ssw16.cuh"

namespace sa {

uint32_t ssw16_max_qlen(const AlignScores& sc) {
    if (sc.match == 0 || sc.match > 16 || sc.mismatch > 64 || sc.gap_open <= sc.gap_extend || sc.gap_extend > 31 ||
        sc.gap_extend > 8 * sc.match)
        return 0;
    return std::min<uint32_t>(SSW16_MAX_QLEN, 1022u / sc.match);
}

void launch_ssw16(const Ssw16Args& a, uint32_t longest) {
    if (a.n_tasks < SSW16_PAIR_TASKS && ssw16_default_gaps(a.sc)) launch_ssw16_pair(a, longest);
    else launch_sizes<false>(a, longest);
}

}  // namespace sa
