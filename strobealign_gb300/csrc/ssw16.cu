// k_ssw16's rules of use, and its launches for many tasks.
#include "ssw16.cuh"

namespace sa {

uint32_t ssw16_max_qlen(const AlignScores& sc) {
    if (sc.match == 0 || sc.match > 16 || sc.mismatch > 64 || sc.gap_open <= sc.gap_extend || sc.gap_extend > 31 ||
        sc.gap_extend > 8 * sc.match)
        return 0;
    // a lane of ceil(L / 8) rows
    const uint32_t by_raise = sc.gap_extend ? 8 * (1024u / sc.gap_extend) : SSW16_MAX_QLEN;
    return std::min({SSW16_MAX_QLEN, 1022u / sc.match, by_raise});
}

void launch_ssw16(const Ssw16Args& a, uint32_t longest) {
    if (a.n_tasks < SSW16_PAIR_TASKS && ssw16_default_gaps(a.sc)) launch_ssw16_pair(a, longest);
    else launch_sizes<false>(a, longest);
}

}  // namespace sa
