// k_ssw16 for few tasks: the byte and the word passes of a task at once.
#include "ssw16.cuh"

namespace sa {

void launch_ssw16_pair(const Ssw16Args& a, uint32_t longest) { launch_sizes<true>(a, longest); }

}  // namespace sa
