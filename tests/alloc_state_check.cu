// Host check of the buffers' state (sim_core.hpp) after an allocation that fails (far more memory than there is,
// or no device at all): prints the size and whether there is memory, before and after.
#include <cstdio>

#include "sim_core.hpp"

namespace sbgpu {
void report_error(int, const std::string&) {}
}  // namespace sbgpu

template <class Buf>
void check(const char* name) {
    Buf b;
    const size_t huge = size_t(1) << 50;
    for (int k = 0; k < 2; ++k) {  // the second time it has to try again
        bool failed = false;
        try {
            k == 0 ? b.alloc(huge) : b.grow(huge);
        } catch (const SbFail&) {
            failed = true;
        }
        std::printf("%s %d %zu %d\n", name, failed ? 1 : 0, b.n, b.p ? 1 : 0);
    }
}

int main() {
    check<DevBuf<double>>("device");
    check<PinnedBuf<double>>("pinned");
    return 0;
}
