// Host check of mlp_gemm_args_ok (sb_mlp.h): a call of each mode with everything it needs, then without one
// array at a time; prints "mode array accepted" lines.
#include <cstdio>
#include <functional>

#include "sb_mlp.h"

using namespace sbgpu;

int main() {
    alignas(16) static char memory[16];
    auto at = [&](auto* p) { return reinterpret_cast<decltype(p)>(memory); };
    const char* names[] = {"none", "A", "B", "bias", "z_out", "h_out", "hT_out", "z_in", "part_out"};
    for (int mode = 0; mode < 3; ++mode)
        for (int k = 0; k < 9; ++k) {
            GemmArgs g;
            g.A = g.B = at(static_cast<bf16*>(nullptr));
            g.lda = g.ldb = g.K = g.k_split = 256;
            g.M = 128;
            g.N = 256;
            g.ldt = 128;
            g.mode = mode;
            g.bias = g.z_in = g.z_out = g.part_out = at(static_cast<float*>(nullptr));
            g.h_out = g.hT_out = at(static_cast<bf16*>(nullptr));
            std::function<void()> drop[] = {[] {}, [&] { g.A = nullptr; }, [&] { g.B = nullptr; }, [&] { g.bias = nullptr; },
                                            [&] { g.z_out = nullptr; }, [&] { g.h_out = nullptr; }, [&] { g.hT_out = nullptr; },
                                            [&] { g.z_in = nullptr; }, [&] { g.part_out = nullptr; }};
            drop[k]();
            std::printf("%d %s %d\n", mode, names[k], mlp_gemm_args_ok(g) ? 1 : 0);
        }
    return 0;
}
