// Host check of the refined Linearized solve's rows (sb_lin_layout.h): for "N C" lines on stdin, prints the
// elements of the residual and the correction in shared memory and then, per CTA, the rows of the system that
// its rows are.
#include <cstdio>

#include "sb_lin_layout.h"

int main() {
    int N, C;
    while (std::scanf("%d %d", &N, &C) == 2) {
        const sbgpu::LinLayout L = sbgpu::LinLayout::make(N, C);
        std::printf("%zu %zu\n", (L.dx - L.rv) / 4, (L.vel - L.dx) / 4);
        for (int rank = 0; rank < C; ++rank) {
            for (int l = 0; l < sbgpu::lin_own_rows(N, C, rank); ++l) std::printf("%d ", sbgpu::lin_row(l, rank, C));
            std::printf("\n");
        }
    }
    return 0;
}
