// Checks snac_gather_plan.h: for every block of nodes, every pair and every
// node, the hexes the node takes lie inside the pair's run of hexes, and the
// run reaches into no more groups than a stage has room for.
#include <algorithm>
#include <cstdio>

#include "snac_gather_plan.h"

using namespace snac;

int main() {
    const int mesh[][3] = {{1, 1, 1}, {1, 3, 1}, {2, 1, 5}, {3, 2, 1}, {7, 1, 1}, {12, 1, 1}, {13, 1, 2}, {1, 1, 40},
                           {5, 3, 7}, {11, 2, 3}, {13, 5, 11}, {63, 2, 2}, {64, 3, 2}, {16, 8, 16}, {37, 21, 43}};
    long long blocks = 0;
    for (const auto& s : mesh)
        for (int threads : {32, 64, 96, 128, 256}) {
            const int nx = s[0], ny = s[1], nz = s[2], nnx = nx + 1, nny = ny + 1, nn = nnx * nny * (nz + 1);
            for (int n0 = 0; n0 < nn; n0 += threads, blocks++) {
                const int n1 = std::min(n0 + threads, nn) - 1;
                for (int c = 0; c < 4; c++) {
                    int lo, hi;
                    pair_hexes(nx, ny, nz, n0, n1, c, lo, hi);
                    if (hi >= lo && (lo < 0 || hi >= nx * ny * nz)) return printf("run outside the mesh\n"), 1;
                    if (hi >= lo && hi / GROUP - lo / GROUP + 1 > gather_groups(threads)) return printf("too many groups\n"), 1;
                    for (int n = n0; n <= n1; n++) {
                        const int i = n % nnx, j = n / nnx % nny, k = n / (nnx * nny);
                        const int ej = j - 1 + (c & 1), ek = k - 1 + (c >> 1);
                        if (ej < 0 || ek < 0 || ej >= ny || ek >= nz) continue;
                        for (int ei = std::max(i - 1, 0); ei <= std::min(i, nx - 1); ei++) {
                            const int e = ei + (ej + ek * ny) * nx;
                            if (e < lo || e > hi) return printf("hex %d of node %d outside its run\n", e, n), 1;
                        }
                    }
                }
            }
        }
    printf("ok %lld blocks\n", blocks);
    return 0;
}
