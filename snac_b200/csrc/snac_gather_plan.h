// snac_gather_plan.h — which groups of hexes a block of the node gathers
// reads (plain C++, so that the host can check it node by node).
//
// Nodes are numbered i + j nnx + k nnx nny and hexes i + j nx + k nx ny.  A node
// (i, j, k) takes terms from up to eight hexes, in four pairs: pair c = 0..3 is
// the hexes (i-1, ej, ek) and (i, ej, ek) with ej = j - 1 + (c & 1) and
// ek = k - 1 + (c >> 1).  Both numberings run row by row, so the hexes that
// the consecutive nodes [n0, n1] of a block take in pair c are a run of
// consecutive hexes, at most one more than the nodes (a row has one hex
// fewer than nodes, and the first node also takes the hex before it).
#pragma once

#ifdef __CUDACC__
#define SNAC_HD __host__ __device__ __forceinline__
#else
#define SNAC_HD inline
#endif

namespace snac {

constexpr int GROUP = 12;  // hexes of an element block, and of a group of per-tet terms

// most groups that `nodes` consecutive nodes touch in one pair: nodes + 1
// consecutive hexes reach into ceil(nodes / GROUP) + 1 groups
SNAC_HD constexpr int gather_groups(int nodes) { return (nodes + GROUP - 1) / GROUP + 1; }

// The run of hexes [lo, hi] that nodes n0..n1 take in pair c (hi < lo: none).
SNAC_HD void pair_hexes(int nx, int ny, int nz, int n0, int n1, int c, int& lo, int& hi) {
    const int nnx = nx + 1, nny = ny + 1;
    {   // the first hex any node from n0 on takes
        const int q = n0 / nnx, i = n0 - q * nnx, k = q / nny, j = q - k * nny;
        int ei = i > 0 ? i - 1 : 0, ej = j - 1 + (c & 1), ek = k - 1 + (c >> 1);
        if (ej < 0) { ej = 0; ei = 0; }
        if (ej >= ny) { ek++; ej = 0; ei = 0; }
        if (ek < 0) { ek = 0; ej = 0; ei = 0; }
        lo = ek >= nz ? nx * ny * nz : ei + (ej + ek * ny) * nx;
    }
    {   // the last hex any node up to n1 takes
        const int q = n1 / nnx, i = n1 - q * nnx, k = q / nny, j = q - k * nny;
        int ei = i < nx ? i : nx - 1, ej = j - 1 + (c & 1), ek = k - 1 + (c >> 1);
        if (ej >= ny) { ej = ny - 1; ei = nx - 1; }
        if (ej < 0) { ek--; ej = ny - 1; ei = nx - 1; }
        if (ek >= nz) { ek = nz - 1; ej = ny - 1; ei = nx - 1; }
        hi = ek < 0 ? -1 : ei + (ej + ek * ny) * nx;
    }
}

}  // namespace snac
