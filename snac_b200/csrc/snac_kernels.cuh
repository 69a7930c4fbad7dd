// snac_kernels.cuh — the kernels of one SNAC step (reference rounding).
//
// Per step, in _Snac_Context_Solve order (Snac/libSnac/src/Context.c:1063-1099):
//   k_heat_flux      Snac_EP_LoopElementsEnergy  temperature/HeatFlux.c:47-200 + HeatFluxBC
//   k_heat_nodes     Snac_EP_LoopNodesEnergy     temperature/Heat.c:47-140
//   k_calc_stresses  Snac_EP_CalcStresses        StrainRate.c + Stress.c + the constitutive hook
//   k_loop_nodes     Snac_EP_LoopNodesMomentum   Force.c + UpdateNode.c
//   k_update_elements Snac_EP_LoopElementsMomentum UpdateElement.c
//   k_sync           AbstractContext_EP_Sync     Context.c:1208-1268
// In a steady step the element update of step n runs fused with the stress
// update of step n+1 (k_fused_step; with temperature k_heat_flux, k_heat_nodes,
// then k_fused_stress, since neither energy hook reads the stress), and the
// minimum length scale of the element update runs fused with Sync
// (k_min_length_scale_sync).
//
// Element kernels run one thread per tetrahedron: a warp holds three
// elements in lanes 0-9, 10-19, 20-29 (lanes 30-31 idle).  Element sums
// (volume, traces) go through shared memory and are added in the
// reference's tet order, so they round like the reference's loops.  Node
// kernels run one thread per node and gather the 8 adjacent hexes x 5 tets in
// the reference's fixed order (Force.c:87-181): no atomics, bit-reproducible.
//
// Geometry (volumes, face areas and normals) is never stored: each kernel
// recomputes it from the coordinates with the reference's formulas, which
// gives the same bits the reference stored in its element structs.
#pragma once

#include "snac_device.cuh"
#include "snac_gather_plan.h"

namespace snac {

struct Mesh {
    int nx, ny, nz, nnx, nny, nnz;
    long long ne, nn;
    int frows;      // rows of a force group: 130 (Config::vonly), 140, or 170 (constant dt)
};

// Per-tet force and energy terms are stored by groups of GROUP hexes (one
// element block each), in rows of GROUP entries: a block's rows leave as one
// contiguous copy.  A tet corner's term (a node takes it from face f of tet t)
// belongs to one of the node gather's four pairs c of hexes (snac_gather_plan.h),
// and the ten corners of a pair are neighbouring rows, so that the gather
// fetches what it needs of a group as one contiguous chunk too:
//   force group: 4 chunks of [3 components][10 corners] rows (constant dt:
//     4 kinds, the inertial-mass term the last), then rows of the ten tets: g rho V / 8
//     (the volume alone with Config::vonly) and, unless vonly or constant dt,
//     the inertial-mass term;
//   heat group: 4 chunks of [10 corners] rows (face energy terms), then Cp rho V / 8 and
//     the thermal stress of the ten tets.
// pair_slot(ne, idx): the place of corner (node_tet, node_face)(ne, idx) among
// the ten of pair ne / 2, chosen so that the element kernels' stores, ten tets times three
// hexes of a row each, fall three to a bank (the least that rows of 12 allow).
__host__ __device__ constexpr int pair_slot(int ne, int idx) {
    constexpr int tab[8][5] = {{0, 6, 4, 3, 1}, {2, 9, 7, 8, 5}, {7, 3, 6, 2, 4}, {1, 8, 5, 0, 9},
                               {7, 0, 4, 6, 2}, {1, 3, 8, 9, 5}, {5, 1, 0, 3, 7}, {2, 9, 4, 8, 6}};
    return tab[ne][idx];
}
// byte f: 16 * pair + slot of the corner that takes face f of tet t
__host__ __device__ constexpr unsigned tet_slots(int t) {
    unsigned w = 0;
    for (int ne = 0; ne < 8; ne++)
        for (int idx = 0; idx < 5; idx++)
            if (node_tet(ne, idx) == t) w |= (unsigned)(16 * (ne / 2) + pair_slot(ne, idx)) << (8 * node_face(ne, idx));
    return w;
}
__device__ const unsigned TET_SLOTS[NT] = {tet_slots(0), tet_slots(1), tet_slots(2), tet_slots(3), tet_slots(4),
                                           tet_slots(5), tet_slots(6), tet_slots(7), tet_slots(8), tet_slots(9)};
// entry of row 0 of the corner that takes face f, in chunks of `rows` rows
__device__ __forceinline__ int corner_row(unsigned slots, int f, int rows) {
    const unsigned v = slots >> (8 * f);
    return (int)((v >> 4) & 3u) * (rows * GROUP) + (int)(v & 15u) * GROUP;
}

struct Fields {
    const double4* pos;      // current coordinates (x, y, z) and temperature (w)
    double4* pos_next;       // written by k_loop_nodes (coordinates are double-buffered)
    double4* vel;            // velocity (x, y, z) and temperature0 (w)
    double4* force;          // damped force (x, y, z) and inertial mass (w)
    double* stress;          // [ne*10][6]
    double* eps_p;           // [ne*10]  plastic strain (plastic, visco-plastic)
    double* pst;             // [ne*10][6] plastic strain tensor (visco-plastic with a Drucker-Prager phase)
    double* visc;            // [ne*10]  viscosity (visco-plastic, Maxwell)
    double* density;         // [ne*10]  only when some phase has alpha or beta != 0
    double* vol;             // [ne*10][2] volume, old volume (Maxwell)
    double* hflux;           // heat groups of HROWS rows
    double* tpre;            // [nn] temperature before the BCs (temperature + density)
    double* fterm;           // force groups of Mesh::frows rows: stress.n.A/6 (Force.c:154-165), g rho V/8 (:173),
                             // the inertial-mass term (:107-140)
    const uchar4* bc;        // per node: velocity-VC index of x, y, z and temperature-VC index (255 = free)
    const double* vbc_val;   // [n_vc][3]
    const double* tbc_val;   // [n_tc]
    const unsigned char* mat;        // [ne] phase, NULL = 0
    const DevMaterial* mats;         // phase table of this model
    double* residual_fr;             // [nn] Winkler residual force of step 1 (winkler/Force.c:154-161)
    double* escal;                   // [ne][4] element strain rate, stress, hydroPressure, aps
                                     // (written on steps with sc->want_scalars; NULL = never)
    const double* coh_scale;         // [ne] or NULL
    const double* fric_scale;        // [ne] or NULL
    const double* visc_scale;        // [ne] or NULL
    DevScalars* sc;
};

struct Config {
    int dt_type, constitutive, temperature, thermal_stress, has_density, time_step_zero;
    double gravity, demf;
    double strain_inert;
    int winkler;          // SnacWinklerForce on Snac_EP_Force
    int traction;         // SnacTractionBC on Snac_EP_Force (after Winkler)
    double topo_kappa, topo_crit;  // surface-topography diffusion
    double pisos, rzbo;   // its isostatic pressure and reference bottom depth
    // one phase, no density coupling, dynamic or wave dt: a tet's gravity and
    // inertial-mass terms are the same multiples of its volume for every tet,
    // so the element kernels store the volume alone (in the gravity rows) and
    // the node gather forms both terms from it with the same operations
    int vonly;
    // phase 0, the only phase of a model without a per-element phase array:
    // the element kernels of such models read it from their parameters
    // (constant-bank operands) instead of loading it from the phase table
    DevMaterial m0;
};

// Resident blocks per SM asked of the compiler (the register budget).  Elastic
// and Maxwell at 5 (96 registers, 56 and 24 bytes of spills): 84 against 88 us at
// 131 k hexes elastic; the hooks with a return map at 4 (128 registers, 8 bytes
// of spills plastic, 40 visco-plastic): 104 against 109 us plastic, 128 against 141 us
// visco-plastic, whose spills at 96 registers miss the small L1 that the
// shared memory leaves.
__host__ __device__ constexpr int elem_minb(int plugin) {
    return plugin == SNAC_RHEOLOGY_ELASTIC || plugin == SNAC_RHEOLOGY_MAXWELL ? 5 : 4;
}
constexpr int ELEM_WARPS = 4;                   // warps per block in the element kernels
constexpr int ELEM_PER_BLOCK = ELEM_WARPS * 3;  // 12 elements per block
constexpr unsigned FULL = 0xffffffffu;
constexpr int FROWS_MAX = 170;
constexpr int ROW10 = NT * GROUP;  // entries of ten rows
static_assert(GROUP == ELEM_PER_BLOCK, "a block writes one group");
constexpr int HROWS = 60;  // rows of a heat group

__device__ __forceinline__ long long node_id(const Mesh& m, int i, int j, int k) {
    return (long long)i + (long long)j * m.nnx + (long long)k * m.nnx * m.nny;
}

// x = i + j a + k a b.  Index arithmetic in 32 bits whenever the index fits:
// a 64-bit integer division is a long software routine on the GPU, a 32-bit
// one a few instructions (the branch is uniform across a launch).
__device__ __forceinline__ void split3(long long x, int a, int b, int& i, int& j, int& k) {
    if (x >= 0 && x < 0x7fffffffLL) {
        const unsigned u = (unsigned)x, q = u / (unsigned)a, r = q / (unsigned)b;
        i = (int)(u - q * (unsigned)a);
        j = (int)(q - r * (unsigned)b);
        k = (int)r;
    } else {
        i = (int)(x % a);
        j = (int)((x / a) % b);
        k = (int)(x / ((long long)a * b));
    }
}

__device__ __forceinline__ void elem_ijk(const Mesh& m, long long e, int& i, int& j, int& k) {
    split3(e, m.nx, m.ny, i, j, k);
}

__device__ __forceinline__ long long corner_node(const Mesh& m, int i, int j, int k, int corner) {
    return node_id(m, i + corner_di(corner), j + corner_dj(corner), k + corner_dk(corner));
}

__device__ __forceinline__ int phase_of(const Fields& F, long long e) { return F.mat ? (int)F.mat[e] : 0; }

// The value of lane (base + u) of this lane's element group.
__device__ __forceinline__ double grp(double v, int base, int u) { return __shfl_sync(FULL, v, base + u); }

// Sum over the 10 tets of the group, added in tet order starting from 0.
__device__ __forceinline__ double grp_sum(double v, int base) {
    double s = 0.0f;
#pragma unroll
    for (int u = 0; u < NT; u++) s += grp(v, base, u);
    return s;
}

// The same sums through shared memory: each lane puts its term (hex_put), and
// after a __syncwarp every lane of the hex reads the ten terms as five 16-byte
// broadcasts (hex_total): 7 data-pipe passes per sum against the 20 of ten
// 64-bit shuffles.
__device__ __forceinline__ void hex_put(double (&h)[3 * 12], int lane, int base, int t, double v) {
    if (lane < 30) h[base / 10 * 12 + t] = v;
}
__device__ __forceinline__ double hex_total(const double (&h)[3 * 12], int base) {
    const double2* p = reinterpret_cast<const double2*>(h + base / 10 * 12);
    double s = 0.0f;
#pragma unroll
    for (int u = 0; u < NT / 2; u++) {
        const double2 w = p[u];
        s += w.x;
        s += w.y;
    }
    return s;
}

struct TetSlot {
    int lane, base, t;
    long long e, q;
    bool active;
};

// ---- element blocks ---------------------------------------------------------------------
// A block takes GROUP consecutive hexes, each of its warps a triple of them:
// 30 tets in lanes 0-29 (lanes 30 and 31 repeat lanes 0 and 1 and store
// nothing).  What a triple reads (the coordinates and velocities of its 24
// corners, the stresses, the plastic strains, the scales) comes to shared
// memory by cp.async, and what it writes leaves shared memory as bulk copies:
// with direct accesses the 24-byte row pieces and 48-byte strides kept the
// load/store unit's data pipe 70 % busy, and the kernels waited for it.  A hex
// past the end of the mesh is read as the last hex, so every lane works on a
// regular tet.  (A persistent form that fetched one group ahead took the load
// stalls from 1.6 to 0.2 per instruction and measured the same within 3 % either way:
// 117 against 121 us plastic, 1.12 against 1.10 ms visco-plastic at 1 M hexes,
// 35 against 33 us at 33 k.)
struct Triple {
    // parts of row hex * 8 + corner: x, y | z, T | vx, vy | vz, T0; PART rows
    // apart, so that the four 16-byte pieces of a node fall in different banks
    static constexpr int PART = 26;
    double2 node[4 * PART];
    double2 stress[90];                          // [30][6]
    double eps_p[30];
    double scale[3][4];                          // cohesion, friction, viscosity scale of each hex
};
struct TripleCoords {  // the part of a Triple that the heat-flux kernels use
    static constexpr int PART = Triple::PART;
    double2 node[2 * PART];
};

__device__ __forceinline__ unsigned smem_addr(const void* p) { return (unsigned)__cvta_generic_to_shared(p); }
__device__ __forceinline__ void cp_async16(void* s, const void* g) {
    asm volatile("cp.async.ca.shared.global [%0], [%1], 16;" ::"r"(smem_addr(s)), "l"(g) : "memory");
}
__device__ __forceinline__ void cp_async16_once(void* s, const void* g) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(smem_addr(s)), "l"(g) : "memory");
}
__device__ __forceinline__ void cp_async8(void* s, const void* g) {
    asm volatile("cp.async.ca.shared.global [%0], [%1], 8;" ::"r"(smem_addr(s)), "l"(g) : "memory");
}
__device__ __forceinline__ void cp_async_wait_all() { asm volatile("cp.async.wait_all;" ::: "memory"); }
// shared memory written by this thread, before another thread's bulk copy reads it
__device__ __forceinline__ void bulk_fence() { asm volatile("fence.proxy.async.shared::cta;" ::: "memory"); }
// bytes: a multiple of 16, both addresses on 16-byte boundaries
__device__ __forceinline__ void bulk_store(void* g, const void* s, unsigned bytes) {
    asm volatile("cp.async.bulk.global.shared::cta.bulk_group [%0], [%1], %2;" ::"l"(g), "r"(smem_addr(s)), "r"(bytes) : "memory");
}
// commits this thread's bulk copies and waits until they have read shared memory
__device__ __forceinline__ void bulk_drain() {
    asm volatile("cp.async.bulk.commit_group;" ::: "memory");
    asm volatile("cp.async.bulk.wait_group.read 0;" ::: "memory");
}

// NEED: 1 velocities (and T0), 2 stresses, 4 plastic strains, 8 parameter scales
template <int NEED, class Tri>
__device__ __forceinline__ void fetch_triple(const Mesh& m, const Fields& F, int lb, Tri& z) {
    const int lane = threadIdx.x & 31;
    long long e0 = (long long)lb * GROUP + (threadIdx.x >> 5) * 3;
    if (e0 >= m.ne) e0 = m.ne - 1;  // a warp past the end of the mesh
    // lanes 0-2: the first corner's node of their hex (32 bits hold any hex or
    // node number of a mesh that fits the device's memory)
    unsigned n0;
    {
        const unsigned e = (unsigned)(e0 + (lane < 2 ? lane : 2)), ne = (unsigned)m.ne;
        const unsigned x = e < ne ? e : ne - 1, q = x / (unsigned)m.nx, k = q / (unsigned)m.ny;
        n0 = (x - q * m.nx) + ((q - k * m.ny) + k * m.nny) * m.nnx;
    }
    // lane: corner lane / 4, part lane % 4 of its 64 bytes
    const int corner = lane >> 2, part = lane & 3;
    const unsigned off = corner_di(corner) + (corner_dj(corner) + corner_dk(corner) * m.nny) * m.nnx;
    const double4* src = part < 2 ? F.pos : F.vel;
    double2* dst = z.node + part * Tri::PART + corner;
#pragma unroll
    for (int g = 0; g < 3; g++) {
        const unsigned n = __shfl_sync(FULL, n0, g) + off;
        if ((NEED & 1) || part < 2) cp_async16(dst + g * 8, reinterpret_cast<const double2*>(src + n) + (part & 1));
    }
    const int nh = (int)(m.ne - e0 < 3 ? m.ne - e0 : 3);
    if constexpr ((NEED & 2) != 0) {
#pragma unroll
        for (int c = 0; c < 3; c++) {
            const int x = lane + c * 32, h = x / 30;
            if (x < 90)
                cp_async16_once(z.stress + x, reinterpret_cast<const double2*>(F.stress + e0 * NT * 6) + (h < nh ? x : x - (h - nh + 1) * 30));
        }
    }
    if constexpr ((NEED & 4) != 0) {
        const int h = lane / 5;
        if (lane < 15)
            cp_async16_once(z.eps_p + lane * 2, F.eps_p + e0 * NT + (h < nh ? lane : lane - (h - nh + 1) * 5) * 2);
    }
    if constexpr ((NEED & 8) != 0) {
        const double* p = part == 0 ? F.coh_scale : part == 1 ? F.fric_scale : F.visc_scale;
        if (corner < 3 && part < 3 && p) cp_async8(&z.scale[part][corner], p + e0 + (corner < nh ? corner : nh - 1));
        if (corner < 3 && part < 3 && !p) z.scale[part][corner] = 1.0;
    }
}

// A lane's tet in a fetched triple
struct TetLane {
    int lane, base, t;
    unsigned rows;  // rows of its corners in the triple, one per byte
};
__device__ __forceinline__ TetLane tet_lane() {
    TetLane L;
    L.lane = threadIdx.x & 31;
    int g = L.lane / 10;
    L.t = L.lane - g * 10;
    if (g >= 3) {  // lanes 30 and 31
        g = 0;
        L.t = L.lane - 30;
    }
    L.base = g * 10;
    L.rows = 0;
#pragma unroll
    for (int q = 0; q < 4; q++) L.rows |= (unsigned)(g * 8 + tet_node_rt(L.t, q)) << (8 * q);
    return L;
}
__device__ __forceinline__ TetSlot tet_slot_of(const Mesh& m, const TetLane& L, int lb) {
    TetSlot s;
    s.lane = L.lane;
    s.base = L.base;
    s.t = L.t;
    const long long e = (long long)lb * GROUP + (threadIdx.x >> 5) * 3 + L.base / 10;
    s.active = L.lane < 30 && e < m.ne;
    s.e = e < m.ne ? e : m.ne - 1;
    s.q = s.e * NT + s.t;
    return s;
}

template <class Tri>
struct TetView {  // a lane's corners in shared memory
    const Tri& z;
    const unsigned rows;
    __device__ __forceinline__ int row(int q) const { return (rows >> (8 * q)) & 0xffu; }
    __device__ __forceinline__ void coords(V3 c[4]) const {
#pragma unroll
        for (int q = 0; q < 4; q++) {
            const double2 a = z.node[row(q)];
            c[q] = {a.x, a.y, z.node[Tri::PART + row(q)].x};
        }
    }
    __device__ __forceinline__ void velocities(V3 v[4]) const {
#pragma unroll
        for (int q = 0; q < 4; q++) {
            const double2 a = z.node[2 * Tri::PART + row(q)];
            v[q] = {a.x, a.y, z.node[3 * Tri::PART + row(q)].x};
        }
    }
    __device__ __forceinline__ double T(int q) const { return z.node[Tri::PART + row(q)].y; }
};

// Shared memory of the element kernels: the warps' triples, the terms of their hex
// sums, and the group of force or heat terms that the block writes.
struct ElemSmem {
    Triple tri[ELEM_WARPS];
    double hex_terms[ELEM_WARPS][2][3 * 12];
    double rows[FROWS_MAX * GROUP];
};
struct HeatSmem {
    TripleCoords tri[ELEM_WARPS];
    double rows[HROWS * GROUP];
};

// Whether the coordinates (and, with VEL, the sizes of the velocities) of
// the warp's triple are tame (see tet_geometry_tame): lane l looks at corner l.
template <bool VEL, class Tri>
__device__ __forceinline__ bool tame_triple(const Tri& z, int lane) {
    bool ok = true;
    if (lane < 24) {
        const double2 a = z.node[lane];
        ok = tame_coordinate(a.x) & tame_coordinate(a.y) & tame_coordinate(z.node[Tri::PART + lane].x);
        if (VEL) {
            const double2 b = z.node[2 * Tri::PART + lane];
            ok = ok & tame_size(b.x) & tame_size(b.y) & tame_size(z.node[3 * Tri::PART + lane].x);
        }
    }
    return ok;
}

// What the constitutive update reads besides the corners and the stress
struct TetIn {
    double eps_p;                 // plastic strain (plastic, visco-plastic)
    double coh, fric, visc;       // per-element parameter scales (1 without them)
    double pst[6];                // plastic strain tensor (Drucker-Prager instances)
};

template <int PLUGIN>
__device__ __forceinline__ TetIn load_tet_in(const Fields& F, const TetSlot& s, const Triple& z) {
    TetIn in;
    in.eps_p = 0.0;
    if (PLUGIN == SNAC_RHEOLOGY_PLASTIC || is_vp(PLUGIN)) in.eps_p = z.eps_p[s.base + s.t];
    for (int a = 0; a < 6; a++) in.pst[a] = 0.0;
    if (PLUGIN == SNAC_VP_DP) {
        const double2* p = reinterpret_cast<const double2*>(F.pst + s.q * 6);
        for (int a = 0; a < 3; a++) {
            const double2 w = p[a];
            in.pst[2 * a] = w.x;
            in.pst[2 * a + 1] = w.y;
        }
    }
    const int h = s.base / 10;
    in.coh = z.scale[0][h];
    in.fric = z.scale[1][h];
    in.visc = z.scale[2][h];
    return in;
}
__host__ __device__ constexpr int stress_need(int plugin) {
    return 1 | 2 | ((plugin == SNAC_RHEOLOGY_PLASTIC || (plugin & SNAC_RHEOLOGY_VISCOPLASTIC)) ? 4 | 8 : 0);
}

// ======================================================================================
// Snac_EP_CalcStresses: StrainRate.c:49-305, Stress.c:53-172 and the constitutive hook
// ======================================================================================
// st holds the tet's stress on entry (already rotated when fused with the
// element update); the new stress, plastic strain, viscosity, density and
// the Force terms are stored.
// The tet's four face areas and normals are needed again by the force terms at
// the end of the stress update.  Across the eigen-solve of a tet that may
// yield (~60 registers) they wait in shared memory: the normals in the places
// that the tet's force terms will take, the areas over the warp's corners,
// which every lane has read by then.
__device__ __forceinline__ void stash_faces(const TetGeom& g, double* r, const int (&row)[4], double* areas, int lane) {
    if (lane >= 30) return;  // lanes 30 and 31 read what lanes 0 and 1 stash
#pragma unroll
    for (int f = 0; f < 4; f++) {
        areas[f * 30 + lane] = g.A[f];
        double* const o = r + row[f];
        o[0] = g.n[f].x;
        o[ROW10] = g.n[f].y;
        o[2 * ROW10] = g.n[f].z;
    }
    asm volatile("" ::: "memory");  // keep the copies in shared memory, not in registers
}
__device__ __forceinline__ void unstash_faces(TetGeom& g, const double* r, const int (&row)[4], const double* areas, int lane) {
    __syncwarp();
    if (lane >= 30) lane -= 30;
#pragma unroll
    for (int f = 0; f < 4; f++) {
        g.A[f] = areas[f * 30 + lane];
        const double* const o = r + row[f];
        g.n[f] = {o[0], o[ROW10], o[2 * ROW10]};
    }
    __syncwarp();
}

// The geometry of any tet, with IEEE roots and quotients throughout: the rare
// triples that are not tame.  Calls that take the corners from shared memory
// and return values in registers, so that the common path neither keeps its
// geometry in local memory nor gives up registers for their arguments (with
// the corners as arguments k_fused_step of the Mohr-Coulomb hooks spilled 32
// and 44 bytes instead of 8 and 40: 1.70 -> 1.68 ms visco-plastic at 1 M hexes).
struct AnyFace {
    double A;
    V3 n;
};
// abc: the corners of the face, four bits each
template <class Tri>
__device__ __noinline__ AnyFace any_face(const Tri* z, unsigned rows, unsigned abc) {
    V3 c[3];
    for (int k = 0; k < 3; k++) {
        const int r = (rows >> (8 * ((abc >> (4 * k)) & 15u))) & 0xffu;
        const double2 a = z->node[r];
        c[k] = {a.x, a.y, z->node[Tri::PART + r].x};
    }
    AnyFace f;
    tet_face(c[0], c[1], c[2], f.A, f.n);
    return f;
}
template <class Tri>
__device__ __noinline__ double any_volume(const Tri* z, unsigned rows) {
    V3 c[4];
    TetView<Tri>{*z, rows}.coords(c);
    return tet_volume(c[0], c[1], c[2], c[3]);
}

// The geometry of this lane's tet; returns whether the whole triple is tame.
template <bool VEL, class Tri>
__device__ __forceinline__ bool triple_geometry(const Tri& z, const TetLane& L, TetGeom& g) {
    bool ok = tame_triple<VEL>(z, L.lane);
    {
        V3 c[4];
        TetView<Tri>{z, L.rows}.coords(c);
        tet_geometry_tame(c, g, ok);
    }
    if (__all_sync(FULL, ok)) return true;
    g.V = any_volume(&z, L.rows);
    g.zV = recip(g.V);
#pragma unroll
    for (int f = 0; f < 4; f++) {
        const AnyFace a = any_face(&z, L.rows, (unsigned)(face_node(f, 0) + 16 * face_node(f, 1) + 256 * face_node(f, 2)));
        g.A[f] = a.A;
        g.n[f] = a.n;
    }
    return false;
}

__device__ __forceinline__ void stage_stress(const TetSlot& s, const Triple& z, double st[6]) {
    const double2* p = z.stress + (s.base + s.t) * 3;
#pragma unroll
    for (int a = 0; a < 3; a++) {
        const double2 v = p[a];
        st[2 * a] = v.x;
        st[2 * a + 1] = v.y;
    }
}
__device__ __forceinline__ void unstage_stress(const TetSlot& s, Triple& z, const double st[6]) {
    double2* p = z.stress + (s.base + s.t) * 3;
#pragma unroll
    for (int a = 0; a < 3; a++) p[a] = make_double2(st[2 * a], st[2 * a + 1]);
}

template <int PLUGIN, bool ONE>
__device__ __forceinline__ void stress_update(const Mesh& m, const Fields& F, const Config& cfg, const TetSlot& s,
                                              Triple& z, double (&hx)[2][3 * 12], double* rows,
                                              const TetView<Triple>& w, TetGeom& g, double sr[6], double st[6],
                                              const double dt, const bool tame) {
    double* const r = rows + (threadIdx.x >> 5) * 3 + s.base / 10;  // the hex's column of the group
    const unsigned slots = TET_SLOTS[s.t];
    const int kinds = m.frows == FROWS_MAX ? 4 : 3;
    auto rows_of = [&](int (&row)[4]) {
#pragma unroll
        for (int f = 0; f < 4; f++) row[f] = corner_row(slots, f, kinds * NT);
    };
    double* const areas = reinterpret_cast<double*>(z.node);
    // element volume: UpdateElement.c:141,267 then 2*volume (StrainRate.c:62)
    // mixed discretisation, StrainRate.c:272-289 (each term trace_u V_u is formed on its own lane)
    const double tsum = sr[0] + sr[1] + sr[2];
    double trace = tame ? markstein(tsum, 3.0, Z3, tsum * Z3) : dv3(tsum);
    hex_put(hx[0], s.lane, s.base, s.t, g.V);
    hex_put(hx[1], s.lane, s.base, s.t, trace * g.V);
    __syncwarp();
    const double vsum = hex_total(hx[0], s.base);
    const double partial = hex_total(hx[1], s.base);
    double elemVolume = 2.0 * (vsum * 0.5);
    const double zE = recip(elemVolume);
    double corr = -1.0f * trace + dvz(partial, elemVolume, zE);
    sr[0] += corr;
    sr[1] += corr;
    sr[2] += corr;
    // scalar element outputs for the dump writers, on the steps that need them
    const bool want = F.escal != nullptr && F.sc->want_scalars;
    if (want) {
        // StrainRate.c:284-304
        double srVolAvg = grp_sum(sr[1] * sr[2] + sr[2] * sr[0] + sr[0] * sr[1], s.base);
        double srOtherAvg = grp_sum(sr[3] * sr[3] + sr[5] * sr[5] + sr[4] * sr[4], s.base);
        srVolAvg = dv10(srVolAvg);
        srOtherAvg = dv10(srOtherAvg);
        if (s.active && s.t == 0) F.escal[s.e * 4 + 0] = 0.5f * sqrt(0.5f * fabs(-1.0f * srVolAvg + srOtherAvg));
    }

    // strain, Stress.c:71-82
    double e[6];
#pragma unroll
    for (int a = 0; a < 6; a++) e[a] = sr[a] * dt;

    const TetIn in = load_tet_in<PLUGIN>(F, s, z);
    const int ph = phase_of(F, s.e);
    const DevMaterial& M = ONE ? cfg.m0 : F.mats[ph];  // ONE: the model has one phase
    double eps_p = in.eps_p, eta = 0.0;
    // what the Drucker-Prager return map needs from the viscous update
    double dp_sd[3] = {0.0, 0.0, 0.0}, dp_S0[6] = {0.0, 0.0, 0.0, 0.0, 0.0, 0.0};
    double dp_vic1 = 0.0, dp_vic2 = 0.0, dp_bulkm = 0.0;

    double sp[3] = {0, 0, 0}, cn[3][3];
    // softening-table lookup results of this tet (for the carry-over between tets)
    double fa = 0.0f, da = 0.0f, co = 0.0f, hd = 0.0f;
    int matched = 0;

    if (PLUGIN == SNAC_RHEOLOGY_ELASTIC) {
        // elastic/Constitutive.c:40-66
        const double a2 = M.lambda;
        const double sh2 = 2.0 * M.mu;
        double tr = e[0] + e[1] + e[2];
        st[0] += sh2 * e[0] + a2 * (tr);
        st[1] += sh2 * e[1] + a2 * (tr);
        st[2] += sh2 * e[2] + a2 * (tr);
        st[3] += sh2 * e[3];
        st[4] += sh2 * e[4];
        st[5] += sh2 * e[5];
    } else if (PLUGIN == SNAC_RHEOLOGY_MAXWELL) {
        // maxwell/Constitutive.c:47-184
        const double bulkm = M.lambda + dv3(2.0f * M.mu);
        double vold = F.vol[s.q * 2 + 1];
        double vcur = F.vol[s.q * 2 + 0];
        double trace_stress = st[0] + st[1] + st[2];
        double trace_strain = dv(vcur, vold) - 1.0f;
        double straind[3], stressd[3];
        const double tn3 = dv3(trace_strain), ts3 = dv3(trace_stress);
        for (int a = 0; a < 3; a++) straind[a] = e[a] - tn3;
        for (int a = 0; a < 3; a++) stressd[a] = st[a] - ts3;
        double srJ2 = sqrt(fabs(straind[1] * straind[2] + straind[2] * straind[0] + straind[0] * straind[1] -
                                e[3] * e[3] - e[4] * e[4] - e[5] * e[5])) /
                      dt;
        if (srJ2 == 0.0f) srJ2 = M.refsrate;
        double avgTemp = 0.0;
        for (int qn = 0; qn < 4; qn++) avgTemp += 0.25 * w.T(qn);
        eta = arrhenius_viscosity(M, M.refvisc, srJ2, avgTemp);
        if (s.active && !isfinite(eta)) report(F.sc, SNAC_GPU_ENAN, s.e);
        if (ph == 0) maxwell_update(st, e, stressd, straind, ts3, trace_strain, M.mu, eta, dt, bulkm);
    } else {
        if (PLUGIN == SNAC_RHEOLOGY_PLASTIC) {
            // elastic trial, plastic/Constitutive.c:114-121
            double tr = e[0] + e[1] + e[2];
            st[0] += (2.0f * M.mu) * e[0] + M.lambda * (tr);
            st[1] += (2.0f * M.mu) * e[1] + M.lambda * (tr);
            st[2] += (2.0f * M.mu) * e[2] + M.lambda * (tr);
            st[3] += (2.0f * M.mu) * e[3];
            st[4] += (2.0f * M.mu) * e[4];
            st[5] += (2.0f * M.mu) * e[5];
            if (s.active && M.plstrain[0] != 0.0) report(F.sc, SNAC_GPU_EINVAL, s.e);
        } else {
            // visco-plastic Maxwell step, viscoplastic/Constitutive.c:158-257
            const double bulkm = M.lambda + dv3(2.0f * M.mu);
            if (cfg.thermal_stress) {
                const unsigned grp = (unsigned)s.e / GROUP, col = (unsigned)s.e - grp * GROUP;
                double ts = F.hflux[(long long)grp * (HROWS * GROUP) + 5 * ROW10 + s.t * GROUP + col];
                st[0] += ts;
                st[1] += ts;
                st[2] += ts;
            }
            if (PLUGIN == SNAC_VP_DP)  // Stress0, viscoplastic/Constitutive.c:165-170
                for (int a = 0; a < 6; a++) dp_S0[a] = st[a];
            double trace_stress = st[0] + st[1] + st[2];
            double trace_strain = e[0] + e[1] + e[2];
            double straind[3], stressd[3];
            const double tn3 = dv3(trace_strain), ts3 = dv3(trace_stress);
            for (int a = 0; a < 3; a++) straind[a] = e[a] - tn3;
            for (int a = 0; a < 3; a++) stressd[a] = st[a] - ts3;
            // viscoplastic/Constitutive.c:189 reads strain[1][0], strain[2][0] and stress[2][0]
            // (the pointer, not the tensor, is indexed); those entries are always zero.
            const double lower = 0.0;
            double srJ2 = sqrt(fabs(straind[1] * straind[2] + straind[2] * straind[0] + straind[0] * straind[1] -
                                    (lower) * (lower) - (lower) * (lower) - (lower) * (lower))) /
                          dt;
            if (srJ2 == 0.0f) srJ2 = M.refsrate;
            double avgTemp = 0.0;
            for (int qn = 0; qn < 4; qn++) avgTemp += 0.25 * w.T(qn);
            double refvisc = M.refvisc;
            refvisc = M.refvisc * in.visc;
            eta = arrhenius_viscosity(M, refvisc, srJ2, avgTemp);
            if (s.active && !isfinite(eta)) report(F.sc, SNAC_GPU_ENAN, s.e);
            maxwell_update(st, e, stressd, straind, ts3, trace_strain, M.mu, eta, dt, bulkm, dp_vic1, dp_vic2);
            if (PLUGIN == SNAC_VP_DP) {
                for (int a = 0; a < 3; a++) dp_sd[a] = stressd[a];
                dp_bulkm = bulkm;
            }
        }
        // piecewise-linear softening (plastic/Constitutive.c:133-159 with break and
        // clamp; viscoplastic/Constitutive.c:279-293 without either: the last
        // matching segment wins)
        const double cs = in.coh;
        const double fsc = in.fric;
        // an angle that is the same at every point of the table keeps its
        // value: 0 / dpl = 0 and angle + 0 * (eps_p - pl1) = angle (dpl finite and not 0)
        for (int i = 0; i < M.nsegments; i++) {
            const double pl1 = M.plstrain[i], pl2 = M.plstrain[i + 1];
            if (eps_p >= pl1 && eps_p <= pl2) {
                const double dpl = pl2 - pl1, zpl = M.zpl[i], dep = eps_p - pl1;  // zpl = RN(1 / dpl)
                const double c0 = M.coh[i] * cs;
                hd = dvz(M.coh[i + 1] * cs - c0, dpl, zpl);
                co = c0 + hd * dep;
                fa = M.fric0;
                da = M.dil0;
                if (!M.angles_const) {
                    const double f0 = M.fric[i] * fsc;
                    double tg[2] = {M.fric[i + 1] * fsc - f0, M.dil[i + 1] - M.dil[i]};
                    dvz_n(tg, dpl, zpl);
                    fa = f0 + tg[0] * dep;
                    da = M.dil[i] + tg[1] * dep;
                }
                matched = 1;
                if (PLUGIN == SNAC_RHEOLOGY_PLASTIC) break;
            } else if (PLUGIN == SNAC_RHEOLOGY_PLASTIC && i == M.nsegments - 1 && eps_p > pl2) {
                fa = M.fric[M.nsegments] * fsc;
                da = M.dil[M.nsegments];
                co = M.coh[M.nsegments] * cs;
                hd = 0.0;
                matched = 1;
                break;
            }
        }
    }

    double pst[6];
    for (int a = 0; a < 6; a++) pst[a] = in.pst[a];
    if (PLUGIN == SNAC_RHEOLOGY_PLASTIC || is_vp(PLUGIN)) {
        double frictionAngle = fa, dilationAngle = da, cohesion = co, hardening = hd;
        double stc, anphi, anpsi, sq_anphi, aP;
        // the usual table: the tet found its segment, angles constant, their
        // sines and tangents evaluated on the host.  The hexes of a warp may
        // be of different phases, so the test itself is the tet's, and every
        // lane takes the vote.
        const bool usual = matched && M.angles_const && M.fric0 > 0.0;
        if (__all_sync(FULL, usual)) {
            stc = M.ten_off;
            const double tmp = dvz(cohesion, M.tan_fric0, M.ztan_fric0);
            if (tmp < stc) stc = tmp;
            anphi = M.anphi0;
            anpsi = M.anpsi0;
            sq_anphi = M.sq_anphi0;
            aP = M.ap0;
        } else {
            // The reference keeps the table values (and the tension cutoff) in
            // variables that outlive the tet loop: a tet whose lookup matched no
            // segment reuses the previous tet's values, 0 before the first match.
            if (__ballot_sync(FULL, s.active && !matched) != 0u) {
                unsigned mb = __ballot_sync(FULL, matched && s.active);
                unsigned mine = (mb >> s.base) & ((1u << (s.t + 1)) - 1u);
                int src = mine ? (31 - __clz(mine)) : -1;
                double src_fa = __shfl_sync(FULL, fa, s.base + (src < 0 ? 0 : src));
                double src_da = __shfl_sync(FULL, da, s.base + (src < 0 ? 0 : src));
                double src_co = __shfl_sync(FULL, co, s.base + (src < 0 ? 0 : src));
                double src_hd = __shfl_sync(FULL, hd, s.base + (src < 0 ? 0 : src));
                frictionAngle = src < 0 ? 0.0f : src_fa;
                dilationAngle = src < 0 ? 0.0f : src_da;
                cohesion = src < 0 ? 0.0f : src_co;
                hardening = src < 0 ? 0.0f : src_hd;
            }
            // tension cutoff st = min(ten_off, c / tan(phi)) when phi > 0, else carried over
            const bool fconst = M.fric_const && frictionAngle == M.fric0;
            bool phi_ok = (PLUGIN == SNAC_RHEOLOGY_PLASTIC) ? (frictionAngle >= 0.0f) : (frictionAngle > 0.0f);
            double st_own = 0.0;
            if (phi_ok) {
                st_own = M.ten_off;
                if (frictionAngle > 0.0) {
                    double tmp = fconst ? dvz(cohesion, M.tan_fric0, M.ztan_fric0) : dv(cohesion, tan_fric(M, frictionAngle));
                    if (tmp < st_own) st_own = tmp;
                }
            }
            stc = st_own;
            if (__ballot_sync(FULL, s.active && !phi_ok) != 0u) {
                unsigned pb = __ballot_sync(FULL, phi_ok && s.active);
                unsigned pm = (pb >> s.base) & ((1u << (s.t + 1)) - 1u);
                int psrc = pm ? (31 - __clz(pm)) : -1;
                double st_c = __shfl_sync(FULL, st_own, s.base + (psrc < 0 ? 0 : psrc));
                stc = psrc < 0 ? 0.0 : st_c;
            }
            if (PLUGIN == SNAC_RHEOLOGY_PLASTIC && s.active && frictionAngle < 0.0f)
                report(F.sc, SNAC_GPU_EPHYSICS, s.e);  // plastic/Constitutive.c:175 abort()
            const double sphi = sin_fric(M, frictionAngle), spsi = sin_dil(M, dilationAngle);
            anphi = fconst ? M.anphi0 : dv(1.0f + sphi, 1.0f - sphi);
            anpsi = (M.dil_const && dilationAngle == M.dil0) ? M.anpsi0 : dv(1.0f + spsi, 1.0f - spsi);
            sq_anphi = fconst ? M.sq_anphi0 : sqrt(anphi);
            aP = fconst ? M.ap0 : sqrt(1.0f + anphi * anphi) + anphi;
        }
        // a Drucker-Prager tet takes a return map of its own (the principal
        // stresses the reference computes first are not used by it); its
        // warp may hold Mohr-Coulomb tets, so it goes through their votes too
        const bool dp = PLUGIN == SNAC_VP_DP && !M.yield_mc;
        const double a1 = M.lambda + 2.0f * M.mu;
        const double a2 = M.lambda;
        // The reference always computes the principal stresses; they only
        // matter when the tet yields.  A tet that provably stays inside the
        // yield surface keeps its trial stress without the eigen-solve.
        const bool may_yield = !dp && !surely_elastic(st, cohesion, anphi, sq_anphi, stc);
        if (__any_sync(FULL, may_yield)) {
            __syncwarp();  // every lane has read its corners
            int row[4];
            rows_of(row);
            stash_faces(g, r, row, areas, s.lane);
            if (may_yield) {
                principal_stresses(st, sp, cn);
                mc_return_map(sp, cn, st, eps_p, cohesion, hardening, anphi, sq_anphi, aP, anpsi, stc, a1, a2);
            }
            unstash_faces(g, r, row, areas, s.lane);
        }
        if (PLUGIN == SNAC_VP_DP && dp && s.active)  // viscoplastic/Constitutive.c:372-518
            dp_return_map(st, dp_sd, dp_S0, e, dp_vic1, dp_vic2, M.mu, dp_bulkm, tan_fric(M, frictionAngle),
                          tan_dil(M, dilationAngle), cohesion, stc, M.dp_tol, M.dp_maxit, pst, eps_p);
    }

    // trace averaging over the 10 tets, Stress.c:87-137
    double traceS = dv3(st[0] + st[1] + st[2]);
    const double traceSV = traceS * g.V;
    __syncwarp();  // every lane has read the volumes
    hex_put(hx[0], s.lane, s.base, s.t, traceSV);
    __syncwarp();
    const double partialS = hex_total(hx[0], s.base);
    const double avgTrace = dvz(partialS, elemVolume, zE);
    double cs2 = -1.0f * traceS + avgTrace;
    st[0] += cs2;
    st[1] += cs2;
    st[2] += cs2;
    if (want) {
        // Stress.c:130-156: the element's scalar stress and hydrostatic pressure
        double sVolAvg = grp_sum((st[1] - avgTrace) * (st[2] - avgTrace) + (st[2] - avgTrace) * (st[0] - avgTrace) +
                                     (st[0] - avgTrace) * (st[1] - avgTrace),
                                 s.base);
        double sOtherAvg = grp_sum(st[3] * st[3] + st[5] * st[5] + st[4] * st[4], s.base);
        double pressure = grp_sum(dv3(st[0] + st[1] + st[2]), s.base);
        sVolAvg = dv10(sVolAvg);
        sOtherAvg = dv10(sOtherAvg);
        pressure = dv10(pressure);
        // plastic/Constitutive.c:239-244, viscoplastic/Constitutive.c:519-523: aps
        double aps = 0.0;
        if (PLUGIN == SNAC_RHEOLOGY_PLASTIC || is_vp(PLUGIN))
            aps = dv(grp_sum(eps_p * g.V, s.base), vsum);
        if (s.active && s.t == 0) {
            F.escal[s.e * 4 + 1] = 0.5f * sqrt(0.5f * fabs(-1.0f * sVolAvg + sOtherAvg));
            F.escal[s.e * 4 + 2] = -1.0 * pressure;
            F.escal[s.e * 4 + 3] = aps;
        }
    }

    if (cfg.has_density) {
        // Stress.c:125-170: pressure = mean tet trace/3, density update
        double ptet = dv3(st[0] + st[1] + st[2]);
        double pressure = 0.0f;
#pragma unroll
        for (int u = 0; u < NT; u++) pressure += grp(ptet, s.base, u);
        pressure = dv10(pressure);
        double avgT = 0.0;
        if (cfg.temperature) {
            // UpdateAverageTemp_LoopElements (Heat.c:143-172) ran before the
            // temperature BCs were re-applied: use the pre-BC temperatures
            avgT = 0.0;
            int ei = 0, ej = 0, ek = 0;  // recomputed here: the slot's i, j, k need not stay live
            elem_ijk(m, s.e, ei, ej, ek);
            for (int qn = 0; qn < 4; qn++) {
                long long n = corner_node(m, ei, ej, ek, tet_node_rt(s.t, qn));
                avgT += F.tpre[n] / (1.0f * 4);
            }
        }
        if (s.active) F.density[s.q] = M.density * (1.0 - M.alpha * (avgT - M.reftemp) + M.beta * pressure);
    }

    // Per-tet terms of Snac_Force (Force.c:107-180), evaluated here where the
    // tet's geometry and new stress already are.  k_loop_nodes adds them in
    // the reference's node-centred order, so the sums keep their bits.
    if (s.lane < 30) {
        const double rho = cfg.has_density ? F.density[s.q] : M.density;
        int row[4];
        rows_of(row);
#pragma unroll
        for (int f = 0; f < 4; f++) {
            const V3& nr = g.n[f];
            const double A = g.A[f];
            double t[3] = {(st[0] * nr.x + st[3] * nr.y + st[4] * nr.z) * A, (st[3] * nr.x + st[1] * nr.y + st[5] * nr.z) * A,
                           (st[4] * nr.x + st[5] * nr.y + st[2] * nr.z) * A};
            dvk_n(t, 6.0, Z6);
            double* const o = r + row[f];
            o[0] = t[0];
            o[ROW10] = t[1];
            o[2 * ROW10] = t[2];
        }
        const double factor4 = 1.0f / 4.0f;
        double* const rg = r + 4 * kinds * ROW10 + s.t * GROUP;
        double* const rm = rg + ROW10;
        if (ONE && cfg.vonly) {  // both terms formed by the node gather
            *rg = g.V;
        } else {
            *rg = cfg.gravity * rho * g.V * 0.125;  // x * 2^-3 rounds as x / 8
            if (cfg.dt_type == SNAC_DT_DYNAMIC) {
                const double sos = F.sc->speed_of_sound;
                const double inertialDensity = ONE ? F.sc->inertial_density0 : dv(M.lambda + 2.0f * M.mu, sos * sos);
                *rm = factor4 * inertialDensity * g.V;
            } else if (cfg.dt_type == SNAC_DT_CONSTANT) {
                const double alpha1 = (M.lambda + 2.0f * M.mu);
                const double nineV = 9.0f * g.V, z9V = recip(nineV);
#pragma unroll
                for (int f = 0; f < 4; f++) {
                    const V3& nr = g.n[f];
                    const double A = g.A[f];
                    double area_sum = 0.0, temp;
                    temp = (nr.x * A) * (nr.x * A);
                    if (temp > area_sum) area_sum = temp;
                    temp = (nr.y * A) * (nr.y * A);
                    if (temp > area_sum) area_sum = temp;
                    temp = (nr.z * A) * (nr.z * A);
                    if (temp > area_sum) area_sum = temp;
                    r[row[f] + 3 * ROW10] = dvz(alpha1 * area_sum, nineV, z9V) * (dt * dt);
                }
            } else {
                *rm = factor4 * rho * g.V;
            }
        }
        unstage_stress(s, z, st);  // the new state replaces the old in the triple
        if (PLUGIN == SNAC_RHEOLOGY_PLASTIC || is_vp(PLUGIN)) z.eps_p[s.base + s.t] = eps_p;
    }

    if (s.active) {
        bool ok = true;
#pragma unroll
        for (int a = 0; a < 6; a++) ok = ok & (bool)isfinite(st[a]);
        if (!ok) report(F.sc, SNAC_GPU_ENAN, s.e);  // Stress.c:161-166
        if (is_vp(PLUGIN) || (PLUGIN == SNAC_RHEOLOGY_MAXWELL && ph == 0)) F.visc[s.q] = eta;
        if (PLUGIN == SNAC_VP_DP) {
            double2* p = reinterpret_cast<double2*>(F.pst + s.q * 6);
            for (int a = 0; a < 3; a++) p[a] = make_double2(pst[2 * a], pst[2 * a + 1]);
        }
    }
}

// The results of group lb leave shared memory: each warp's triple, then the
// group of force terms once every warp has written its columns.
template <int PLUGIN, bool TERMS>
__device__ __forceinline__ void store_group(const Mesh& m, const Fields& F, int lb, const Triple& z,
                                            const double* rows) {
    bulk_fence();
    __syncwarp();
    if ((threadIdx.x & 31) == 0) {
        const long long e0 = (long long)lb * GROUP + (threadIdx.x >> 5) * 3, left = m.ne - e0;
        const unsigned nh = left < 3 ? (left > 0 ? (unsigned)left : 0u) : 3u;
        if (nh) {
            bulk_store(F.stress + e0 * NT * 6, z.stress, nh * NT * 48);
            if (TERMS && (PLUGIN == SNAC_RHEOLOGY_PLASTIC || is_vp(PLUGIN))) bulk_store(F.eps_p + e0 * NT, z.eps_p, nh * NT * 8);
        }
    }
    if (TERMS) {
        __syncthreads();
        if (threadIdx.x == 0) bulk_store(F.fterm + (long long)lb * (m.frows * GROUP), rows, (unsigned)m.frows * GROUP * 8);
    }
    if ((threadIdx.x & 31) == 0) bulk_drain();
}

// The tet's share of the minimum length scale, min over its faces of |V / A|
// (UpdateElement.c:109-139) = RN(V / max_f A_f), as correctly rounded
// division is monotonic; faces with A = 0 (or NaN) are skipped as in the
// reference.
__device__ __forceinline__ double tet_length_scale(const TetGeom& g) {
    double ls = 1.0e+27f, A = 0.0;
#pragma unroll
    for (int f = 0; f < 4; f++)
        if (g.A[f] > A) A = g.A[f];
    if (A) {
        const double l = fabs(dv(g.V, A));
        if (ls > l) ls = l;
    }
    return ls;
}

// UpdateElement.c:84-91 volume bookkeeping (Maxwell reads V/V_old) and the
// Jaumann rotation of the stress (:145-265) of one tet; st: the stress,
// rotated in place.
template <int PLUGIN>
__device__ __forceinline__ void element_update_tet(const Fields& F, const Config& cfg, const TetSlot& s,
                                                   const double (&r)[3], const TetGeom& g, double dt, double st[6]) {
    if (PLUGIN == SNAC_RHEOLOGY_MAXWELL && s.active) {
        double vc = F.vol[s.q * 2 + 0];
        F.vol[s.q * 2 + 1] = cfg.time_step_zero ? g.V : vc;
        F.vol[s.q * 2 + 0] = g.V;
    }
    rotate_stress(r, dt, st);
}

// The stress update of group lb; FUSED: after the pending element update of the
// step before (dt_rot), whose geometry and velocities are the same: one
// geometry evaluation, one stress read-modify-write.
template <int PLUGIN, bool ONE, bool FUSED>
__device__ __forceinline__ void stress_group(ElemSmem& S, const Mesh& m, const Fields& F, const Config& cfg, int lb) {
    Triple& z = S.tri[threadIdx.x >> 5];
    fetch_triple<stress_need(PLUGIN)>(m, F, lb, z);
    const TetLane L = tet_lane();
    const TetSlot s = tet_slot_of(m, L, lb);
    const double dt = F.sc->dt, dt_rot = FUSED ? F.sc->dt_rot : 0.0;
    cp_async_wait_all();
    __syncwarp();
    const TetView<Triple> w{z, L.rows};
    TetGeom g;
    const bool tame = triple_geometry<true>(z, L, g);
    double r[3], sr[6], st[6];
    {
        V3 v[4];
        w.velocities(v);
        if (FUSED)
            spin_and_strain_rates(v, g, r, sr, tame);
        else
            tet_strain_rate(v, g, sr, tame);
    }
    asm volatile("" ::: "memory");  // the stress is loaded when the velocities have gone
    stage_stress(s, z, st);
    if (FUSED) element_update_tet<PLUGIN>(F, cfg, s, r, g, dt_rot, st);
    stress_update<PLUGIN, ONE>(m, F, cfg, s, z, S.hex_terms[threadIdx.x >> 5], S.rows, w, g, sr, st, dt, tame);
    store_group<PLUGIN, true>(m, F, lb, z, S.rows);
}

template <int PLUGIN, bool ONE>
__global__ void __launch_bounds__(ELEM_WARPS * 32, elem_minb(PLUGIN)) k_calc_stresses(Mesh m, Fields F, Config cfg) {
    __shared__ __align__(16) ElemSmem S;
    stress_group<PLUGIN, ONE, false>(S, m, F, cfg, blockIdx.x);
}

// The end of step n (element update with dt_n, whose geometry and velocities
// are already final) fused with the stress update of step n+1.  Used when no
// energy hook sits between the two.
__device__ __forceinline__ void count_step(const Fields& F) {  // _AbstractContext_Execute_Hook
    F.sc->time_step += 1;
    F.sc->current_time += F.sc->dt;
}
template <int PLUGIN, bool ONE>
__global__ void __launch_bounds__(ELEM_WARPS * 32, elem_minb(PLUGIN)) k_fused_step(Mesh m, Fields F, Config cfg) {
    if (blockIdx.x == 0 && threadIdx.x == 0) count_step(F);
    __shared__ __align__(16) ElemSmem S;
    stress_group<PLUGIN, ONE, true>(S, m, F, cfg, blockIdx.x);
}

// Temperature runs: the element update of step n is deferred past the heat
// flux and temperature update of step n+1 (neither reads the stress) into
// the stress kernel of step n+1, which recomputes the same geometry anyway;
// the step counters were advanced by the heat-flux kernel.
template <int PLUGIN, bool ONE>
__global__ void __launch_bounds__(ELEM_WARPS * 32, elem_minb(PLUGIN)) k_fused_stress(Mesh m, Fields F, Config cfg) {
    __shared__ __align__(16) ElemSmem S;
    stress_group<PLUGIN, ONE, true>(S, m, F, cfg, blockIdx.x);
}

// ======================================================================================
// Snac_EP_LoopElementsMomentum: UpdateElement.c:54-269 and the minLengthScale
// reduction of _Snac_Context_LoopElements (Context.c:1156-1184)
// ======================================================================================
template <int PLUGIN>
__device__ __forceinline__ void update_group(const Mesh& m, const Fields& F, const Config& cfg, int pending, int lb) {
    __shared__ __align__(16) Triple tri[ELEM_WARPS];
    Triple& z = tri[threadIdx.x >> 5];
    fetch_triple<1 | 2>(m, F, lb, z);
    const TetLane L = tet_lane();
    const TetSlot s = tet_slot_of(m, L, lb);
    const double dt = pending ? F.sc->dt_rot : F.sc->dt;
    cp_async_wait_all();
    __syncwarp();
    const TetView<Triple> w{z, L.rows};
    TetGeom g;
    const bool tame = triple_geometry<true>(z, L, g);
    double r[3], st[6];
    {
        V3 v[4];
        w.velocities(v);
        spin_rates(v, g, r, tame);
    }
    stage_stress(s, z, st);
    element_update_tet<PLUGIN>(F, cfg, s, r, g, dt, st);
    if (s.lane < 30) unstage_stress(s, z, st);
    store_group<PLUGIN, false>(m, F, lb, z, nullptr);
    if (pending) return;  // the minimum length scale of this geometry is already known
    double ls = tet_length_scale(g);
    if (s.active && g.V == 0.0) report(F.sc, SNAC_GPU_EVOLUME, s.e);
    // global minimum (exact: min does not round)
    for (int o = 16; o > 0; o >>= 1) ls = fmin(ls, __shfl_xor_sync(FULL, ls, o));
    if ((threadIdx.x & 31) == 0) atomicMin(&F.sc->minls_bits, (unsigned long long)__double_as_longlong(ls));
}

template <int PLUGIN>
__global__ void __launch_bounds__(ELEM_WARPS * 32, 5) k_update_elements(Mesh m, Fields F, Config cfg,
                                                                                     int pending) {
    update_group<PLUGIN>(m, F, cfg, pending, blockIdx.x);
}

// The minimum over all tets and faces of |V/A| (UpdateElement.c:109-139) for
// the current coordinates, without the rest of the element update.  For a
// tet, min_f RN(V/A_f) = RN(V / max_f A_f) because correctly rounded
// division is monotonic, and max_f A_f = RN(sqrt(max_f s_f))/2 for the same
// reason; faces with A = 0 are skipped as in the reference.
__device__ __forceinline__ double hex_min_length_scale(const Mesh& m, const Fields& F, int lb) {
    long long e = (long long)lb * blockDim.x + threadIdx.x;
    double ls = 1.0e+27f;
    if (e < m.ne) {
        int i, j, k;
        elem_ijk(m, e, i, j, k);
        V3 corner[8];
#pragma unroll
        for (int cc = 0; cc < 8; cc++) {
            double4 p = F.pos[corner_node(m, i, j, k, cc)];
            corner[cc] = {p.x, p.y, p.z};
        }
#pragma unroll
        for (int t = 0; t < NT; t++) {
            V3 c[4];
#pragma unroll
            for (int qn = 0; qn < 4; qn++) c[qn] = corner[tet_node(t, qn)];
            double V = tet_volume(c[0], c[1], c[2], c[3]);
            double smax = 0.0;
#pragma unroll
            for (int f = 0; f < 4; f++) {
                const V3 &c1 = c[face_node(f, 0)], &c2 = c[face_node(f, 1)], &c3 = c[face_node(f, 2)];
                double x2 = c2.x - c1.x, y2 = c2.y - c1.y, z2 = c2.z - c1.z;
                double x3 = c3.x - c1.x, y3 = c3.y - c1.y, z3 = c3.z - c1.z;
                double a = y2 * z3 - z2 * y3;
                double b = z2 * x3 - x2 * z3;
                double cc = x2 * y3 - y2 * x3;
                double sq = a * a + b * b + cc * cc;
                if (sq > smax) smax = sq;
            }
            double A = sqrt(smax) * 0.5;  // rounds as / 2
            if (A) {
                double l = fabs(dv(V, A));
                if (ls > l) ls = l;
            }
            if (V == 0.0) report(F.sc, SNAC_GPU_EVOLUME, e);
        }
    }
    return ls;
}

__device__ __forceinline__ void k_min_length_scale_body(const Mesh& m, const Fields& F, int lb) {
    double ls = hex_min_length_scale(m, F, lb);
    for (int o = 16; o > 0; o >>= 1) ls = fmin(ls, __shfl_xor_sync(FULL, ls, o));
    if ((threadIdx.x & 31) == 0) atomicMin(&F.sc->minls_bits, (unsigned long long)__double_as_longlong(ls));
}


// ======================================================================================
// Snac_EP_LoopNodesMomentum: Snac_Force (Force.c:53-188), then
// Snac_UpdateNodeMomentum_PreProcess (UpdateNode.c:74-158) and
// Snac_UpdateNodeMomentum (UpdateNode.c:60-72) for every node.  Coordinates
// are read from pos and written to pos_next, so every force sees the old
// geometry, as in the reference where all forces are summed before any node moves.
// ======================================================================================
// SnacWinklerForce (Snac/plugins/winkler/Force.c:56-168), appended to the
// force of a bottom node (j == 0): for each incident element, the isostatic
// pressure corrected by the element's bottom height acts on its bottom face
// (tets 1, 2, 6, 8, faces 0, 1, 2, 2); at step 1 the node's total y force is
// kept as a residual and subtracted from then on.
// The force-BC plugins run for a few boundary nodes only, as calls.  Their
// arguments are plain values: a reference to the kernel's parameter structs
// (or to the caller's force registers) would make every thread copy those to
// its stack before the call.
struct WinklerArgs {
    const double4* pos;
    const unsigned char* mat;
    const DevMaterial* mats;
    double* residual_fr;
    long long time_step;
    double pisos, gravity, rzbo;
};

inline __device__ __noinline__ V3 winkler_force(WinklerArgs a, int nx, int ny, int nz, long long n, int i, int k, V3 f) {
    Mesh m{};
    m.nx = nx;
    m.ny = ny;
    m.nz = nz;
    m.nnx = nx + 1;
    m.nny = ny + 1;
    double fx = f.x, fy = f.y, fz = f.z;
    const double factor4 = 1.0f / 4.0f;
    const double y_node = a.pos[n].y;
    const double nodeT = 0.0;  // the temperature lookup is compiled out in the reference (#if 0)
    for (int ne = 0; ne < 8; ne++) {
        const int ei = i - 1 + (ne & 1), ej = -1 + ((ne >> 1) & 1), ek = k - 1 + ((ne >> 2) & 1);
        if (ei < 0 || ej < 0 || ek < 0 || ei >= m.nx || ej >= m.ny || ek >= m.nz) continue;
        const long long e = (long long)ei + (long long)ej * m.nx + (long long)ek * m.nx * m.ny;
        const DevMaterial& M = a.mats[a.mat ? (int)a.mat[e] : 0];
        V3 corner[8];
#pragma unroll
        for (int cc = 0; cc < 8; cc++) {
            double4 p = a.pos[corner_node(m, ei, ej, ek, cc)];
            corner[cc] = {p.x, p.y, p.z};
        }
        const double phsDensity = M.density, drosub = 0.0f;
        const double p_est = a.pisos + 0.5f * (phsDensity + drosub) * a.gravity * (y_node - a.rzbo);
        const double rosubg = a.gravity * (phsDensity + drosub) * (1.0 - M.alpha * (nodeT - M.reftemp) + M.beta * p_est);
        const double dhE = factor4 * (corner[0].y + corner[1].y + corner[4].y + corner[5].y);
        const int ft[4][2] = {{1, 0}, {2, 1}, {6, 2}, {8, 2}};
        double area = 0.0f, A[4];
        V3 nr[4];
#pragma unroll
        for (int q = 0; q < 4; q++) {
            const int t = ft[q][0], f = ft[q][1];
            tet_face(corner[tet_node(t, face_node(f, 0))], corner[tet_node(t, face_node(f, 1))],
                     corner[tet_node(t, face_node(f, 2))], A[q], nr[q]);
            area += A[q];
        }
        const double nx_ = factor4 * (nr[0].x + nr[1].x + nr[2].x + nr[3].x);
        const double ny_ = -1.0f * factor4 * (nr[0].y + nr[1].y + nr[2].y + nr[3].y);
        const double nz_ = factor4 * (nr[0].z + nr[1].z + nr[2].z + nr[3].z);
        area *= 0.5f;
        const double press_norm = a.pisos + rosubg * (a.rzbo - dhE);
        fx += factor4 * (press_norm * area * nx_);
        fy += factor4 * (press_norm * area * ny_);
        fz += factor4 * (press_norm * area * nz_);
    }
    if (a.time_step == 1) {  // restartTimestep == 0
        const double Fy = fy;
        if (Fy != 0.0) a.residual_fr[n] = Fy;
    }
    fy -= a.residual_fr[n];
    return V3{fx, fy, fz};
}

// SnacTractionBC's active branch (Snac/plugins/tractionBC/Force.c:43-268):
// on a right-wall node (i == nx), each incident element's right face (the
// triangles (1,2,6) and (1,6,5)) carries the fixed stress sxx = 1e8 Pa.
inline __device__ __noinline__ V3 traction_force(const double4* pos, int nx, int ny, int nz, int j, int k, V3 f) {
    Mesh m{};
    m.nx = nx;
    m.ny = ny;
    m.nz = nz;
    m.nnx = nx + 1;
    m.nny = ny + 1;
    double fx = f.x, fy = f.y, fz = f.z;
    const double factor4 = 1.0f / 4.0f;
    const double s00 = 1.0e+08, s01 = 0.0, s02 = 0.0, s10 = 0.0, s11 = 0.0, s12 = 0.0, s20 = 0.0, s21 = 0.0, s22 = 0.0;
    const int i = m.nnx - 1;
    for (int ne = 0; ne < 8; ne++) {
        const int ei = i - 1 + (ne & 1), ej = j - 1 + ((ne >> 1) & 1), ek = k - 1 + ((ne >> 2) & 1);
        if (ei < 0 || ej < 0 || ek < 0 || ei >= m.nx || ej >= m.ny || ek >= m.nz) continue;
        auto P = [&](int c) {
            const double4 p = pos[corner_node(m, ei, ej, ek, c)];
            return V3{p.x, p.y, p.z};
        };
        const V3 c1 = P(1), c2 = P(2), c5 = P(5), c6 = P(6);
        double a1, a2;
        V3 n1, n2;
        tet_face(c1, c2, c6, a1, n1);
        tet_face(c1, c6, c5, a2, n2);
        const double area = a1 + a2;
        const double nx_ = 0.5f * (n1.x + n2.x), ny_ = 0.5f * (n1.y + n2.y), nz_ = 0.5f * (n1.z + n2.z);
        fx += factor4 * area * (s00 * nx_ + s01 * ny_ + s02 * nz_);
        fy += factor4 * area * (s10 * nx_ + s11 * ny_ + s12 * nz_);
        fz += factor4 * area * (s20 * nx_ + s21 * ny_ + s22 * nz_);
    }
    return V3{fx, fy, fz};
}

// The tail of the node loop for node n with its summed force and inertial
// mass: force-BC plugins, FLAC local damping with the pre-update velocity
// (UpdateNode.c:102-104), v and x update, BC override; returns the node's
// max-BC-speed candidate.
__device__ __forceinline__ double node_update(const Mesh& m, const Fields& F, const Config& cfg, long long n, int i,
                                              int j, int k, double4 w, double4 p, uchar4 b, double fx, double fy,
                                              double fz, double imass) {
    const double dt = F.sc->dt;
    if (cfg.winkler && cfg.gravity > 0.0 && j == 0) {
        const WinklerArgs a{F.pos, F.mat, F.mats, F.residual_fr, F.sc->time_step, cfg.pisos, cfg.gravity, cfg.rzbo};
        const V3 r = winkler_force(a, m.nx, m.ny, m.nz, n, i, k, V3{fx, fy, fz});
        fx = r.x;
        fy = r.y;
        fz = r.z;
    }
    if (cfg.traction && i == m.nnx - 1) {
        const V3 r = traction_force(F.pos, m.nx, m.ny, m.nz, j, k, V3{fx, fy, fz});
        fx = r.x;
        fy = r.y;
        fz = r.z;
    }
    const double demf = cfg.demf;
    auto sgn = [](double x) { return x < 0 ? -1.0f : x > 0 ? +1.0f : 0.0f; };
    fx -= demf * sgn(w.x) * fabs(fx);
    fy -= demf * sgn(w.y) * fabs(fy);
    fz -= demf * sgn(w.z) * fabs(fz);
    double dw[3] = {dt * fx, dt * fy, dt * fz};
    dvz_n(dw, imass, recip(imass));
    w.x += dw[0];
    w.y += dw[1];
    w.z += dw[2];
    if (b.x != 255) w.x = F.vbc_val[b.x * 3 + 0];
    if (b.y != 255) w.y = F.vbc_val[b.y * 3 + 1];
    if (b.z != 255) w.z = F.vbc_val[b.z * 3 + 2];
    p.x += dt * w.x;
    p.y += dt * w.y;
    p.z += dt * w.z;
    F.pos_next[n] = p;
    F.vel[n] = w;
    F.force[n] = make_double4(fx, fy, fz, imass);
    if (!(isfinite(w.x) && isfinite(w.y) && isfinite(w.z))) report(F.sc, SNAC_GPU_ENAN, n);
    return (b.x != 255 || b.y != 255 || b.z != 255) ? sqrt(w.x * w.x + w.y * w.y + w.z * w.z) : 0.0;
}

// ---- what a block of nodes gathers -------------------------------------------------------
// A block takes blockDim.x consecutive nodes.  For each pair c of incident hexes
// it fetches the pair's chunk and the per-tet rows of every group that its nodes touch
// (gather_groups at most) into shared memory by bulk copies, so that all of
// a pair's terms are on their way at once without holding registers (direct
// loads kept 27 warps of 64 registers waiting on memory latency), and every
// thread then adds its own terms in the reference's order.  With one stage a
// pair is fetched when the block is done with the one before; grids that
// leave room in the SMs take two or four stages, which hide a small mesh's latency.
struct GatherSmem {
    unsigned long long full[4];  // mbarrier of each pair
    int g0[4], ng[4];            // first group and number of groups of each pair
    int gave_up;                 // a pair did not arrive in time: the block gathers no further tile
};
extern __shared__ __align__(16) unsigned char g_gather[];

// Waits for the phase of parity `phase` of an mbarrier, false if it has not
// completed after `limit` ns of the device's clock.  The usual wait ends
// within a few tries, each of which may suspend the thread for a time of the
// hardware's choosing; the clock is read, and the barrier only tested, after those.
__device__ __forceinline__ unsigned long long global_ns() {
    unsigned long long t;
    asm volatile("mov.u64 %0, %globaltimer;" : "=l"(t));
    return t;
}
__device__ __forceinline__ bool mbarrier_wait(unsigned bar, unsigned phase, unsigned long long limit) {
    unsigned done;
    for (int tries = 0; tries < 32; tries++) {
        asm volatile("{\n\t.reg .pred p;\n\t"
                     "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
                     "selp.u32 %0, 1, 0, p;\n\t}" : "=r"(done) : "r"(bar), "r"(phase) : "memory");
        if (done) return true;
    }
    for (const unsigned long long t0 = global_ns(); global_ns() - t0 < limit;) {
        asm volatile("{\n\t.reg .pred p;\n\t"
                     "mbarrier.test_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
                     "selp.u32 %0, 1, 0, p;\n\t}" : "=r"(done) : "r"(bar), "r"(phase) : "memory");
        if (done) return true;
    }
    return false;
}
constexpr unsigned long long GATHER_LIMIT = 1000000000ull;  // ns

template <int CHUNK, int TAIL>  // rows of a pair's chunk; rows after the four chunks
struct Gather {
    static constexpr int ROWS = CHUNK + TAIL;
    GatherSmem& S;
    const double* src;   // the groups
    int frows, stages, stage_entries;
    unsigned phase;      // parity of the mbarriers (blocks that take several tiles use them again)
    unsigned long long limit = GATHER_LIMIT;  // of the wait for a pair

    __device__ __forceinline__ double* stage(int c) const {
        return reinterpret_cast<double*>(g_gather) + (c % stages) * stage_entries;
    }
    __device__ __forceinline__ void plan(const Mesh& m, int lb) const {
        if (threadIdx.x < 4) {
            int lo, hi;
            const int n0 = lb * (int)blockDim.x, last = (int)m.nn - 1, n1 = n0 + (int)blockDim.x - 1;
            pair_hexes(m.nx, m.ny, m.nz, n0, n1 < last ? n1 : last, threadIdx.x, lo, hi);
            S.g0[threadIdx.x] = lo / GROUP;
            S.ng[threadIdx.x] = hi < lo ? 0 : hi / GROUP - lo / GROUP + 1;
        }
    }
    // by the whole of warp 0
    __device__ __forceinline__ void fetch(int c) const {
        const int lane = threadIdx.x, ng = S.ng[c];
        const unsigned bar = smem_addr(&S.full[c]);
        if (lane == 0)
            asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"(ng * ROWS * GROUP * 8) : "memory");
        __syncwarp();
        if (lane < ng) {
            const double* g = src + (long long)(S.g0[c] + lane) * (frows * GROUP);
            double* d = stage(c) + lane * (ROWS * GROUP);
            bulk_load(d, g + c * (CHUNK * GROUP), CHUNK * GROUP * 8, bar);
            if (TAIL > 0) bulk_load(d + CHUNK * GROUP, g + 4 * (CHUNK * GROUP), TAIL * GROUP * 8, bar);
        }
    }
    static __device__ __forceinline__ void bulk_load(double* d, const double* s, unsigned bytes, unsigned bar) {
        asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(
                         smem_addr(d)), "l"(s), "r"(bytes), "r"(bar) : "memory");
    }
    __device__ __forceinline__ bool wait(int c) const { return mbarrier_wait(smem_addr(&S.full[c]), phase, limit); }
    // Runs add(ne, base) for the hexes ne = 0..7 of node (i, j, k) in the reference's order
    // (HexaEL.c:529-573: pair by pair, i - 1 before i; absent hexes are
    // skipped, Force.c:92), base the hex's entry of row 0 of pair c's stage.
    // False in the threads for which a pair has not arrived within the limit: they
    // add nothing from it on, and warp 0 then fetches no more (so that the other
    // warps' waits run out too).
    template <class Add>
    __device__ __forceinline__ bool run(const Mesh& m, int lb, bool active, int i, int j, int k, Add&& add) const {
        plan(m, lb);
        __syncthreads();
        if (threadIdx.x < 32)
            for (int c = 0; c < stages; c++) fetch(c);
        int fetched = stages;
        bool ok = true;
#pragma unroll
        for (int c = 0; c < 4; c++) {
            if (ok && !wait(c)) {
                ok = false;
                S.gave_up = 1;
            }
            const int ej = j - 1 + (c & 1), ek = k - 1 + (c >> 1);
            if (ok && active && ej >= 0 && ej < m.ny && ek >= 0 && ek < m.nz) {
                const int row = (ej + ek * m.ny) * m.nx, g0 = S.g0[c] * GROUP;
                const double* const d = stage(c);
#pragma unroll
                for (int s = 0; s < 2; s++) {
                    const int ei = i - 1 + s;
                    if (ei < 0 || ei >= m.nx) continue;
                    const unsigned x = (unsigned)(row + ei - g0), g = x / GROUP;
                    add(2 * c + s, d + g * (ROWS * GROUP) + (x - g * GROUP));
                }
            }
            if (c + stages < 4) {
                __syncthreads();
                if (threadIdx.x < 32 && __all_sync(FULL, ok)) {
                    fetch(c + stages);
                    fetched++;
                }
            }
        }
        // the block stays until its copies have arrived, or the limit has passed again
        if (!ok && threadIdx.x < 32)
            for (int c = 0; c < fetched; c++) wait(c);
        return ok;
    }
};
// thread 0 of a block, before its first gather
__device__ __forceinline__ void gather_init(GatherSmem& S) {
    if (threadIdx.x == 0) {
#pragma unroll
        for (int c = 0; c < 4; c++)
            asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(smem_addr(&S.full[c])) : "memory");
        S.gave_up = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
}
// rows of a momentum gather's chunk and tail (see the group layouts above)
__host__ __device__ constexpr int force_chunk(bool constant_dt) { return constant_dt ? 40 : 30; }
__host__ __device__ constexpr int force_tail(bool constant_dt, bool vonly) { return vonly || constant_dt ? 10 : 20; }
__host__ __device__ constexpr size_t gather_stage_bytes(int rows, int threads) {
    return (size_t)gather_groups(threads) * rows * GROUP * sizeof(double);
}

// Snac_Force (Force.c:53-188) and the node update for the nodes of block lb.  With
// cfg.vonly the tet rows hold the volume: (g rho) V / 8 and (1/4 rho_i) V
// are formed here exactly as the element kernel forms them.
// VONLY: cfg.vonly (a template argument, so that the gather loop of each
// instance is straight-line code)
template <int DTTYPE, bool VONLY>
__device__ __forceinline__ void k_loop_nodes_body(GatherSmem& S, const Mesh& m, const Fields& F, const Config& cfg,
                                                  int lb, int stages, unsigned phase) {
    constexpr bool CDT = DTTYPE == SNAC_DT_CONSTANT;
    using G = Gather<force_chunk(CDT), force_tail(CDT, VONLY)>;
    const int n = lb * (int)blockDim.x + (int)threadIdx.x;
    const bool active = n < (int)m.nn;
    int i = 0, j = 0, k = 0;
    double4 w = make_double4(0.0, 0.0, 0.0, 0.0), p = w;
    uchar4 b = make_uchar4(255, 255, 255, 255);
    if (active) {  // on their way while the terms are fetched
        split3(n, m.nnx, m.nny, i, j, k);
        w = F.vel[n];
        p = F.pos[n];
        b = F.bc[n];
    }
    double fx = 0.0, fy = 0.0, fz = 0.0, imass = 0.0f;
    const double gr = VONLY ? cfg.gravity * cfg.m0.density : 0.0;
    const double f4r =
        VONLY ? (1.0f / 4.0f) * (DTTYPE == SNAC_DT_DYNAMIC ? F.sc->inertial_density0 : cfg.m0.density) : 0.0;
    const G gather{S, F.fterm, m.frows, stages, gather_groups(blockDim.x) * G::ROWS * GROUP, phase};
    const bool ok = gather.run(m, lb, active, i, j, k, [&](int ne, const double* r) {
#pragma unroll
        for (int idx = 0; idx < 5; idx++) {
            const double* const o = r + pair_slot(ne, idx) * GROUP;
            const double vg = r[(force_chunk(CDT) + node_tet(ne, idx)) * GROUP];
            imass += VONLY ? f4r * vg : CDT ? o[3 * ROW10] : r[(force_chunk(CDT) + NT + node_tet(ne, idx)) * GROUP];
            fx += o[0];
            fy += o[ROW10];
            fz += o[2 * ROW10];
            fy -= VONLY ? gr * vg * 0.125 : vg;
        }
    });
    if (!ok) report(F.sc, SNAC_GPU_ETIMEDOUT, n);
    double vcand = 0.0;
    if (active) vcand = node_update(m, F, cfg, n, i, j, k, w, p, b, fx, fy, fz, imass);
    // max |v| over velocity-BC nodes for Sync (exact: max does not round)
    for (int o = 16; o > 0; o >>= 1) vcand = fmax(vcand, __shfl_xor_sync(FULL, vcand, o));
    if ((threadIdx.x & 31) == 0 && vcand > 0.0)
        atomicMax(&F.sc->vmax_bits, (unsigned long long)__double_as_longlong(vcand));
}

// Nodes (threads) of a block.  Measured at 131 k / 1 M hexes, one stage: 64 threads 39 / 202 us, 128
// threads 40 / 208, 32 threads 40 / 199, two stages 41 / 215 (more blocks do
// more than more stages); direct loads, the form before, 41 / 232.
constexpr int NODE_THREADS = 64;
template <int DTTYPE, bool VONLY>
__global__ void __launch_bounds__(NODE_THREADS) k_loop_nodes(Mesh m, Fields F, Config cfg, int stages) {
    __shared__ GatherSmem S;
    gather_init(S);
    k_loop_nodes_body<DTTYPE, VONLY>(S, m, F, cfg, blockIdx.x, stages, 0);
}

// Slab launches of the step with the state in host memory: the same bodies
// over blocks [b0, b0 + gridDim.x) of the whole-mesh launch, so a slab's
// hexes (nodes) get exactly the arithmetic of the whole-mesh kernels.
template <int PLUGIN, bool ONE>
__global__ void __launch_bounds__(ELEM_WARPS * 32, elem_minb(PLUGIN)) k_calc_stresses_slab(Mesh m, Fields F, Config cfg,
                                                                                        int b0) {
    __shared__ __align__(16) ElemSmem S;
    stress_group<PLUGIN, ONE, false>(S, m, F, cfg, b0 + (int)blockIdx.x);
}

// UpdateElement.c:54-269 with this step's dt and the minimum length scale
// of the new geometry (the unfused element update)
template <int PLUGIN>
__global__ void __launch_bounds__(ELEM_WARPS * 32, 5) k_update_elements_slab(Mesh m, Fields F, Config cfg,
                                                                                          int b0) {
    update_group<PLUGIN>(m, F, cfg, 0, b0 + (int)blockIdx.x);
}

template <int DTTYPE, bool VONLY>
__global__ void __launch_bounds__(NODE_THREADS) k_loop_nodes_slab(Mesh m, Fields F, Config cfg, int b0, int stages) {
    __shared__ GatherSmem S;
    gather_init(S);
    k_loop_nodes_body<DTTYPE, VONLY>(S, m, F, cfg, b0 + (int)blockIdx.x, stages, 0);
}

// ======================================================================================
// Snac_EP_LoopElementsEnergy: Snac_HeatFlux (temperature/HeatFlux.c:60-200) and
// SnacTemperature_HeatFluxBC (temperature/VariableConditions.c:280-413)
// ======================================================================================
template <bool ONE>
__device__ __forceinline__ void heat_flux_tet(const Mesh& m, const Fields& F, const Config& cfg, const TetSlot& s,
                                              const TetView<TripleCoords>& w, const TetGeom& g, double* rows) {
    const DevMaterial& M = ONE ? cfg.m0 : F.mats[phase_of(F, s.e)];
    int ei, ej, ek;
    elem_ijk(m, s.e, ei, ej, ek);
    const double T[4] = {w.T(0), w.T(1), w.T(2), w.T(3)};
    double q[3], tsr = 0.0;
    const double zV = g.zV;
#pragma unroll
    for (int d = 0; d < 3; d++)
        q[d] = 1.0f * M.thermal_conduct *
               (T[0] * comp(g.n[1], d) * g.A[1] + T[1] * comp(g.n[2], d) * g.A[2] + T[2] * comp(g.n[3], d) * g.A[3] +
                T[3] * comp(g.n[0], d) * g.A[0]);
    dvk_n(q, 3.0, Z3);
    dvz_n(q, g.V, zV);
    if (cfg.thermal_stress) {
        const double bulkm = M.lambda + dv3(2.0f * M.mu);
        double temp = 0.25f * (T[0] + T[1] + T[2] + T[3]);
        double T0[4];
#pragma unroll
        for (int q = 0; q < 4; q++) T0[q] = F.vel[corner_node(m, ei, ej, ek, tet_node_rt(s.t, q))].w;
        double temp0 = 0.25f * (T0[0] + T0[1] + T0[2] + T0[3]);
        tsr = -1.0f * M.alpha * bulkm * (temp - temp0);
    }
    // flux BC on the x and z walls: remove the wall-normal part of grad T
    const bool on_wall = ei == 0 || ei == m.nx - 1 || ek == 0 || ek == m.nz - 1;
    double nrm[4][3];
    // (tet, face) pairs averaged for each wall, VariableConditions.c:311-367;
    // the shuffles run only in warps that hold a wall element (warp-uniform)
    if (__any_sync(FULL, on_wall)) {
        const int W[4][4][2] = {{{0, 2}, {1, 2}, {5, 0}, {6, 0}},
                                {{2, 0}, {3, 0}, {7, 0}, {8, 0}},
                                {{0, 1}, {2, 2}, {6, 1}, {7, 1}},
                                {{1, 1}, {3, 2}, {5, 1}, {8, 1}}};
#pragma unroll
        for (int w = 0; w < 4; w++)
#pragma unroll
            for (int d = 0; d < 3; d++) {
                double a[4];
#pragma unroll
                for (int r = 0; r < 4; r++) {
                    const int f = W[w][r][1];
                    double val = f == 0 ? comp(g.n[0], d) : f == 1 ? comp(g.n[1], d) : f == 2 ? comp(g.n[2], d) : comp(g.n[3], d);
                    a[r] = __shfl_sync(FULL, val, s.base + W[w][r][0]);
                }
                nrm[w][d] = 0.25f * (a[0] + a[1] + a[2] + a[3]);
            }
    }
    if (on_wall) {
        double normal[3];
        if (ei == 0)
            for (int d = 0; d < 3; d++) normal[d] = nrm[0][d];
        if (ei == m.nx - 1)
            for (int d = 0; d < 3; d++) normal[d] = nrm[1][d];
        if (ek == 0)
            for (int d = 0; d < 3; d++) normal[d] = nrm[2][d];
        if (ek == m.nz - 1)
            for (int d = 0; d < 3; d++) normal[d] = nrm[3][d];
        double gd[3];
        for (int d = 0; d < 3; d++)
            gd[d] = dvz(dv3(-1.0f * (T[0] * comp(g.n[1], d) * g.A[1] + T[1] * comp(g.n[2], d) * g.A[2] +
                                     T[2] * comp(g.n[3], d) * g.A[3] + T[3] * comp(g.n[0], d) * g.A[0])),
                        g.V, zV);
        double Fn = 0.0f;
        for (int d = 0; d < 3; d++) Fn += gd[d] * normal[d];
        for (int d = 0; d < 3; d++) q[d] -= Fn * normal[d];
    }
    // Per-tet terms of Snac_Heat (temperature/Heat.c:88-126) for the node
    // gather: (q . n) A / 6 of each face, the lumped heat capacity
    // Cp rho V / 8, and the thermal stress for the visco-plastic hook.
    if (s.lane < 30) {
        double* const h = rows + (threadIdx.x >> 5) * 3 + s.base / 10;
        const unsigned slots = TET_SLOTS[s.t];
        double hf[4];
#pragma unroll
        for (int f = 0; f < 4; f++) hf[f] = (q[0] * g.n[f].x + q[1] * g.n[f].y + q[2] * g.n[f].z) * g.A[f];
        dvk_n(hf, 6.0, Z6);
#pragma unroll
        for (int f = 0; f < 4; f++) h[corner_row(slots, f, NT)] = hf[f];
        // tetra density is set from TimeStepZero on, so the reference's
        // "density == 0" fallback (Heat.c:120-125) is never taken
        const double rho = cfg.has_density ? F.density[s.q] : M.density;
        h[4 * ROW10 + s.t * GROUP] = M.heat_capacity * ((rho)*g.V) * 0.125;  // rounds as / 8
        h[5 * ROW10 + s.t * GROUP] = tsr;
        // Heat.c:127-135, once per element; with one phase every element
        // gives the same value, so only element 0 (the first the reference
        // checks) evaluates it
        if (s.active && s.t == 0 && (!ONE || s.e == 0)) {
            double dt_thermal_to_mech = sqrt((M.lambda + 2.0f * M.mu) / M.density) * F.sc->min_length_scale /
                                        (M.thermal_conduct / (M.heat_capacity * M.density));
            if (!(dt_thermal_to_mech > 1.0)) report(F.sc, SNAC_GPU_EPHYSICS, s.e);
        }
    }
}

// The heat flux of group lb; MINLS: returns the tet's share of the minimum length scale.
template <bool ONE, bool MINLS>
__device__ __forceinline__ double heat_group(HeatSmem& S, const Mesh& m, const Fields& F, const Config& cfg, int lb) {
    TripleCoords& z = S.tri[threadIdx.x >> 5];
    fetch_triple<0>(m, F, lb, z);
    const TetLane L = tet_lane();
    const TetSlot s = tet_slot_of(m, L, lb);
    cp_async_wait_all();
    __syncwarp();
    TetGeom g;
    triple_geometry<false>(z, L, g);
    heat_flux_tet<ONE>(m, F, cfg, s, TetView<TripleCoords>{z, L.rows}, g, S.rows);
    bulk_fence();
    __syncthreads();
    if (threadIdx.x == 0) bulk_store(F.hflux + (long long)lb * (HROWS * GROUP), S.rows, HROWS * GROUP * 8);
    double ls = 1.0e+27f;
    if (MINLS) {
        ls = tet_length_scale(g);
        if (s.active && g.V == 0.0) report(F.sc, SNAC_GPU_EVOLUME, s.e);
    }
    if (threadIdx.x == 0) bulk_drain();
    return ls;
}

#ifndef SNAC_HEAT_MINB
#define SNAC_HEAT_MINB 6  // resident blocks per SM asked of the heat-flux kernel (80 registers; measured best)
#endif
template <bool ONE>
__global__ void __launch_bounds__(ELEM_WARPS * 32, SNAC_HEAT_MINB) k_heat_flux(Mesh m, Fields F, Config cfg,
                                                                           int opens_step) {
    if (opens_step && blockIdx.x == 0 && threadIdx.x == 0) count_step(F);  // the step's first kernel
    __shared__ __align__(16) HeatSmem S;
    heat_group<ONE, false>(S, m, F, cfg, blockIdx.x);
}


// ======================================================================================
// Snac_EP_LoopNodesEnergy: Snac_Heat for every node (temperature/Heat.c:64-140),
// the tet mean temperatures and the temperature BCs (Heat.c:47-62)
// ======================================================================================
constexpr int HEAT_CHUNK = 10, HEAT_TAIL = 10;  // face energy terms of a pair; lumped capacities
__device__ __forceinline__ void k_heat_nodes_body(GatherSmem& S, const Mesh& m, const Fields& F, const Config& cfg,
                                                  int lb, int stages, unsigned phase) {
    using G = Gather<HEAT_CHUNK, HEAT_TAIL>;
    const int n = lb * (int)blockDim.x + (int)threadIdx.x;
    const bool active = n < (int)m.nn;
    // only the w slots are written: other threads read this node's x, y, z
    double* const pw = reinterpret_cast<double*>(const_cast<double4*>(F.pos) + n) + 3;
    const double dt = F.sc->dt;
    int i = 0, j = 0, k = 0;
    double Told = 0.0;
    uchar4 b = make_uchar4(255, 255, 255, 255);
    if (active) {
        split3(n, m.nnx, m.nny, i, j, k);
        Told = *pw;
        b = F.bc[n];
    }
    double energy = 0.0f, lumpVolume = 0.0f;
    // the volumetric source of Snac_Heat is called with sourceterm = 0
    // (Heat.c:59), which adds +0 to the energy
    const double source = 0.0f;
    const G gather{S, F.hflux, HROWS, stages, gather_groups(blockDim.x) * G::ROWS * GROUP, phase};
    const bool ok = gather.run(m, lb, active, i, j, k, [&](int ne, const double* r) {
#pragma unroll
        for (int idx = 0; idx < 5; idx++) {
            energy += r[pair_slot(ne, idx) * GROUP];
            lumpVolume += r[(HEAT_CHUNK + node_tet(ne, idx)) * GROUP];
        }
    });
    if (!ok) report(F.sc, SNAC_GPU_ETIMEDOUT, n);
    if (!active) return;
    double Tnew = Told + dv((energy + source) * -1.0f * dt, lumpVolume);
    if (F.tpre) F.tpre[n] = Tnew;
    if (b.w != 255) Tnew = F.tbc_val[b.w];
    reinterpret_cast<double*>(F.vel + n)[3] = Told;
    *pw = Tnew;
    if (!isfinite(Tnew)) report(F.sc, SNAC_GPU_ENAN, n);
}

// Slab launches of the energy hooks for the step with the state in host
// memory (see k_calc_stresses_slab): blocks [b0, b0 + gridDim.x) of the
// whole-mesh launch; the step was counted by its first kernel.
template <bool ONE>
__global__ void __launch_bounds__(ELEM_WARPS * 32, SNAC_HEAT_MINB) k_heat_flux_slab(Mesh m, Fields F, Config cfg,
                                                                                   int b0) {
    __shared__ __align__(16) HeatSmem S;
    heat_group<ONE, false>(S, m, F, cfg, b0 + (int)blockIdx.x);
}

// ======================================================================================
// AbstractContext_EP_Sync: _Snac_Context_Sync (Context.c:1208-1268), one thread
// ======================================================================================
__device__ __forceinline__ void sync_one(const Config& cfg, DevScalars* sc, double wave_speed) {
    // the reductions are read where the other blocks' atomics left them (L2)
    double vmax = __longlong_as_double((long long)atomicOr(&sc->vmax_bits, 0ull));
    const double vlb = 3.0e-11f;
    if (vmax < vlb) vmax = vlb;
    sc->vmax = vmax;
    double minLS = __longlong_as_double((long long)atomicOr(&sc->minls_bits, 0ull));
    sc->min_length_scale = minLS;
    if (sc->time_step == 0) sc->init_min_length_scale = minLS;
    sc->dt_rot = sc->dt;  // the element update of this step (done now, or deferred into the next kernel) used this dt
    if (cfg.dt_type == SNAC_DT_DYNAMIC) {
        sc->dt = minLS * 0.45f * cfg.strain_inert / vmax;
        sc->speed_of_sound = minLS * 0.5f / sc->dt;
        // Force.c:112-114 for phase 0, once per step instead of once per tet
        sc->inertial_density0 = dv(cfg.m0.lambda + 2.0f * cfg.m0.mu, sc->speed_of_sound * sc->speed_of_sound);
    } else if (cfg.dt_type == SNAC_DT_WAVE) {
        sc->speed_of_sound = wave_speed;
        sc->dt = 0.5f * minLS / sc->speed_of_sound;
    }
    sc->vmax_bits = 0ull;
    sc->minls_bits = 0x7ff0000000000000ull;  // +inf
}

// The minimum length scale of the new coordinates and Sync in one launch:
// the last block to finish (counted in DevScalars, reset by that block) runs
// Sync on the completed reductions.
// PER_TET: a thread per tet instead of a thread per hex.  A hex's ten tets share
// their corner loads and edge differences in one thread, which is the better
// form once the GPU is full (131 k hexes: 21 against 42 us); a small mesh's one
// wave is done sooner with a tenth of the work per thread.
constexpr int MINLS_THREADS = 128;
static_assert(MINLS_THREADS == ELEM_WARPS * 32, "both forms have blocks of one size");
template <bool PER_TET>
__global__ void __launch_bounds__(MINLS_THREADS) k_min_length_scale_sync(Mesh m, Fields F, Config cfg,
                                                                         double wave_speed) {
    double ls;
    if (PER_TET) {
        __shared__ __align__(16) TripleCoords tri[ELEM_WARPS];
        TripleCoords& z = tri[threadIdx.x >> 5];
        fetch_triple<0>(m, F, blockIdx.x, z);
        const TetLane L = tet_lane();
        const TetSlot s = tet_slot_of(m, L, blockIdx.x);
        cp_async_wait_all();
        __syncwarp();
        TetGeom g;
        triple_geometry<false>(z, L, g);
        ls = tet_length_scale(g);
        if (s.active && g.V == 0.0) report(F.sc, SNAC_GPU_EVOLUME, s.e);
    } else {
        ls = hex_min_length_scale(m, F, blockIdx.x);
    }
    for (int o = 16; o > 0; o >>= 1) ls = fmin(ls, __shfl_xor_sync(FULL, ls, o));
    // the block's minimum in one atomic (fewer atomics on the one address),
    // fenced so that it is visible device-wide before the block is counted
    __shared__ double wmin[MINLS_THREADS / 32];
    __shared__ bool last;
    if ((threadIdx.x & 31) == 0) wmin[threadIdx.x >> 5] = ls;
    __syncthreads();
    if (threadIdx.x == 0) {
        double b = wmin[0];
#pragma unroll
        for (int w = 1; w < MINLS_THREADS / 32; w++) b = fmin(b, wmin[w]);
        atomicMin(&F.sc->minls_bits, (unsigned long long)__double_as_longlong(b));
        __threadfence();
        last = atomicAdd(&F.sc->blocks_done, 1u) == gridDim.x - 1;
    }
    __syncthreads();
    if (last && threadIdx.x == 0) {
        __threadfence();
        sync_one(cfg, F.sc, wave_speed);
        F.sc->blocks_done = 0u;
    }
}

// Temperature runs: the minimum length scale of step n together with the
// heat flux of step n+1 (Snac_HeatFlux, temperature/HeatFlux.c:60-200, and
// its wall BC), which reads the same coordinates x^{n+1} and node
// temperatures T^{n+1}: one geometry evaluation instead of two.  One thread
// per tet, as k_heat_flux; each block's minimum goes to one of 32 slots
// (non-returning atomics spread over addresses, so that the many small
// blocks neither queue on one address nor wait for a counter), and
// k_slots_sync then takes the minimum of the slots and runs Sync.  The tet's
// share of the minimum is RN(V / max_f A_f) from the heat flux's own face areas:
// max_f RN(RN(sqrt(s_f)) / 2) = RN(RN(sqrt(max_f s_f)) / 2), square root and
// halving being monotonic and correctly rounded (faces with a NaN area are
// skipped by both forms), so the minimum has the bits of
// hex_min_length_scale.
#ifndef SNAC_HEAT_MINLS_MINB
#define SNAC_HEAT_MINLS_MINB 6  // resident blocks per SM asked of the kernel below (80 registers: 400 us at 1 M hexes; 5: 414, 4: 447)
#endif
template <bool ONE>
__global__ void __launch_bounds__(ELEM_WARPS * 32, SNAC_HEAT_MINLS_MINB)
    k_heat_flux_min_length_scale(Mesh m, Fields F, Config cfg) {
    __shared__ __align__(16) HeatSmem S;
    double ls = heat_group<ONE, true>(S, m, F, cfg, blockIdx.x);
    for (int o = 16; o > 0; o >>= 1) ls = fmin(ls, __shfl_xor_sync(FULL, ls, o));
    __shared__ double wmin[ELEM_WARPS];
    if ((threadIdx.x & 31) == 0) wmin[threadIdx.x >> 5] = ls;
    __syncthreads();
    if (threadIdx.x == 0) {
        double b = wmin[0];
#pragma unroll
        for (int w = 1; w < ELEM_WARPS; w++) b = fmin(b, wmin[w]);
        atomicMin(&F.sc->minls_slot[blockIdx.x & 31], (unsigned long long)__double_as_longlong(b));
    }
}

}  // namespace snac
