// snac_kernels_api.cuh — the kernels that only snac_api.cu launches: the
// temperature of the nodes, Sync, topography diffusion, transfers, the
// self-test, and the batch's and the adjoint's launches over models and nodes.
// (The other headers hold templates and device functions; the files that
// instantiate the element kernels include them too, see snac_launch.cuh.)
#pragma once

#include <math_constants.h>

#include "snac_adjoint.cuh"
#include "snac_batch.cuh"
#include "snac_kernels.cuh"

namespace snac {

// ---- energy hooks: the node loop (k_heat_nodes_body) ------------------------------------
// opens_step: the step's first kernel (its heat flux was formed at the end
// of the previous step): timeStep++, currentTime += dt
__global__ void __launch_bounds__(NODE_THREADS) k_heat_nodes(Mesh m, Fields F, Config cfg, int opens_step, int stages) {
    if (opens_step && blockIdx.x == 0 && threadIdx.x == 0) count_step(F);
    __shared__ GatherSmem S;
    gather_init(S);
    k_heat_nodes_body(S, m, F, cfg, blockIdx.x, stages, 0);
}

__global__ void __launch_bounds__(NODE_THREADS) k_heat_nodes_slab(Mesh m, Fields F, Config cfg, int b0, int stages) {
    __shared__ GatherSmem S;
    gather_init(S);
    k_heat_nodes_body(S, m, F, cfg, b0 + (int)blockIdx.x, stages, 0);
}

// ---- Sync ----------------------------------------------------------------------------
// One warp after k_heat_flux_min_length_scale: the minimum over its
// slots (exact: min does not round), the slots reset, then Sync.
__global__ void k_slots_sync(Config cfg, DevScalars* sc, double wave_speed) {
    const int l = threadIdx.x;
    unsigned long long v = sc->minls_slot[l];
    sc->minls_slot[l] = 0x7ff0000000000000ull;
    for (int o = 16; o > 0; o >>= 1) {
        const unsigned long long w = __shfl_xor_sync(FULL, v, o);
        v = w < v ? w : v;
    }
    if (l == 0) {
        if (v < sc->minls_bits) sc->minls_bits = v;
        sync_one(cfg, sc, wave_speed);
    }
}

__global__ void k_sync(Config cfg, DevScalars* sc, double wave_speed) {
    if (threadIdx.x != 0 || blockIdx.x != 0) return;
    sync_one(cfg, sc, wave_speed);
}

// max |v| over the velocity-BC nodes from the current velocities, for a
// Sync that does not follow the node loop (step zero, hook-by-hook callers)
__device__ __forceinline__ void k_vmax_body(const Mesh& m, const Fields& F, int lb) {
    long long n = (long long)lb * blockDim.x + threadIdx.x;
    double vcand = 0.0;
    if (n < m.nn) {
        uchar4 b = F.bc[n];
        if (b.x != 255 || b.y != 255 || b.z != 255) {
            double4 w = F.vel[n];
            vcand = sqrt(w.x * w.x + w.y * w.y + w.z * w.z);
        }
    }
    for (int o = 16; o > 0; o >>= 1) vcand = fmax(vcand, __shfl_xor_sync(FULL, vcand, o));
    if ((threadIdx.x & 31) == 0 && vcand > 0.0)
        atomicMax(&F.sc->vmax_bits, (unsigned long long)__double_as_longlong(vcand));
}

// With Sync in the same launch, run by the last block as in k_min_length_scale_sync
// (both are latency alone: one launch less per hook-by-hook step).
__global__ void __launch_bounds__(256) k_vmax_sync(Mesh m, Fields F, Config cfg, double wave_speed) {
    k_vmax_body(m, F, blockIdx.x);
    __threadfence();  // each warp's maximum is visible device-wide before the block is counted
    __syncthreads();
    if (threadIdx.x != 0 || atomicAdd(&F.sc->blocks_done, 1u) != gridDim.x - 1) return;
    __threadfence();
    sync_one(cfg, F.sc, wave_speed);
    F.sc->blocks_done = 0u;
}

// ======================================================================================
// Surface-topography diffusion (UpdateNode.c:161-857, cartesian), after the node update.
// The reference runs getMaxTopoGrad, DiffTopo + UpdateInteriorTopo and
// AdjustEdgeTopo inside its node loop, node after node: a top node sees its
// -x and -z neighbours already finished (moved, diffused, edge-copied) and
// its +x and +z neighbours not yet moved this step (their start-of-step
// coordinates).  That is a wavefront over the top surface's anti-diagonals
// i + k = d: one block walks the diagonals in order, the nodes of a diagonal
// in parallel.  topoGradMax is the running max in node order (a prefix max,
// exact in any association), never reset between steps.
// old: start-of-step coordinates; cur: after this step's node update (updated in place).
// tgrad: scratch of (nnx * nnz) doubles.
// ======================================================================================
__global__ void __launch_bounds__(1024) k_topo(Mesh m, const double4* __restrict__ old, double4* cur, Config cfg,
                                               DevScalars* sc, double* tgrad) {
    __shared__ double chunk_max[1024];
    if (sc->time_step <= 1) return;
    const int nnx = m.nnx, nnz = m.nnz, T = blockDim.x, tid = threadIdx.x;
    const long long top = (long long)(m.nny - 1) * nnx, plane = (long long)nnx * m.nny;
    const long long N = (long long)nnx * nnz;
    auto id = [&](int i, int k) { return (long long)i + top + (long long)k * plane; };
    auto interior = [&](int i, int k) { return i > 0 && i < nnx - 1 && k > 0 && k < nnz - 1; };
    // getMaxTopoGrad (:161-260), called from UpdateNodeMomentum when topo_kappa > 0
    for (long long p = tid; p < N; p += T) {
        const int i = (int)(p % nnx), k = (int)(p / nnx);
        double g = -CUDART_INF;
        if (cfg.topo_kappa > 0 && interior(i, k)) {
            const double4 X0 = cur[id(i, k)], xR = old[id(i + 1, k)], xF = old[id(i, k + 1)];
            const double dydx = (xR.y - X0.y) / (xR.x - X0.x);
            const double dydz = (xF.y - X0.y) / (xF.z - X0.z);
            g = sqrt(dydx * dydx + dydz * dydz);
        }
        tgrad[p] = g;
    }
    __syncthreads();
    // running max in node order: each thread a contiguous chunk, then the chunk prefixes
    const long long C = (N + T - 1) / T, lo = tid * C, hi = lo + C < N ? lo + C : N;
    double cm = -CUDART_INF;
    for (long long p = lo; p < hi; p++) cm = cm > tgrad[p] ? cm : tgrad[p];
    chunk_max[tid] = cm;
    __syncthreads();
    if (tid == 0) {
        double run = sc->topo_grad_max;
        for (int t = 0; t < T; t++) {
            const double c = chunk_max[t];
            chunk_max[t] = run;  // the max before chunk t
            run = run > c ? run : c;
        }
        sc->topo_grad_max = run;
    }
    __syncthreads();
    double run = chunk_max[tid];
    for (long long p = lo; p < hi; p++) {
        run = run > tgrad[p] ? run : tgrad[p];
        tgrad[p] = run;  // topoGradMax as node p's DiffTopo sees it
    }
    __syncthreads();
    const double kdt = cfg.topo_kappa * sc->dt;
    for (int d = 0; d <= (nnx - 1) + (nnz - 1); d++) {
        const int i0 = d - (nnz - 1) > 0 ? d - (nnz - 1) : 0, i1 = d < nnx - 1 ? d : nnx - 1;
        for (int i = i0 + tid; i <= i1; i += T) {
            const int k = d - i;
            if (tgrad[i + (long long)k * nnx] < cfg.topo_crit) continue;  // "topoGradMax < topoGradCriterion"
            double4& X0 = cur[id(i, k)];
            if (interior(i, k)) {
                // DiffTopo (:359-506) and UpdateInteriorTopo (:647-715)
                const double4 xR = old[id(i + 1, k)], xF = old[id(i, k + 1)];
                const double4 xL = cur[id(i - 1, k)], xB = cur[id(i, k - 1)];
                const double dydx1 = (xR.y - X0.y) / (xR.x - X0.x);
                const double dydx2 = (X0.y - xL.y) / (X0.x - xL.x);
                const double d2ydx2 = (dydx1 - dydx2) / (0.5f * (xR.x - xL.x));
                const double dydz1 = (xF.y - X0.y) / (xF.z - X0.z);
                const double dydz2 = (X0.y - xB.y) / (X0.z - xB.z);
                const double d2ydz2 = (dydz1 - dydz2) / (0.5f * (xF.z - xB.z));
                const double lapl_topo = d2ydx2 + d2ydz2;
                X0.y += kdt * lapl_topo;
            } else {
                // AdjustEdgeTopo (:716-857): copy the neighbour's height inward
                bool h1 = false, h2 = false;
                double y1 = 0.0, y2 = 0.0;
                if (i == 0) {
                    h1 = true;
                    y1 = old[id(1, k)].y;
                } else if (i == nnx - 1) {
                    h1 = true;
                    y1 = cur[id(nnx - 2, k)].y;
                }
                if (k == 0) {
                    h2 = true;
                    y2 = old[id(i, 1)].y;
                } else if (k == nnz - 1) {
                    h2 = true;
                    y2 = cur[id(i, nnz - 2)].y;
                }
                if (h1 && !h2) X0.y = y1;
                else if (!h1 && h2) X0.y = y2;
                else if (h1 && h2) X0.y = 0.5f * (y1 + y2);
            }
        }
        __syncthreads();
    }
}

// ---- self-test of the straight-line division against the IEEE quotient -------------------
__device__ __forceinline__ unsigned long long splitmix64(unsigned long long& x) {
    unsigned long long z = (x += 0x9e3779b97f4a7c15ull);
    z = (z ^ (z >> 30)) * 0xbf58476d1ce4e5b9ull;
    z = (z ^ (z >> 27)) * 0x94d049bb133111ebull;
    return z ^ (z >> 31);
}
__device__ __forceinline__ bool same_bits(double a, double b) {
    return __double_as_longlong(a) == __double_as_longlong(b) || (a != a && b != b);
}
__global__ void k_selftest_division(long long n, unsigned long long seed, unsigned long long* bad) {
    long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    unsigned long long st = seed ^ (0x632be59bd9b4e019ull * (unsigned long long)(i + 1));
    unsigned long long local = 0;
    for (; i < n; i += (long long)gridDim.x * blockDim.x) {
        unsigned long long a = splitmix64(st), b = splitmix64(st), c = splitmix64(st);
        // random significands, exponents spread over +-300 (x) and +-130 (y), random signs
        double x = __longlong_as_double((long long)((a & 0x800fffffffffffffull) | ((unsigned long long)(1023 + (int)(c % 601) - 300) << 52)));
        double y = __longlong_as_double((long long)((b & 0x800fffffffffffffull) | ((unsigned long long)(1023 + (int)((c >> 20) % 261) - 130) << 52)));
        if ((c >> 40) % 5 == 0) x = rint(x * 1e-3) * y;         // quotients that are exact or near ties
        if ((c >> 44) % 97 == 0) x = ((c >> 50) & 1) ? 0.0 : -0.0;
        // about 1 in 16: an operand drawn from every exponent (subnormals,
        // zeros' neighbours, overflow range, Inf and NaN) to exercise the window tests
        unsigned long long d = splitmix64(st);
        if ((d & 15) == 0) x = __longlong_as_double((long long)((a & 0x800fffffffffffffull) | ((d >> 8) % 2048) << 52));
        if (((d >> 4) & 15) == 0) y = __longlong_as_double((long long)((b & 0x800fffffffffffffull) | ((d >> 20) % 2048) << 52));
        local += !same_bits(dv(x, y), x / y);
        local += !same_bits(dvz(x, y, recip(y)), x / y);
        const double y1 = __longlong_as_double((long long)((a & 0x000fffffffffffffull) | ((unsigned long long)(1023 + (int)((c >> 12) % 64)) << 52)));
        if (__double2loint(y1) != -1) local += !same_bits(recip_mid(y1), 1.0 / y1);
        // the joint root and reciprocal of tet_geometry_tame over its range, but
        // for the roots its caller turns away
        const double q = __longlong_as_double((long long)((b & 0x000fffffffffffffull) | ((unsigned long long)(1023 + (int)((c >> 8) % 1283) - 714) << 52)));
        double root, zroot;
        sqrt_recip(q, root, zroot);
        if (__double2loint(root) != -1) local += !same_bits(root, sqrt(q)) + !same_bits(zroot, 1.0 / root);
        local += !same_bits(dv3(x), x / 3.0) + !same_bits(dv6(x), x / 6.0);
        local += !same_bits(dv9(x), x / 9.0) + !same_bits(dv10(x), x / 10.0);
    }
    if (local) atomicAdd(bad, local);
}

// the short root and reciprocals of n given operands
__global__ void k_selftest_roots(long long n, const double* q, double* root, double* recip_root, double* recip) {
    const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    sqrt_recip(q[i], root[i], recip_root[i]);
    recip[i] = recip_mid(q[i]);
}

// ---- self-test of the gather's bounded wait ---------------------------------------------
// One block gathers a small mesh's heat groups twice, with `stages` stages and
// `limit` ns for each wait.  The barrier of pair `late` (none if it is not 0 to 3) is
// told to expect 16 bytes more than the copies bring: that pair never completes,
// although every copy arrives.  out: threads whose first gather succeeded, whose
// second did, and the hexes added by all threads in the first.
__global__ void __launch_bounds__(NODE_THREADS) k_selftest_gather(Mesh m, const double* groups, int stages, int late,
                                                                  unsigned long long limit, int* out) {
    __shared__ GatherSmem S;
    gather_init(S);
    if (threadIdx.x == 0 && late >= 0 && late < 4)
        asm volatile("mbarrier.expect_tx.relaxed.cta.shared::cta.b64 [%0], 16;" ::"r"(smem_addr(&S.full[late])) : "memory");
    int i = 0, j = 0, k = 0;
    const bool active = threadIdx.x < m.nn;
    if (active) split3(threadIdx.x, m.nnx, m.nny, i, j, k);
    for (int pass = 0; pass < 2; pass++) {
        const Gather<HEAT_CHUNK, HEAT_TAIL> G{S, groups, HROWS, stages,
                                              gather_groups(NODE_THREADS) * (HEAT_CHUNK + HEAT_TAIL) * GROUP,
                                              (unsigned)pass, limit};
        int added = 0;
        const bool ok = G.run(m, 0, active, i, j, k, [&](int, const double* r) { added += *r == 0.0; });
        if (ok) atomicAdd(out + pass, 1);
        if (pass == 0 && added) atomicAdd(out + 2, added);
        __syncthreads();
        if (S.gave_up) break;
    }
}

// ---- host transfers: node fields between the packed double4 layout and
// the reference's interleaved (x, y, z) / scalar arrays -------------------------------------
// what: 0 = x, y, z of each double4 <-> 3 doubles per node; 1 = w <-> 1 double per node
__global__ void k_pack_nodes(const double4* __restrict__ src, double* __restrict__ dst, long long nn, int what) {
    long long n = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (n >= nn) return;
    double4 a = src[n];
    if (what == 0) {
        dst[n * 3 + 0] = a.x;
        dst[n * 3 + 1] = a.y;
        dst[n * 3 + 2] = a.z;
    } else {
        dst[n] = a.w;
    }
}

__global__ void k_unpack_nodes(double4* __restrict__ dst, const double* __restrict__ src, long long nn, int what) {
    long long n = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (n >= nn) return;
    double* d = reinterpret_cast<double*>(dst + n);
    if (what == 0) {
        d[0] = src[n * 3 + 0];
        d[1] = src[n * 3 + 1];
        d[2] = src[n * 3 + 2];
    } else {
        d[3] = src[n];
    }
}

// ---- arrays between the device and page-locked host memory that the device maps ---------
// A few dozen copies of a state's pieces cost several microseconds each,
// whatever their size; a kernel that writes the host's arrays itself costs
// one launch.  Rows: consecutive doubles of the host array; what: 0 the
// same doubles on the device, 1 the x, y, z of a double4 per three, 2 the w of a double4 per one.
struct HostRows {
    double* host;
    double* dev;
    long long n;   // doubles
    int what;
};
struct HostJob {
    static constexpr int MAX = 10;
    HostRows rows[MAX];
    long long first[MAX + 1];  // first unit (two doubles) of each piece
    int count;
};
__device__ __forceinline__ double* dev_double(const HostRows& r, long long i) {
    return r.what == 0 ? r.dev + i : r.what == 1 ? r.dev + i / 3 * 4 + i % 3 : r.dev + i * 4 + 3;
}
__global__ void __launch_bounds__(256) k_host_rows(HostJob J) {
    const long long stride = (long long)gridDim.x * blockDim.x;
    for (long long u = (long long)blockIdx.x * blockDim.x + threadIdx.x; u < J.first[J.count]; u += stride) {
        int a = 0;
        while (u >= J.first[a + 1]) a++;
        // pairs that start on 16-byte boundaries of the host array: where it
        // starts between two, its first unit is a single double
        const HostRows& r = J.rows[a];
        const int odd = (int)((unsigned long long)r.host >> 3) & 1;
        const long long i = (u - J.first[a]) * 2 - odd;
        if (i >= 0 && i + 1 < r.n) {
            *reinterpret_cast<double2*>(r.host + i) = make_double2(*dev_double(r, i), *dev_double(r, i + 1));
        } else {
            const long long x = i < 0 ? 0 : i;
            if (x < r.n) r.host[x] = *dev_double(r, x);
        }
    }
}

// The node state of nodes [0, nn) between the host's rows (3 doubles of
// coordinates, 3 of velocity, 1 of temperature per node) and the device's
// double4 rows (pos: x, y, z, T; vel: vx, vy, vz and the previous T, which
// stays); pos and vel always hold nn rows, a null host row (c, t, v) is
// skipped.
__global__ void k_unpack_node_state(double4* __restrict__ pos, const double* __restrict__ c,
                                    const double* __restrict__ t, double4* __restrict__ vel,
                                    const double* __restrict__ v, long long nn) {
    long long n = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (n >= nn) return;
    double* p = reinterpret_cast<double*>(pos + n);
    if (c) {
        p[0] = c[n * 3 + 0];
        p[1] = c[n * 3 + 1];
        p[2] = c[n * 3 + 2];
    }
    if (t) p[3] = t[n];
    if (v) {
        double* w = reinterpret_cast<double*>(vel + n);
        w[0] = v[n * 3 + 0];
        w[1] = v[n * 3 + 1];
        w[2] = v[n * 3 + 2];
    }
}

__global__ void k_pack_node_state(const double4* __restrict__ pos, double* __restrict__ c, double* __restrict__ t,
                                  const double4* __restrict__ vel, double* __restrict__ v, long long nn) {
    long long n = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (n >= nn) return;
    const double4 x = pos[n];
    if (c) {
        c[n * 3 + 0] = x.x;
        c[n * 3 + 1] = x.y;
        c[n * 3 + 2] = x.z;
    }
    if (t) t[n] = x.w;
    if (v) {
        const double4 w = vel[n];
        v[n * 3 + 0] = w.x;
        v[n * 3 + 1] = w.y;
        v[n * 3 + 2] = w.z;
    }
}

// _AbstractContext_Execute_Hook: timeStep++ and dt = dtFactor * dt (AbstractContext.c:874-890)
__global__ void k_begin_step(DevScalars* sc) {
    if (threadIdx.x == 0 && blockIdx.x == 0) {
        sc->time_step += 1;
        sc->dt = 1.0 * sc->dt;
        sc->current_time += sc->dt;
    }
}

// ---- batch: launches over the models -------------------------------------------------
// _Snac_Context_Sync of every model: one thread per model
__global__ void kb_sync(const ModelDesc* __restrict__ D, int n) {
    int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n) sync_one(D[i].cfg, D[i].F.sc, D[i].wave_speed);
}

// _AbstractContext_Execute_Hook of every model (a step that does not start
// with the fused kernel): timeStep++ and dt = dtFactor * dt
__global__ void kb_begin_step(const ModelDesc* __restrict__ D, int n) {
    int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n) {
        DevScalars* sc = D[i].F.sc;
        sc->time_step += 1;
        sc->dt = 1.0 * sc->dt;
        sc->current_time += sc->dt;
    }
}

__global__ void kb_status(const ModelDesc* __restrict__ D, int n, ModelStatus* out) {
    int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n) {
        const DevScalars* sc = D[i].F.sc;
        out[i].status = sc->status;
        out[i].pad = 0;
        out[i].err_index = sc->err_index;
        out[i].time_step = sc->time_step;
    }
}

// ---- adjoint: launches over nodes and hexes --------------------------------------------
// Node adjoints: gather the corner adjoints of tet pass n (fixed order), then
// the reverse of the node update of step n-1:
//   x^n = x^{n-1} + dt v^n,  v^n_c = v^{n-1}_c + dt F_d,c / m  (free components)
//   F_d = F (1 - demf sgn(v^{n-1}) sgn(F))
// cur = S^n (its force holds F_d and m of step n-1), prev = S^{n-1} (velocities).
__global__ void __launch_bounds__(NODE_THREADS) k_adj_nodes(Mesh m, Fields F, AdjState cur, AdjState prev, AdjBufs B,
                                                           int gather, int update, double dt, double demf, int stages) {
    __shared__ GatherSmem S;
    const int n = blockIdx.x * NODE_THREADS + threadIdx.x;
    const bool active = n < (int)m.nn;
    double4 xb = make_double4(0.0, 0.0, 0.0, 0.0), vb = xb;
    if (active) {
        xb = B.xbar[n];
        vb = B.vbar[n];
    }
    if (gather) {
        gather_init(S);
        int i = 0, j = 0, k = 0;
        if (active) split3(n, m.nnx, m.nny, i, j, k);
        const Gather<CCHUNK, 0> G{S, B.cbuf, CROWS, stages, gather_groups(NODE_THREADS) * CCHUNK * GROUP, 0};
        const bool ok = G.run(m, blockIdx.x, active, i, j, k, [&](int ne, const double* r) {
#pragma unroll
            for (int idx = 0; idx < 5; idx++) {
                const double* const o = r + pair_slot(ne, idx) * GROUP;
                xb.x += o[0];
                xb.y += o[ROW10];
                xb.z += o[2 * ROW10];
                vb.x += o[3 * ROW10];
                vb.y += o[4 * ROW10];
                vb.z += o[5 * ROW10];
            }
        });
        if (!ok) report(F.sc, SNAC_GPU_ETIMEDOUT, n);
    }
    if (!active) return;
    if (update) {
        vb.x += dt * xb.x;
        vb.y += dt * xb.y;
        vb.z += dt * xb.z;
        const double4 fd = cur.force[n];
        const double4 vp = prev.vel[n];
        const uchar4 bc = F.bc[n];
        const double mass = fd.w;
        double fb[3], mb = 0.0;
        const double vbc[3] = {vb.x, vb.y, vb.z};
        const double fdc[3] = {fd.x, fd.y, fd.z};
        const double vpc[3] = {vp.x, vp.y, vp.z};
        const bool fixed[3] = {bc.x != 255, bc.y != 255, bc.z != 255};
        double vout[3];
        const double im = 1.0 / mass;
        for (int c = 0; c < 3; c++) {
            if (fixed[c]) {
                fb[c] = 0.0;
                vout[c] = 0.0;
            } else {
                const double fdb = vbc[c] * dt * im;
                mb += -vbc[c] * dt * fdc[c] * (im * im);
                fb[c] = fdb * (1.0 - demf * sgnd(vpc[c]) * sgnd(fdc[c]));
                vout[c] = vbc[c];
            }
        }
        B.fbar[n] = make_double4(fb[0], fb[1], fb[2], mb);
        vb = make_double4(vout[0], vout[1], vout[2], 0.0);
    }
    B.xbar[n] = xb;
    B.vbar[n] = vb;
}

// loss on the top surface (j = nny - 1): per node w_v (v_y - tv)^2 + w_h (y - ty)^2,
// its gradient seeds the adjoints; every other node's adjoint starts at zero
__global__ void k_adj_loss(Mesh m, const double4* pos, const double4* vel, const double* tv, const double* ty,
                           double wv, double wh, double* terms, AdjBufs B) {
    long long n = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (n >= m.nn) return;
    int i, j, k;
    split3(n, m.nnx, m.nny, i, j, k);
    double4 xb = make_double4(0, 0, 0, 0), vb = make_double4(0, 0, 0, 0);
    if (j == m.nny - 1) {
        long long t = (long long)i + (long long)k * m.nnx;
        const double dv_ = vel[n].y - tv[t], dy = pos[n].y - ty[t];
        terms[t] = wv * dv_ * dv_ + wh * dy * dy;
        vb.y = 2.0 * wv * dv_;
        xb.y = 2.0 * wh * dy;
    }
    B.xbar[n] = xb;
    B.vbar[n] = vb;
    B.fbar[n] = make_double4(0, 0, 0, 0);
}

// up to 6 array copies in one launch (checkpoint save / restore), 64-bit words
struct CopyJob {
    unsigned long long* dst[7];
    const unsigned long long* src[7];
    long long n[7];
    int count;
};
__global__ void __launch_bounds__(256) k_copy_many(CopyJob J) {
    const long long stride = (long long)gridDim.x * blockDim.x;
    for (int a = 0; a < J.count; a++) {
        unsigned long long* d = J.dst[a];
        const unsigned long long* s = J.src[a];
        for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < J.n[a]; i += stride) d[i] = s[i];
    }
}

// per-element gradients: sum of the element's 10 tets in tet order
__global__ void k_adj_reduce(long long ne, const double* pbar, double* gc, double* gf, double* gv) {
    long long e = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (e >= ne) return;
    double a = 0, b = 0, c = 0;
    for (int t = 0; t < NT; t++) {
        a += pbar[(e * NT + t) * 3 + 0];
        b += pbar[(e * NT + t) * 3 + 1];
        c += pbar[(e * NT + t) * 3 + 2];
    }
    gc[e] = a;
    gf[e] = b;
    gv[e] = c;
}

}  // namespace snac
