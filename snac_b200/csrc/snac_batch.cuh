// snac_batch.cuh — one launch per kernel type for a whole ensemble of models.
//
// Every model of a batch keeps its own device buffers (the same layout as a
// single-model handle).  A batch adds a table of per-model descriptors
// (mesh, field pointers, configuration) and, for each kind of launch, a list
// of work tiles: (model, block index within that model).  A tile is exactly
// the work one block of the single-model kernel does, so the per-model
// results are the single-model results bit for bit; only the launch
// geometry changes.  A block copies its tile's descriptor to shared memory
// and calls the same kernel body as the single-model kernel.  With a grid
// smaller than the tile list, blocks stride over the list (a persistent
// grid whose size the autotuner chooses).
#pragma once

#include "snac_kernels.cuh"

namespace snac {

struct ModelDesc {
    Mesh m;
    Fields F;
    Config cfg;
    double wave_speed;
};
static_assert(sizeof(ModelDesc) % 8 == 0, "descriptor is copied as 64-bit words");

// per-model status gathered after a batch of steps
struct ModelStatus {
    int status;
    int pad;
    long long err_index;
    long long time_step;
};

// BOP_FUSED: the step's first element launch (models without temperature:
// pending element update + stress update; with temperature: the heat flux,
// the element update waiting for BOP_FUSED_STRESS after the energy hooks)
enum {
    BOP_FUSED = 0,
    BOP_HEAT_FLUX = 1,
    BOP_STRESS = 2,
    BOP_LOOP_NODES = 3,
    BOP_HEAT_NODES = 4,
    BOP_MINLS = 5,
    BOP_FUSED_STRESS = 6
};

__device__ __forceinline__ void load_desc(ModelDesc& dst, const ModelDesc* __restrict__ src) {
    constexpr int W = sizeof(ModelDesc) / 8;
    const long long* s = reinterpret_cast<const long long*>(src);
    long long* d = reinterpret_cast<long long*>(&dst);
    for (int i = threadIdx.x; i < W; i += blockDim.x) d[i] = s[i];
}

// What a tile costs beyond the single-model kernel's block is the chain list
// entry -> descriptor -> first loads, and the registers held across the body.
// The tiles of one block: at(i) is tile i of the list, whose model's descriptor
// is then in md for the whole block (the previous tile is done).  The list
// entry of the block's next tile is fetched a tile ahead, and a descriptor
// that is there already stays: consecutive tiles mostly are of one model.
struct Tiles {
    const ModelDesc* __restrict__ D;
    const int2* __restrict__ list;
    int n;
    int2 next;
    int model = -1;
    __device__ __forceinline__ Tiles(const ModelDesc* __restrict__ D_, const int2* __restrict__ l, int n_)
        : D(D_), list(l), n(n_), next(l[blockIdx.x]) {}  // (the grid is at most n blocks)
    __device__ __forceinline__ int at(int i, ModelDesc& md) {
        const int2 t = next;
        if (i + (int)gridDim.x < n) next = list[i + gridDim.x];
        __syncthreads();  // the previous tile is done with md and the staging
        if (t.x != model) {
            load_desc(md, D + t.x);
            model = t.x;
            __syncthreads();
        }
        return t.y;
    }
};

// the element bodies for a tile's model: phase 0 from the descriptor (in
// shared memory) when the model has one phase, else the model's phase table
union TileSmem {
    ElemSmem elem;
    HeatSmem heat;
};
template <int P, bool FUSED>
__device__ __forceinline__ void stress_any(TileSmem& S, const ModelDesc& md, int lb) {
    if (md.F.mat)
        stress_group<P, false, FUSED>(S.elem, md.m, md.F, md.cfg, lb);
    else
        stress_group<P, true, FUSED>(S.elem, md.m, md.F, md.cfg, lb);
}
__device__ __forceinline__ void heat_flux_any(TileSmem& S, const ModelDesc& md, int lb) {
    if (md.F.mat)
        heat_group<false, false>(S.heat, md.m, md.F, md.cfg, lb);
    else
        heat_group<true, false>(S.heat, md.m, md.F, md.cfg, lb);
}
// a model's first launch of a fused step: timeStep++, currentTime += dt
// (once per model), then the pending element update with the stress update,
// or with temperature the heat flux
__device__ __forceinline__ void open_step(const ModelDesc& md, int lb) {
    if (lb == 0 && threadIdx.x == 0) count_step(md.F);
}

// One element tile: OP for a model of plugin P
template <int OP, int P>
__device__ __forceinline__ void elem_tile(TileSmem& S, const ModelDesc& md, int lb, bool temperature) {
    if (OP == BOP_FUSED) {
        open_step(md, lb);
        if (temperature)
            heat_flux_any(S, md, lb);
        else
            stress_any<P, true>(S, md, lb);
    } else if (OP == BOP_FUSED_STRESS) {
        stress_any<P, true>(S, md, lb);
    } else if (OP == BOP_STRESS) {
        stress_any<P, false>(S, md, lb);
    } else {
        heat_flux_any(S, md, lb);
    }
}

// Element-tile kernels: the fused end-of-step/next-stress kernel (or its
// heat variant for models with temperature), the heat flux, the stress update.
template <int OP>
__global__ void __launch_bounds__(ELEM_WARPS * 32, 4)
    kb_elements(const ModelDesc* __restrict__ D, const int2* __restrict__ tiles, int ntiles) {
    __shared__ ModelDesc md;
    __shared__ __align__(16) TileSmem S;
    Tiles T(D, tiles, ntiles);
    for (int i = blockIdx.x; i < ntiles; i += gridDim.x) {
        const int b = T.at(i, md);
        const bool temp = md.cfg.temperature != 0;
        switch (md.cfg.constitutive) {
            case SNAC_RHEOLOGY_ELASTIC: elem_tile<OP, SNAC_RHEOLOGY_ELASTIC>(S, md, b, temp); break;
            case SNAC_RHEOLOGY_PLASTIC: elem_tile<OP, SNAC_RHEOLOGY_PLASTIC>(S, md, b, temp); break;
            case SNAC_RHEOLOGY_VISCOPLASTIC: elem_tile<OP, SNAC_RHEOLOGY_VISCOPLASTIC>(S, md, b, temp); break;
            default: elem_tile<OP, SNAC_RHEOLOGY_MAXWELL>(S, md, b, temp); break;
        }
    }
}

// The same element-tile kernels specialised for one rheology class (plugin,
// temperature on/off): the tile lists are grouped by class, and each class
// present gets its own launch, without the run-time switch (fewer registers).
// Resident blocks per SM asked of a class's kernel: as the single-model
// kernels, but five of the heat flux (with both forms of the phase table and the
// descriptor it spills twice as much at six; 24 models of up to 48x24x48: 460 us a
// step with four for every class, 456 so).
__host__ __device__ constexpr int tile_minb(int op, int plugin, bool temp) {
    return op == BOP_HEAT_FLUX || (op == BOP_FUSED && temp) ? 5 : elem_minb(plugin);
}
template <int OP, int P, int TEMP>
__global__ void __launch_bounds__(ELEM_WARPS * 32, tile_minb(OP, P, TEMP != 0))
    kb_elements_c(const ModelDesc* __restrict__ D, const int2* __restrict__ tiles, int ntiles) {
    __shared__ ModelDesc md;
    __shared__ __align__(16) TileSmem S;
    Tiles T(D, tiles, ntiles);
    for (int i = blockIdx.x; i < ntiles; i += gridDim.x) {
        const int b = T.at(i, md);
        elem_tile<OP, P>(S, md, b, TEMP != 0);
    }
}

// rheology classes of a batch: index = plugin slot * 2 + temperature
constexpr int NCLASS = 8;
__host__ __device__ constexpr int plugin_slot(int constitutive) {
    return constitutive == SNAC_RHEOLOGY_ELASTIC ? 0 : constitutive == SNAC_RHEOLOGY_PLASTIC ? 1
           : constitutive == SNAC_RHEOLOGY_VISCOPLASTIC                                  ? 2
                                                                                          : 3;
}

// Node-tile kernels (one thread per node, or per element for the minimum
// length scale); the block size is the tile size the tile list was built for.
// The gathers have one stage (node_stage_bytes of dynamic shared memory).
__host__ __device__ constexpr size_t node_stage_bytes(int op, int threads) {
    return gather_stage_bytes(op == BOP_HEAT_NODES ? HEAT_CHUNK + HEAT_TAIL : 50, threads);
}
constexpr int NODE_TILE_MAX = 256;  // nodes (threads) of the largest node tile
template <int OP>
__global__ void __launch_bounds__(NODE_TILE_MAX) kb_nodes(const ModelDesc* __restrict__ D, const int2* __restrict__ tiles, int ntiles) {
    __shared__ ModelDesc md;
    __shared__ GatherSmem S;
    if (OP != BOP_MINLS) gather_init(S);
    unsigned phase = 0;
    Tiles T(D, tiles, ntiles);
    for (int i = blockIdx.x; i < ntiles; i += gridDim.x, phase ^= 1) {
        const int b = T.at(i, md);
        if (OP != BOP_MINLS && S.gave_up) break;  // (T.at is a barrier: the whole block sees the same)
        if (OP == BOP_LOOP_NODES) {
            const bool vo = md.cfg.vonly != 0;
            switch (md.cfg.dt_type) {
                case SNAC_DT_CONSTANT:
                    k_loop_nodes_body<SNAC_DT_CONSTANT, false>(S, md.m, md.F, md.cfg, b, 1, phase);
                    break;
                case SNAC_DT_DYNAMIC:
                    if (vo) k_loop_nodes_body<SNAC_DT_DYNAMIC, true>(S, md.m, md.F, md.cfg, b, 1, phase);
                    else k_loop_nodes_body<SNAC_DT_DYNAMIC, false>(S, md.m, md.F, md.cfg, b, 1, phase);
                    break;
                default:
                    if (vo) k_loop_nodes_body<SNAC_DT_WAVE, true>(S, md.m, md.F, md.cfg, b, 1, phase);
                    else k_loop_nodes_body<SNAC_DT_WAVE, false>(S, md.m, md.F, md.cfg, b, 1, phase);
                    break;
            }
        } else if (OP == BOP_HEAT_NODES) {
            k_heat_nodes_body(S, md.m, md.F, md.cfg, b, 1, phase);
        } else {
            k_min_length_scale_body(md.m, md.F, b);
        }
    }
}

}  // namespace snac
