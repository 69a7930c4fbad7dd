// snac_launch.cuh — launches of the element kernels, which are compiled in
// files of their own.
//
// The compiler allocates the registers of a kernel together with those of the
// functions it calls (ieee_div, any_face, dp_return_map, its own slow paths), and
// those with the other kernels that call them.  In one file the result
// depended on how that file was cut among threads, which changes from build to
// build: k_fused_step of the plastic hook took 116 registers or 128 with
// 32 bytes spilled, the plastic class tiles spilled 0 or 236 bytes, and
// 24 models of up to 48x24x48 took 568 or 651 us a step.  So each file holds the
// kernels of one budget (resident blocks per SM: elem_minb, and the bounds beside the
// other kernels) and is compiled in one piece; the code is then the same in every build.
//   elements_mohr_coulomb.cu   plastic, visco-plastic: 4 blocks per SM
//   elements_drucker_prager.cu visco-plastic with a Drucker-Prager phase: 4
//   elements_linear.cu         elastic, Maxwell, element update: 5
//   heat.cu                    heat flux: 6
//   batch_yielding.cu          class tiles, plastic and visco-plastic: 4
//   batch_linear.cu            class tiles, the others and the heat flux: 5
//   batch_any.cu               tiles with the run-time switch: 4
//   adjoint_tets.cu            reverse of a tet: 1
// The templates below are defined beside their instantiations.
#pragma once

#include <atomic>

#include "snac_adjoint.cuh"
#include "snac_batch.cuh"
#include "snac_kernels.cuh"

namespace snac {

struct ElemGrid {
    unsigned blocks;
    cudaStream_t stream;
};

// one_phase: the model has no phase array (the kernels' ONE)
template <int P>
void run_calc_stresses(ElemGrid g, bool one_phase, const Mesh& m, const Fields& F, const Config& c);
template <int P>
void run_calc_stresses_slab(ElemGrid g, bool one_phase, const Mesh& m, const Fields& F, const Config& c, int b0);
template <int P>
void run_fused_step(ElemGrid g, bool one_phase, const Mesh& m, const Fields& F, const Config& c);
template <int P>
void run_fused_stress(ElemGrid g, bool one_phase, const Mesh& m, const Fields& F, const Config& c);
template <int P>
void run_update_elements(ElemGrid g, const Mesh& m, const Fields& F, const Config& c, int pending);
template <int P>
void run_update_elements_slab(ElemGrid g, const Mesh& m, const Fields& F, const Config& c, int b0);

void run_heat_flux(ElemGrid g, bool one_phase, const Mesh& m, const Fields& F, const Config& c, int opens_step);
void run_heat_flux_slab(ElemGrid g, bool one_phase, const Mesh& m, const Fields& F, const Config& c, int b0);
void run_heat_flux_min_length_scale(ElemGrid g, bool one_phase, const Mesh& m, const Fields& F, const Config& c);

template <int OP>
void run_tiles(ElemGrid g, const ModelDesc* D, const int2* tiles, int n);
template <int OP, int P, int TEMP>
void run_class_tiles(ElemGrid g, const ModelDesc* D, const int2* tiles, int n);

// returns the status of raising the kernel's limit of shared memory
template <int P>
cudaError_t run_adj_tet(int device, ElemGrid g, const Mesh& m, const Fields& F, const Config& c, const AdjState& S,
                        const AdjBufs& B, int rotate, int first_rev, double dt);

// Raises a kernel's limit of dynamic shared memory to `most`, the largest size
// that any launch of it asks for.  The limit belongs to the kernel on a
// device, not to a handle: were it set to what each launch needs, one thread
// could lower it between another's call and launch.  So it takes one value only.
template <auto KERNEL>
cudaError_t allow_smem(int device, size_t most) {
    static std::atomic<unsigned long long> done{0};  // devices 0 to 63
    const unsigned long long bit = device < 64 ? 1ull << device : 0ull;
    if (done.load(std::memory_order_acquire) & bit) return cudaSuccess;
    const cudaError_t e = cudaFuncSetAttribute(KERNEL, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)most);
    if (e == cudaSuccess) done.fetch_or(bit, std::memory_order_release);
    return e;
}

}  // namespace snac
