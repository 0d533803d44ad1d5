// launch.h -- host-side launchers of the kernel translation units.
#pragma once

#include <cuda_runtime.h>

#include "layout.h"

namespace dmd {

// Launch with programmatic stream serialisation: the kernel may be set up on the
// device while the kernel before it in the stream still runs, and waits for
// that kernel's completion in its own chain_wait() (device.cuh).  Saves about
// 1 us of launch latency per kernel of the step's chain.
// The rule for such a kernel: every thread that stays calls chain_wait(); before
// it, a kernel stores nothing and loads only what the kernel directly before it
// does not write (k_kick_drift, k_shake, k_kick2, k_rattle, k_replica_update and
// k_pme_convert load ahead; the others call it first).  Whatever ran earlier is
// complete by then: chain_wait() lets the next kernel be set up only after its
// own wait, so a kernel's blocks start when the one two before it has ended.
template <typename... P, typename... A>
inline void launch_chained_smem(void (*kernel)(P...), int grid, int block, int smem, cudaStream_t st, A... args) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(static_cast<unsigned>(grid));
    cfg.blockDim = dim3(static_cast<unsigned>(block));
    cfg.dynamicSmemBytes = static_cast<size_t>(smem);
    cfg.stream = st;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    cudaLaunchKernelEx(&cfg, kernel, static_cast<P>(args)...);
}
template <typename... P, typename... A>
inline void launch_chained(void (*kernel)(P...), int grid, int block, cudaStream_t st, A... args) {
    launch_chained_smem(kernel, grid, block, 0, st, args...);
}

// k_list.cu: spatial sort + pair-list build for replicas whose `rebuild` flag
// is set, as one cooperative launch (returns at once when no replica rebuilds).
// chained: launched as launch_chained does.  Only in tables without a PME chain:
// 1,000 LJ atoms 1,721 -> 1,618 us per 100 steps, decane 4k 2,189 -> 2,095; with
// one, the pair kernel's blocks then come before the chain's first ones and
// water 9k went from 3,106 to 3,156 us per 50 steps.
void launch_rebuild(const Dev& d, const int* bin_rep, int n_sm, bool chained, cudaStream_t st, long long* nlaunch);

// k_nonbonded.cu: LJ + real-space Ewald over the pair list (replicas with `eval`).
// Pair energies and virial are summed only for replicas whose `want_e` is set.
// The mixed-precision kernels are persistent with blocks_per_sm blocks of 256
// threads per SM (1..3, LJ only 1..4) and come in two forms -- one warp per
// 32 x 32 chunk, or one warp per 8-atom i-cluster over its rows (needs d.cl_j).
// The form is the caller's option; the blocks follow from the list's size, a
// single system with a PME chain timing the other shapes too.  Results do not
// depend on the launch shape (one warp per work item, fixed-point sums).
enum NbForm { NB_CHUNK32 = 0, NB_CLUSTER8 = 1 };
// The FP64 kernel's blocks per SM, whatever blocks_per_sm says: what its registers
// and its shared memory allow.
constexpr int NB64_BLOCKS_PER_SM = 2;
void launch_nonbonded(const Dev& d, bool fp64, bool phys, int n_sm, int blocks_per_sm, int form,
                      cudaStream_t st, long long* nlaunch);
// Whether a kernel function (cudaGraphKernelNodeGetParams' func) is one of the
// pair kernels: the step graph gives every other kernel the higher priority.
bool is_nonbonded_kernel(const void* func);
// Per-device function attributes of the pair kernels (the shared-memory
// carveout and limit); called once per context before the first launch.  False
// where the device refuses the FP64 kernel's shared memory.
bool configure_nonbonded_kernels();

// k_forces.cu
// bonds, angles, dihedrals and the exclusion correction in one launch
void launch_bonded(const Dev& d, bool fp64, bool phys, cudaStream_t st, long long* nlaunch);
void launch_pme_spread(const Dev& d, bool fp64, cudaStream_t st, long long* nlaunch);
void launch_pme_convert(const Dev& d, bool fp64, int n_blocks, cudaStream_t st, long long* nlaunch);
void launch_pme_influence(const Dev& d, bool fp64, int n_blocks, cudaStream_t st,
                          long long* nlaunch);
void launch_pme_gather(const Dev& d, bool fp64, cudaStream_t st, long long* nlaunch);

// k_integrate.cu
// PASS_SECOND_ONLY: the second pass of a step whose first evaluation was not
// issued (REF: no replica needs it)
enum EvalPass { PASS_FIRST = 1, PASS_SECOND = 2, PASS_SINGLE = 3, PASS_SECOND_ONLY = 4 };
// What follows a step in the same launch, begun by k_replica_update: nothing, a
// step, or (REF) a step without its first evaluation.
enum NextStep { NEXT_NONE = 0, NEXT_STEP = 1, NEXT_SKIPS = 2 };
void launch_eval_begin(const Dev& d, int pass, cudaStream_t st, long long* nlaunch);
// the evaluation n_steps from now forms energies (a slot's own target aside)
void launch_mark_read(const Dev& d, int n_steps, cudaStream_t st, long long* nlaunch);
void launch_clear_forces(const Dev& d, cudaStream_t st, long long* nlaunch);
void launch_eval_end(const Dev& d, cudaStream_t st, long long* nlaunch);
void launch_kick_drift(const Dev& d, bool fp64, cudaStream_t st, long long* nlaunch);
// chained: the launch before it in the stream is the only thing it waits for
// (no join of other streams)
void launch_kick2(const Dev& d, bool andersen_ref, bool andersen_phys, bool chained, cudaStream_t st,
                  long long* nlaunch);
void launch_shake(const Dev& d, cudaStream_t st, long long* nlaunch);
void launch_rattle(const Dev& d, cudaStream_t st, long long* nlaunch);
void launch_replica_update(const Dev& d, int next, cudaStream_t st, long long* nlaunch);
void launch_apply_scale(const Dev& d, bool fp64, cudaStream_t st, long long* nlaunch);
void launch_finalize_velocities(const Dev& d, cudaStream_t st, long long* nlaunch);
// atoms a0 .. a0 + n - 1 (one replica's) to and from pinned host memory: which 0
// positions, 1 velocities, 2 forces (export only); rows: [n][3], otherwise three
// arrays `stride` doubles apart
void launch_export_state(const Dev& d, int a0, int n, int which, bool rows, long long stride, double* out,
                         cudaStream_t st, long long* nlaunch);
void launch_import_state(const Dev& d, int r, int a0, int n, int which, bool rows, long long stride, const double* in,
                         cudaStream_t st, long long* nlaunch);
void launch_request_rebuild(const Dev& d, int r, cudaStream_t st, long long* nlaunch);
void launch_energy_reduce(const Dev& d, cudaStream_t st, long long* nlaunch);
// replica r's frame (step, time, box, positions, velocities) into `out`
// (3 + 6 n_atoms doubles), state unchanged
void launch_frame_snapshot(const Dev& d, int r, int n_atoms, double* out, cudaStream_t st, long long* nlaunch);
void launch_write_mirror(const Dev& d, bool fp64, cudaStream_t st, long long* nlaunch);

}  // namespace dmd
