// prog_kernels.cuh -- host-side launchers of the solver kernels (implemented in prog_gs.cu and
// prog_kernels.cu).  Every launcher enqueues on the given stream and returns immediately.
#pragma once

#include <cuda_runtime.h>

#include "prog_common.cuh"

namespace gral {

// Boundary-condition event lists (PrognosticFlowfield.cs:595-696): for the W/E pass one list per
// row j of the columns i (ascending) that copy inflow; for the S/N pass one list per column i.
// Entry = index | (west_or_south << 16) | (east_or_north << 17).
struct BcLists {
    const int *we_ptr, *we_ev;   // we_ptr[j]..we_ptr[j+1]
    const int *sn_ptr, *sn_ev;   // sn_ptr[i]..sn_ptr[i+1]
};

// Full-height staging copies of the host fields of one situation: [NII+2][NJJ+2][NKK+2].
struct Staging {
    float *uk, *vk, *wk, *turb, *tdiss;
    size_t stride;   // floats between situations
};

// A launch that is set up while the launch before it on the stream runs (its kernel calls grid_wait first).
template <class... P, class... A>
void launch_after(void (*kernel)(P...), dim3 grid, dim3 block, cudaStream_t st, const A &...args) {
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at[0].val.programmaticStreamSerializationAllowed = 1;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = grid;
    cfg.blockDim = block;
    cfg.stream = st;
    cfg.attrs = at;
    cfg.numAttrs = 1;
    cudaLaunchKernelEx(&cfg, kernel, P(args)...);
}

// Buffers of the row-chain schedule (prog_chain.cu): column records of the units in flight, stamped
// words between claims, the pressure sweep's elimination table per i-direction.
struct ChainBufs {
    float2 *rec;                 // records [unit][col][pair][KMAX_LEVELS]; pressure: DIV/DTIME [unit][col][KS]
    unsigned long long *words;   // [situation][claim][column][values][KMAX_LEVELS]
    const float2 *ptab;          // [dir][col][KS] {T, P}
    const int *epoch;            // iterations run in this context, part of the word stamps
    int unit_lo, unit_n;         // situations (positions in the active list) of a launch
    int ctr_slot;                // task-counter slot of the launch
};

int gs_num_variants();
int gs_block_threads(bool il, int variant);
cudaError_t gs_prepare(bool il, int ks, int model);
cudaError_t gs_occupancy(bool il, int kind, int model, int simd, int ks, int variant, int *blocks_per_sm);
// one Gauss-Seidel phase (kind = PH_PRESSURE, PH_U, PH_V, PH_W or PH_TKE) of the loaded model
void launch_gs(int kind, const KArgs &a, const SweepGeom &g, int grid, cudaStream_t st);
// strip schedule of the slab family's model-1 sweeps (kind = PH_PRESSURE, PH_U, PH_V, PH_W): a
// block per strip of strip_rows(variant) sweep rows, hand-offs inside a strip in shared memory
int strip_num_variants();
int strip_rows(int variant);
int strip_block_threads(int variant);
cudaError_t strip_occupancy(int kind, int variant, int *blocks_per_sm);
void launch_strip(int kind, const KArgs &a, const SweepGeom &g, int variant, int grid, cudaStream_t st);
// pressure, velocity correction, averages and model-1 U in one launch on the strip schedule:
// claims (per situation) alternate pressure strips and U strips, 2*strips+1 of them
cudaError_t fused_strip_occupancy(int *blocks_per_sm);
int fused_strip_claims(const SweepGeom &gp);
void launch_fused_strip(const KArgs &a, const FusedGeom &fg, int grid, cudaStream_t st);
// pressure + velocity correction + averages + model-1 U in one wavefront launch (slab family)
cudaError_t fused_occupancy(int *blocks_per_sm);
void launch_fused_pvau(const KArgs &a, const FusedGeom &fg, int grid, cudaStream_t st);

// row-chain schedule of the slab family's sweeps: coefficient launch and chain launch of one
// phase (kind = PH_PRESSURE, PH_U, PH_V, PH_W, PH_TKE); bufs.unit_n situations at a time
size_t chain_record_bytes(int model);
size_t chain_unit_words(int nii, int njj);      // words of one unit
int chain_claims(int ni);                               // claims of a sweep of ni rows
cudaError_t chain_grid(int kind, const KArgs &a, long long claims, int *grid);
void launch_chain(int kind, const KArgs &a, const SweepGeom &g, const ChainBufs &bufs, int grid, cudaStream_t st);
// passes [first, first + passes) of the elimination table; changed[p] (zeroed) says whether pass p
// changed a value, and the table is complete when its last pass did not
void launch_pressure_tab(const KArgs &a, float2 *tab, int *changed, int first, int passes, cudaStream_t st);

void launch_bc(const KArgs &a, const BcLists &bc, cudaStream_t st);
void launch_velcorr(const KArgs &a, cudaStream_t st);
void launch_average(const KArgs &a, cudaStream_t st);
void launch_bookkeeping(const KArgs &a, cudaStream_t st);

// set-up and tear-down of a batch (PrognosticFlowfield.cs:295-329, 410-579); varw = per
// (situation, column) vertical-variance term of the TURB initialisation (model != 1), or null
void launch_setup(const KArgs &a, const Staging &sg, int model, const float *varw, const float *z0_init,
                  cudaStream_t st);
void launch_gather(const KArgs &a, const Staging &sg, int model, cudaStream_t st);
void launch_scatter(const KArgs &a, const Staging &sg, int model, cudaStream_t st);
// post-checks (PrognosticFlowfield.cs:1193-1243); counts[s*4 + 0..3] = UK, VK, WK, non-finite
void launch_postcheck(const KArgs &a, int *counts, cudaStream_t st);

// DiagnosticFlowfield.Calculate (DiagnosticFlowfield.cs:24-436) and the final vertical velocity of
// the columns outside the prognostic sub-domains (MicroscaleFlat.cs:389-462), on full-height
// fields: `a` describes them as a slab layout with KS = NKK+2 and a.dpm the diagnostic DPM.
cudaError_t diag_prepare(int ks);
cudaError_t diag_occupancy(int ks, int *blocks_per_sm);
void launch_diag_dtime(const KArgs &a, int kadvmax, float *dtime, cudaStream_t st);
void launch_diag_pressure(const KArgs &a, const SweepGeom &g, const DiagTabs &t, int grid, cudaStream_t st);
void launch_diag_velcorr(const KArgs &a, const DiagTabs &t, cudaStream_t st);
// the same sweeps on row chains (prog_chain_diag.cu): one iteration, pressure sweep and velocity
// correction, on DPM in planes; levels = levels per lane (diag_chain_levels, 0: too many for a warp)
struct DiagChainBufs {
    int levels, units, grid;         // units: situations whose DIV/DTIME is held at once
    float *div, *dpm;                // levels/2 planes [units or all situations][col][64]
    unsigned long long *words;       // zeroed before the first iteration
    const int *stamps;               // [iteration-1], distinct
};
int diag_chain_levels(int nkk);
size_t diag_chain_words(int nii, int njj, int levels);   // words of one situation
cudaError_t diag_chain_grid(int levels, int ni, int units, int *grid);
void launch_diag_chain(const KArgs &a, const SweepGeom &g, const DiagTabs &t, const DiagChainBufs &buf, cudaStream_t st);
void launch_diag_wfinal(const KArgs &a, const DiagTabs &t, cudaStream_t st);

}  // namespace gral
