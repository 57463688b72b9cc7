// Kernel launchers of the fluid time step (definitions in kernels.cu).
#pragma once

#include <cuda.h>
#include <cuda_runtime.h>

#include "device.cuh"

namespace fb {

constexpr int kRedSlot = 65536;  // block partials per reduction slot

cudaError_t kernels_configure();   // shared-memory limits (once per device)
void launch_cfl(const Dev &d, cudaStream_t s);
// keep the scalars and the status word beside them (scal + kScalNoted)
void launch_note(const Dev &d, cudaStream_t s);
void launch_boucdq(const Dev &d, double ga, double ro, cudaStream_t s);
// TMA descriptors of the fields that the stencil tiles stage (q2, q3, pr for
// k_nl_rhs_tma, dph for k_updvp_prcalc_tma): 2-D arrays (j - 1 fastest, row k,
// k = 0 .. n3), one box per tile and field
struct alignas(64) NlMaps {
    CUtensorMap q2, q3, pr, dph;
};
int encode_nl_maps(NlMaps *m, const Dev &d);   // FB_OK, or an error (no maps)
// pend / deferred: the fused step's deferred pr_submean of RK3 substeps 1 and 2.
// extra: the fused step's work on the same launch (kNlBoucdq: boucdq of this
// substep in a block of its own; kNlCfl: the CFL number and the mean w of the
// field the tiles hold; kNlMeans: the step before left all its pressure means to
// be subtracted, and a block of its own brings the entries of pr that updvp does
// not rewrite up to date)
constexpr int kNlBoucdq = 1, kNlCfl = 2, kNlMeans = 4;
void launch_nl_rhs(const Dev &d, double al, double ga, double ro, cudaStream_t s, bool pend,
                   const NlMaps &maps, int extra = 0);
void launch_lgrdist(const Dev &d, cudaStream_t s);
// find: the nearest nodes (lgrdistribution) in the same launch
void launch_mls_setup(const Dev &d, cudaStream_t s, bool find = false);
// clear: empty the spreading table behind k_spread_chains (substep 1); cfl: check
// the CFL number of nl_rhs (kNlCfl) ahead of the forcing
void launch_mls_interp(const Dev &d, cudaStream_t s, bool clear, bool cfl);
// empty the spreading table behind a set-up that no interpolation follows
void launch_table_clear(const Dev &d, cudaStream_t s);
void launch_mls_spread(const Dev &d, cudaStream_t s);
void launch_spread_chains(const Dev &d, cudaStream_t s);
void launch_helsolve(const Dev &d, const SubDev &sd, cudaStream_t s);
// rmax (may be null): n2m row maxima of |dph| accumulated for the INT8 digit cut
// extra: the fused step's work on the same launch (kDivBoucqt: boucqt;
// kDivCfl: the CFL number of nl_rhs made the step's, and its check, which the
// forcing has made before where there are markers)
constexpr int kDivBoucqt = 1, kDivCfl = 2;
void launch_divg(const Dev &d, double usdtal, cudaStream_t s, double *rmax = nullptr, int extra = 0);
// slot: a scalar slot that keeps the pressure mean beside S_PRAVG (-1: none)
void launch_updvp_prcalc(const Dev &d, double al, double be, cudaStream_t s, bool pend, const NlMaps &maps,
                         int slot = -1);
// mbox[0] = *d.status, mbox[1..8] = d.forces[0..7] (when forces); mbox in
// mapped host memory
void launch_publish(const Dev &d, bool forces, double *mbox, cudaStream_t s);
// deferred: the end of the fused step (boucqt has run with divg)
void launch_submean_boucqt(const Dev &d, cudaStream_t s, bool deferred = false);
// the probes alone; finish: with press and tau of every marker that has a
// tangent of its own, for launch_step_close
void launch_loads_probe(const Dev &d, cudaStream_t s, bool pend, bool finish);
// the rest of the loads and the rigid update of a loosely coupled step in one
// launch, for the marker counts that step_closes
bool step_closes(int nlm);
void launch_step_close(const Dev &d, int hist_rows, cudaStream_t s);
// pend: pr still lacks the subtraction of its mean (S_PRAVG)
void launch_loads(const Dev &d, cudaStream_t s, bool pend = false);
void launch_diag(const Dev &d, int hist_rows, cudaStream_t s);
enum RigidMode { RIGID_STEP = 0, RIGID_PLACE = 1, RIGID_FORCES = 2, RIGID_COMMIT = 3 };
// mbox (mapped host memory, may be null; RIGID_STEP and RIGID_COMMIT): the status
// word and the forcecomp row, written at the end as k_publish does
void launch_rigid(const Dev &d, int hist_rows, cudaStream_t s, int mode = RIGID_STEP, const double *fin = nullptr,
                  double *mbox = nullptr);

// grouped forms (one launch over a group of cases; substep n 0-based)
void glaunch_nl_rhs(const Group &g, int n, cudaStream_t s, bool pend, int extra);
void glaunch_marker_setup(const Group &g, cudaStream_t s);   // nearest nodes and MLS weights, spreading chains
void glaunch_forcing(const Group &g, int n, cudaStream_t s); // interpolation and spreading
void glaunch_divg(const Group &g, int n, cudaStream_t s, int extra);
void glaunch_updvp_prcalc(const Group &g, int n, cudaStream_t s, bool pend, int slot);
void glaunch_submean_boucqt(const Group &g, cudaStream_t s, bool deferred = false);
void glaunch_loads(const Group &g, cudaStream_t s);
void glaunch_rigid(const Group &g, cudaStream_t s, int mode = RIGID_STEP);
void glaunch_diag(const Group &g, cudaStream_t s);

}  // namespace fb
