// Programmatic dependent launch: kernels of one stream launched with the
// programmatic-stream-serialization attribute may be scheduled while the
// kernel before them drains.  Every block of such a kernel passes FB_GRID_WAIT,
// which returns once the preceding grid has completed and its writes are
// visible.
#pragma once

#include <cuda_runtime.h>

#include <cstdlib>
#include <cstring>
#include <utility>

// After its wait, every block lets the next kernel of the stream launch: that
// kernel's blocks take free SM slots while this grid's last blocks run and
// wait in their own FB_GRID_WAIT, so the launch latency is hidden.  Since a
// block triggers only once it is running, the next grid launches after all of
// this grid's blocks have started: a waiting grid never holds slots that this
// one still needs.
//
// What a kernel may do before its wait: the kernel before it has triggered,
// that is, every block of it has passed its own wait, so everything earlier is
// complete and visible; only what the kernel directly before it writes is not.
// So a kernel may load what that one does not write, and work on it, ahead of
// its wait; it stores nothing and raises no status there.  These load early, each
// marked with what the kernel before it writes, and may follow directly only
// kernels that leave the rest alone:
//   k_nl_rhs_tma        ru2, ru3: not behind nl_rhs itself
//   k_mls_interp        q2, q3, markers, MLS weights: not behind updvp, helsolve,
//                       the marker set-up, or a launch that moves the markers
//   k_mls_spread        rhs2, rhs3 and the chains: not behind nl_rhs or the chains
//   k_helsolve_win      q2, q3 and its coefficients: not behind updvp or itself
//   k_updvp_prcalc_tma  q2, q3, pr: not behind helsolve or itself
//   k_loads_probe       markers: not behind a launch that moves them
//   k_step_close        markers, body state, scalars: behind the probes only
//   k_ymodes, k_i8x8_gemm, the 3xTF32 products: constants and the base operand
// Kernels that find their case in device memory (grouped launches) wait first.
// A caller that cannot promise the order makes the next launch an ordinary one
// (pdl_full_next): it then starts behind the complete kernel before it.
#define FB_GRID_WAIT() asm volatile("griddepcontrol.wait;\n\tgriddepcontrol.launch_dependents;" ::: "memory")

namespace fb {

inline bool pdl_enabled() {
    static const bool on = [] {
        const char *v = std::getenv("FRIBOIS2D_PDL");
        return !(v && std::strcmp(v, "0") == 0);
    }();
    return on;
}

// set by this thread for its next launch, which clears it
inline thread_local bool pdl_full_next = false;

template <typename... KArgs, typename... Args>
inline void pdl(void (*kern)(KArgs...), dim3 grid, dim3 block, size_t smem, cudaStream_t st, Args &&...args) {
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = grid;
    cfg.blockDim = block;
    cfg.dynamicSmemBytes = smem;
    cfg.stream = st;
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = at;
    cfg.numAttrs = (pdl_enabled() && !std::exchange(pdl_full_next, false)) ? 1 : 0;
    cudaLaunchKernelEx(&cfg, kern, std::forward<Args>(args)...);
}

}  // namespace fb
