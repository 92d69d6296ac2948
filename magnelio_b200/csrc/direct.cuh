// Arguments and launchers of the direct stencil kernels (stencil.cu): 16 bytes
// of cells or one cell per thread, any number of field sets.
#pragma once
#include "fitb_common.cuh"

namespace fitb {

// One-edge lumped ports that may step inside the E kernel.
constexpr int kDirectLumped = 16;
// The CPML faces of one axis: [0] the layers 0 .. n[0] - 1, [1] the layers
// lo1 .. lo1 + n[1] - 1 (lo1 = INT_MAX: none).  Entry of cell (i, j, k):
// s0 i + s1 j + k with the layer in place of the axis coordinate.  psi, air:
// the first of the side's (E or H) two auxiliaries, the second `slab` entries
// further on, a field set's `set` entries apart; air null without PEC masks.
struct AxisSlabs {
    int lo1;
    int n[2], s0[2], s1[2];
    unsigned slab[2];
    size_t set[2];
    const void* psi[2];
    void* psi_out[2];
    const void* bcc[2];
    const unsigned char* air[2];
};
// Division by a fixed n (direct_div).
struct DirectDiv {
    unsigned m;
    int s;
};
// What the direct kernels take beside StencilArgs: the launcher fills the
// division and the slab bounds, the caller the planes per thread (0: one), the
// one-edge lumped ports that step inside the E kernel (their cell and
// component; `ports` the device table in the same order) and the step counter
// the H kernel advances (null: not advanced there).
struct DirectArgs {
    int np;
    // vectors of a row: n_low in the near z slab, n_mid clear of both, n_edge
    // = all but the n_mid; a plane's first mid_threads threads take the clear ones
    int n_low, n_mid, n_edge;
    unsigned mid_threads;
    DirectDiv mid_div, edge_div;
    AxisSlabs ax[2][3];  // E side, H side
    int ping_pong;       // the new fields and psi go to the *_next buffers
    int slab_bits;       // E with the slab step's roundings
    int n_lumped;
    int4 lumped[kDirectLumped];
    const LumpedDev* ports;
    PortsArgs pa;
    long long* advance;
};
// which: 0 = E update, 1 = H update
template <typename T>
void launch_direct_half(const StencilArgs<T>& a, const DirectArgs& d, int which, cudaStream_t s);
// Planes per thread and grid (x, y, z) of those launches for np (0: their own).
template <typename T>
void direct_shape(const StencilArgs<T>& a, int np, int* out);
// flags[side] (zeroed by the caller): bit 0 set when alpha is not (beta != 0),
// bit 1 when it is not 1 everywhere.
template <typename T>
void launch_unit_alpha(const StencilArgs<T>& a, int* flags, cudaStream_t s);

}  // namespace fitb
