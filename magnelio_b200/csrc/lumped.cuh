// One step of a lumped element (Thevenin source with a series R-L-C
// companion; reference: src/magnelio/ports/_lumped/operator.py:134-166,
// src/magnelio/circuit/companion.py:45-112), shared by the port kernel and by
// the E update that steps one-edge ports itself.
#pragma once
#include "fitb_common.cuh"

namespace fitb {

// The port current of step n from the element voltage v_total; advances the
// companion state of field set b.
__device__ __forceinline__ double lumped_current(const LumpedDev& d, const PortsArgs& pa, int b, long long n,
                                                 double v_total) {
    const double v_src = (n < d.n_src) ? d.src[(long long)b * d.n_src + n] : 0.0;
    double* st = d.st + 4 * b;
    const double dt = pa.dt_lumped;
    const double i_prev = st[0];
    double r_eq = (d.R >= 0.0) ? d.R : 0.0;
    if (d.L >= 0.0) r_eq += 2.0 * d.L / dt;
    if (d.C >= 0.0) r_eq += dt / (2.0 * d.C);
    double v_hist = 0.0;
    if (d.L >= 0.0) v_hist += -(2.0 * d.L / dt) * i_prev - st[1];
    if (d.C >= 0.0) v_hist += st[2] + (dt / (2.0 * d.C)) * i_prev;
    const double z_eff = r_eq + d.beta_sum;
    const double i_port = (v_src - v_hist - v_total) / z_eff;
    if (d.L >= 0.0) st[1] = (2.0 * d.L / dt) * (i_port - i_prev) - st[1];
    if (d.C >= 0.0) st[2] = st[2] + (dt / (2.0 * d.C)) * (i_port + i_prev);
    st[0] = i_port;
    st[3] = i_port;
    return i_port;
}

// Recorder: V re-projected from the corrected field, I = the port current.
__device__ __forceinline__ void lumped_record(const LumpedDev& d, const PortsArgs& pa, int b, long long n, double v,
                                              double i_port) {
    const long long r = ((long long)b * pa.rec.cap + n) * pa.rec.nch + d.channel;
    pa.rec.V[r] = v * d.rec_scale;
    pa.rec.I[r] = i_port * d.rec_scale;
}

// A port of one edge whose updated field value is `e`: the value to store.
template <typename T>
__device__ __forceinline__ T lumped_edge_step(const LumpedDev& d, const PortsArgs& pa, int b, T e) {
    const long long n = *pa.step;
    const double sign = d.sign[0];
    const double i_port = lumped_current(d, pa, b, n, sign * (double)e);
    const T out = (T)((double)e + sign * d.beta[0] * i_port);
    lumped_record(d, pa, b, n, sign * (double)out, i_port);
    return out;
}

}  // namespace fitb
