// Pool ODEs of one site: the resident kernel, the Update of the streaming path, the generic kernels
// and the surrogate-driven gating step them here.
#pragma once
#include "model.h"

// Cytosol pool ODE of one site (CaSim/CytosolPool.cpp:217-288). NI > 0 fixes the ion count at
// compile time here and below: the loops unroll and the site's values stay in registers.
template <int NI = 0>
__device__ __forceinline__ void cb_pool_step(const cb_model& m, cb_site_scalars& q, double dt) {
    const int ni = NI > 0 ? NI : m.n_ions;
    double evo_i[CB_MAX_IONS], evo_p[CB_MAX_CPAIRS];
    int ipd = 0, is = 0;
#pragma unroll
    for (int j = 0; j < ni; ++j) {
        double react = 0;
        for (int p = 0; p < m.c_n_pairs; ++p) {
            if (m.c_pair_ion[p] != j) continue;
            double R1 = m.c_koff[p] * q.c_pairs[p] - m.c_kon[p] * q.c_ions[j] * q.c_free[m.c_pair_buf[p]];
            evo_p[p] = -R1;
            react += R1;
            if (m.c_in_dyad[p]) {
                evo_p[p] += q.efflux[ni + ipd];
                ++ipd;
            }
        }
        evo_i[j] = react + q.efflux[j];
        if (m.c_serca[j]) {
            const double i2 = q.c_ions[j] * q.c_ions[j];
            evo_i[j] -= m.c_Jmax[is] * (i2 / (i2 + m.c_Kup[is] * m.c_Kup[is]) - m.c_rest[is]);
            ++is;
        }
    }
#pragma unroll
    for (int j = 0; j < ni; ++j) {
        evo_i[j] -= m.c_onetau_ion[j] * (q.c_ions[j] - m.c_bg[j]);
        q.c_ions[j] += evo_i[j] * dt;
    }
    ipd = 0;
    for (int p = 0; p < m.c_n_pairs; ++p) {
        evo_p[p] -= m.c_onetau_pair[p] * (q.c_pairs[p] - m.c_init[p]);
        q.c_pairs[p] += evo_p[p] * dt;
        if (m.c_in_dyad[p]) q.c_bnd[ipd++] = q.c_pairs[p];
    }
    for (int b = 0; b < m.c_n_buf; ++b) q.c_free[b] = m.c_Ctot[b];
    for (int p = 0; p < m.c_n_pairs; ++p) q.c_free[m.c_pair_buf[p]] -= q.c_pairs[p];
}

// dt / beta of the jSR (CaSim/SRPool.cpp:70-80), beta = 1 + sum_j a_j / s_j^2 with a_j = n_j K_j CQ
// and s_j = K_j + jSR_j: over the common denominator, so that the one warp that steps a site's
// pools waits for one FP64 division instead of a chain of two or more.
template <int NI = 0>
__device__ __forceinline__ double cb_jsr_dt_beta(const cb_model& m, const double* jsr, double dt) {
    double num = 1, den = 1;  // beta = den / num
#pragma unroll
    for (int j = 0; j < (NI > 0 ? NI : m.n_ions); ++j) {
        const double s = m.K_CQ[j] + jsr[j], s2 = s * s;
        den = den * s2 + num * (m.nCQ[j] * m.K_CQ[j] * m.CQ);
        num *= s2;
    }
    return dt * num / den;
}

// jSR pool ODE of one site (CaSim/SRPool.cpp:70-89) with the site's own beta.
template <int NI = 0>
__device__ __forceinline__ void cb_jsr_step(const cb_model& m, cb_site_scalars& q, double dt) {
    if (m.jsr_const) return;
    const double db = cb_jsr_dt_beta<NI>(m, q.jsr, dt);
#pragma unroll
    for (int i = 0; i < (NI > 0 ? NI : m.n_ions); ++i)
        q.jsr_new[i] = q.jsr[i] + db * (m.inv_tau[i] * (q.nsr[i] - q.jsr[i]) - q.IjSR[i] * m.inv_V_jsr);
    if (m.ca_idx >= 0) q.release += q.IjSR[m.ca_idx] * dt;
}

