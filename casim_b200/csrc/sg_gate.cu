// Surrogate-driven gating, two warps per site: n time steps of RyR gating with the held mouth
// values, the jSR ODE and the RyR currents (one warp), and of the cytosol pool ODE, which nothing
// in a window depends on (the other), without the RD step. The gating consumes the site's MRG32k3a
// stream in the reference's order (CaSim/DyadChannels.cpp:97-130: one draw per
// RyR test, one more per transition) with the warp-parallel scheme of the
// resident kernel: a ring of draws generated 16 per lane from jumped-ahead
// states, 32 RyRs resolved per ballot, one re-evaluation per transition. A step is a chain of
// dependent FP64 operations, so it is kept short: every lane carries the jSR in registers (no
// exchange through shared memory), the mouth values sit in shared memory. 2048 sites of 20 RyRs,
// 20 windows of 20 steps with start and readback (the network and the feature and mouth kernels in
// it took a third of the gain): 5.87 ms with the pools and the jSR on lane 0 and the mouths read
// from global memory, 2.80 ms so (3.00 with the pool's divisions done one by one).
#include "engine.h"
#include "pools.cuh"
#include "resident_kernel.cuh"

namespace {

using namespace cbres;

constexpr int SG_MAXCH = 256;  // RyRs per site this kernel serves (two draws each fit one refill)
constexpr int SG_WARPS = 4;    // sites per block

template <int NI>
struct sg_warp_smem {
    double ring[RING];
    double p[2][SG_MAXCH];  // transition probability per step of each RyR when closed / open
    double mo[NI][SG_MAXCH];  // held mouth concentrations
    int state[SG_MAXCH];
    cb_site_scalars q;
};

template <int NI>
__global__ void __launch_bounds__(64 * SG_WARPS) k_sg_warp(const __grid_constant__ cb_model m, int S, int NS, long long n,
                                                          const cb_site* __restrict__ sites, cb_site_scalars* __restrict__ sc,
                                                          int* __restrict__ ch_state, const double* __restrict__ mouth,
                                                          const double* __restrict__ spx0, const double* __restrict__ spc0,
                                                          const double* __restrict__ spx1, const double* __restrict__ spc1,
                                                          const unsigned long long* __restrict__ pow2) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    const int w = (threadIdx.x >> 5) % SG_WARPS, lane = threadIdx.x & 31;
    const bool pool = threadIdx.x >= 32 * SG_WARPS;  // the site's second warp
    const int s = blockIdx.x * SG_WARPS + w;
    const bool mine = s < S;
    sg_warp_smem<NI>& W = ((sg_warp_smem<NI>*)smem_raw)[w];
    const double dt = m.dt;
    cb_site st{};
    if (mine) {
        st = sites[s];
        if (!pool) {
            const unsigned int* src = (const unsigned int*)(sc + s);
            unsigned int* dst = (unsigned int*)&W.q;
            for (int k = lane; k < (int)(sizeof(cb_site_scalars) / 4); k += 32) dst[k] = src[k];
        }
    }
    __syncthreads();
    const int nch = st.n_ch;
    if (mine && pool) {
        if (lane == 0 && m.cyto_type == CB_CYTO_POOL)
            for (long long it = 0; it < n; ++it) cb_pool_step<NI>(m, W.q, dt);
    } else if (mine) {
        for (int c = lane; c < nch; c += 32) {
            const double* mo = mouth + (size_t)(st.ch_off + c) * NS;
            const double mg = m.mg_idx >= 0 ? mo[m.mg_idx] : 0.0;
            W.state[c] = ch_state[st.ch_off + c];
            W.p[0][c] = cb_rate(m, spx0, spc0, spx1, spc1, 0, mo[m.ca_idx], mg) * dt;
            W.p[1][c] = cb_rate(m, spx0, spc0, spx1, spc1, 1, mo[m.ca_idx], mg) * dt;
#pragma unroll
            for (int j = 0; j < NI; ++j) W.mo[j][c] = mo[j];
        }
        cbrng::State gl;
        for (int i = 0; i < 6; ++i) gl.s[i] = W.q.rng[i];
        rng_jump(pow2, gl, 2ULL * LANE_DRAWS * lane);  // lane l: draw l*LANE_DRAWS of the first refill
        // jSR pool (CaSim/SRPool.cpp:55-89), the same on every lane
        double jsr[NI], jnew[NI], I[NI], nsr[NI], tot[NI];
#pragma unroll
        for (int j = 0; j < NI; ++j) {
            jsr[j] = W.q.jsr[j];
            jnew[j] = W.q.jsr_new[j];
            I[j] = W.q.IjSR[j];
            nsr[j] = W.q.nsr[j];
            tot[j] = W.q.total[j];
        }
        double release = W.q.release;
        __syncwarp();
        long long D = 0, we = 0;
        for (long long it = 0; it < n; ++it) {
            if (!m.jsr_const) {
                const double db = cb_jsr_dt_beta<NI>(m, jsr, dt);
#pragma unroll
                for (int j = 0; j < NI; ++j) {
                    jnew[j] = jsr[j] + db * (m.inv_tau[j] * (nsr[j] - jsr[j]) - I[j] * m.inv_V_jsr);
                    if (j == m.ca_idx) release += I[j] * dt;
                }
            }
            if (we - D < 2LL * nch) {  // ring refill: at least two draws per RyR available
                const long long base = we + (long long)lane * LANE_DRAWS;
                for (int i = 0; i < LANE_DRAWS; ++i) W.ring[(base + i) & (RING - 1)] = u01d_fast(gl);
                jump_row(pow2, gl, JUMP_ROW);
                we += WINDOW;
            }
            __syncwarp();
#pragma unroll
            for (int j = 0; j < NI; ++j) tot[j] = 0;
            for (int b0 = 0; b0 < nch; b0 += 32) {
                const int c = b0 + lane;
                const int cnt = min(32, nch - b0);
                const bool act = lane < cnt;
                int stt = act ? W.state[c] : 0;
                const double p = act ? W.p[stt][c] : 0.0;
                int start = 0;
                while (start < cnt) {
                    const bool rem = act && lane >= start;
                    const double u = rem ? W.ring[(D + (lane - start)) & (RING - 1)] : 2.0;
                    const unsigned int t = __ballot_sync(0xffffffffu, rem && (u < p));
                    if (t == 0u) {
                        D += cnt - start;
                        break;
                    }
                    const int f = __ffs(t) - 1;
                    if (lane == f) W.state[c] = stt = 1 - stt;
                    D += (f - start) + 2;
                    start = f + 1;
                }
                // RyR currents from the held mouth values
                if (act)
#pragma unroll
                    for (int j = 0; j < NI; ++j) tot[j] += stt * (m.g[j] * (jnew[j] - W.mo[j][c]));
            }
#pragma unroll
            for (int o = 16; o > 0; o >>= 1)
#pragma unroll
                for (int j = 0; j < NI; ++j) tot[j] += __shfl_xor_sync(0xffffffffu, tot[j], o);
            if (!m.jsr_const)
#pragma unroll
                for (int j = 0; j < NI; ++j) {
                    I[j] = tot[j] * m.V_elem;
                    nsr[j] = m.nsr[j];
                    jsr[j] = jnew[j];
                }
        }
        if (lane == 0) {
            cbrng::State gd;  // stream state at the next unconsumed draw
            for (int i = 0; i < 6; ++i) gd.s[i] = W.q.rng[i];
            rng_jump(pow2, gd, 2ULL * (unsigned long long)D);
            for (int i = 0; i < 6; ++i) W.q.rng[i] = gd.s[i];
            W.q.draws += (unsigned long long)D;
#pragma unroll
            for (int j = 0; j < NI; ++j) {
                W.q.jsr[j] = jsr[j];
                W.q.jsr_new[j] = jnew[j];
                W.q.IjSR[j] = I[j];
                W.q.nsr[j] = nsr[j];
                W.q.total[j] = tot[j];
            }
            W.q.release = release;
        }
    }
    __syncthreads();
    if (mine && !pool) {
        const unsigned int* src = (const unsigned int*)&W.q;
        unsigned int* dst = (unsigned int*)(sc + s);
        for (int k = lane; k < (int)(sizeof(cb_site_scalars) / 4); k += 32) dst[k] = src[k];
        for (int c = lane; c < nch; c += 32) ch_state[st.ch_off + c] = W.state[c];
    }
}

template <int NI>
cudaError_t launch(cb_dev& d, long long n, cudaStream_t st, bool capturing) {
    const size_t smem = sizeof(sg_warp_smem<NI>) * SG_WARPS;
    if (!capturing) {  // set before any capture (the first call runs eagerly)
        const cudaError_t e = cudaFuncSetAttribute(k_sg_warp<NI>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
        if (e != cudaSuccess) return e;
    }
    k_sg_warp<NI><<<(d.S + SG_WARPS - 1) / SG_WARPS, 64 * SG_WARPS, smem, st>>>(d.m, d.S, d.NS, n, d.sites, d.sc, d.ch_state, d.mouth, d.spx[0],
                                                                               d.spc[0], d.spx[1], d.spc[1], d.rs_pow2);
    return cudaGetLastError();
}

}  // namespace

// the warp-per-site kernel when every site has at most SG_MAXCH RyRs
cudaError_t cb_sg_steps_warp(cb_dev& d, long long n, cudaStream_t st, bool* used) {
    *used = false;
    if (d.max_ch > SG_MAXCH) return cudaSuccess;
    cudaError_t e = cb_ensure_pow2(d);
    if (e != cudaSuccess) return e;
    cudaStreamCaptureStatus cap = cudaStreamCaptureStatusNone;
    if ((e = cudaStreamIsCapturing(st, &cap)) != cudaSuccess) return e;
    const bool capturing = cap != cudaStreamCaptureStatusNone;
    switch (d.m.n_ions) {
    case 1: e = launch<1>(d, n, st, capturing); break;
    case 2: e = launch<2>(d, n, st, capturing); break;
    case 3: e = launch<3>(d, n, st, capturing); break;
    default: e = launch<4>(d, n, st, capturing); break;
    }
    *used = true;
    return e;
}
