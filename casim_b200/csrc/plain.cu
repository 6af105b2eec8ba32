// Plain path: one time step = one launch sequence over HBM-resident fields. Layouts of 1-2 ions, up to
// 4 pairs and 1 or 3 cleft layers run the specialised kernels of stream_kernels.cuh (cytosol, cleft,
// gating with pools and Update: two or three launches per step), others the generic ones here:
//
//   k_pre     one thread per site: cytosol pool ODE (CaSim/CytosolPool.cpp:217-268),
//             jSR pool ODE (CaSim/SRPool.cpp:70-89), two-state gating
//             (CaSim/DyadChannels.cpp:97-130) with the site's MRG32k3a stream
//   k_cyto    RD3D cytosol stencil (this project's 3D cytosol; no reference analog)
//   k_rd      cleft RD step of every interior node (CaSim/DyadRD2DCPU.cpp:394-490,
//             CaSim/DyadRDCPU.cpp:404-506), ping-pong buffers
//   k_update  one block per site: mouth gather, Dirichlet edges, efflux,
//             RyR currents, jSR coupling (CaSim/ParallelHybridSolver.cpp:159-175)
//
// The generic kernels are the straightforward GPU formulation of the reference step; they
// handle any site size and layout.
#include <algorithm>
#include <climits>
#include <cstring>
#include <vector>

#include "engine.h"
#include "mrg32k3a.cuh"
#include "mwc.h"
#include "physics.cuh"
#include "pools.cuh"
#include "stream_kernels.cuh"

namespace {

template <typename R>
__global__ void k_reset(cb_model m, const cb_site* __restrict__ sites, R* __restrict__ A, R* __restrict__ B,
                        R* __restrict__ cur, cb_site_scalars* __restrict__ sc, int* __restrict__ ch_state, int* __restrict__ err) {
    const int s = blockIdx.y;
    if (s == 0 && blockIdx.x == 0 && threadIdx.x == 0) *err = 0;  // the state is valid again
    const cb_site st = sites[s];
    const int F = m.F;
    R* a = A + st.node_base * F;
    R* b = B + st.node_base * F;
    R* c = cur + st.node_base * m.n_ions;
    for (int n = blockIdx.x * blockDim.x + threadIdx.x; n < st.npad; n += gridDim.x * blockDim.x) {
        for (int f = 0; f < F; ++f) {
            R v = (R)(f < m.n_ions ? m.Cb[f] : m.pair_init[f - m.n_ions]);
            a[(long long)f * st.npad + n] = v;
            b[(long long)f * st.npad + n] = v;
        }
        for (int j = 0; j < m.n_ions; ++j) c[(long long)j * st.npad + n] = (R)0;
    }
    if (blockIdx.x == 0) {
        for (int k = threadIdx.x; k < st.n_ch; k += blockDim.x) ch_state[st.ch_off + k] = 0;
        if (threadIdx.x == 0) {
            cb_site_scalars& q = sc[s];
            for (int i = 0; i < CB_MAX_IONS; ++i) {
                q.jsr[i] = q.jsr_new[i] = q.jsr0[i];
                q.IjSR[i] = 0;
                q.nsr[i] = q.jsr0[i];
                q.total[i] = 0;
                q.c_ions[i] = i < m.n_ions ? m.c_bg[i] : 0.0;
            }
            for (int k = 0; k < CB_MAX_SPECIES; ++k) q.efflux[k] = 0;
            for (int b2 = 0; b2 < m.c_n_buf; ++b2) q.c_free[b2] = m.c_Ctot[b2];
            for (int p = 0; p < m.c_n_pairs; ++p) {
                q.c_pairs[p] = m.c_init[p];
                q.c_free[m.c_pair_buf[p]] -= m.c_init[p];
            }
            for (int p = 0; p < m.n_pairs; ++p)
                q.c_bnd[p] = m.dyad_c_pair[p] >= 0 ? m.c_init[m.dyad_c_pair[p]] : m.pair_init[p];
            q.release = 0;
        }
    }
}

template <typename R>
__global__ void k_cyto_reset(cb_model m, int nc, R* __restrict__ A, R* __restrict__ B, double* __restrict__ cin) {
    const int s = blockIdx.y;
    const int CS = m.n_ions + m.c_n_pairs;
    const int mc2 = m.mc * m.mc;
    for (int n = blockIdx.x * blockDim.x + threadIdx.x; n < nc; n += gridDim.x * blockDim.x)
        for (int k = 0; k < CS; ++k) {
            R v = (R)(k < m.n_ions ? m.c_bg[k] : m.c_init[k - m.n_ions]);
            long long o = ((long long)s * CS + k) * nc + n;
            A[o] = v;
            B[o] = v;
            if (n < mc2) cin[((long long)s * CS + k) * mc2 + n] = 0.0;
        }
}

__global__ void k_init_open(const cb_site* __restrict__ sites, const int* __restrict__ first, int lo, int hi,
                            cb_site_scalars* __restrict__ sc, int* __restrict__ ch_state, int* __restrict__ ch_micro,
                            const cb_mwc_tab* __restrict__ mwc) {
    int s = lo + blockIdx.x * blockDim.x + threadIdx.x;
    if (s >= hi) return;
    const cb_site st = sites[s];
    cb_site_scalars& q = sc[s];
    cbrng::State g;
    for (int i = 0; i < 6; ++i) g.s[i] = q.rng[i];
    // CaSim/DyadChannels.cpp:83-95: one draw per channel (SetMacroState(0, .)),
    // then one more for the channel that is opened
    // (SingleSiteMWC: each draw picks the micro-state of the macro state from the
    // stationary distribution, CaSim/QMatrixModel.cpp:38-58)
    for (int c = 0; c < st.n_ch; ++c) {
        const double u = cbrng::u01d_fold(g);
        ch_state[st.ch_off + c] = 0;
        if (mwc) ch_micro[st.ch_off + c] = cb_mwc_pick(*mwc, 0, u, ch_micro[st.ch_off + c]);
    }
    const double u = cbrng::u01d_fold(g);
    int f = first[s - lo];
    if (f >= 0 && f < st.n_ch) {
        ch_state[st.ch_off + f] = 1;
        if (mwc) {
            const int mi = cb_mwc_pick(*mwc, 1, u, ch_micro[st.ch_off + f]);
            ch_micro[st.ch_off + f] = mi;
            ch_state[st.ch_off + f] = mi >= CB_MWC_OPEN;
        }
    }
    q.draws += (unsigned long long)st.n_ch + 1;
    for (int i = 0; i < 6; ++i) q.rng[i] = g.s[i];
}

__global__ void k_pre(cb_model m, int S, int NS, const cb_site* __restrict__ sites, cb_site_scalars* __restrict__ sc,
                      int* __restrict__ ch_state, const double* __restrict__ mouth, const double* __restrict__ spx0,
                      const double* __restrict__ spc0, const double* __restrict__ spx1, const double* __restrict__ spc1,
                      int* __restrict__ ch_micro, const cb_mwc_tab* __restrict__ mwc) {
    int s = blockIdx.x * blockDim.x + threadIdx.x;
    if (s >= S) return;
    const cb_site st = sites[s];
    cb_site_scalars& q = sc[s];
    const double dt = m.dt;
    if (m.cyto_type == CB_CYTO_POOL) cb_pool_step(m, q, dt);
    cb_jsr_step(m, q, dt);
    cbrng::State g;
    for (int i = 0; i < 6; ++i) g.s[i] = q.rng[i];
    unsigned long long draws = 0;
    for (int c = 0; c < st.n_ch; ++c) {
        const double* mo = mouth + (long long)(st.ch_off + c) * NS;
        double ca = mo[m.ca_idx];
        double mg = m.mg_idx >= 0 ? mo[m.mg_idx] : 0.0;
        if (mwc) {
            // SingleSiteMWC: escape rate of the micro-state, the second draw picks where to
            const int mi = ch_micro[st.ch_off + c];
            const double r = cb_mwc_exit(*mwc, mi, ca, mg);
            ++draws;
            if (cbrng::u01d_fold(g) < r * dt) {
                const double u2 = cbrng::u01d_fold(g);
                ++draws;
                const int nx = cb_mwc_next(*mwc, mi, ca, mg, r, u2);
                ch_micro[st.ch_off + c] = nx;
                ch_state[st.ch_off + c] = nx >= CB_MWC_OPEN;
            }
            continue;
        }
        int state = ch_state[st.ch_off + c];
        double r = cb_rate(m, spx0, spc0, spx1, spc1, state, ca, mg);
        ++draws;
        if (cbrng::u01d_fold(g) < r * dt) {
            (void)cbrng::u01d_fold(g);
            ++draws;
            ch_state[st.ch_off + c] = 1 - state;
        }
    }
    q.draws += draws;
    for (int i = 0; i < 6; ++i) q.rng[i] = g.s[i];
}

template <typename R>
__global__ void __launch_bounds__(256) k_cyto(cb_model m, int nc, const R* __restrict__ in, R* __restrict__ out,
                                              const double* __restrict__ cin) {
    const int s = blockIdx.y;
    const int n = blockIdx.x * blockDim.x + threadIdx.x;
    if (n >= nc) return;
    const int mc = m.mc, px = m.cpx, mc2 = mc * px;  // mc2: a stored plane
    const int i = n % px, j = (n / px) % mc, k = n / mc2;
    if (i == 0 || i >= mc - 1 || j == 0 || j == mc - 1 || k == mc - 1) return;
    const int CS = m.n_ions + m.c_n_pairs;
    const R* u = in + (long long)s * CS * nc;
    R* o = out + (long long)s * CS * nc;
    const int zl = k == 0 ? n + mc2 : n - mc2, zr = n + mc2;
    const R ih2 = (R)m.inv_hc2;
    R evo[CB_MAX_CSPECIES];
    for (int c = 0; c < CS; ++c) {
        const R* v = u + (long long)c * nc;
        R D = (R)(c < m.n_ions ? m.D_ion[c] : m.c_D_pair[c - m.n_ions]);
        R cc = v[n];
        evo[c] = D * ((v[n + 1] - 2 * cc + v[n - 1]) * ih2 + (v[n + px] - 2 * cc + v[n - px]) * ih2 + (v[zr] - 2 * cc + v[zl]) * ih2);
    }
    R fr[CB_MAX_CBUF];
    for (int b = 0; b < m.c_n_buf; ++b) fr[b] = (R)m.c_Ctot[b];
    for (int p = 0; p < m.c_n_pairs; ++p) fr[m.c_pair_buf[p]] -= u[(long long)(m.n_ions + p) * nc + n];
    int is = 0;
    for (int j2 = 0; j2 < m.n_ions; ++j2) {
        R ion = u[(long long)j2 * nc + n];
        R react = 0;
        for (int p = 0; p < m.c_n_pairs; ++p) {
            if (m.c_pair_ion[p] != j2) continue;
            R B = u[(long long)(m.n_ions + p) * nc + n];
            R R1 = (R)m.c_koff[p] * B - (R)m.c_kon[p] * ion * fr[m.c_pair_buf[p]];
            evo[m.n_ions + p] += -R1;
            react += R1;
        }
        evo[j2] += react;
        if (m.c_serca[j2]) {
            R i2 = ion * ion;
            R K2 = (R)(m.c_Kup[is] * m.c_Kup[is]);
            R b2 = (R)(m.c_bg[is] * m.c_bg[is]);
            evo[j2] -= (R)m.c_Jmax[is] * (i2 / (i2 + K2) - b2 / (b2 + K2));
            ++is;
        }
    }
    const R dt = (R)m.dt;
    for (int c = 0; c < CS; ++c) {
        R e = evo[c];
        if (k == 0) e += (R)cin[((long long)s * CS + c) * mc * mc + i + mc * j];
        o[(long long)c * nc + n] = u[(long long)c * nc + n] + e * dt;
    }
}

template <typename R>
__global__ void __launch_bounds__(256) k_rd(cb_model m, const cb_site* __restrict__ sites, const R* __restrict__ in,
                                            R* __restrict__ out, const R* __restrict__ curg) {
    const int s = blockIdx.y;
    const cb_site st = sites[s];
    const int n = blockIdx.x * blockDim.x + threadIdx.x;
    const int nxy = st.px * st.ny;
    if (n >= nxy * st.nz) return;
    const int F = m.F;
    const R* u = in + st.node_base * F;
    R* o = out + st.node_base * F;
    const int x = n % st.px, y = (n / st.px) % st.ny, z = n / nxy;
    if (x == 0 || x >= st.nx - 1 || y == 0 || y == st.ny - 1) {
        for (int f = 0; f < F; ++f) o[(long long)f * st.npad + n] = u[(long long)f * st.npad + n];
        return;
    }
    const R idx2 = (R)m.inv_dx2, idy2 = (R)m.inv_dy2, idz2 = (R)m.inv_dz2;
    int zl = n, zr = n;
    if (m.dim == 3) {
        zl = z == 0 ? n + nxy : n - nxy;
        zr = z == st.nz - 1 ? n - nxy : n + nxy;
    }
    R val[CB_MAX_SPECIES], evo[CB_MAX_SPECIES];
    for (int f = 0; f < F; ++f) {
        const R* v = u + (long long)f * st.npad;
        R c = v[n];
        val[f] = c;
        R D = (R)(f < m.n_ions ? m.D_ion[f] : m.D_pair[f - m.n_ions]);
        if (D != (R)0) {
            R lap = (v[n + 1] - 2 * c + v[n - 1]) * idx2 + (v[n + st.px] - 2 * c + v[n - st.px]) * idy2;
            if (m.dim == 3) lap = lap + (v[zr] - 2 * c + v[zl]) * idz2;
            evo[f] = D * lap;
        } else {
            evo[f] = 0;
        }
    }
    R fr[CB_MAX_BUF];
    for (int b = 0; b < m.n_buf; ++b) fr[b] = (R)m.Ctot[b];
    for (int p = 0; p < m.n_pairs; ++p) fr[m.pair_buf[p]] -= val[m.n_ions + p];
    R Rj[CB_MAX_IONS];
    for (int j = 0; j < m.n_ions; ++j) Rj[j] = 0;
    for (int p = 0; p < m.n_pairs; ++p) {
        int j = m.pair_ion[p];
        R R1 = (R)m.koff[p] * val[m.n_ions + p] - (R)m.kon[p] * val[j] * fr[m.pair_buf[p]];
        evo[m.n_ions + p] += -R1;
        Rj[j] += R1;
    }
    const R dt = (R)m.dt;
    const R* cg = curg + st.node_base * m.n_ions;
    const bool sl_layer = (m.dim == 2) || (z == st.nz - 1);
    for (int j = 0; j < m.n_ions; ++j) {
        R e = evo[j] + Rj[j];
        e += cg[(long long)j * st.npad + n];
        if (sl_layer && m.has_sl[j]) {
            R s1 = (R)m.K1[j] + val[j];
            R s2 = (R)m.K2[j] + val[j];
            e *= (R)1 / ((R)1 + (R)(m.N1[j] * m.K1[j]) / (s1 * s1) + (R)(m.N2[j] * m.K2[j]) / (s2 * s2));
        }
        o[(long long)j * st.npad + n] = val[j] + e * dt;
    }
    for (int p = 0; p < m.n_pairs; ++p) o[(long long)(m.n_ions + p) * st.npad + n] = val[m.n_ions + p] + evo[m.n_ions + p] * dt;
}

// Deterministic block sum of `v` (blockDim.x == 256).
__device__ double block_sum(double v, double* red) {
    red[threadIdx.x] = v;
    __syncthreads();
    for (int w = blockDim.x >> 1; w > 0; w >>= 1) {
        if (threadIdx.x < w) red[threadIdx.x] += red[threadIdx.x + w];
        __syncthreads();
    }
    double r = red[0];
    __syncthreads();
    return r;
}

template <typename R>
__global__ void __launch_bounds__(256) k_update(cb_model m, int NS, const cb_site* __restrict__ sites, R* __restrict__ fld,
                                                R* __restrict__ curg, const int* __restrict__ ch_node,
                                                const int* __restrict__ ch_owner, const int* __restrict__ ch_state,
                                                double* __restrict__ mouth, cb_site_scalars* __restrict__ sc, int nc,
                                                const R* __restrict__ cyto, double* __restrict__ cin,
                                                const int* __restrict__ rim_cnode, const int* __restrict__ dep_ptr,
                                                const int* __restrict__ dep_term) {
    extern __shared__ double smem[];
    double* red = smem;            // 256
    double* terms = smem + 256;    // RD3D: max_terms * F deposit values
    const int s = blockIdx.x;
    const cb_site st = sites[s];
    cb_site_scalars& q = sc[s];
    const int F = m.F;
    R* u = fld + st.node_base * F;
    const int nx = st.nx, ny = st.ny, nz = st.nz, px = st.px, nxy = px * ny;
    const long long np = st.npad;
    // 1. mouth values: ions, pairs, free buffers (CaSim/DyadRD2DCPU.cpp:361-380)
    for (int c = threadIdx.x; c < st.n_ch; c += blockDim.x) {
        int node = ch_node[st.ch_off + c];
        double* mo = mouth + (long long)(st.ch_off + c) * NS;
        double fr[CB_MAX_BUF];
        for (int b = 0; b < m.n_buf; ++b) fr[b] = m.Ctot[b];
        for (int f = 0; f < F; ++f) {
            double v = (double)u[f * np + node];
            mo[f] = v;
            if (f >= m.n_ions) fr[m.pair_buf[f - m.n_ions]] -= v;
        }
        for (int b = 0; b < m.n_buf; ++b) mo[F + b] = fr[b];
    }
    __syncthreads();
    // 2. Dirichlet edges from the cytosol (CaSim/DyadRD2DCPU.cpp:274-303)
    const int nrim = cb_rim_count(nx, ny);
    const int CS = m.n_ions + m.c_n_pairs;
    const R* cy = cyto ? cyto + (long long)s * CS * nc : nullptr;
    for (int t = threadIdx.x; t < nrim * nz; t += blockDim.x) {
        int r = t % nrim, z = t / nrim, x, y;
        cb_rim_xy(r, nx, ny, x, y);
        int node = x + px * y + nxy * z;
        if (m.cyto_type == CB_CYTO_POOL) {
            for (int j = 0; j < m.n_ions; ++j) u[j * np + node] = (R)q.c_ions[j];
            for (int p = 0; p < m.n_pairs; ++p) u[(m.n_ions + p) * np + node] = (R)q.c_bnd[p];
        } else {
            int cn = rim_cnode[st.rim_off + r];
            for (int j = 0; j < m.n_ions; ++j) u[j * np + node] = cy[(long long)j * nc + cn];
            for (int p = 0; p < m.n_pairs; ++p) {
                int cq = m.dyad_c_pair[p];
                u[(m.n_ions + p) * np + node] = cq >= 0 ? cy[(long long)(m.n_ions + cq) * nc + cn] : (R)m.pair_init[p];
            }
        }
    }
    __syncthreads();
    // 3. efflux (CaSim/DyadRD2DCPU.cpp:305-350): per-term values, block sums
    const int zmax = m.dim == 2 ? 1 : nz - 1;
    const int T = cb_efflux_terms(nx, ny, zmax);
    double part[CB_MAX_SPECIES];
    for (int f = 0; f < F; ++f) part[f] = 0;
    const bool rd3d = m.cyto_type == CB_CYTO_RD3D;
    for (int t = threadIdx.x; t < T; t += blockDim.x) {
        int x0, y0, x1, y1, x2, y2, z;
        int sel = cb_efflux_term(t, nx, ny, zmax, x0, y0, x1, y1, x2, y2, z);
        double sf = sel == 0 ? m.sx : m.sy;
        int n0 = x0 + px * y0 + nxy * z, n1 = x1 + px * y1 + nxy * z, n2 = x2 + px * y2 + nxy * z;
        for (int f = 0; f < F; ++f) {
            double D = f < m.n_ions ? m.D_ion[f] : m.D_pair[f - m.n_ions];
            double g = 2 * (double)u[f * np + n1] - 1.5 * (double)u[f * np + n0] - 0.5 * (double)u[f * np + n2];
            if (!rd3d) {
                part[f] += D * m.grad_mult * sf * g;
            } else {
                double v = D * sf * g * m.inv_hc3;
                part[f] += v;
                terms[(long long)t * F + f] = v;
            }
        }
    }
    for (int f = 0; f < F; ++f) {
        double tot = block_sum(part[f], red);
        if (threadIdx.x == 0) q.efflux[f] = tot;
    }
    // 4. RD3D: deposit into the cytosol layer z = 0 in term order
    if (rd3d) {
        __syncthreads();
        const int mc2 = m.mc * m.mc;
        const int* ptr = dep_ptr + (long long)s * (mc2 + 1);
        for (int cn = threadIdx.x; cn < mc2; cn += blockDim.x) {
            int lo = ptr[cn], hi = ptr[cn + 1];
            for (int c = 0; c < CS; ++c) {
                int f = c < m.n_ions ? c : m.c_dyad_pair[c - m.n_ions];
                if (f >= 0 && c >= m.n_ions) f += m.n_ions;
                double acc = 0;
                if (f >= 0)
                    for (int k = lo; k < hi; ++k) acc += terms[(long long)dep_term[st.term_off + k] * F + f];
                cin[((long long)s * CS + c) * mc2 + cn] = acc;
            }
        }
    }
    // 5. RyR currents (CaSim/DyadRD2DCPU.cpp:243-264, CaSim/PassiveIonChannel.cpp:28-34)
    R* cg = curg + st.node_base * m.n_ions;
    double tot[CB_MAX_IONS];
    for (int j = 0; j < m.n_ions; ++j) tot[j] = 0;
    for (int c = threadIdx.x; c < st.n_ch; c += blockDim.x) {
        int node = ch_node[st.ch_off + c];
        int state = ch_state[st.ch_off + c];
        for (int j = 0; j < m.n_ions; ++j) {
            double flux = state * (m.g[j] * (q.jsr_new[j] - (double)u[j * np + node]));
            if (ch_owner[st.ch_off + c]) cg[j * np + node] = (R)flux;
            tot[j] += flux;
        }
    }
    for (int j = 0; j < m.n_ions; ++j) {
        double t = block_sum(tot[j], red);
        if (threadIdx.x == 0) q.total[j] = t;
    }
    // 6. jSR coupling (CaSim/SRPool.cpp:55-68)
    if (threadIdx.x == 0 && !m.jsr_const)
        for (int i = 0; i < m.n_ions; ++i) {
            q.IjSR[i] = q.total[i] * m.V_elem;
            q.nsr[i] = m.nsr[i];
            q.jsr[i] = q.jsr_new[i];
        }
}

// A kernel's cap on dynamic shared memory is common to all handles, whose needs differ: always the
// most a block can have, so that no handle (nor another thread) lowers it between this and a launch.
cudaError_t allow_most_smem(const void* kern) {
    cudaFuncAttributes fa;
    int dev = 0, most = 0;
    cudaError_t e = cudaFuncGetAttributes(&fa, kern);
    if (e == cudaSuccess) e = cudaGetDevice(&dev);
    if (e == cudaSuccess) e = cudaDeviceGetAttribute(&most, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev);
    if (e != cudaSuccess) return e;
    return cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, most - (int)fa.sharedSizeBytes);
}

// jump table of the warp-parallel gating: row l < 32 holds A^(2l), both components, stored
// entry-major (row 31, A^62, also takes a lane from one chunk of 32 draws to the next)
bool pre_jump(cb_dev& d) {
    if (d.pre_jump) return true;
    std::vector<unsigned long long> t(32 * 18);
    const cbrng::Mat3 a1 = cbrng::step_matrix1(), a2 = cbrng::step_matrix2();
    cbrng::Mat3 p1{{{1, 0, 0}, {0, 1, 0}, {0, 0, 1}}}, p2 = p1;  // A^(2l)
    for (int l = 0; l < 32; ++l) {
        for (int i = 0; i < 9; ++i) {
            t[32 * i + l] = p1.a[i / 3][i % 3];
            t[32 * (9 + i) + l] = p2.a[i / 3][i % 3];
        }
        for (int k = 0; k < 2; ++k) {
            p1 = cbrng::matmul(a1, p1, cbrng::M1);
            p2 = cbrng::matmul(a2, p2, cbrng::M2);
        }
    }
    if (cudaMalloc(&d.pre_jump, sizeof(unsigned long long) * t.size()) != cudaSuccess) {
        d.pre_jump = nullptr;
        return false;
    }
    if (cudaMemcpy(d.pre_jump, t.data(), sizeof(unsigned long long) * t.size(), cudaMemcpyHostToDevice) != cudaSuccess) {
        cudaFree(d.pre_jump);
        d.pre_jump = nullptr;
        return false;
    }
    return true;
}

// The specialised stencils (stream_kernels.cuh) serve 1-2 ions with up to 4 pairs
// and a cleft of one layer (2D) or three (3D) at every site; the first step lists
// the cleft blocks (site, first group). Returns the tile count, 0 if not covered.
int stream_tiles(cb_dev& d) {
    if (d.st_nz >= 0) return d.st_nz > 0 ? d.st_ntiles : 0;
    d.st_nz = 0;
    const int np = d.m.n_pairs, ncp = d.m.c_n_pairs;
    if (d.m.n_ions < 1 || d.m.n_ions > 2 || np > 4 || ncp > 4) return 0;
    std::vector<cb_site> hs(d.S);
    if (cudaMemcpy(hs.data(), d.sites, sizeof(cb_site) * d.S, cudaMemcpyDeviceToHost) != cudaSuccess) return 0;
    const int nz = d.m.dim == 2 ? 1 : 3;
    const int V = stream::rd_vec(d.precision == 0 ? 8 : 4);
    std::vector<int4> tiles;
    std::vector<stream::rd_tile> runs;
    const int tn = stream::rdt_threads(d.precision == 0 ? 8 : 4) * V;
    static_assert(CB_SITE_NODES % 128 == 0 && stream::rdt_threads(4) * stream::rd_vec(4) % 128 == 0 && stream::rdt_threads(8) * stream::rd_vec(8) % 128 == 0,
                  "a tile's RyR bits begin on 16 bytes");
    int px_min = INT32_MAX, px_max = 0;
    bool two_rims = false;  // a tile may hold a site's first and last row
    for (int s = 0; s < d.S; ++s) {
        if (hs[s].nz != nz || (long long)hs[s].npad * d.m.F > INT32_MAX) return 0;
        // the row of a column by a multiply and a shift: floor(2^32 (2^w - px) / px) + 1, w =
        // ceil(log2 px), exact below 2^31 (Granlund and Montgomery 1994)
        unsigned w = 0;
        while ((1u << w) < (unsigned)hs[s].px) ++w;
        const unsigned mul = (unsigned)(((1ull << 32) * ((1ull << w) - hs[s].px)) / hs[s].px + 1);
        const int groups = hs[s].px * hs[s].ny / V;
        for (int c = 0; c < groups; c += stream::RD_THREADS) tiles.push_back(make_int4(s, c, (int)mul, (int)w));
        for (int c = 0; c < groups * V; c += tn) {
            stream::rd_tile t{};
            t.node_base = hs[s].node_base;
            t.site = s;
            t.col0 = c;
            t.np = hs[s].npad;
            t.px = hs[s].px;
            t.nx = hs[s].nx;
            t.ny = hs[s].ny;
            t.rim_off = hs[s].rim_off;
            t.mul = mul;
            t.sh = w;
            runs.push_back(t);
        }
        px_min = std::min(px_min, hs[s].px);
        px_max = std::max(px_max, hs[s].px);
        two_rims = two_rims || hs[s].px * (hs[s].ny - 2) <= tn;
    }
    if (tiles.empty() || tiles.size() > (size_t)INT32_MAX) return 0;
    if (cudaMalloc(&d.st_tiles, sizeof(int4) * tiles.size()) != cudaSuccess) return 0;
    if (cudaMemcpy(d.st_tiles, tiles.data(), sizeof(int4) * tiles.size(), cudaMemcpyHostToDevice) != cudaSuccess) {
        cudaFree(d.st_tiles);
        d.st_tiles = nullptr;
        return 0;
    }
    d.st_ntiles = (int)tiles.size();
    // the columns that hold a RyR: bit (node_base + x + px*y), one word per 32 nodes
    // (the last tile of a site may read up to a tile's bits past the end)
    std::vector<unsigned> bits((size_t)(d.total_nodes + 31) / 32 + 64, 0u);
    std::vector<int> chn((size_t)d.total_ch);
    if (d.total_ch && cudaMemcpy(chn.data(), d.ch_node, sizeof(int) * chn.size(), cudaMemcpyDeviceToHost) != cudaSuccess) return 0;
    for (int s = 0; s < d.S; ++s)
        for (int c = 0; c < hs[s].n_ch; ++c) {
            const long long b = hs[s].node_base + chn[hs[s].ch_off + c] % (hs[s].px * hs[s].ny);
            bits[b >> 5] |= 1u << (b & 31);
        }
    if (cudaMalloc(&d.st_chcol, sizeof(unsigned) * bits.size()) != cudaSuccess) return 0;
    if (cudaMemcpy(d.st_chcol, bits.data(), sizeof(unsigned) * bits.size(), cudaMemcpyHostToDevice) != cudaSuccess) return 0;
    if (!pre_jump(d)) return 0;
    // per RyR its node and flags
    std::vector<int2> chv((size_t)d.total_ch);
    std::vector<int> own((size_t)d.total_ch);
    if (d.total_ch && cudaMemcpy(own.data(), d.ch_owner, sizeof(int) * own.size(), cudaMemcpyDeviceToHost) != cudaSuccess) return 0;
    for (int s = 0; s < d.S; ++s)
        for (int c = hs[s].ch_off; c < hs[s].ch_off + hs[s].n_ch; ++c) {
            const int x = chn[c] % hs[s].px, y = (chn[c] / hs[s].px) % hs[s].ny;
            const bool rim = x == 0 || x == hs[s].nx - 1 || y == 0 || y == hs[s].ny - 1;
            chv[c] = make_int2(chn[c], (own[c] ? stream::CH_OWNER : 0) | (rim ? stream::CH_RIM : 0));
        }
    if (cudaMalloc(&d.st_ch, sizeof(int2) * std::max<size_t>(chv.size(), 1)) != cudaSuccess) return 0;
    if (cudaMemcpy(d.st_ch, chv.data(), sizeof(int2) * chv.size(), cudaMemcpyHostToDevice) != cudaSuccess) return 0;
    if (cudaMalloc(&d.st_prob, sizeof(double) * (size_t)std::max<long long>(d.total_ch, 1) * (d.mwc ? 3 : 1)) != cudaSuccess) return 0;
    // shared-memory carve of the asynchronous kernel's stages. It is used where at least two
    // blocks (FP64) or three (FP32) fit an SM, 12 computing warps; with fewer it is no faster than
    // k_rd_v (2048 sites, FP32: three blocks 189 us, two 270, k_rd_v 262)
    {
        const int rsz = d.precision == 0 ? 8 : 4;
        stream::rd_stage g{};
        auto up = [](int v) { return (v + 127) / 128 * 128; };
        int off = sizeof(stream::rd_tile);
        g.bits = off;
        off = up(off + tn / 8);
        g.rim = off;
        off = up(off + (2 * (tn / px_min + 2) + (two_rims ? 2 : 1) * px_max) * d.m.F * rsz);
        g.halo = px_max + 16 / rsz;
        for (int f = 0; f < d.m.F; ++f) {
            const bool diff = (f < d.m.n_ions ? d.m.D_ion[f] : d.m.D_pair[f - d.m.n_ions]) != 0;
            g.plane[f] = off;
            g.stride[f] = up((tn + (diff ? 2 * g.halo : 0)) * rsz);
            off += g.stride[f] * nz;
        }
        g.bytes = off;
        const long long block = (long long)off * stream::RDT_STAGES + 2048;
        if (block * (rsz == 4 ? 3 : 2) <= 228 * 1024) {
            if (cudaMalloc(&d.st_runs, sizeof(stream::rd_tile) * runs.size()) != cudaSuccess) return 0;
            if (cudaMemcpy(d.st_runs, runs.data(), sizeof(stream::rd_tile) * runs.size(), cudaMemcpyHostToDevice) != cudaSuccess) return 0;
            d.st_nruns = (int)runs.size();
            static_assert(sizeof(g) <= sizeof(d.st_stage), "carve");
            std::memcpy(d.st_stage, &g, sizeof(g));
        }
    }
    d.st_nz = nz;
    return d.st_ntiles;
}

stream::gate_args gating(const cb_dev& d) {
    stream::gate_args g{};
    g.spx0 = d.spx[0];
    g.spc0 = d.spc[0];
    g.spx1 = d.spx[1];
    g.spc1 = d.spc[1];
    g.J = d.pre_jump;
    g.gates = d.gates;
    g.site_gate = d.site_gate;
    g.mwc = d.mwc;
    g.ch_state = d.ch_state;
    g.ch_micro = d.ch_micro;
    g.prob = d.st_prob;
    g.pcm = d.st_prob + d.total_ch;
    return g;
}

// gate: a time step's gating, pools and Update, right after the cleft kernel; else the Update alone
template <typename R, int NI, int NP, bool RD3D>
cudaError_t launch_update_s(cb_dev& d, cudaStream_t st, bool gate, bool want) {
    stream::dep_args dep{};
    if (RD3D) {
        dep.pos = d.st_dpos;
        dep.node_ptr = d.st_dnptr;
        dep.node = d.st_dnode;
        dep.max_nodes = d.st_max_dn;
        for (int c = 0; c < d.CS; ++c) {
            const int p = c < NI ? -1 : d.m.c_dyad_pair[c - NI];
            if (c >= NI && p < 0) continue;
            dep.f[dep.n] = c < NI ? c : NI + p;
            dep.c[dep.n++] = c;
        }
    }
    size_t smem = (size_t)(d.max_ch + 7) / 8 * 8;
    if (RD3D) smem += (size_t)d.max_terms * dep.n * sizeof(double) + (size_t)dep.max_nodes * sizeof(int3);
    auto kern = gate ? stream::k_update_s<R, NI, NP, RD3D, true> : stream::k_update_s<R, NI, NP, RD3D, false>;
    if (smem > 40 * 1024 && !d.up_smem_set[gate]) {
        const cudaError_t e = allow_most_smem((const void*)kern);
        if (e != cudaSuccess) return e;
        d.up_smem_set[gate] = true;
    }
    // the rim reads the cytosol as it was before its latest step (RD3D coupling)
    kern<<<d.S, stream::UP_THREADS, smem, st>>>(d.m, gating(d), dep, d.NS, want, d.sites, (R*)d.fields[d.cur], (const R*)d.fields[1 - d.cur],
                                                (R*)d.curgrid, d.st_ch, d.mouth, d.sc, d.nc, (const R*)d.cyto[1 - d.ccur], d.cin, d.rim_cnode,
                                                d.max_ch, d.max_terms);
    return cudaGetLastError();
}

template <typename R, int NI, bool RD3D>
cudaError_t launch_update_np(cb_dev& d, cudaStream_t st, bool gate, bool want) {
    switch (d.m.n_pairs) {
    case 0: return launch_update_s<R, NI, 0, RD3D>(d, st, gate, want);
    case 1: return launch_update_s<R, NI, 1, RD3D>(d, st, gate, want);
    case 2: return launch_update_s<R, NI, 2, RD3D>(d, st, gate, want);
    case 3: return launch_update_s<R, NI, 3, RD3D>(d, st, gate, want);
    default: return launch_update_s<R, NI, 4, RD3D>(d, st, gate, want);
    }
}

template <typename R>
cudaError_t launch_update(cb_dev& d, cudaStream_t st, bool gate = false, bool want = true) {
    if (stream_tiles(d) > 0) {
        const bool rd3d = d.m.cyto_type == CB_CYTO_RD3D;
        if (d.m.n_ions == 1)
            return rd3d ? launch_update_np<R, 1, true>(d, st, gate, want) : launch_update_np<R, 1, false>(d, st, gate, want);
        return rd3d ? launch_update_np<R, 2, true>(d, st, gate, want) : launch_update_np<R, 2, false>(d, st, gate, want);
    }
    size_t smem = 256 * sizeof(double);
    if (d.m.cyto_type == CB_CYTO_RD3D) smem += (size_t)d.max_terms * d.m.F * sizeof(double);
    if (smem > 48 * 1024 && !d.up_smem_set[0]) {
        const cudaError_t e = allow_most_smem((const void*)k_update<R>);
        if (e != cudaSuccess) return e;
        d.up_smem_set[0] = true;
    }
    // the rim reads the cytosol as it was before its latest step (RD3D coupling)
    k_update<R><<<d.S, 256, smem, st>>>(d.m, d.NS, d.sites, (R*)d.fields[d.cur], (R*)d.curgrid, d.ch_node, d.ch_owner,
                                        d.ch_state, d.mouth, d.sc, d.nc, (const R*)d.cyto[1 - d.ccur], d.cin, d.rim_cnode,
                                        d.dep_ptr, d.dep_term);
    return cudaGetLastError();
}

// constants of the cleft stencil
template <typename R>
stream::rd_const<R> rd_constants(const cb_dev& d) {
    const cb_model& m = d.m;
    stream::rd_const<R> k{};
    for (int f = 0; f < m.F; ++f) {
        const double D = f < m.n_ions ? m.D_ion[f] : m.D_pair[f - m.n_ions];
        k.ax[f] = stream::both((R)(D * m.dt * m.inv_dx2));
        k.ay[f] = stream::both((R)(D * m.dt * m.inv_dy2));
        k.az[f] = stream::both((R)(D * m.dt * m.inv_dz2));
        k.diff[f] = D != 0;
        const int cq = f < m.n_ions ? f : m.dyad_c_pair[f - m.n_ions];
        k.src[f] = f < m.n_ions ? f : cq >= 0 ? m.n_ions + cq : -1;
        k.init[f] = (R)(f < m.n_ions ? m.Cb[f] : m.pair_init[f - m.n_ions]);
    }
    for (int p = 0; p < m.n_pairs; ++p) {
        k.mkon[p] = stream::both((R)(-m.kon[p] * m.dt));
        k.koff[p] = stream::both((R)(m.koff[p] * m.dt));
        k.ctot[p] = stream::both((R)m.Ctot[m.pair_buf[p]]);
        k.pion[p] = m.pair_ion[p];
        for (int q = 0; q < m.n_pairs; ++q)
            if (m.pair_buf[q] == m.pair_buf[p]) k.same[p] |= 1u << q;
    }
    for (int j = 0; j < m.n_ions; ++j) {
        k.has_sl[j] = m.has_sl[j];
        k.K1[j] = (R)m.K1[j];
        k.K2[j] = (R)m.K2[j];
        k.A1[j] = (R)(m.N1[j] * m.K1[j]);
        k.A2[j] = (R)(m.N2[j] * m.K2[j]);
    }
    k.dt = stream::both((R)m.dt);
    k.CS = d.CS;
    k.nc = d.nc;
    return k;
}

// constants of the RD3D cytosol stencil
template <typename R>
stream::cy_const<R> cy_constants(const cb_dev& d) {
    const cb_model& m = d.m;
    stream::cy_const<R> k{};
    for (int c = 0; c < d.CS; ++c) k.a[c] = stream::both((R)((c < m.n_ions ? m.D_ion[c] : m.c_D_pair[c - m.n_ions]) * m.dt * m.inv_hc2));
    for (int p = 0; p < m.c_n_pairs; ++p) {
        k.mkon[p] = stream::both((R)(-m.c_kon[p] * m.dt));
        k.koff[p] = stream::both((R)(m.c_koff[p] * m.dt));
        k.ctot[p] = stream::both((R)m.c_Ctot[m.c_pair_buf[p]]);
        k.pion[p] = m.c_pair_ion[p];
        for (int q = 0; q < m.c_n_pairs; ++q)
            if (m.c_pair_buf[q] == m.c_pair_buf[p]) k.same[p] |= 1u << q;
    }
    int is = 0;
    for (int j = 0; j < m.n_ions; ++j)
        if ((k.serca[j] = m.c_serca[j]) != 0) {
            const double K2 = m.c_Kup[is] * m.c_Kup[is], b2 = m.c_bg[is] * m.c_bg[is];
            k.mjmax[j] = stream::both((R)(-m.c_Jmax[is] * m.dt));
            k.k2[j] = stream::both((R)K2);
            k.mrest[j] = stream::both((R)(-(b2 / (b2 + K2))));
            ++is;
        }
    k.dt = (R)m.dt;
    k.mc = m.mc;
    k.px = m.cpx;
    k.nplane = m.mc * m.cpx;
    k.nc = d.nc;
    return k;
}

template <typename R, int NI, int NP>
cudaError_t launch_rd_s(cb_dev& d, cudaStream_t st) {
    constexpr int V = stream::rd_vec(sizeof(R));
    const R* in = (const R*)d.fields[d.cur];
    R* out = (R*)d.fields[1 - d.cur];
    // the cytosol as it was before its latest step (k_cyto flipped ccur already)
    const R* cy = d.m.cyto_type == CB_CYTO_RD3D ? (const R*)d.cyto[1 - d.ccur] : nullptr;
    if (d.st_runs) {
        stream::rd_stage g;
        std::memcpy(&g, d.st_stage, sizeof(g));
        const int smem = g.bytes * stream::RDT_STAGES;
        auto kern = d.st_nz == 1 ? stream::k_rd_t<R, NI, NP, 1, V, stream::RDT_STAGES> : stream::k_rd_t<R, NI, NP, 3, V, stream::RDT_STAGES>;
        cudaError_t e;
        if (d.st_grid == 0) {
            if ((e = allow_most_smem((const void*)kern)) != cudaSuccess) return e;
            int dev = 0, sms = 0, per = 0;
            if ((e = cudaGetDevice(&dev)) != cudaSuccess) return e;
            if ((e = cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev)) != cudaSuccess) return e;
            if ((e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per, kern, stream::rdt_threads(sizeof(R)) + 32, smem)) != cudaSuccess) return e;
            d.st_grid = std::max(1, std::min(sms * per, d.st_nruns));
        }
        kern<<<d.st_grid, stream::rdt_threads(sizeof(R)) + 32, smem, st>>>(rd_constants<R>(d), g, (const stream::rd_tile*)d.st_runs, d.st_nruns, in,
                                                                          out, (const R*)d.curgrid, cy, d.rim_cnode, d.st_chcol, d.err_flag);
        return cudaGetLastError();
    }
    auto kern = d.st_nz == 1 ? stream::k_rd_v<R, NI, NP, 1, V> : stream::k_rd_v<R, NI, NP, 3, V>;
    kern<<<d.st_ntiles, stream::RD_THREADS, 0, st>>>(rd_constants<R>(d), d.sites, d.st_tiles, in, out, (const R*)d.curgrid, cy,
                                                     d.rim_cnode, d.st_chcol);
    return cudaGetLastError();
}

template <typename R, int NI>
cudaError_t launch_rd_np(cb_dev& d, cudaStream_t st) {
    switch (d.m.n_pairs) {
    case 0: return launch_rd_s<R, NI, 0>(d, st);
    case 1: return launch_rd_s<R, NI, 1>(d, st);
    case 2: return launch_rd_s<R, NI, 2>(d, st);
    case 3: return launch_rd_s<R, NI, 3>(d, st);
    default: return launch_rd_s<R, NI, 4>(d, st);
    }
}

template <typename R, int NI, int NCP>
cudaError_t launch_cyto_s(cb_dev& d, cudaStream_t st) {
    constexpr int V = CB_CYTO_VEC;
    const R* in = (const R*)d.cyto[d.ccur];
    R* out = (R*)d.cyto[1 - d.ccur];
    const int planes = d.m.mc - 1;
    if (d.m.mc == 25) {
        // the planes of a site in 1, 2 or 3 chunks (each but the first loads a plane or two
        // more) so that a small batch fills the chip; FP32, us for 1 / 2 / 3 / 4 chunks: 2048 sites
        // 148 / 154 / 166 / 177, 512 sites 51.5 / 45.9 / 47.3 / 47.4, 128 sites 19.2 / 16.6 / 15.2 / 15.4
        const int chunks = d.S >= 1024 ? 1 : d.S >= 256 ? 2 : 3, chunk = (planes + chunks - 1) / chunks;
        constexpr int stages = stream::cyt_stages(sizeof(R), NI + NCP);
        constexpr int smem = stages * (NI + NCP) * stream::cyt_planes<sizeof(R)>() * 25 * ((25 + V - 1) / V * V) * (int)sizeof(R);
        auto kern = stream::k_cyto_t<R, NI, NCP, V, 25, stages>;
        if (!d.st_cyt_ready) {
            const cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
            if (e != cudaSuccess) return e;
            d.st_cyt_ready = true;
        }
        kern<<<dim3(d.S, chunks), stream::CY_THREADS + 32, smem, st>>>(cy_constants<R>(d), chunk, in, out, d.cin, d.err_flag);
        return cudaGetLastError();
    }
    // a layer of fewer groups takes one block of its own size
    constexpr int W = stream::cyv_vec(sizeof(R)), most = stream::cyv_threads(sizeof(R), NI + NCP);
    const int groups = d.m.mc * d.m.cpx / W, thr = std::min(most, (groups + 31) / 32 * 32);
    stream::k_cyto_v<R, NI, NCP, W><<<dim3(d.S, (groups + thr - 1) / thr), thr, 0, st>>>(cy_constants<R>(d), in, out, d.cin);
    return cudaGetLastError();
}

template <typename R, int NI>
cudaError_t launch_cyto_np(cb_dev& d, cudaStream_t st) {
    switch (d.m.c_n_pairs) {
    case 0: return launch_cyto_s<R, NI, 0>(d, st);
    case 1: return launch_cyto_s<R, NI, 1>(d, st);
    case 2: return launch_cyto_s<R, NI, 2>(d, st);
    case 3: return launch_cyto_s<R, NI, 3>(d, st);
    default: return launch_cyto_s<R, NI, 4>(d, st);
    }
}

// One time step, the `first` or `last` of its call. ev (optional, 5 events): recorded before the
// gating kernel (specialised kernels: the probabilities of a call's first gating; the gating runs
// in the Update kernel) and after each of the gating, cytosol, cleft and Update kernels.
template <typename R>
cudaError_t launch_step(cb_dev& d, cudaStream_t st, bool first, bool last, cudaEvent_t* ev = nullptr) {
    auto mark = [&](int k) { return ev ? cudaEventRecord(ev[k], st) : cudaSuccess; };
    cudaError_t e0 = mark(0);
    if (e0 != cudaSuccess) return e0;
    const bool fast = stream_tiles(d) > 0;
    if (fast) {
        if (first) stream::k_prob<<<d.S, 64, 0, st>>>(d.m, gating(d), d.NS, d.sites, d.mouth);
    } else if (d.site_gate) {
        return cudaErrorNotSupported;  // per-site models need the specialised kernels
    } else {
        k_pre<<<(d.S + 127) / 128, 128, 0, st>>>(d.m, d.S, d.NS, d.sites, d.sc, d.ch_state, d.mouth, d.spx[0], d.spc[0],
                                                   d.spx[1], d.spc[1], d.ch_micro, d.mwc);
    }
    if ((e0 = mark(1)) != cudaSuccess) return e0;
    if (d.m.cyto_type == CB_CYTO_RD3D) {
        if (fast) {
            e0 = d.m.n_ions == 1 ? launch_cyto_np<R, 1>(d, st) : launch_cyto_np<R, 2>(d, st);
            if (e0 != cudaSuccess) return e0;
        } else {
            dim3 g((d.nc + 255) / 256, d.S);
            k_cyto<R><<<g, 256, 0, st>>>(d.m, d.nc, (const R*)d.cyto[d.ccur], (R*)d.cyto[1 - d.ccur], d.cin);
        }
        d.ccur ^= 1;
    }
    if ((e0 = mark(2)) != cudaSuccess) return e0;
    if (fast) {
        e0 = d.m.n_ions == 1 ? launch_rd_np<R, 1>(d, st) : launch_rd_np<R, 2>(d, st);
        if (e0 != cudaSuccess) return e0;
    } else {
        dim3 g((d.max_nodes + 255) / 256, d.S);
        k_rd<R><<<g, 256, 0, st>>>(d.m, d.sites, (const R*)d.fields[d.cur], (R*)d.fields[1 - d.cur], (const R*)d.curgrid);
    }
    d.cur ^= 1;
    if ((e0 = mark(3)) != cudaSuccess) return e0;
    if ((e0 = launch_update<R>(d, st, fast, last)) != cudaSuccess) return e0;
    return mark(4);
}

// ---- surrogate-driven gating (no RD): the mouth Ca comes from the surrogate network

// features of every site (one thread per feature): per RyR slot its open flag and
// grid position scaled to [-1, 1] by the cleft half-widths, then the jSR Ca of
// the first ion / 1000 uM, then each dyad buffer total relative to its config value
__global__ void k_sg_features(int S, int n_buf, int max_ch, int ld, const cb_site* __restrict__ sites, const int* __restrict__ ch_node,
                              const int* __restrict__ ch_state, const cb_site_scalars* __restrict__ sc, float* __restrict__ X) {
    const long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x;
    if (i >= (long long)S * ld) return;
    const int s = (int)(i / ld), k = (int)(i - (long long)s * ld), c = k / 3, what = k - 3 * c;
    float v = 0.0f;
    if (k < 3 * max_ch) {
        const cb_site st = sites[s];
        if (c < st.n_ch) {
            const int node = ch_node[st.ch_off + c];
            const float hx = 0.5f * (st.nx - 1), hy = 0.5f * (st.ny - 1);
            v = what == 0 ? (float)ch_state[st.ch_off + c] : what == 1 ? (node % st.px - hx) / hx : ((node / st.px) % st.ny - hy) / hy;
        }
    } else if (k == 3 * max_ch) {
        v = (float)(sc[s].jsr_new[0] / 1000.0);
    } else if (k <= 3 * max_ch + n_buf) {
        v = 1.0f;
    }
    X[i] = v;
}

// mouth Ca of every RyR from the network output: ca_ref * 10^y (a thread per site and slot)
__global__ void k_sg_mouth(int S, int NS, int ca_idx, double ca_ref, int ld, const cb_site* __restrict__ sites,
                           const float* __restrict__ Y, double* __restrict__ mouth, int slots) {
    const long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x;
    const int s = (int)(i / slots), c = (int)(i - (long long)s * slots);
    if (s >= S) return;
    const cb_site st = sites[s];
    if (c < st.n_ch) mouth[(size_t)(st.ch_off + c) * NS + ca_idx] = ca_ref * exp10((double)Y[(size_t)s * ld + c]);
}

// n time steps of one site without the RD step: cytosol pool and jSR ODEs and
// RyR gating in the order of k_pre, then the part of Update that needs no
// field: RyR currents from the held mouth values and the jSR coupling
__global__ void k_sg_steps(cb_model m, int S, int NS, long long n, const cb_site* __restrict__ sites, cb_site_scalars* __restrict__ sc,
                           int* __restrict__ ch_state, const double* __restrict__ mouth, const double* __restrict__ spx0,
                           const double* __restrict__ spc0, const double* __restrict__ spx1, const double* __restrict__ spc1) {
    const int s = blockIdx.x * blockDim.x + threadIdx.x;
    if (s >= S) return;
    const cb_site st = sites[s];
    cb_site_scalars& q = sc[s];
    const double dt = m.dt;
    cbrng::State g;
    for (int i = 0; i < 6; ++i) g.s[i] = q.rng[i];
    unsigned long long draws = 0;
    // the mouth values are held, so the transition probability of each state is
    // fixed for the whole call: computed once for the first SG_CACHE RyRs
    constexpr int SG_CACHE = 32;
    double pc[2][SG_CACHE];
    const int ncache = st.n_ch < SG_CACHE ? st.n_ch : SG_CACHE;
    for (int c = 0; c < ncache; ++c) {
        const double* mo = mouth + (long long)(st.ch_off + c) * NS;
        const double ca = mo[m.ca_idx];
        const double mg = m.mg_idx >= 0 ? mo[m.mg_idx] : 0.0;
        pc[0][c] = cb_rate(m, spx0, spc0, spx1, spc1, 0, ca, mg) * dt;
        pc[1][c] = cb_rate(m, spx0, spc0, spx1, spc1, 1, ca, mg) * dt;
    }
    for (long long it = 0; it < n; ++it) {
        if (m.cyto_type == CB_CYTO_POOL) cb_pool_step(m, q, dt);
        cb_jsr_step(m, q, dt);
        for (int c = 0; c < st.n_ch; ++c) {
            const int state = ch_state[st.ch_off + c];
            double p;
            if (c < ncache) {
                p = pc[state][c];
            } else {
                const double* mo = mouth + (long long)(st.ch_off + c) * NS;
                const double mg = m.mg_idx >= 0 ? mo[m.mg_idx] : 0.0;
                p = cb_rate(m, spx0, spc0, spx1, spc1, state, mo[m.ca_idx], mg) * dt;
            }
            ++draws;
            if (cbrng::u01d_fold(g) < p) {
                (void)cbrng::u01d_fold(g);
                ++draws;
                ch_state[st.ch_off + c] = 1 - state;
            }
        }
        double tot[CB_MAX_IONS];
        for (int j = 0; j < m.n_ions; ++j) tot[j] = 0;
        for (int c = 0; c < st.n_ch; ++c) {
            const int state = ch_state[st.ch_off + c];
            const double* mo = mouth + (long long)(st.ch_off + c) * NS;
            for (int j = 0; j < m.n_ions; ++j) tot[j] += state * (m.g[j] * (q.jsr_new[j] - mo[j]));
        }
        for (int j = 0; j < m.n_ions; ++j) q.total[j] = tot[j];
        if (!m.jsr_const)
            for (int i = 0; i < m.n_ions; ++i) {
                q.IjSR[i] = q.total[i] * m.V_elem;
                q.nsr[i] = m.nsr[i];
                q.jsr[i] = q.jsr_new[i];
            }
    }
    q.draws += draws;
    for (int i = 0; i < 6; ++i) q.rng[i] = g.s[i];
}

template <typename R>
cudaError_t reset_impl(cb_dev& d, cudaStream_t st) {
    dim3 g(std::max(1, std::min(64, (d.max_nodes + 255) / 256)), d.S);
    k_reset<R><<<g, 256, 0, st>>>(d.m, d.sites, (R*)d.fields[0], (R*)d.fields[1], (R*)d.curgrid, d.sc, d.ch_state, d.err_flag);
    d.cur = 0;
    if (d.m.cyto_type == CB_CYTO_RD3D) {
        dim3 gc((d.nc + 255) / 256, d.S);
        k_cyto_reset<R><<<gc, 256, 0, st>>>(d.m, d.nc, (R*)d.cyto[0], (R*)d.cyto[1], d.cin);
        d.ccur = 0;
    }
    return cudaGetLastError();
}

}  // namespace

cudaError_t cb_plain_reset(cb_dev& d, cudaStream_t st) {
    return d.precision == 0 ? reset_impl<double>(d, st) : reset_impl<float>(d, st);
}

cudaError_t cb_plain_init_opening(cb_dev& d, const int* d_first, int lo, int hi, cudaStream_t st) {
    int n = hi - lo;
    if (n <= 0) return cudaSuccess;
    k_init_open<<<(n + 127) / 128, 128, 0, st>>>(d.sites, d_first, lo, hi, d.sc, d.ch_state, d.ch_micro, d.mwc);
    return cudaGetLastError();
}

cudaError_t cb_plain_update(cb_dev& d, cudaStream_t st, long long* launches) {
    if (launches) *launches += 1;
    return d.precision == 0 ? launch_update<double>(d, st) : launch_update<float>(d, st);
}

bool cb_plain_streaming(cb_dev& d) { return stream_tiles(d) > 0; }

bool cb_plain_gating_ready(cb_dev& d) { return stream_tiles(d) > 0 && !d.mwc; }

cudaError_t cb_plain_step_marked(cb_dev& d, cudaStream_t st, cudaEvent_t* ev) {
    return d.precision == 0 ? launch_step<double>(d, st, true, true, ev) : launch_step<float>(d, st, true, true, ev);
}

cudaError_t cb_plain_step(cb_dev& d, long long n, cudaStream_t st, long long* launches) {
    const bool fast = stream_tiles(d) > 0;
    const int per = (fast ? 2 : 3) + (d.m.cyto_type == CB_CYTO_RD3D ? 1 : 0);
    for (long long i = 0; i < n; ++i) {
        const bool first = i == 0, last = i == n - 1;
        cudaError_t e = d.precision == 0 ? launch_step<double>(d, st, first, last) : launch_step<float>(d, st, first, last);
        if (e != cudaSuccess) return e;
        if (launches) *launches += per + (fast && first ? 1 : 0);
    }
    return cudaSuccess;
}

namespace {
__global__ void k_gather_mouth(long long n, int NS, int species, const double* __restrict__ mouth, double* __restrict__ out) {
    const long long c = blockIdx.x * (long long)blockDim.x + threadIdx.x;
    if (c < n) out[c] = mouth[c * NS + species];
}
}  // namespace

cudaError_t cb_gather_mouth(const cb_dev& d, int species, double* out, cudaStream_t st) {
    k_gather_mouth<<<(unsigned)((d.total_ch + 255) / 256), 256, 0, st>>>(d.total_ch, d.NS, species, d.mouth, out);
    return cudaGetLastError();
}

cudaError_t cb_sg_features(cb_dev& d, int max_ch, int ld, float* X, cudaStream_t st) {
    k_sg_features<<<(unsigned)(((long long)d.S * ld + 255) / 256), 256, 0, st>>>(d.S, d.m.n_buf, max_ch, ld, d.sites, d.ch_node, d.ch_state, d.sc, X);
    return cudaGetLastError();
}

cudaError_t cb_sg_mouth(cb_dev& d, const float* Y, int ld, double ca_ref, cudaStream_t st) {
    const int slots = std::max(1, std::min(d.max_ch, ld));
    k_sg_mouth<<<(unsigned)(((long long)d.S * slots + 255) / 256), 256, 0, st>>>(d.S, d.NS, d.m.ca_idx, ca_ref, ld, d.sites, Y, d.mouth, slots);
    return cudaGetLastError();
}

namespace {
// per site: the largest relative error of the network's mouth Ca over its open RyRs (the
// mouths whose Ca sets the release flux; a site with none open has error 0); the max over
// sites (non-negative doubles order as their bit patterns) and the failing sites
__global__ void k_sg_residual(int S, int NS, int ca_idx, double ca_ref, int ld, double tol, const cb_site* __restrict__ sites,
                              const int* __restrict__ ch_state, const float* __restrict__ Y, const double* __restrict__ mouth,
                              unsigned long long* __restrict__ out) {
    const int s = blockIdx.x * blockDim.x + threadIdx.x;
    if (s >= S) return;
    const cb_site st = sites[s];
    double e = 0;
    for (int c = 0; c < st.n_ch && c < ld; ++c) {
        if (!ch_state[st.ch_off + c]) continue;
        const double rd = mouth[(size_t)(st.ch_off + c) * NS + ca_idx];
        const double pr = ca_ref * exp10((double)Y[(size_t)s * ld + c]);
        const double r = fabs(pr - rd) / fabs(rd);
        e = r > e ? r : (r != r ? INFINITY : e);
    }
    atomicMax(out, (unsigned long long)__double_as_longlong(e));
    if (!(e <= tol)) atomicAdd(out + 1, 1ULL);
}
}  // namespace

cudaError_t cb_sg_residual(const cb_dev& d, const float* Y, int ld, double ca_ref, double tol, unsigned long long* scratch,
                           double* worst, double* fail_fraction, cudaStream_t st) {
    cudaError_t e = cudaMemsetAsync(scratch, 0, 2 * sizeof(unsigned long long), st);
    if (e != cudaSuccess) return e;
    k_sg_residual<<<(d.S + 127) / 128, 128, 0, st>>>(d.S, d.NS, d.m.ca_idx, ca_ref, ld, tol, d.sites, d.ch_state, Y, d.mouth, scratch);
    if ((e = cudaGetLastError()) != cudaSuccess) return e;
    unsigned long long h[2];
    if ((e = cudaMemcpyAsync(h, scratch, sizeof(h), cudaMemcpyDeviceToHost, st)) != cudaSuccess) return e;
    if ((e = cudaStreamSynchronize(st)) != cudaSuccess) return e;
    double w;
    std::memcpy(&w, &h[0], sizeof(w));
    *worst = w;
    *fail_fraction = d.S ? (double)h[1] / d.S : 0.0;
    return cudaSuccess;
}

cudaError_t cb_sg_steps(cb_dev& d, long long n, cudaStream_t st) {
    bool used = false;
    cudaError_t e = cb_sg_steps_warp(d, n, st, &used);
    if (e != cudaSuccess || used) return e;
    k_sg_steps<<<(d.S + 127) / 128, 128, 0, st>>>(d.m, d.S, d.NS, n, d.sites, d.sc, d.ch_state, d.mouth, d.spx[0], d.spc[0],
                                                  d.spx[1], d.spc[1]);
    return cudaGetLastError();
}
