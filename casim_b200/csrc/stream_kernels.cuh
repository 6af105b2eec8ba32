// Streaming stencils of the plain path, specialised per species layout.
//
// The plain path keeps every field in HBM and sweeps it once per time step. With a thread
// per node the stencils were bound by instruction issue, not by HBM: 162 thread
// instructions per cleft node, 6.4 ns per 1000 nodes whether the batch fitted L2 or not
// (HBM at its measured copy rate: 3.7). So a thread takes V adjacent nodes of a row (the
// stored rows are padded to whole groups of V) and loads and stores them as one word, the
// x neighbours inside the group come from its registers, the species counts are fixed at
// compile time, and every product of model constants is formed once on the host and read
// as a kernel-parameter operand. Each thread holds a column of groups (the cleft's z layers,
// the cytosol's planes), so the z neighbours are its own. Work is listed per block (site,
// first group) so that sites of uneven size leave no idle blocks. The node update is the
// reference's (CaSim/DyadRD2DCPU.cpp:394-490, CaSim/DyadRDCPU.cpp:404-506), as in the generic
// kernels k_rd and k_cyto, which stay in use for layouts these do not cover; FP32 fields
// divide with the approximate reciprocal in the sarcolemmal buffer factor and the SERCA
// term, as the resident path.
#pragma once

namespace stream {

// FP32: the approximate reciprocal (2 ulp), as the resident path; FP64: IEEE division
__device__ __forceinline__ float sdiv(float a, float b) { return __fdividef(a, b); }
__device__ __forceinline__ double sdiv(double a, double b) { return a / b; }

// V adjacent nodes as one word
template <typename R, int V>
struct word_of;
template <>
struct word_of<float, 1> { typedef float T; };
template <>
struct word_of<float, 2> { typedef float2 T; };
template <>
struct word_of<float, 4> { typedef float4 T; };
template <>
struct word_of<double, 1> { typedef double T; };
template <>
struct word_of<double, 2> { typedef double2 T; };

template <typename R, int V>
struct group {
    R v[V];
};
template <int V, typename R>
__device__ __forceinline__ group<R, V> load_group(const R* p) {
    typedef typename word_of<R, V>::T W;
    const W w = *(const W*)p;
    return *(const group<R, V>*)&w;
}
// outputs are read back only in the next time step, after the whole state has passed
// through L2: cache-streaming stores leave L2 to the rows neighbouring blocks read
template <int V, typename R>
__device__ __forceinline__ void store_group(R* p, const group<R, V>& g) {
    typedef typename word_of<R, V>::T W;
    __stcs((W*)p, *(const W*)&g);
}

// a model constant, twice: a packed operand of two nodes
template <typename R>
struct pair_of {
    R v[2];
};
template <typename R>
__host__ __device__ __forceinline__ pair_of<R> both(R x) {
    return {{x, x}};
}

// Arithmetic on groups. FP32 groups run two nodes per instruction (fma/add/mul.rn.f32x2, each
// result rounded as the scalar one): the stencils are bound by issue slots and latency once
// their reads are asynchronous.
template <int V>
__device__ __forceinline__ group<float, V> gfma(const group<float, V>& a, const group<float, V>& b, const group<float, V>& c) {
    group<float, V> r;
#pragma unroll
    for (int e = 0; e < V; e += 2) {
        const float2 t = __ffma2_rn(make_float2(a.v[e], a.v[e + 1]), make_float2(b.v[e], b.v[e + 1]), make_float2(c.v[e], c.v[e + 1]));
        r.v[e] = t.x;
        r.v[e + 1] = t.y;
    }
    return r;
}
template <int V>
__device__ __forceinline__ group<double, V> gfma(const group<double, V>& a, const group<double, V>& b, const group<double, V>& c) {
    group<double, V> r;
#pragma unroll
    for (int e = 0; e < V; ++e) r.v[e] = fma(a.v[e], b.v[e], c.v[e]);
    return r;
}
template <int V>
__device__ __forceinline__ group<float, V> gadd(const group<float, V>& a, const group<float, V>& b) {
    group<float, V> r;
#pragma unroll
    for (int e = 0; e < V; e += 2) {
        const float2 t = __fadd2_rn(make_float2(a.v[e], a.v[e + 1]), make_float2(b.v[e], b.v[e + 1]));
        r.v[e] = t.x;
        r.v[e + 1] = t.y;
    }
    return r;
}
template <int V>
__device__ __forceinline__ group<double, V> gadd(const group<double, V>& a, const group<double, V>& b) {
    group<double, V> r;
#pragma unroll
    for (int e = 0; e < V; ++e) r.v[e] = a.v[e] + b.v[e];
    return r;
}
template <int V>
__device__ __forceinline__ group<float, V> gmul(const group<float, V>& a, const group<float, V>& b) {
    group<float, V> r;
#pragma unroll
    for (int e = 0; e < V; e += 2) {
        const float2 t = __fmul2_rn(make_float2(a.v[e], a.v[e + 1]), make_float2(b.v[e], b.v[e + 1]));
        r.v[e] = t.x;
        r.v[e + 1] = t.y;
    }
    return r;
}
template <int V>
__device__ __forceinline__ group<double, V> gmul(const group<double, V>& a, const group<double, V>& b) {
    group<double, V> r;
#pragma unroll
    for (int e = 0; e < V; ++e) r.v[e] = a.v[e] * b.v[e];
    return r;
}
template <int V, typename R>
__device__ __forceinline__ group<R, V> gall(const pair_of<R>& k) {
    group<R, V> r;
#pragma unroll
    for (int e = 0; e < V; ++e) r.v[e] = k.v[e & 1];
    return r;
}
template <int V, typename R>
__device__ __forceinline__ group<R, V> gall(R k) {
    group<R, V> r;
#pragma unroll
    for (int e = 0; e < V; ++e) r.v[e] = k;
    return r;
}
// (p - 2 c) + q: second difference of c between its neighbours p and q
template <typename R, int V>
__device__ __forceinline__ group<R, V> diff2(const group<R, V>& p, const group<R, V>& c, const group<R, V>& q) {
    return gadd(gfma(c, gall<V>((R)-2), p), q);
}
// the same along x, left and right: the nodes beside the group
template <typename R, int V>
__device__ __forceinline__ group<R, V> diff2x(R left, const group<R, V>& c, R right) {
    group<R, V> r;
#pragma unroll
    for (int e = 0; e < V; ++e)
        r.v[e] = fma((R)-2, c.v[e], e == V - 1 ? right : c.v[e < V - 1 ? e + 1 : 0]) + (e == 0 ? left : c.v[e > 0 ? e - 1 : 0]);
    return r;
}

constexpr int MAX_F = 6;  // species of the specialised layouts: 2 ions, 4 pairs

// Constants of the cleft stencil in the field precision, each rounded once from the
// double-precision product noted.
template <typename R>
struct rd_const {
    pair_of<R> ax[MAX_F], ay[MAX_F], az[MAX_F];  // D dt / h^2 per direction
    int diff[MAX_F];                    // D != 0
    pair_of<R> mkon[4], koff[4];        // -kon dt, koff dt
    pair_of<R> ctot[4];                 // total of the pair's buffer
    unsigned same[4];                   // bit q: pair q binds pair p's buffer
    int pion[4];
    pair_of<R> dt;
    int has_sl[2];
    R K1[2], K2[2], A1[2], A2[2];       // sarcolemma: N1 K1, N2 K2
    int src[MAX_F];                     // rim: cytosol species (RD3D), or -1 for init
    R init[MAX_F];
    int CS, nc;                         // RD3D cytosol: species and stored nodes per site
};

constexpr int RD_THREADS = 256;                                     // k_rd_v
constexpr int rd_vec(int w) { return w == 4 ? CB_CLEFT_VEC : 2; }  // nodes per thread and layer
// computing threads of k_rd_t and its blocks per SM. 4096 uneven sites of 40 to 120 nodes a
// side, F = 3, GB/s of algorithmic bytes: FP32 128 threads 5550, 160 5380, 192 5270; FP64 256
// threads 5710, 192 5020. Fewer, smaller blocks drift apart more, so that some compute while
// others wait; below that the halo rows weigh.
__host__ __device__ constexpr int rdt_threads(int w) { return w == 4 ? 128 : 256; }
constexpr int RDT_STAGES = 2;
__host__ __device__ constexpr int rdt_blocks(int w, int F, int NZ) { return w == 4 ? (F * NZ <= 9 ? 4 : F * NZ <= 12 ? 3 : 2) : (F * NZ <= 9 ? 2 : 1); }
// blocks of k_rd_v per SM asked of the compiler, for the registers a column of groups takes
constexpr int rd_min_blocks(int w, int F, int NZ, int V) {
    const int words = F * NZ * V * w / 4;  // registers of the column itself
    return words <= 18 ? 5 : words <= 24 ? 4 : words <= 36 ? 3 : words <= 54 ? 2 : 1;
}

// The part of a node's rate of change (times dt, evo) that needs no neighbour, layer z: binding,
// RyR currents (layer 0), the sarcolemmal buffer factor.
template <typename R, int NI, int NP, int NZ, int V>
__device__ __forceinline__ void node_reactions(const rd_const<R>& k, const group<R, V> (&c)[NI + NP][NZ], int z, const group<R, V> (&cur)[NI],
                                               group<R, V> (&evo)[NI + NP]) {
    // binding: R1 = koff B - kon ion free, free = the buffer's total less every pair bound to it,
    // in pair order
#pragma unroll
    for (int p = 0; p < NP; ++p) {
        group<R, V> fr = gall<V>(k.ctot[p]), ion = c[0][z];
        if (NI == 1) {
            fr = gfma(c[NI + p][z], gall<V>((R)-1), fr);  // one ion: every buffer has one pair
        } else {
#pragma unroll
            for (int q = 0; q < NP; ++q)
                if (k.same[p] >> q & 1u) fr = gfma(c[NI + q][z], gall<V>((R)-1), fr);
#pragma unroll
            for (int i = 1; i < NI; ++i)
                if (k.pion[p] == i) ion = c[i][z];
        }
        const group<R, V> r1 = gfma(gmul(ion, gall<V>(k.mkon[p])), fr, gmul(c[NI + p][z], gall<V>(k.koff[p])));
        evo[NI + p] = gfma(r1, gall<V>((R)-1), evo[NI + p]);
#pragma unroll
        for (int i = 0; i < NI; ++i)
            if (NI == 1 || k.pion[p] == i) evo[i] = gadd(evo[i], r1);
    }
#pragma unroll
    for (int j = 0; j < NI; ++j) {
        if (z == 0) evo[j] = gfma(cur[j], gall<V>(k.dt), evo[j]);
        if ((NZ == 1 || z == NZ - 1) && k.has_sl[j]) {
#pragma unroll
            for (int e = 0; e < V; ++e) {
                const R s1 = k.K1[j] + c[j][z].v[e], s2 = k.K2[j] + c[j][z].v[e];
                evo[j].v[e] *= sdiv((R)1, (R)1 + sdiv(k.A1[j], s1 * s1) + sdiv(k.A2[j], s2 * s2));
            }
        }
    }
}

// Cleft step of the groups [tile.y, tile.y + 256) of site tile.x (tile.z, tile.w: the
// division by the row pitch). The rim takes the Dirichlet values that the Update would set
// right after this step (CaSim/DyadRD2DCPU.cpp:274-303), from the same sources: the cytosol as
// it was before its latest step (cyto, RD3D) or the pool values of this step (sc); the Update
// then leaves the rim alone (k_update_s with prev set).
template <typename R, int NI, int NP, int NZ, int V>
__global__ void __launch_bounds__(RD_THREADS, rd_min_blocks(sizeof(R), NI + NP, NZ, V))
    k_rd_v(const __grid_constant__ rd_const<R> k, const cb_site* __restrict__ sites, const int4* __restrict__ tiles,
           const R* __restrict__ in, R* __restrict__ out, const R* __restrict__ curg, const cb_site_scalars* __restrict__ sc,
           const R* __restrict__ cyto, const int* __restrict__ rim_cnode, const unsigned* __restrict__ chcol) {
    constexpr int F = NI + NP;
    const int4 tl = tiles[blockIdx.x];
    const cb_site st = sites[tl.x];
    const int nx = st.nx, ny = st.ny, px = st.px, pxy = px * ny, np = st.npad;
    const int col = (tl.y + (int)threadIdx.x) * V;
    if (col >= pxy) return;
    const R* __restrict__ u = in + st.node_base * F + col;
    R* __restrict__ o = out + st.node_base * F + col;
    const int y = (int)((__umulhi((unsigned)col, (unsigned)tl.z) + (unsigned)col) >> tl.w), x = col - y * px;
    auto rim_values = [&](int ri, R(&b)[F]) {
        if (cyto) {
            const R* cy = cyto + (long long)tl.x * k.CS * k.nc + rim_cnode[st.rim_off + ri];
#pragma unroll
            for (int f = 0; f < F; ++f) b[f] = k.src[f] >= 0 ? cy[k.src[f] * k.nc] : k.init[f];
        } else {
            const cb_site_scalars& q = sc[tl.x];
#pragma unroll
            for (int f = 0; f < F; ++f) b[f] = (R)(f < NI ? q.c_ions[f < NI ? f : 0] : q.c_bnd[f < NI ? 0 : f - NI]);
        }
    };
    if (y == 0 || y == ny - 1) {
#pragma unroll
        for (int e = 0; e < V; ++e) {
            R b[F];
            rim_values(cb_rim_index(min(x + e, nx - 1), y, nx, ny), b);
#pragma unroll
            for (int f = 0; f < F; ++f)
#pragma unroll
                for (int z = 0; z < NZ; ++z) o[f * np + z * pxy + e] = b[f];
        }
        return;
    }
    group<R, V> c[F][NZ];
#pragma unroll
    for (int f = 0; f < F; ++f)
#pragma unroll
        for (int z = 0; z < NZ; ++z) c[f][z] = load_group<V>(u + f * np + z * pxy);
    // the first and the last group of a row hold one rim node each (and the padding): their
    // values are loaded first and put in last
    const bool edge = x == 0 || x + V >= nx;
    R b[F];
    if (edge) rim_values(x == 0 ? y : ny + y, b);
    // RyR currents exist only in the columns that hold a RyR (bits of the site's words in
    // chcol), in layer 0; elsewhere the current grid is zero and is not read
    const long long bit = st.node_base + col;
    const bool has_ch = (chcol[bit >> 5] >> (bit & 31)) & ((1u << V) - 1u);
    const R* cg = curg + st.node_base * NI + col;
    group<R, V> cur[NI];
#pragma unroll
    for (int j = 0; j < NI; ++j) {
        if (has_ch) cur[j] = load_group<V>(cg + j * np);
#pragma unroll
        for (int e = 0; e < V; ++e) cur[j].v[e] = has_ch ? cur[j].v[e] : (R)0;
    }
#pragma unroll
    for (int z = 0; z < NZ; ++z) {
        // reflecting z boundaries: z = 0 and z = nz-1 see their inner neighbour twice
        const int zl = z == 0 ? (NZ > 1 ? 1 : 0) : z - 1;
        const int zr = z == NZ - 1 ? (NZ > 1 ? NZ - 2 : 0) : z + 1;
        group<R, V> evo[F];
#pragma unroll
        for (int f = 0; f < F; ++f) {
            const group<R, V>& cc = c[f][z];
            if (k.diff[f]) {
                const R* v = u + f * np + z * pxy;
                const group<R, V> dn = load_group<V>(v - px), up = load_group<V>(v + px);
                const R left = v[-1], right = v[V];
                evo[f] = gfma(diff2(up, cc, dn), gall<V>(k.ay[f]), gmul(diff2x(left, cc, right), gall<V>(k.ax[f])));
                if (NZ > 1) evo[f] = gfma(diff2(c[f][zr], cc, c[f][zl]), gall<V>(k.az[f]), evo[f]);
            } else {
                evo[f] = gall<V>((R)0);
            }
        }
        node_reactions<R, NI, NP, NZ, V>(k, c, z, cur, evo);
#pragma unroll
        for (int f = 0; f < F; ++f) {
            group<R, V> w = gadd(c[f][z], evo[f]);
#pragma unroll
            for (int e = 0; e < V; ++e)
                if (edge && (x + e == 0 || x + e >= nx - 1)) w.v[e] = b[f];
            store_group(o + f * np + z * pxy, w);
        }
    }
}

// ---- bulk copies and their barriers (one block only; every wait is bounded)
__device__ __forceinline__ uint32_t smem_addr(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }
__device__ __forceinline__ void bar_init(uint64_t* b, int count) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_addr(b)), "r"(count) : "memory");
}
__device__ __forceinline__ void bar_arrive(uint64_t* b) {
    asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_addr(b)) : "memory");
}
__device__ __forceinline__ void bar_expect(uint64_t* b, uint32_t bytes) {
    asm volatile("mbarrier.expect_tx.relaxed.cta.shared::cta.b64 [%0], %1;" ::"r"(smem_addr(b)), "r"(bytes) : "memory");
}
// false when the phase did not complete within the bound (far above any copy's time)
__device__ __forceinline__ bool bar_wait(uint64_t* b, uint32_t parity) {
    const uint32_t a = smem_addr(b);
    for (int i = 0; i < (1 << 17); ++i) {
        uint32_t ok;
        asm volatile(
            "{\n\t.reg .pred p;\n\tmbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
            "selp.u32 %0, 1, 0, p;\n\t}\n"
            : "=r"(ok)
            : "r"(a), "r"(parity)
            : "memory");
        if (ok) return true;
    }
    return false;
}
// bytes: a multiple of 16; both addresses 16-byte aligned
__device__ __forceinline__ void bulk_load(void* dst, const void* src, uint32_t bytes, uint64_t* b) {
    asm volatile("cp.async.bulk.shared::cta.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(smem_addr(dst)), "l"(src),
                 "r"(bytes), "r"(smem_addr(b))
                 : "memory");
}

// A tile of the cleft: a group per computing thread of site `site` from stored node `col0` on.
struct __align__(16) rd_tile {
    long long node_base;
    int site, col0, np, px, nx, ny, rim_off;
    unsigned mul, sh;  // division by px: (umulhi(n, mul) + n) >> sh
    int pad[3];
};

// Shared-memory carve of one stage of k_rd_t (bytes), from the species and the widest row.
struct rd_stage {
    int bits, rim, plane[MAX_F], bytes;  // offsets after the tile; plane[f]: its first layer
    int stride[MAX_F];                   // bytes between a species' layers
    int halo;                            // nodes kept on each side of a diffusing species' tile
};

// The same step by persistent blocks that read through shared memory: a producer warp
// keeps STAGES tiles in flight ahead of the computing warps, each tile one bulk copy
// per species and layer (a flattened run of nodes, with a row and a group on each side
// where the species diffuses), its RyR bits and the rim values of its rows. Reading the
// neighbours from global memory, the kernel waited for the chain tile -> site -> fields ->
// rim and fetched rows from L2 once per block that touches them: 6.2 to 6.5 ns per 1000
// nodes whatever the group width or occupancy.
template <typename R, int NI, int NP, int NZ, int V, int STAGES>
__global__ void __launch_bounds__(rdt_threads(sizeof(R)) + 32, rdt_blocks(sizeof(R), NI + NP, NZ))
    k_rd_t(const __grid_constant__ rd_const<R> k, const __grid_constant__ rd_stage g, const rd_tile* __restrict__ tiles, int ntiles,
           const R* __restrict__ in, R* __restrict__ out, const R* __restrict__ curg, const cb_site_scalars* __restrict__ sc,
           const R* __restrict__ cyto, const int* __restrict__ rim_cnode, const unsigned* __restrict__ chcol, int* __restrict__ err) {
    constexpr int F = NI + NP, THREADS = rdt_threads(sizeof(R)), TN = THREADS * V, EXT = 16 / (int)sizeof(R);
    extern __shared__ __align__(128) unsigned char rd_smem[];
    __shared__ __align__(8) uint64_t full[STAGES], empty[STAGES];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    if (threadIdx.x == 0) {
#pragma unroll
        for (int i = 0; i < STAGES; ++i) {
            bar_init(&full[i], 1);
            bar_init(&empty[i], THREADS / 32);
        }
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    __syncthreads();
    if (warp == THREADS / 32) {
        // ---- producer
        rd_tile nt;
        if ((int)blockIdx.x < ntiles) nt = tiles[blockIdx.x];
        int it = 0;
        bool ok = true;
        for (int t = blockIdx.x; t < ntiles; t += gridDim.x, ++it) {
            const rd_tile tl = nt;
            if (t + (int)gridDim.x < ntiles) nt = tiles[t + gridDim.x];
            const int s = it % STAGES;
            unsigned char* st = rd_smem + (size_t)s * g.bytes;
            if (it >= STAGES && !(ok = bar_wait(&empty[s], (uint32_t)((it / STAGES - 1) & 1)))) break;
            const int pxy = tl.px * tl.ny;
            const int n = min(TN, pxy - tl.col0);
            if (lane == 0) {
                // a diffusing species' run: a row and 16 bytes more on each side, inside the layer
                const int lo = max(tl.col0 - tl.px - EXT, 0), hi = min(tl.col0 + n + tl.px + EXT, pxy);
                const long long b0 = tl.node_base * F;
                uint32_t bytes = TN / 8;
#pragma unroll
                for (int f = 0; f < F; ++f) bytes += NZ * (uint32_t)sizeof(R) * (uint32_t)(k.diff[f] ? hi - lo : n);
                bar_expect(&full[s], bytes);
#pragma unroll
                for (int f = 0; f < F; ++f) {
                    const int from = k.diff[f] ? lo : tl.col0, len = k.diff[f] ? hi - lo : n;
                    const int at = k.diff[f] ? g.halo - (tl.col0 - lo) : 0;
#pragma unroll
                    for (int z = 0; z < NZ; ++z)
                        bulk_load(st + g.plane[f] + z * g.stride[f] + at * (int)sizeof(R),
                                  in + b0 + (long long)f * tl.np + z * pxy + from, (uint32_t)(len * sizeof(R)), &full[s]);
                }
                bulk_load(st + g.bits, chcol + ((tl.node_base + tl.col0) >> 5), TN / 8, &full[s]);
                *(rd_tile*)st = tl;
            }
            // Dirichlet values: the first and last node of each row of the tile, [row][side][F],
            // and, after them, the whole first and last row of the site where the tile meets them
            R* rv = (R*)(st + g.rim);
            const int y0 = (int)((__umulhi((unsigned)tl.col0, tl.mul) + (unsigned)tl.col0) >> tl.sh);
            const int ce = tl.col0 + n - 1;
            const int y1 = (int)((__umulhi((unsigned)ce, tl.mul) + (unsigned)ce) >> tl.sh);
            const int side = 2 * (y1 - y0 + 1), top = y0 == 0 ? tl.nx : 0, bot = y1 == tl.ny - 1 ? tl.nx : 0;
            for (int i = lane; i < side + top + bot; i += 32) {
                int ri;
                if (i < side) ri = (i & 1 ? tl.ny : 0) + y0 + (i >> 1);
                else if (i < side + top) ri = cb_rim_index(i - side, 0, tl.nx, tl.ny);
                else ri = cb_rim_index(i - side - top, tl.ny - 1, tl.nx, tl.ny);
                if (cyto) {
                    const R* cy = cyto + (long long)tl.site * k.CS * k.nc + rim_cnode[tl.rim_off + ri];
#pragma unroll
                    for (int f = 0; f < F; ++f) rv[i * F + f] = k.src[f] >= 0 ? cy[k.src[f] * k.nc] : k.init[f];
                } else {
                    const cb_site_scalars& q = sc[tl.site];
#pragma unroll
                    for (int f = 0; f < F; ++f) rv[i * F + f] = (R)(f < NI ? q.c_ions[f < NI ? f : 0] : q.c_bnd[f < NI ? 0 : f - NI]);
                }
            }
            __syncwarp();
            if (lane == 0) bar_arrive(&full[s]);
        }
        if (!ok) {  // the consumers gave up: let the copies in flight land before the block ends
            if (lane == 0) *err = 1;
            for (int i = max(it - STAGES, 0); i < it; ++i) bar_wait(&full[i % STAGES], (uint32_t)((i / STAGES) & 1));
        }
        return;
    }
    // ---- consumers
    int it = 0;
    for (int t = blockIdx.x; t < ntiles; t += gridDim.x, ++it) {
        const int s = it % STAGES;
        if (!bar_wait(&full[s], (uint32_t)((it / STAGES) & 1))) {
            if (lane == 0) *err = 1;
            break;
        }
        const unsigned char* stg = rd_smem + (size_t)s * g.bytes;
        const rd_tile& tl = *(const rd_tile*)stg;
        const int nx = tl.nx, ny = tl.ny, px = tl.px, pxy = px * ny, np = tl.np, col0 = tl.col0;
        const int gi = (int)threadIdx.x * V, col = col0 + gi;
        if (col < pxy) {
            const long long b0 = tl.node_base;
            R* __restrict__ o = out + b0 * F + col;
            const int y = (int)((__umulhi((unsigned)col, tl.mul) + (unsigned)col) >> tl.sh), x = col - y * px;
            const int y0 = (int)((__umulhi((unsigned)col0, tl.mul) + (unsigned)col0) >> tl.sh);
            const R* rv = (const R*)(stg + g.rim);
            if (y == 0 || y == ny - 1) {
                const int ce = min(col0 + TN, pxy) - 1;
                const int y1 = (int)((__umulhi((unsigned)ce, tl.mul) + (unsigned)ce) >> tl.sh);
                const R* row = rv + (2 * (y1 - y0 + 1) + (y == 0 || y0 > 0 ? 0 : nx)) * F;
#pragma unroll
                for (int f = 0; f < F; ++f) {
                    group<R, V> w;
#pragma unroll
                    for (int e = 0; e < V; ++e) w.v[e] = row[min(x + e, nx - 1) * F + f];
#pragma unroll
                    for (int z = 0; z < NZ; ++z) store_group(o + f * np + z * pxy, w);
                }
            } else {
                const bool has_ch = (((const unsigned*)(stg + g.bits))[gi >> 5] >> (gi & 31)) & ((1u << V) - 1u);
                group<R, V> cur[NI];
                const R* cg = curg + b0 * NI + col;
#pragma unroll
                for (int j = 0; j < NI; ++j) {
                    if (has_ch) cur[j] = load_group<V>(cg + j * np);
#pragma unroll
                    for (int e = 0; e < V; ++e) cur[j].v[e] = has_ch ? cur[j].v[e] : (R)0;
                }
                const bool edge = x == 0 || x + V >= nx;
                const R* er = rv + (2 * (y - y0) + (x == 0 ? 0 : 1)) * F;
                group<R, V> c[F][NZ];
#pragma unroll
                for (int f = 0; f < F; ++f) {
                    const unsigned char* pf = stg + g.plane[f] + (gi + (k.diff[f] ? g.halo : 0)) * (int)sizeof(R);
#pragma unroll
                    for (int z = 0; z < NZ; ++z) c[f][z] = load_group<V>((const R*)(pf + z * g.stride[f]));
                }
                // layer 0 last: its RyR currents come from global memory
#pragma unroll
                for (int zz = 0; zz < NZ; ++zz) {
                    const int z = NZ - 1 - zz;
                    const int zl = z == 0 ? (NZ > 1 ? 1 : 0) : z - 1;
                    const int zr = z == NZ - 1 ? (NZ > 1 ? NZ - 2 : 0) : z + 1;
                    group<R, V> evo[F];
#pragma unroll
                    for (int f = 0; f < F; ++f) {
                        const group<R, V>& cc = c[f][z];
                        if (k.diff[f]) {
                            const R* v = (const R*)(stg + g.plane[f] + z * g.stride[f]) + g.halo + gi;
                            const group<R, V> dn = load_group<V>(v - px), up = load_group<V>(v + px);
                            const R left = v[-1], right = v[V];
                            evo[f] = gfma(diff2(up, cc, dn), gall<V>(k.ay[f]), gmul(diff2x(left, cc, right), gall<V>(k.ax[f])));
                            if (NZ > 1) evo[f] = gfma(diff2(c[f][zr], cc, c[f][zl]), gall<V>(k.az[f]), evo[f]);
                        } else {
                            evo[f] = gall<V>((R)0);
                        }
                    }
                    node_reactions<R, NI, NP, NZ, V>(k, c, z, cur, evo);
#pragma unroll
                    for (int f = 0; f < F; ++f) {
                        group<R, V> w = gadd(c[f][z], evo[f]);
#pragma unroll
                        for (int e = 0; e < V; ++e)
                            if (edge && (x + e == 0 || x + e >= nx - 1)) w.v[e] = er[f];
                        store_group(o + f * np + z * pxy, w);
                    }
                }
            }
        }
        __syncwarp();
        if (lane == 0) bar_arrive(&empty[s]);
    }
}

// Constants of the RD3D cytosol stencil, as rd_const.
template <typename R>
struct cy_const {
    pair_of<R> a[MAX_F];         // D dt / h^2
    pair_of<R> mkon[4], koff[4], ctot[4];  // -kon dt, koff dt, total of the pair's buffer
    unsigned same[4];
    int pion[4];
    int serca[2];
    pair_of<R> mjmax[2], k2[2], mrest[2];  // -Jmax dt, Kup^2, less the uptake share at rest
    R dt;
    int mc, px, nplane, nc;      // nodes per edge, row pitch, stored nodes of a plane and of a species
};

// The part of a cytosol node's rate of change (times dt) that needs no neighbour: binding, SERCA.
template <typename R, int NI, int NCP, int V>
__device__ __forceinline__ void cyto_reactions(const cy_const<R>& k, const group<R, V> (&cu)[NI + NCP], group<R, V> (&evo)[NI + NCP]) {
#pragma unroll
    for (int j2 = 0; j2 < NI; ++j2) {
        const group<R, V>& ion = cu[j2];
#pragma unroll
        for (int p = 0; p < NCP; ++p) {
            if (NI > 1 && k.pion[p] != j2) continue;
            group<R, V> fr = gall<V>(k.ctot[p]);
            if (NI == 1) {
                fr = gfma(cu[NI + p], gall<V>((R)-1), fr);
            } else {
#pragma unroll
                for (int q = 0; q < NCP; ++q)
                    if (k.same[p] >> q & 1u) fr = gfma(cu[NI + q], gall<V>((R)-1), fr);
            }
            const group<R, V> r1 = gfma(gmul(ion, gall<V>(k.mkon[p])), fr, gmul(cu[NI + p], gall<V>(k.koff[p])));
            evo[NI + p] = gfma(r1, gall<V>((R)-1), evo[NI + p]);
            evo[j2] = gadd(evo[j2], r1);
        }
        if (k.serca[j2]) {
            const group<R, V> i2 = gmul(ion, ion), d = gadd(i2, gall<V>(k.k2[j2]));
            group<R, V> up;
#pragma unroll
            for (int e = 0; e < V; ++e) up.v[e] = sdiv(i2.v[e], d.v[e]);
            evo[j2] = gfma(gadd(up, gall<V>(k.mrest[j2])), gall<V>(k.mjmax[j2]), evo[j2]);
        }
    }
}

// blocks of k_cyto_t per SM asked of the compiler, and stages a block keeps in flight
constexpr int cyt_blocks(int w, int CS) { return w == 4 ? (CS <= 3 ? 3 : 2) : (CS <= 3 ? 2 : 1); }
constexpr int CYT_STAGES = 4;
constexpr int CY_THREADS = 352;  // 13 groups x 25 rows of the shipped grid in 11 warps
constexpr int cy_min_blocks(int w, int CS) { return w == 4 ? (CS <= 3 ? 3 : 2) : (CS <= 3 ? 2 : 1); }

// RD3D cytosol step on any grid: a thread per group of V nodes of a layer (blockIdx.y: groups
// [y * CY_THREADS, ..)), marching the mc - 1 updated planes (the top plane is the bath) with planes
// k-1 .. k+1 of its own nodes in registers and planes k+2, k+3 loaded ahead; plane 0 mirrors and
// takes the efflux deposits. The bath columns copy themselves so that every memory sector is
// written whole (a partly written sector is read back from memory when it leaves L2).
template <typename R, int NI, int NCP, int V>
__global__ void __launch_bounds__(CY_THREADS, cy_min_blocks(sizeof(R), NI + NCP))
    k_cyto_v(const __grid_constant__ cy_const<R> k, const R* __restrict__ in, R* __restrict__ out, const double* __restrict__ cin) {
    constexpr int CS = NI + NCP;
    const int mc = k.mc, px = k.px, npl = k.nplane, nc = k.nc;
    const int col = ((int)blockIdx.y * CY_THREADS + (int)threadIdx.x) * V;
    if (col >= npl) return;
    const int s = blockIdx.x, j = col / px, i = col - j * px;
    const bool bath = j == 0 || j == mc - 1;  // a whole row of the bath
    const bool edge = i == 0 || i + V >= mc;  // the row's first or last node among these
    const R* __restrict__ u = in + (long long)s * CS * nc + col;
    R* __restrict__ o = out + (long long)s * CS * nc + col;
    group<R, V> lo[CS], cu[CS], hi[CS], p2[CS], p3[CS];
#pragma unroll
    for (int c = 0; c < CS; ++c) {
        const R* v = u + c * nc;
        cu[c] = load_group<V>(v);
        hi[c] = load_group<V>(v + npl);
        p2[c] = load_group<V>(v + min(2, mc - 1) * npl);
        p3[c] = load_group<V>(v + min(3, mc - 1) * npl);
        lo[c] = hi[c];
    }
#pragma unroll 4
    for (int kp = 0; kp < mc - 1; ++kp) {
        const int n = kp * npl;
        if (bath) {
#pragma unroll
            for (int c = 0; c < CS; ++c) store_group(o + c * nc + n, cu[c]);
        } else {
            group<R, V> evo[CS];
#pragma unroll
            for (int c = 0; c < CS; ++c) {
                const R* v = u + c * nc + n;
                const group<R, V> dn = load_group<V>(v - px), up = load_group<V>(v + px);
                const R left = v[-1], right = v[V];
                evo[c] = gmul(gadd(gadd(diff2x(left, cu[c], right), diff2(up, cu[c], dn)), diff2(hi[c], cu[c], lo[c])), gall<V>(k.a[c]));
            }
            cyto_reactions<R, NI, NCP, V>(k, cu, evo);
            if (kp == 0) {
                const double* ci = cin + (long long)s * CS * mc * mc + i + mc * j;
#pragma unroll
                for (int c = 0; c < CS; ++c)
#pragma unroll
                    for (int e = 0; e < V; ++e) evo[c].v[e] = fma((R)ci[c * mc * mc + min(e, mc - 1 - i)], k.dt, evo[c].v[e]);
            }
#pragma unroll
            for (int c = 0; c < CS; ++c) {
                group<R, V> w = gadd(cu[c], evo[c]);
#pragma unroll
                for (int e = 0; e < V; ++e)
                    if (edge && (i + e == 0 || i + e >= mc - 1)) w.v[e] = cu[c].v[e];
                store_group(o + c * nc + n, w);
            }
        }
#pragma unroll
        for (int c = 0; c < CS; ++c) {
            lo[c] = cu[c];
            cu[c] = hi[c];
            hi[c] = p2[c];
            p2[c] = p3[c];
            if (kp + 4 < mc) p3[c] = load_group<V>(u + c * nc + n + 4 * npl);
        }
    }
}

// The same step on a grid of MC^3 nodes fixed at compile time (25, the shipped configs), the
// planes read through shared memory: a producer warp keeps STAGES stages of PS planes of every
// species in flight, each one bulk copy per species (PS planes are a multiple of 16 bytes), and
// the computing threads take the neighbours in the plane from there. One block per site and chunk
// of planes. 2048 sites, one ion and two buffers, FP32 / FP64: 148 / 259 us (5190 / 5920 GB/s of
// algorithmic bytes), a thread per column and neighbours through L1 173 / 305 us.
template <int w>
__host__ __device__ constexpr int cyt_planes() { return w == 4 ? 2 : 1; }
template <typename R, int NI, int NCP, int V, int MC, int STAGES>
__global__ void __launch_bounds__(CY_THREADS + 32, cyt_blocks(sizeof(R), NI + NCP))
    k_cyto_t(const __grid_constant__ cy_const<R> k, int chunk, const R* __restrict__ in, R* __restrict__ out,
             const double* __restrict__ cin, int* __restrict__ err) {
    constexpr int CS = NI + NCP, px = (MC + V - 1) / V * V, npl = MC * px, PS = cyt_planes<sizeof(R)>();
    constexpr int nc = (MC * npl + 3) / 4 * 4;  // stored nodes of a species
    constexpr uint32_t SPB = PS * npl * sizeof(R);  // bytes of a species in a stage
    extern __shared__ __align__(128) unsigned char rd_smem[];
    __shared__ __align__(8) uint64_t full[STAGES], empty[STAGES];
    R* const ring = (R*)rd_smem;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int s = blockIdx.x, k0 = blockIdx.y * chunk, k1 = min(k0 + chunk, MC - 1);
    const int kb = k0 == 0 ? 0 : (k0 - 1) / PS * PS;  // first plane loaded
    if (tid == 0) {
#pragma unroll
        for (int i = 0; i < STAGES; ++i) {
            bar_init(&full[i], 1);
            bar_init(&empty[i], CY_THREADS / 32);
        }
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    __syncthreads();
    const R* __restrict__ u = in + (long long)s * CS * nc;
    if (warp == CY_THREADS / 32) {
        if (lane == 0) {
            const int nq = (k1 - kb) / PS + 1;  // up to the stage of plane k1
            bool ok = true;
            int q = 0;
            for (; q < nq; ++q) {
                const int st = q % STAGES, kk = kb + q * PS;
                if (q >= STAGES && !(ok = bar_wait(&empty[st], (uint32_t)((q / STAGES - 1) & 1)))) break;
                // the last plane of the grid may be alone in its stage: whole 16 bytes, within nc
                const uint32_t bytes = (uint32_t)(min(PS * npl, nc - kk * npl) * (int)sizeof(R)) & ~15u;
                bar_expect(&full[st], CS * bytes);
#pragma unroll
                for (int c = 0; c < CS; ++c) bulk_load(ring + (size_t)(st * CS + c) * PS * npl, u + (size_t)c * nc + kk * npl, bytes, &full[st]);
                bar_arrive(&full[st]);
            }
            if (!ok) {  // the computing warps gave up: let the copies in flight land before the block ends
                *err = 1;
                for (int i = max(q - STAGES, 0); i < q; ++i) bar_wait(&full[i % STAGES], (uint32_t)((i / STAGES) & 1));
            }
        }
        return;
    }
    const int g = min(tid, npl / V - 1), col = g * V;  // surplus threads repeat the last group and store nothing
    const int j = col / px, i = col - j * px;
    const bool mine = tid < npl / V;
    const bool bath = j == 0 || j == MC - 1, edge = i == 0 || i + V >= MC;
    R* __restrict__ o = out + (long long)s * CS * nc + col;
    auto plane = [&](int kp, int c) { return ring + (size_t)((kp - kb) / PS % STAGES * CS + c) * PS * npl + (kp - kb) % PS * npl + col; };
    auto wait_full = [&](int kp) { return bar_wait(&full[(kp - kb) / PS % STAGES], (uint32_t)((kp - kb) / PS / STAGES & 1)); };
    auto done = [&](int kp) {  // plane kp was the last of its stage
        __syncwarp();
        if (lane == 0) bar_arrive(&empty[(kp - kb) / PS % STAGES]);
    };
    group<R, V> lo[CS], cu[CS], hi[CS];
    bool ok = true;
    if (k0 > 0) {
        ok = wait_full(k0 - 1);
#pragma unroll
        for (int c = 0; c < CS; ++c) lo[c] = load_group<V>(plane(k0 - 1, c));
        if ((k0 - kb) % PS == 0) done(k0 - 1);
    }
    ok = ok && wait_full(k0);
#pragma unroll
    for (int c = 0; c < CS; ++c) cu[c] = load_group<V>(plane(k0, c));
#pragma unroll PS
    for (int kp = k0; kp < k1; ++kp) {
        if ((kp + 1 - kb) % PS == 0) ok = ok && wait_full(kp + 1);
        if (!ok) break;
#pragma unroll
        for (int c = 0; c < CS; ++c) {
            hi[c] = load_group<V>(plane(kp + 1, c));
            if (kp == 0) lo[c] = hi[c];
        }
        const int n = kp * npl;
        if (bath) {
#pragma unroll
            for (int c = 0; c < CS; ++c)
                if (mine) store_group(o + c * nc + n, cu[c]);
        } else {
            group<R, V> evo[CS];
#pragma unroll
            for (int c = 0; c < CS; ++c) {
                const R* v = plane(kp, c);
                const group<R, V> dn = load_group<V>(v - px), up = load_group<V>(v + px);
                const R left = v[-1], right = v[V];
                evo[c] = gmul(gadd(gadd(diff2x(left, cu[c], right), diff2(up, cu[c], dn)), diff2(hi[c], cu[c], lo[c])), gall<V>(k.a[c]));
            }
            cyto_reactions<R, NI, NCP, V>(k, cu, evo);
            if (kp == 0) {
                const double* ci = cin + (long long)s * CS * MC * MC + i + MC * j;
#pragma unroll
                for (int c = 0; c < CS; ++c)
#pragma unroll
                    for (int e = 0; e < V; ++e) evo[c].v[e] = fma((R)ci[c * MC * MC + min(e, MC - 1 - i)], k.dt, evo[c].v[e]);
            }
#pragma unroll
            for (int c = 0; c < CS; ++c) {
                group<R, V> w = gadd(cu[c], evo[c]);
#pragma unroll
                for (int e = 0; e < V; ++e)
                    if (edge && (i + e == 0 || i + e >= MC - 1)) w.v[e] = cu[c].v[e];
                if (mine) store_group(o + c * nc + n, w);
            }
        }
        if ((kp + 1 - kb) % PS == 0) done(kp);
#pragma unroll
        for (int c = 0; c < CS; ++c) {
            lo[c] = cu[c];
            cu[c] = hi[c];
        }
    }
    if (!ok && lane == 0) *err = 1;
}

}  // namespace stream

namespace stream {

constexpr int UP_THREADS = 256;

// Sum of each of the K per-thread values over the block (UP_THREADS threads) in a fixed
// order: warp butterflies, then the warp partials in warp order; every thread gets the
// sums. red holds (UP_THREADS / 32) * K doubles.
template <int K>
__device__ __forceinline__ void block_sums(double (&v)[K], double* red) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1)
#pragma unroll
        for (int k = 0; k < K; ++k) v[k] += __shfl_xor_sync(0xffffffffu, v[k], o);
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    __syncthreads();  // red may still be read from its previous use
    if (lane == 0)
#pragma unroll
        for (int k = 0; k < K; ++k) red[warp * K + k] = v[k];
    __syncthreads();
#pragma unroll
    for (int k = 0; k < K; ++k) {
        double s = red[k];
#pragma unroll
        for (int w = 1; w < UP_THREADS / 32; ++w) s += red[w * K + k];
        v[k] = s;
    }
}

// The Update of one site per block (CaSim/ParallelHybridSolver.cpp:159-175): mouth
// values, Dirichlet rim from the cytosol, efflux through the rim, the RD3D deposits
// into cytosol layer 0, RyR currents and the jSR coupling; the steps, their order and
// the values they read are those of the generic k_update, the per-node quantities in
// registers and the block sums by warp shuffles.
template <typename R, int NI, int NP, bool RD3D>
__global__ void __launch_bounds__(UP_THREADS) k_update_s(const __grid_constant__ cb_model m, int NS, const cb_site* __restrict__ sites,
                                                         R* __restrict__ fld, R* __restrict__ curg, const int* __restrict__ ch_node,
                                                         const int* __restrict__ ch_owner, const int* __restrict__ ch_state,
                                                         double* __restrict__ mouth, cb_site_scalars* __restrict__ sc, int nc,
                                                         const R* __restrict__ cyto, double* __restrict__ cin,
                                                         const int* __restrict__ rim_cnode, const int* __restrict__ dep_ptr,
                                                         const int* __restrict__ dep_term, const R* __restrict__ prev, int max_terms) {
    constexpr int F = NI + NP;
    constexpr int CSM = NI + 4;  // cytosol species slots (ions + at most 4 pairs)
    const int CS = m.n_ions + m.c_n_pairs;
    extern __shared__ double smem[];
    double* red = smem;                   // (UP_THREADS / 32) * (F + NI)
    double* terms = smem + 8 * (F + NI);  // RD3D: [term][F] efflux values
    const int s = blockIdx.x;
    const cb_site st = sites[s];
    cb_site_scalars& q = sc[s];
    R* u = fld + st.node_base * F;
    const int nx = st.nx, ny = st.ny, nz = st.nz, px = st.px, nxy = px * ny;
    const long long np = st.npad;
    // RD3D: the site's deposit lists (per layer-0 cytosol node its efflux terms, in term
    // order) staged in shared memory behind the terms, loaded here so that the loads
    // overlap the phases before the deposit sums
    const int zmax0 = nz == 1 ? 1 : nz - 1;
    const int T0 = cb_efflux_terms(nx, ny, zmax0);
    int* s_ptr = (int*)(terms + (size_t)max_terms * F);
    int* s_term = s_ptr + (RD3D ? m.mc * m.mc + 1 : 0);
    if (RD3D) {
        const int mc2 = m.mc * m.mc;
        const int* ptr = dep_ptr + (long long)s * (mc2 + 1);
        for (int k = threadIdx.x; k <= mc2; k += UP_THREADS) s_ptr[k] = ptr[k];
        const int* dtm = dep_term + st.term_off;
        for (int k = threadIdx.x; k < T0; k += UP_THREADS) s_term[k] = dtm[k];
    }
    // 1. mouth values: ions, pairs, free buffers (CaSim/DyadRD2DCPU.cpp:361-380). After
    // k_rd_v (prev set) the rim holds its Dirichlet values already; a RyR on the rim
    // reads the value the step carried over there, which is prev's
    for (int c = threadIdx.x; c < st.n_ch; c += UP_THREADS) {
        const int node = ch_node[st.ch_off + c];
        double* mo = mouth + (long long)(st.ch_off + c) * NS;
        const R* src = u;
        if (prev) {
            const int cx = node % px, cyy = (node / px) % ny;
            if (cx == 0 || cx == nx - 1 || cyy == 0 || cyy == ny - 1) src = prev + st.node_base * F;
        }
        double v[F];
#pragma unroll
        for (int f = 0; f < F; ++f) v[f] = (double)src[f * np + node];
#pragma unroll
        for (int f = 0; f < F; ++f) mo[f] = v[f];
        for (int b = 0; b < m.n_buf; ++b) {
            double fr = m.Ctot[b];
#pragma unroll
            for (int p = 0; p < NP; ++p)
                if (m.pair_buf[p] == b) fr -= v[NI + p];
            mo[F + b] = fr;
        }
    }
    __syncthreads();
    // 2. Dirichlet edges from the cytosol (CaSim/DyadRD2DCPU.cpp:274-303), unless k_rd_v
    // set them (prev set)
    const int nrim = prev ? 0 : cb_rim_count(nx, ny);
    const R* cy = RD3D ? cyto + (long long)s * CS * nc : nullptr;
    for (int t = threadIdx.x; t < nrim * nz; t += UP_THREADS) {
        const int z = t / nrim, r = t - z * nrim;
        int x, y;
        cb_rim_xy(r, nx, ny, x, y);
        const int node = x + px * y + nxy * z;
        if (!RD3D) {
#pragma unroll
            for (int j = 0; j < NI; ++j) u[j * np + node] = (R)q.c_ions[j];
#pragma unroll
            for (int p = 0; p < NP; ++p) u[(NI + p) * np + node] = (R)q.c_bnd[p];
        } else {
            const int cn = rim_cnode[st.rim_off + r];
#pragma unroll
            for (int j = 0; j < NI; ++j) u[j * np + node] = cy[(long long)j * nc + cn];
#pragma unroll
            for (int p = 0; p < NP; ++p) {
                const int cq = m.dyad_c_pair[p];
                u[(NI + p) * np + node] = cq >= 0 ? cy[(long long)(NI + cq) * nc + cn] : (R)m.pair_init[p];
            }
        }
    }
    __syncthreads();
    // 3. efflux (CaSim/DyadRD2DCPU.cpp:305-350): per-term values, block sums
    const int zmax = nz == 1 ? 1 : nz - 1;
    const int T = cb_efflux_terms(nx, ny, zmax);
    double part[F];
#pragma unroll
    for (int f = 0; f < F; ++f) part[f] = 0;
    for (int t = threadIdx.x; t < T; t += UP_THREADS) {
        int x0, y0, x1, y1, x2, y2, z;
        const int sel = cb_efflux_term(t, nx, ny, zmax, x0, y0, x1, y1, x2, y2, z);
        const double sf = sel == 0 ? m.sx : m.sy;
        const int n0 = x0 + px * y0 + nxy * z, n1 = x1 + px * y1 + nxy * z, n2 = x2 + px * y2 + nxy * z;
        double a0[F], a1[F], a2[F];
#pragma unroll
        for (int f = 0; f < F; ++f) {
            a0[f] = (double)u[f * np + n0];
            a1[f] = (double)u[f * np + n1];
            a2[f] = (double)u[f * np + n2];
        }
#pragma unroll
        for (int f = 0; f < F; ++f) {
            const double D = f < NI ? m.D_ion[f] : m.D_pair[f - NI];
            const double g = 2 * a1[f] - 1.5 * a0[f] - 0.5 * a2[f];
            if (!RD3D) {
                part[f] += D * m.grad_mult * sf * g;
            } else {
                const double v = D * sf * g * m.inv_hc3;
                part[f] += v;
                terms[(long long)t * F + f] = v;
            }
        }
    }
    block_sums<F>(part, red);  // its barriers also publish the terms
    if (threadIdx.x == 0)
#pragma unroll
        for (int f = 0; f < F; ++f) q.efflux[f] = part[f];
    // 4. RD3D: deposit into the cytosol layer z = 0 in term order
    if (RD3D) {
        const int mc2 = m.mc * m.mc;
        const int* ptr = s_ptr;
        const int* dtm = s_term;
        for (int cn = threadIdx.x; cn < mc2; cn += UP_THREADS) {
            const int lo = ptr[cn], hi = ptr[cn + 1];
            double acc[CSM];
#pragma unroll
            for (int c = 0; c < CSM; ++c) acc[c] = 0;
            for (int k = lo; k < hi; ++k) {
                const int t = dtm[k];
#pragma unroll
                for (int c = 0; c < CSM; ++c) {
                    if (c >= CS) break;
                    int f = c < NI ? c : m.c_dyad_pair[c - NI];
                    if (f >= 0 && c >= NI) f += NI;
                    if (f >= 0) acc[c] += terms[(long long)t * F + f];
                }
            }
#pragma unroll
            for (int c = 0; c < CSM; ++c)
                if (c < CS) cin[((long long)s * CS + c) * mc2 + cn] = acc[c];
        }
    }
    // 5. RyR currents (CaSim/DyadRD2DCPU.cpp:243-264, CaSim/PassiveIonChannel.cpp:28-34)
    R* cg = curg + st.node_base * NI;
    double tot[NI];
#pragma unroll
    for (int j = 0; j < NI; ++j) tot[j] = 0;
    for (int c = threadIdx.x; c < st.n_ch; c += UP_THREADS) {
        const int node = ch_node[st.ch_off + c];
        const int state = ch_state[st.ch_off + c];
        const int own = ch_owner[st.ch_off + c];
#pragma unroll
        for (int j = 0; j < NI; ++j) {
            const double flux = state * (m.g[j] * (q.jsr_new[j] - (double)u[j * np + node]));
            if (own) cg[j * np + node] = (R)flux;
            tot[j] += flux;
        }
    }
    block_sums<NI>(tot, red);
    if (threadIdx.x == 0) {
#pragma unroll
        for (int j = 0; j < NI; ++j) q.total[j] = tot[j];
        // 6. jSR coupling (CaSim/SRPool.cpp:55-68)
        if (!m.jsr_const)
#pragma unroll
            for (int i = 0; i < NI; ++i) {
                q.IjSR[i] = q.total[i] * m.V_elem;
                q.nsr[i] = m.nsr[i];
                q.jsr[i] = q.jsr_new[i];
            }
    }
}

// Pools and two-state gating of one site per warp (CaSim/CytosolPool.cpp:217-268,
// CaSim/SRPool.cpp:70-89, CaSim/DyadChannels.cpp:97-130). The site's MRG32k3a stream is
// consumed in the reference's order (one draw per RyR test in RyR order, one more per
// transition) without a serial loop: lane l jumps to draw l of the stream (jump table J,
// row l: A^(2l)), the lanes draw 32 consecutive values at a time (then jump by A^62,
// row 31, to their draw of the next 32), and 32 RyRs are resolved per ballot, one more
// ballot after each transition. The stream state left behind is that at the first
// unused draw, as after the serial loop. With site_gate set, site s gates by
// gates[site_gate[s]] (per-site gating models) instead of the batch's model.
// MWC60: the 60-state model (mwc.h): the lanes form 32 escape rates at a time, a
// transition's second draw picks the micro-state it goes to (100 2D sites of 20 RyRs, FP64,
// 200 steps and readback: 89.4 ms with a thread per site, 6.4 ms here).
constexpr int PRE_WARPS = 4;
template <bool MWC60>
__global__ void __launch_bounds__(32 * PRE_WARPS) k_pre_r(const __grid_constant__ cb_model m, int S, int NS,
                                                          const cb_site* __restrict__ sites, cb_site_scalars* __restrict__ sc,
                                                          int* __restrict__ ch_state, const double* __restrict__ mouth,
                                                          const double* __restrict__ spx0, const double* __restrict__ spc0,
                                                          const double* __restrict__ spx1, const double* __restrict__ spc1,
                                                          const unsigned long long* __restrict__ J, const cb_gate* __restrict__ gates,
                                                          const int* __restrict__ site_gate, int* __restrict__ ch_micro,
                                                          const cb_mwc_tab* __restrict__ mwc) {
    __shared__ double s_u[PRE_WARPS][64];  // draws [we - 64, we), slot = draw & 63
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    const int s = blockIdx.x * PRE_WARPS + w;
    if (s >= S) return;  // whole warp
    const cb_site st = sites[s];
    cb_site_scalars& q = sc[s];
    const double dt = m.dt;
    if (lane == 0) {
        if (m.cyto_type == CB_CYTO_POOL) cb_pool_step(m, q, dt);
        cb_jsr_step(m, q, dt);
    }
    cbrng::State gl;  // this lane's draw we + lane
#pragma unroll
    for (int i = 0; i < 6; ++i) gl.s[i] = q.rng[i];
    cbrng::jump_by(J + 18 * lane, gl);
    cbrng::State gs = gl;  // state at this lane's draw of the latest chunk
    long long D = 0, we = 0;
    const int nch = st.n_ch;
    for (int c0 = 0; c0 < nch; c0 += 32) {
        const int cnt = min(32, nch - c0);
        const int c = c0 + lane;
        const bool act = lane < cnt;
        double p = 0, exit_rate = 0, ca = 0, mg = 0;
        int stt = 0;
        if (act) {
            const double* mo = mouth + (long long)(st.ch_off + c) * NS;
            ca = mo[m.ca_idx];
            mg = m.mg_idx >= 0 ? mo[m.mg_idx] : 0.0;
            stt = MWC60 ? ch_micro[st.ch_off + c] : ch_state[st.ch_off + c];
            if (MWC60) {
                exit_rate = cb_mwc_exit(*mwc, stt, ca, mg);
                p = exit_rate * dt;
            } else if (site_gate) {  // the site's own gating model
                const cb_gate& g = gates[site_gate[s]];
                p = cb_rate(g, g.spx[0], g.spc[0], g.spx[1], g.spc[1], stt, ca, mg) * dt;
            } else {
                p = cb_rate(m, spx0, spc0, spx1, spc1, stt, ca, mg) * dt;
            }
        }
        int start = 0;
        while (start < cnt) {
            // draws D .. D + (cnt - start) - 1 must be in the ring (MWC60: one more, the last
            // RyR's second draw; D + 33 at most, and chunks of 32 keep 64 draws)
            while (we < D + (cnt - start) + (MWC60 ? 1 : 0)) {
                gs = gl;
                s_u[w][(we + lane) & 63] = cbrng::u01d_fold(gl);
                cbrng::jump_by(J + 18 * 31, gl);
                we += 32;
                __syncwarp();
            }
            const bool rem = act && lane >= start;
            const double u = rem ? s_u[w][(D + (lane - start)) & 63] : 2.0;
            const unsigned int t = __ballot_sync(0xffffffffu, rem && (u < p));
            if (t == 0u) {
                D += cnt - start;
                break;
            }
            const int f = __ffs(t) - 1;
            if (lane == f) {
                if (MWC60) {
                    const int to = cb_mwc_next(*mwc, stt, ca, mg, exit_rate, s_u[w][(D + (f - start) + 1) & 63]);
                    ch_micro[st.ch_off + c] = to;
                    ch_state[st.ch_off + c] = to >= CB_MWC_OPEN;
                } else {
                    ch_state[st.ch_off + c] = 1 - stt;
                }
            }
            D += (f - start) + 2;
            start = f + 1;
        }
        __syncwarp();
    }
    // the state at draw D: lane D - (we - 32) of the latest chunk before its draw, or, past
    // the chunk, lane D - we at its next chunk's draw (D - we is 0 or 1)
    const bool in_chunk = D < we;
    const int k = in_chunk ? (int)(D - (we - 32)) : (int)(D - we);
    unsigned int out[6];
#pragma unroll
    for (int i = 0; i < 6; ++i) out[i] = __shfl_sync(0xffffffffu, in_chunk ? gs.s[i] : gl.s[i], k);
    if (lane == 0) {
        q.draws += (unsigned long long)D;
#pragma unroll
        for (int i = 0; i < 6; ++i) q.rng[i] = out[i];
    }
}

}  // namespace stream
