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
// (keep: nodes that the Update reads right after the step)
template <int V, typename R>
__device__ __forceinline__ void store_group(R* p, const group<R, V>& g, bool keep = false) {
    typedef typename word_of<R, V>::T W;
    if (keep) *(W*)p = *(const W*)&g;
    else __stcs((W*)p, *(const W*)&g);
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
// division by the row pitch). With the RD3D cytosol the rim takes the Dirichlet values of this
// step's Update (CaSim/DyadRD2DCPU.cpp:274-303), the cytosol as it was before its latest step; with
// the pool (cyto null) it carries its values over and the Update sets it.
template <typename R, int NI, int NP, int NZ, int V>
__global__ void __launch_bounds__(RD_THREADS, rd_min_blocks(sizeof(R), NI + NP, NZ, V))
    k_rd_v(const __grid_constant__ rd_const<R> k, const cb_site* __restrict__ sites, const int4* __restrict__ tiles,
           const R* __restrict__ in, R* __restrict__ out, const R* __restrict__ curg, const R* __restrict__ cyto, const int* __restrict__ rim_cnode, const unsigned* __restrict__ chcol) {
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
        const R* cy = cyto + (long long)tl.x * k.CS * k.nc + rim_cnode[st.rim_off + ri];
#pragma unroll
        for (int f = 0; f < F; ++f) b[f] = k.src[f] >= 0 ? cy[k.src[f] * k.nc] : k.init[f];
    };
    const bool carry = cyto == nullptr;
    if (y == 0 || y == ny - 1) {
        if (carry) {
#pragma unroll
            for (int f = 0; f < F; ++f)
#pragma unroll
                for (int z = 0; z < NZ; ++z) store_group(o + f * np + z * pxy, load_group<V>(u + f * np + z * pxy));
            return;
        }
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
    if (edge && !carry) rim_values(x == 0 ? y : ny + y, b);
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
                if (edge && (x + e == 0 || x + e >= nx - 1)) w.v[e] = carry ? c[f][z].v[e] : b[f];
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
           const R* __restrict__ in, R* __restrict__ out, const R* __restrict__ curg, const R* __restrict__ cyto, const int* __restrict__ rim_cnode, const unsigned* __restrict__ chcol, int* __restrict__ err) {
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
            for (int i = cyto ? lane : INT_MAX; i < side + top + bot; i += 32) {
                int ri;
                if (i < side) ri = (i & 1 ? tl.ny : 0) + y0 + (i >> 1);
                else if (i < side + top) ri = cb_rim_index(i - side, 0, tl.nx, tl.ny);
                else ri = cb_rim_index(i - side - top, tl.ny - 1, tl.nx, tl.ny);
                const R* cy = cyto + (long long)tl.site * k.CS * k.nc + rim_cnode[tl.rim_off + ri];
#pragma unroll
                for (int f = 0; f < F; ++f) rv[i * F + f] = k.src[f] >= 0 ? cy[k.src[f] * k.nc] : k.init[f];
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
            const bool carry = cyto == nullptr;
            if (carry && (y == 0 || y == ny - 1)) {
#pragma unroll
                for (int f = 0; f < F; ++f)
#pragma unroll
                    for (int z = 0; z < NZ; ++z)
                        store_group(o + f * np + z * pxy,
                                    load_group<V>((const R*)(stg + g.plane[f] + z * g.stride[f]) + gi + (k.diff[f] ? g.halo : 0)));
            } else if (y == 0 || y == ny - 1) {
                const int ce = min(col0 + TN, pxy) - 1;
                const int y1 = (int)((__umulhi((unsigned)ce, tl.mul) + (unsigned)ce) >> tl.sh);
                const R* row = rv + (2 * (y1 - y0 + 1) + (y == 0 || y0 > 0 ? 0 : nx)) * F;
#pragma unroll
                for (int f = 0; f < F; ++f) {
                    group<R, V> w;
#pragma unroll
                    for (int e = 0; e < V; ++e) w.v[e] = row[min(x + e, nx - 1) * F + f];
#pragma unroll
                    for (int z = 0; z < NZ; ++z) store_group(o + f * np + z * pxy, w, true);
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
                const bool keep = x <= 2 || x + V > nx - 3 || y < 3 || y >= ny - 3;
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
                            if (edge && (x + e == 0 || x + e >= nx - 1)) w.v[e] = carry ? c[f][z].v[e] : er[f];
                        store_group(o + f * np + z * pxy, w, keep || (has_ch && z == 0));
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

// blocks of k_cyto_t per SM asked of the compiler, and stages a block keeps in flight: four, three
// where four of six FP32 species would leave room for one block (2 ions, 4 pairs, 256 sites: 78 us with
// four, 57 with three; a thread per node from global memory 68)
constexpr int cyt_blocks(int w, int CS) { return w == 4 ? (CS <= 3 ? 3 : 2) : (CS <= 3 ? 2 : 1); }
__host__ __device__ constexpr int cyt_stages(int w, int CS) { return w == 4 && CS > 5 ? 3 : 4; }
constexpr int CY_THREADS = 352;  // 13 groups x 25 rows of the shipped grid in 11 warps

// k_cyto_v: nodes per thread, the most threads of a block, blocks per SM asked of the compiler and
// planes loaded ahead of the next. A column's planes have to fit the registers: pairs of FP64 nodes, or
// five species and more, in blocks of 352 threads spilled up to 1100 bytes, and layers of a few nodes left
// most of such a block idle. Us of that shape / a thread per node with no planes ahead / this one: FP64,
// three species, 1024 sites of 9^3 40 / 17 / 15, of 30^3 556 / 366 / 384, 256 of 40^3 364 / 244 / 209, six
// species, 256 of 30^3 577 / 241 / 247; FP32, 1024 of 9^3 17.1 / 13.3 / 13.3, six species, 256 of 30^3
// 206 / 163 / 124 (but of 24^3, which 352 threads hold whole, 76 / 108 / 85).
constexpr int cyv_vec(int w) { return w == 4 ? CB_CYTO_VEC : 1; }
constexpr int cyv_threads(int w, int CS) { return w == 4 && CS <= 4 ? 352 : 128; }
constexpr int cyv_blocks(int w, int CS) { return w == 4 ? (CS <= 3 ? 3 : CS <= 4 ? 2 : 4) : (CS <= 3 ? 6 : CS <= 4 ? 4 : 3); }
__host__ __device__ constexpr int cyv_ahead(int w, int CS) { return w == 4 ? (CS <= 4 ? 2 : 1) : (CS <= 5 ? 2 : 1); }

// RD3D cytosol step on any grid: a thread per group of V nodes of a layer (blockIdx.y: groups
// [y * blockDim.x, ..)), marching the mc - 1 updated planes (the top plane is the bath) with planes
// k-1 .. k+1 of its own nodes in registers and up to two more loaded ahead; plane 0 mirrors and
// takes the efflux deposits. The bath columns copy themselves so that every memory sector is
// written whole (a partly written sector is read back from memory when it leaves L2).
template <typename R, int NI, int NCP, int V>
__global__ void __launch_bounds__(cyv_threads(sizeof(R), NI + NCP), cyv_blocks(sizeof(R), NI + NCP))
    k_cyto_v(const __grid_constant__ cy_const<R> k, const R* __restrict__ in, R* __restrict__ out, const double* __restrict__ cin) {
    constexpr int CS = NI + NCP, AHEAD = cyv_ahead(sizeof(R), CS), ROT = AHEAD + 2;
    constexpr bool KEEP = sizeof(R) == 8;  // FP64 stores past L2 took 2 to 4 % longer
    const int mc = k.mc, px = k.px, npl = k.nplane, nc = k.nc;
    const int col = ((int)blockIdx.y * (int)blockDim.x + (int)threadIdx.x) * V;
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
        if (AHEAD > 1) p3[c] = load_group<V>(v + min(3, mc - 1) * npl);
        lo[c] = hi[c];
    }
#pragma unroll ROT
    for (int kp = 0; kp < mc - 1; ++kp) {
        const int n = kp * npl;
        if (bath) {
#pragma unroll
            for (int c = 0; c < CS; ++c) store_group(o + c * nc + n, cu[c], KEEP);
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
                store_group(o + c * nc + n, w, KEEP);
            }
        }
#pragma unroll
        for (int c = 0; c < CS; ++c) {
            lo[c] = cu[c];
            cu[c] = hi[c];
            hi[c] = p2[c];
            if (AHEAD > 1) p2[c] = p3[c];
            group<R, V>& far = AHEAD > 1 ? p3[c] : p2[c];
            if (kp + 2 + AHEAD < mc) far = load_group<V>(u + c * nc + n + (2 + AHEAD) * npl);
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

// RyR gating of one site by one warp (CaSim/DyadChannels.cpp:97-130), the transition
// probabilities prob given. The site's MRG32k3a stream is consumed in the reference's order (one
// draw per RyR test in RyR order, one more per transition) without a serial loop: lane l jumps
// to draw l of the stream (jump table J, row l: A^(2l)), the lanes draw 32 consecutive values at
// a time (then jump by A^62, row 31, to their draw of the next 32), and 32 RyRs are resolved per
// ballot, one more ballot after each transition. The stream state left behind is that at the
// first unused draw, as after the serial loop. (J is stored entry-major, [18][32 rows], so that the
// lanes' rows load coalesced.) ring: 64 draws, [we - 64, we), slot = draw & 63.
// The new open flags go to s_open as well. With mwc (60-state model) a transition's second draw
// picks the micro-state, at the mouth concentrations pcm.
__device__ __forceinline__ void gate_warp(const cb_site& st, cb_site_scalars& q, const double* __restrict__ prob, const double* __restrict__ pcm,
                                          int* __restrict__ ch_state, int* __restrict__ ch_micro, const cb_mwc_tab* __restrict__ mwc,
                                          const unsigned long long* __restrict__ J, double* ring, unsigned char* s_open) {
    const int lane = threadIdx.x & 31;
    cbrng::State gl;  // this lane's draw we + lane
#pragma unroll
    for (int i = 0; i < 6; ++i) gl.s[i] = q.rng[i];
    auto jump = [&](int row) {
        unsigned long long a[18];
#pragma unroll
        for (int i = 0; i < 18; ++i) a[i] = J[32 * i + row];
        cbrng::jump_by(a, gl);
    };
    jump(lane);
    cbrng::State gs = gl;  // state at this lane's draw of the latest chunk
    long long D = 0, we = 0;
    const int nch = st.n_ch, extra = mwc ? 1 : 0;
    for (int c0 = 0; c0 < nch; c0 += 32) {
        const int cnt = min(32, nch - c0);
        const int c = c0 + lane;
        const bool act = lane < cnt;
        const double p = act ? prob[st.ch_off + c] : 0.0;
        int open = act ? ch_state[st.ch_off + c] : 0;
        int start = 0;
        while (start < cnt) {
            // draws D .. D + (cnt - start) - 1 must be in the ring (60-state: one more, the last
            // RyR's second draw; D + 33 at most, and chunks of 32 keep 64 draws)
            while (we < D + (cnt - start) + extra) {
                gs = gl;
                ring[(we + lane) & 63] = cbrng::u01d_fold(gl);
                jump(31);
                we += 32;
                __syncwarp();
            }
            const bool rem = act && lane >= start;
            const double u = rem ? ring[(D + (lane - start)) & 63] : 2.0;
            const unsigned int t = __ballot_sync(0xffffffffu, rem && (u < p));
            if (t == 0u) {
                D += cnt - start;
                break;
            }
            const int f = __ffs(t) - 1;
            if (lane == f) {
                if (mwc) {
                    const int mi = ch_micro[st.ch_off + c];
                    const double ca = pcm[2 * (st.ch_off + c)], mg = pcm[2 * (st.ch_off + c) + 1];
                    const int to = cb_mwc_next(*mwc, mi, ca, mg, cb_mwc_exit(*mwc, mi, ca, mg), ring[(D + (f - start) + 1) & 63]);
                    ch_micro[st.ch_off + c] = to;
                    open = to >= CB_MWC_OPEN;
                } else {
                    open = 1 - open;
                }
                ch_state[st.ch_off + c] = open;
            }
            D += (f - start) + 2;
            start = f + 1;
        }
        if (act) s_open[c] = (unsigned char)open;
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

// What the gating of the next step needs of RyR c: its transition probability at the mouth
// concentrations (and, 60-state, the concentrations).
struct gate_args {
    const double *spx0, *spc0, *spx1, *spc1;
    const unsigned long long* J;
    const cb_gate* gates;      // per-site gating models, or null
    const int* site_gate;
    const cb_mwc_tab* mwc;     // 60-state model, or null
    int* ch_state;
    int* ch_micro;
    double* prob;              // [RyR] scratch of one casim_b200_step call
    double* pcm;               // [RyR][2]: mouth Ca and Mg (60-state)
};
__device__ __forceinline__ void store_prob(const cb_model& m, const gate_args& g, int s, int c, int open, double ca, double mg) {
    double r;
    if (g.mwc) {
        r = cb_mwc_exit(*g.mwc, g.ch_micro[c], ca, mg);
        g.pcm[2 * c] = ca;
        g.pcm[2 * c + 1] = mg;
    } else if (g.site_gate) {
        const cb_gate& o = g.gates[g.site_gate[s]];
        r = cb_rate(o, o.spx[0], o.spc[0], o.spx[1], o.spc[1], open, ca, mg);
    } else {
        r = cb_rate(m, g.spx0, g.spc0, g.spx1, g.spc1, open, ca, mg);
    }
    g.prob[c] = r * m.dt;
}

// the probabilities for the first step of a call, from the mouth values and RyR states as they are
__global__ void k_prob(const __grid_constant__ cb_model m, const __grid_constant__ gate_args g, int NS, const cb_site* __restrict__ sites,
                       const double* __restrict__ mouth) {
    const cb_site st = sites[blockIdx.x];
    for (int c = threadIdx.x; c < st.n_ch; c += blockDim.x) {
        const double* mo = mouth + (long long)(st.ch_off + c) * NS;
        store_prob(m, g, blockIdx.x, st.ch_off + c, g.ch_state[st.ch_off + c], mo[m.ca_idx], m.mg_idx >= 0 ? mo[m.mg_idx] : 0.0);
    }
}

// RD3D deposits of a site: its efflux terms are stored grouped by receiving layer-0 cytosol
// node; slot k feeds cytosol species c[k] from dyad species f[k]
struct dep_args {
    const int* pos;       // [term_off + term]: its place in the grouped order
    const int* node_ptr;  // [site]: the first of its receiving nodes, [S]: their count
    const int3* node;     // cytosol node (i + mc*j), first and end term
    int max_nodes, n, f[MAX_F], c[MAX_F];
};

constexpr int CH_OWNER = 1, CH_RIM = 2;  // flags of a RyR beside its node: takes the node's flux; lies on the rim

// One site per block. GATE (a time step): first the RyR gating (warp 0) and the pool ODEs (warp
// 1), which nothing before them in the step needs, while the other warps form the efflux; then
// the Update (CaSim/ParallelHybridSolver.cpp:159-175): mouth values, Dirichlet rim from the
// cytosol (RD3D: k_rd_t set it), efflux through the rim, the RD3D deposits into cytosol layer 0 (each
// receiving node's terms in a fixed order of eight interleaved partial sums, equal to their sum in term
// order within rounding),
// RyR currents, the jSR coupling and the probabilities of the next gating. Without GATE (the
// public Update) no time passes and the rim is always set here. want: also write what only
// the getters read (mouth values, RD3D: efflux sums), for the last step of a call.
//
// The kernel is a chain of short latency-bound phases per site, so they overlap: gating in a
// launch of its own took 18 us of a 64-site step and this kernel 21 us, most of it waiting; the
// efflux indices took integer divisions, the deposits went through an index list, the RyRs'
// nodes were fetched twice and the sums reduced twice.
// 4096 dyads, FP32: 45 + 131 us in two launches, 127 us in this one, of which the mouth and rim
// gathers (a sector per value of an x edge) take over half.
template <typename R, int NI, int NP, bool RD3D, bool GATE>
__global__ void __launch_bounds__(UP_THREADS, 4)
    k_update_s(const __grid_constant__ cb_model m, const __grid_constant__ gate_args ga, const __grid_constant__ dep_args dep, int NS, bool want,
               const cb_site* __restrict__ sites, R* __restrict__ fld, const R* __restrict__ prev, R* __restrict__ curg,
               const int2* __restrict__ ch, double* __restrict__ mouth, cb_site_scalars* __restrict__ sc,
               int nc, const R* __restrict__ cyto, double* __restrict__ cin, const int* __restrict__ rim_cnode, int max_ch, int max_terms) {
    constexpr int F = NI + NP;
    extern __shared__ double up_smem[];
    __shared__ double red[UP_THREADS / 32 * (F + NI)], s_ring[64], s_jsr[NI];
    __shared__ R s_rim[F];
    unsigned char* s_open = (unsigned char*)up_smem;                    // [max_ch]
    double* terms = up_smem + (max_ch + 7) / 8;                         // RD3D: [dep.n][max_terms]
    int3* s_node = (int3*)(terms + (RD3D ? dep.n * max_terms : 0));     // RD3D: [dep.max_nodes]
    const int s = blockIdx.x, tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const cb_site st = sites[s];
    cb_site_scalars& q = sc[s];
    R* u = fld + st.node_base * F;
    const R* before = GATE ? prev + st.node_base * F : u;
    const int nx = st.nx, ny = st.ny, nz = st.nz, px = st.px, nxy = px * ny, np = st.npad;
    const int2* chs = ch + st.ch_off;
    // the warps of the efflux: all, or those that neither gate nor (RD3D) step the jSR
    constexpr int E0 = !GATE ? 0 : RD3D ? 64 : 32, EN = UP_THREADS - E0;
    const int et = tid - E0;
    // 1. mouth values: ions, pairs, free buffers (CaSim/DyadRD2DCPU.cpp:361-380): the new fields, a
    // RyR on the rim what the step carried over there, which is before's (GATE: the rim is set
    // already or set below). Each thread keeps its first RyR's.
    int2 ch0 = make_int2(0, 0);
    R v0[F];
    for (int c = tid; c < st.n_ch; c += UP_THREADS) {
        const int2 cc = chs[c];
        const R* src = cc.y & CH_RIM ? before : u;
        R v[F];
#pragma unroll
        for (int f = 0; f < F; ++f) v[f] = src[f * np + cc.x];
        if (c == tid) {
            ch0 = cc;
#pragma unroll
            for (int f = 0; f < F; ++f) v0[f] = v[f];
        }
        if (!want) break;
        double* mo = mouth + (long long)(st.ch_off + c) * NS;
#pragma unroll
        for (int f = 0; f < F; ++f) mo[f] = (double)v[f];
        for (int b = 0; b < m.n_buf; ++b) {
            double fr = m.Ctot[b];
#pragma unroll
            for (int p = 0; p < NP; ++p)
                if (m.pair_buf[p] == b) fr -= (double)v[NI + p];
            mo[F + b] = fr;
        }
    }
    auto efflux_sync = [&]() {
        if (GATE) {
            __syncwarp();
            asm volatile("bar.sync 1, %0;" ::"n"(EN) : "memory");
        } else {
            __syncthreads();
        }
    };
    double part[F];
#pragma unroll
    for (int f = 0; f < F; ++f) part[f] = 0;
    if (GATE && warp == 0) {
        gate_warp(st, q, ga.prob, ga.pcm, ga.ch_state, ga.ch_micro, ga.mwc, ga.J, s_ring, s_open);
    } else if (GATE && RD3D && warp == 1) {
        if (lane == 0) {
            cb_jsr_step<NI>(m, q, m.dt);
#pragma unroll
            for (int j = 0; j < NI; ++j) s_jsr[j] = q.jsr_new[j];
        }
    } else {
        if (et == 0) {
            if (GATE && !RD3D) cb_pool_step<NI>(m, q, m.dt);
#pragma unroll
            for (int j = 0; j < NI; ++j) s_rim[j] = (R)q.c_ions[j];
#pragma unroll
            for (int p = 0; p < NP; ++p) s_rim[NI + p] = (R)q.c_bnd[p];
        }
        __syncwarp();
        // RD3D: the site's deposit nodes, staged while the efflux loads are in flight
        int nd = 0;
        if (RD3D) {
            const int d0 = dep.node_ptr[s];
            nd = dep.node_ptr[s + 1] - d0;
            for (int i = et; i < nd; i += EN) s_node[i] = dep.node[d0 + i];
        }
        // 2. Dirichlet edges from the cytosol (CaSim/DyadRD2DCPU.cpp:274-303)
        auto set_rim = [&]() {
            const int nrim = cb_rim_count(nx, ny);
            const R* cy = RD3D ? cyto + (long long)s * (m.n_ions + m.c_n_pairs) * nc : nullptr;
            for (int r = et; r < nrim; r += EN) {
                int x, y;
                cb_rim_xy(r, nx, ny, x, y);
                R b[F];
                if (!RD3D) {
#pragma unroll
                    for (int f = 0; f < F; ++f) b[f] = s_rim[f];
                } else {
                    const int cn = rim_cnode[st.rim_off + r];
#pragma unroll
                    for (int j = 0; j < NI; ++j) b[j] = cy[j * nc + cn];
#pragma unroll
                    for (int p = 0; p < NP; ++p) {
                        const int cq = m.dyad_c_pair[p];
                        b[NI + p] = cq >= 0 ? cy[(NI + cq) * nc + cn] : (R)m.pair_init[p];
                    }
                }
                for (int z = 0; z < nz; ++z)
#pragma unroll
                    for (int f = 0; f < F; ++f) u[f * np + x + px * y + nxy * z] = b[f];
            }
        };
        if (!GATE) {
            efflux_sync();
            set_rim();
            efflux_sync();
        }
        // 3. efflux (CaSim/DyadRD2DCPU.cpp:305-350) in the reference's term order: x-edges (x = 0,
        // then nx-1) over y = 1..ny-2, y-edges over x, layers innermost (the top one has no rim).
        // A thread's NB terms are loaded together. Pool, GATE: the rim nodes read s_rim.
        constexpr int NB = 2;
        constexpr bool POOL = GATE && !RD3D;
        const int zs = nz == 1 ? 0 : 1, nye = ny - 2, T = (2 * nye + 2 * nx) << zs;
        const int* pos = RD3D ? dep.pos + st.term_off : nullptr;
        bool synced = !POOL;
        for (int t0 = et; t0 < T || !synced; t0 += NB * EN) {
            R a0[NB][F], a1[NB][F], a2[NB][F];
            int at[NB];
            double sf[NB];
            bool end[NB];
#pragma unroll
            for (int i = 0; i < NB; ++i) {
                const int t = t0 + i * EN;
                if (t >= T) break;
                const int z = zs ? t & 1 : 0;
                int a = t >> zs, n0, step;
                const bool xe = a < 2 * nye;
                if (xe) {
                    const bool far = a >= nye;
                    n0 = px * (1 + a - (far ? nye : 0)) + (far ? nx - 1 : 0);
                    step = far ? -1 : 1;
                    end[i] = false;
                } else {
                    a -= 2 * nye;
                    const bool far = a >= nx;
                    a -= far ? nx : 0;
                    n0 = a + (far ? px * (ny - 1) : 0);
                    step = far ? -px : px;
                    end[i] = a == 0 || a == nx - 1;  // the line runs along the rim
                }
                n0 += nxy * z;
                sf[i] = xe ? m.sx : m.sy;
#pragma unroll
                for (int f = 0; f < F; ++f) {
                    if (!POOL) a0[i][f] = u[f * np + n0];
                    a1[i][f] = u[f * np + n0 + step];
                    a2[i][f] = u[f * np + n0 + 2 * step];
                }
                at[i] = RD3D ? pos[t] : 0;
            }
            if (!synced) {  // the pool's new values
                efflux_sync();
                synced = true;
            }
#pragma unroll
            for (int i = 0; i < NB; ++i) {
                if (t0 + i * EN >= T) break;
#pragma unroll
                for (int f = 0; f < F; ++f) {
                    if (POOL) {
                        a0[i][f] = s_rim[f];
                        if (end[i]) a1[i][f] = a2[i][f] = s_rim[f];
                    }
                    const double D = f < NI ? m.D_ion[f] : m.D_pair[f - NI];
                    const double g = 2 * (double)a1[i][f] - 1.5 * (double)a0[i][f] - 0.5 * (double)a2[i][f];
                    if (!RD3D) {
                        part[f] += D * m.grad_mult * sf[i] * g;
                    } else {
                        const double v = D * sf[i] * g * m.inv_hc3;
                        part[f] += v;
#pragma unroll
                        for (int k = 0; k < F; ++k)
                            if (k < dep.n && dep.f[k] == f) terms[k * max_terms + at[i]] = v;
                    }
                }
            }
        }
        if (POOL) {
            set_rim();
            if (et == 0) {
                cb_jsr_step<NI>(m, q, m.dt);
            }
        }
        if (!RD3D || !GATE) {
            if (et == 0)
#pragma unroll
                for (int j = 0; j < NI; ++j) s_jsr[j] = q.jsr_new[j];
        }
        // 4. RD3D: deposits into the cytosol layer z = 0 (the other nodes' deposits stay zero): 8
        // lanes per receiving node, every 8th of its terms each (most nodes have 8, those under
        // the corners of a cleft wider than the cytosol dozens)
        if (RD3D) {
            efflux_sync();
            const int mc2 = m.mc * m.mc;
            for (int i = et >> 3; i < (nd + EN / 8 - 1) / (EN / 8) * (EN / 8); i += EN / 8) {
                const int3 dn = i < nd ? s_node[i] : make_int3(0, 0, 0);
                double acc[F];
#pragma unroll
                for (int k = 0; k < F; ++k) acc[k] = 0;
                for (int t = dn.y + (lane & 7); t < dn.z; t += 8)
#pragma unroll
                    for (int k = 0; k < F; ++k)
                        if (k < dep.n) acc[k] += terms[k * max_terms + t];
#pragma unroll
                for (int o = 4; o > 0; o >>= 1)
#pragma unroll
                    for (int k = 0; k < F; ++k)
                        if (k < dep.n) acc[k] += __shfl_xor_sync(0xffffffffu, acc[k], o);
                if (i < nd && (lane & 7) == 0)
#pragma unroll
                    for (int k = 0; k < F; ++k)
                        if (k < dep.n) cin[((long long)s * (m.n_ions + m.c_n_pairs) + dep.c[k]) * mc2 + dn.x] = acc[k];
            }
        }
    }
    __syncthreads();
    // 5. RyR currents (CaSim/DyadRD2DCPU.cpp:243-264, CaSim/PassiveIonChannel.cpp:28-34) and the
    // next gating's probabilities
    R* cg = curg + st.node_base * NI;
    double sums[F + NI];
#pragma unroll
    for (int f = 0; f < F; ++f) sums[f] = part[f];
#pragma unroll
    for (int j = 0; j < NI; ++j) sums[F + j] = 0;
    for (int c = tid; c < st.n_ch; c += UP_THREADS) {
        const int2 cc = c == tid ? ch0 : chs[c];
        const int open = GATE ? (int)s_open[c] : ga.ch_state[st.ch_off + c];
        const R* src = cc.y & CH_RIM ? before : u;
        double ca = 0, mg = 0;
#pragma unroll
        for (int j = 0; j < NI; ++j) {
            const R mv = c == tid ? v0[j] : src[j * np + cc.x];
            // the flux reads the node after the rim is set
            const R at = !(cc.y & CH_RIM) ? mv : GATE && !RD3D ? s_rim[j] : u[j * np + cc.x];
            const double flux = open * (m.g[j] * (s_jsr[j] - (double)at));
            if (cc.y & CH_OWNER) cg[j * np + cc.x] = (R)flux;
            sums[F + j] += flux;
            if (j == m.ca_idx) ca = (double)mv;
            if (j == m.mg_idx) mg = (double)mv;
        }
        if (GATE) store_prob(m, ga, s, st.ch_off + c, open, ca, mg);
    }
    if (!RD3D || !GATE || want) {
        block_sums<F + NI>(sums, red);
    } else {
        double tot[NI];
#pragma unroll
        for (int j = 0; j < NI; ++j) tot[j] = sums[F + j];
        block_sums<NI>(tot, red);
#pragma unroll
        for (int j = 0; j < NI; ++j) sums[F + j] = tot[j];
    }
    if (tid == 0) {
        if (!RD3D || !GATE || want)
#pragma unroll
            for (int f = 0; f < F; ++f) q.efflux[f] = sums[f];
#pragma unroll
        for (int j = 0; j < NI; ++j) q.total[j] = sums[F + j];
        // 6. jSR coupling (CaSim/SRPool.cpp:55-68)
        if (!m.jsr_const)
#pragma unroll
            for (int i = 0; i < NI; ++i) {
                q.IjSR[i] = sums[F + i] * m.V_elem;
                q.nsr[i] = m.nsr[i];
                q.jsr[i] = s_jsr[i];
            }
    }
}

}  // namespace stream
