// cluster.cu -- largest solid-glycine cluster (get_greatestCluster) on the GPU.
//
// The reference (Source/mod_cluster.f90:15-83) builds per-molecule centres,
// a centre cell list, a density list within denscut, a recursive flood fill
// over "solid" molecules (denstrack >= densmin), a histogram, the largest
// cluster by strict '>' in discovery order, and appends adjacent non-solid
// molecules.  The partition into clusters is independent of the visiting
// order, so the flood fill is replaced by a union of the list's edges whose labels
// are the smallest molecule index of each component; ranking the roots in
// ascending order gives exactly the reference's discovery numbering.  The
// integer result is therefore bit-identical.
//
// Compiled with -fmad=false like the other reference-semantics kernels.
#include "common.cuh"

namespace {

constexpr unsigned FULL = 0xffffffffu;
constexpr int DCAP = 256;  // density-list entries per molecule

__device__ __forceinline__ double shift_real4(double d, float box, float ibox) {
    // box*nint(d*ibox) with the product in real*4 (mod_build_ptta.f90:158-160,
    // mod_neighbor_cluster.f90:104-106)
    int n = (int)round(d * (double)ibox);
    return (double)(box * (float)n);
}

struct ClusterArgs {
    int n_gly, apg, densmin, mncellD, mncellT;
    float box, ibox;
    double mrcut2, denscut2, imrn;
    double *ptta;
    double *com;
    int *mcell, *cell_count, *cell_start, *cell_fill, *cell_list;
    int *denstrack, *densvl, *label, *rank, *csize, *surf;
    int *status;
    int *result;  // [0] size, [1] greatest_belongsto (in/out)
};

// The analysis is a chain of six short launches: refresh, centres, cells, density
// lists, components, result.  Everything per molecule is spread over the GPU; only
// the scan of the cells and the final bookkeeping (3,500 molecules: a few passes of
// one block) stay in one block.  As one block with serial loops of its first thread
// over cells, molecules and clusters, the whole took 660 us at 3,500 glycines
// against the launches' 30 us, which are bound by their latency.

// build_ptta_wrap_cluster2, Source/mod_build_ptta.f90:116-132: the atom whose
// global id equals n_gly*apg is never refreshed (`id.lt.flag`).  Also clears the
// cell counts and the status words.
__global__ void k_ptta_refresh(int np, const float4 *__restrict__ pos,
                               const int *__restrict__ gid, int flag, ClusterArgs a) {
    SOFIA_PDL_ENTRY();
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    for (int c = i; c <= a.mncellT; c += gridDim.x * blockDim.x) {
        a.cell_count[c] = 0;
        a.cell_fill[c] = 0;
    }
    if (i < sofia::ST_NSLOTS) a.status[i] = 0;
    if (i >= np) return;
    int id = gid[i];
    if (id >= 1 && id < flag) {
        float4 p = pos[i];
        a.ptta[(size_t)(id - 1) * 3 + 0] = (double)p.x;
        a.ptta[(size_t)(id - 1) * 3 + 1] = (double)p.y;
        a.ptta[(size_t)(id - 1) * 3 + 2] = (double)p.z;
    }
}

// unwrap about the first atom + unweighted centre + wrap to [0, box]
// (mod_build_ptta.f90:135-163, mod_cluster.f90:803-884), one thread per molecule
__global__ void k_cluster_centres(ClusterArgs a) {
    SOFIA_PDL_ENTRY();
    const int m = blockIdx.x * blockDim.x + threadIdx.x;
    if (m >= a.n_gly) return;
    const double boxd = (double)a.box;
    double *base = a.ptta + (size_t)m * a.apg * 3;
    const double x1 = base[0], y1 = base[1], z1 = base[2];
    double xc = 0.0, yc = 0.0, zc = 0.0;
    for (int j = 0; j < a.apg; ++j) {
        double *pj = base + (size_t)j * 3;
        double x2 = pj[0], y2 = pj[1], z2 = pj[2];
        if (j > 0) {
            x2 = x2 - shift_real4(x2 - x1, a.box, a.ibox);
            y2 = y2 - shift_real4(y2 - y1, a.box, a.ibox);
            z2 = z2 - shift_real4(z2 - z1, a.box, a.ibox);
            pj[0] = x2;
            pj[1] = y2;
            pj[2] = z2;
        }
        xc += x2;
        yc += y2;
        zc += z2;
    }
    const double na = (double)(float)a.apg;
    double c[3] = {xc / na, yc / na, zc / na};
    for (int d = 0; d < 3; ++d) {
        int guard = 0;
        while (c[d] > boxd && guard++ < 64) c[d] = c[d] - boxd;
        while (c[d] < 0.0 && guard++ < 128) c[d] = c[d] + boxd;
        a.com[(size_t)m * 3 + d] = c[d];
    }
    // mol_xyz2bin, mod_neighbor_cluster.f90:668-709
    const int D = a.mncellD;
    int ix = (c[0] < boxd) ? (int)(c[0] * a.imrn) : D - 1;
    int iy = (c[1] < boxd) ? (int)(c[1] * a.imrn) : D - 1;
    int iz = (c[2] < boxd) ? (int)(c[2] * a.imrn) : D - 1;
    if (ix >= D) ix = D - 1;
    if (iy >= D) iy = D - 1;
    if (iz >= D) iz = D - 1;
    if (ix < 0) ix = 0;
    if (iy < 0) iy = 0;
    if (iz < 0) iz = 0;
    const int cell = ix + iy * D + iz * D * D;
    a.mcell[m] = cell;
    a.label[m] = m;
    atomicAdd(&a.cell_count[cell], 1);
}

// Inclusive scan over the block's 1024 threads; s_w holds 32 words.
__device__ __forceinline__ int block_scan(int v, int *s_w) {
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
#pragma unroll
    for (int off = 1; off < 32; off <<= 1) {
        const int x = __shfl_up_sync(FULL, v, off);
        if (lane >= off) v += x;
    }
    __syncthreads();  // the words may still be read from the previous call
    if (lane == 31) s_w[w] = v;
    __syncthreads();
    if (w == 0) {
        int x = s_w[lane];
#pragma unroll
        for (int off = 1; off < 32; off <<= 1) {
            const int y = __shfl_up_sync(FULL, x, off);
            if (lane >= off) x += y;
        }
        s_w[lane] = x;
    }
    __syncthreads();
    return v + (w > 0 ? s_w[w - 1] : 0);
}

// Exclusive scan of the cell counts, then the molecules of every cell; one block.
__global__ void __launch_bounds__(1024) k_cluster_cells(ClusterArgs a) {
    SOFIA_PDL_ENTRY();
    __shared__ int s_w[32];
    const int t = threadIdx.x;
    int carry = 0;
    for (int base = 0; base <= a.mncellT; base += 1024) {
        const int v = (base + t < a.mncellT) ? a.cell_count[base + t] : 0;
        const int incl = block_scan(v, s_w);
        if (base + t <= a.mncellT) a.cell_start[base + t] = carry + incl - v;
        carry += s_w[31];
    }
    __syncthreads();
    for (int m = t; m < a.n_gly; m += 1024) {
        const int c = a.mcell[m];
        const int s = atomicAdd(&a.cell_fill[c], 1);
        a.cell_list[a.cell_start[c] + s] = m;
    }
}

// mol_build_neighbor_nosort (mod_neighbor_cluster.f90:57-176): the 26 stencil
// cells with minimum image, then the own cell without it.  Counts include
// repeated cells when mncellD < 3, as there.  One warp per molecule: lane k holds
// stencil cell k (the 27th is the own cell) and the cells' molecules are streamed
// over the lanes as one sequence; the order of a list's entries does not matter.
__global__ void __launch_bounds__(128) k_cluster_density(ClusterArgs a) {
    SOFIA_PDL_ENTRY();
    __shared__ int s_seg[4][2][32];  // per warp and stencil cell: first entry, end in the sequence
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    const int p1 = blockIdx.x * 4 + w;
    if (p1 >= a.n_gly) return;
    const double x1 = a.com[(size_t)p1 * 3], y1 = a.com[(size_t)p1 * 3 + 1],
                 z1 = a.com[(size_t)p1 * 3 + 2];
    const int D = a.mncellD;
    const int cell = a.mcell[p1];
    int start = 0, len = 0;
    if (lane < 27) {
        const int icz = cell / (D * D);
        const int icy = (cell - icz * D * D) / D;
        const int icx = cell - icy * D - icz * D * D;
        int zc = icz + lane / 9 - 1, yc = icy + (lane / 3) % 3 - 1, xc = icx + lane % 3 - 1;
        zc = zc < 0 ? zc + D : (zc >= D ? zc - D : zc);
        yc = yc < 0 ? yc + D : (yc >= D ? yc - D : yc);
        xc = xc < 0 ? xc + D : (xc >= D ? xc - D : xc);
        const int cn = xc + yc * D + zc * D * D;
        start = a.cell_start[cn];
        len = a.cell_start[cn + 1] - start;
    }
    int incl = len;
#pragma unroll
    for (int off = 1; off < 32; off <<= 1) {
        const int v = __shfl_up_sync(FULL, incl, off);
        if (lane >= off) incl += v;
    }
    const int total = __shfl_sync(FULL, incl, 31);
    s_seg[w][0][lane] = start;
    s_seg[w][1][lane] = incl;
    __syncwarp();
    int cnt = 0, seg = 0;
    int *dv = a.densvl + (size_t)p1 * DCAP;
    for (int base = 0; base < total; base += 32) {
        const int q = base + lane;
        bool in = false;
        int p2 = 0;
        if (q < total) {
            while (s_seg[w][1][seg] <= q) ++seg;  // ends: offset of the last one is total
            const bool own = seg == 13;
            p2 = a.cell_list[s_seg[w][0][seg] + (q - (seg > 0 ? s_seg[w][1][seg - 1] : 0))];
            double dx = x1 - a.com[(size_t)p2 * 3];
            double dy = y1 - a.com[(size_t)p2 * 3 + 1];
            double dz = z1 - a.com[(size_t)p2 * 3 + 2];
            if (!own) {
                dx = dx + (-shift_real4(dx, a.box, a.ibox));
                dy = dy + (-shift_real4(dy, a.box, a.ibox));
                dz = dz + (-shift_real4(dz, a.box, a.ibox));
            }
            const double dr2 = dx * dx + dy * dy + dz * dz;
            in = dr2 < a.mrcut2 && dr2 < a.denscut2 && !(own && p2 == p1);
        }
        const unsigned m = __ballot_sync(FULL, in);
        if (in) {
            const int at = cnt + __popc(m & ((1u << lane) - 1u));
            if (at < DCAP) dv[at] = p2;
        }
        cnt += __popc(m);
    }
    if (lane == 0) {
        if (cnt > DCAP) atomicAdd(&a.status[sofia::ST_DENSOVER], 1);
        a.denstrack[p1] = cnt;
    }
}

// Root of u.  A parent's index is never larger than its child's, so the walk ends;
// the parents are read past L1, where another SM's hook may not show.
__device__ __forceinline__ int find_root(const int *parent, int u) {
    int p = __ldcg(parent + u);
    while (p != u) {
        u = p;
        p = __ldcg(parent + u);
    }
    return u;
}

// Connected components of the solid molecules: every density-list edge hooks the
// larger of its two roots to the smaller, so a component's root is its smallest
// index whatever the order of the hooks.  One warp per molecule, lanes over its
// list.  A failed hook has met a smaller parent and continues from there, so each
// retry moves to a smaller index.
__global__ void __launch_bounds__(128) k_cluster_hook(ClusterArgs a) {
    SOFIA_PDL_ENTRY();
    const int lane = threadIdx.x & 31;
    const int u = blockIdx.x * 4 + (threadIdx.x >> 5);
    if (u >= a.n_gly || a.denstrack[u] < a.densmin) return;
    const int cnt = min(a.denstrack[u], DCAP);
    const int *dv = a.densvl + (size_t)u * DCAP;
    for (int l = lane; l < cnt; l += 32) {
        const int v = dv[l];
        if (v >= u || a.denstrack[v] < a.densmin) continue;  // the mirror edge hooks v > u
        int x = find_root(a.label, u), y = find_root(a.label, v);
        while (x != y) {
            if (x < y) {
                const int s = x;
                x = y;
                y = s;
            }
            const int old = atomicCAS(&a.label[x], x, y);
            if (old == x) break;
            x = find_root(a.label, old);
            y = find_root(a.label, y);
        }
    }
}

// Cluster numbers, sizes, the largest cluster and its surface; one block.
__global__ void __launch_bounds__(1024) k_cluster_result(ClusterArgs a, int greatest_in) {
    SOFIA_PDL_ENTRY();
    __shared__ int s_w[32];
    __shared__ int s_cluster, s_surface;
    __shared__ unsigned long long s_best;
    const int t = threadIdx.x, n = a.n_gly;
    int *root = a.mcell;  // the cells are done with
    if (t == 0) {
        s_surface = 0;
        s_best = 0ull;
    }
    // rank roots in ascending index = buildClusters discovery numbering (:228-246)
    int carry = 0;
    for (int base = 0; base < n; base += 1024) {
        const int u = base + t;
        const bool solid = u < n && a.denstrack[u] >= a.densmin;
        const int r = solid ? find_root(a.label, u) : -1;
        const int incl = block_scan(r == u && solid ? 1 : 0, s_w);
        if (u < n) {
            root[u] = r;
            a.rank[u] = carry + incl;
            a.csize[u] = 0;
        }
        carry += s_w[31];
    }
    const int nclus = carry;
    __syncthreads();
    for (int u = t; u < n; u += 1024) {
        const int b = root[u] >= 0 ? a.rank[root[u]] : 0;
        a.label[u] = b;  // label now holds belongsto
        a.surf[u] = 0;
        if (b > 0) atomicAdd(&a.csize[b - 1], 1);
    }
    __syncthreads();
    // the largest cluster, the first of equals (strict '>' in discovery order)
    for (int c = t; c < nclus; c += 1024)
        atomicMax(&s_best, ((unsigned long long)a.csize[c] << 32) | (unsigned)(~c));
    __syncthreads();
    const int greatest = (int)(s_best >> 32);
    if (t == 0) {
        s_cluster = greatest > 0 ? (int)~(unsigned)s_best + 1 : greatest_in;
        a.result[1] = s_cluster;
    }
    __syncthreads();
    // append_surface_molecules (mod_cluster.f90:163-194)
    const int cluster = s_cluster;
    for (int u = t; u < n; u += 1024) {
        if (a.label[u] != cluster) continue;
        const int cnt = min(a.denstrack[u], DCAP);
        const int *dv = a.densvl + (size_t)u * DCAP;
        for (int l = 0; l < cnt; ++l) {
            const int v = dv[l];
            if (a.denstrack[v] < a.densmin) a.surf[v] = 1;
        }
    }
    __syncthreads();
    int mine = 0;
    for (int u = t; u < n; u += 1024)
        if (a.surf[u]) {
            mine++;
            a.label[u] = cluster;
        }
    if (mine) atomicAdd(&s_surface, mine);
    __syncthreads();
    if (t == 0) {
        a.result[0] = greatest + s_surface;
        a.result[2] = a.status[sofia::ST_DENSOVER];
    }
}

}  // namespace

extern "C" int sofia_greatest_cluster(sofia_nb_ctx *ctx, int np, const sofia_ainfo *position,
                                      const int32_t *global_id, int n_gly, int atoms_per_gly,
                                      float box, double mrcut, double denscut, int densmin,
                                      double *ptta_full, int32_t *greatest_belongsto,
                                      int32_t *size_out, int32_t *denstrack,
                                      int32_t *belongsto) {
    if (!ctx) return SOFIA_EINVAL;
    if (np <= 0 || !position || !global_id || n_gly < 0 || atoms_per_gly <= 0 || !ptta_full ||
        !greatest_belongsto || !size_out || !(box > 0.0f) || !(mrcut > 0.0) || !(denscut > 0.0))
        return sofia::fail(ctx, SOFIA_EINVAL, "bad args%s");
    if (n_gly == 0) {
        *size_out = 0;
        return SOFIA_OK;
    }
    SOFIA_CUDA(ctx, cudaSetDevice(ctx->device));
    sofia::HostCopies copies(ctx);
    cudaStream_t st = ctx->stream;
    int rc;
    const void *dpos, *dgid;
    if ((rc = sofia::stage_in(ctx, position, sizeof(float4) * (size_t)np, 0, &dpos))) return rc;
    if ((rc = sofia::stage_in(ctx, global_id, sizeof(int) * (size_t)np, 1, &dgid))) return rc;
    sofia::OutArg o_ptta;
    const size_t ptta_bytes = sizeof(double) * 3 * (size_t)n_gly * atoms_per_gly;
    if ((rc = sofia::stage_out(ctx, ptta_full, ptta_bytes, 2, &o_ptta, true))) return rc;
    // cell grid of check_allocation_cluster (mod_neighbor_cluster.f90:546-548)
    const float ibox = (float)(1.0 / (double)box);
    volatile float vb2 = box * box;
    volatile float vol = vb2 * box;
    const int nside = (int)((double)box / mrcut);
    if (nside < 1) return sofia::fail(ctx, SOFIA_EINVAL, "box smaller than mrcut%s");
    volatile float mrn_f = box / (float)nside;
    const double mrn = (double)mrn_f;
    const int mncellT = (int)lround((double)vol / ((mrn * mrn) * mrn));
    const int mncellD = (int)lround(pow((double)mncellT, 1.0 / 3.0));
    if ((long)mncellD * mncellD * mncellD != mncellT)
        return sofia::fail(ctx, SOFIA_EINVAL, "invalid cluster cell grid%s");
    const size_t n = (size_t)n_gly;
    SOFIA_CUDA(ctx, ctx->cl_buf[0].ensure(sizeof(double) * 3 * n));
    SOFIA_CUDA(ctx, ctx->cl_buf[1].ensure(sizeof(int) * n * 4));
    SOFIA_CUDA(ctx, ctx->cl_buf[2].ensure(sizeof(int) * ((size_t)mncellT + 1) * 3));
    SOFIA_CUDA(ctx, ctx->cl_buf[3].ensure(sizeof(int) * n * DCAP));
    SOFIA_CUDA(ctx, ctx->cl_buf[4].ensure(sizeof(int) * (n + 1) * 4));
    SOFIA_CUDA(ctx, ctx->cl_buf[5].ensure(sizeof(int) * 4));
    ClusterArgs a;
    a.n_gly = n_gly;
    a.apg = atoms_per_gly;
    a.densmin = densmin;
    a.mncellD = mncellD;
    a.mncellT = mncellT;
    a.box = box;
    a.ibox = ibox;
    a.mrcut2 = mrcut * mrcut;
    a.denscut2 = denscut * denscut;
    a.imrn = 1.0 / mrn;
    a.ptta = (double *)o_ptta.dev;
    a.com = ctx->cl_buf[0].as<double>();
    int *b1 = ctx->cl_buf[1].as<int>();
    a.mcell = b1;
    a.cell_list = b1 + n;
    a.denstrack = b1 + 2 * n;
    int *b2 = ctx->cl_buf[2].as<int>();
    a.cell_count = b2;
    a.cell_start = b2 + (mncellT + 1);
    a.cell_fill = b2 + 2 * (mncellT + 1);
    a.densvl = ctx->cl_buf[3].as<int>();
    int *b4 = ctx->cl_buf[4].as<int>();
    a.label = b4;
    a.rank = b4 + (n + 1);
    a.csize = b4 + 2 * (n + 1);
    a.surf = b4 + 3 * (n + 1);
    a.status = ctx->d_status;
    a.result = ctx->cl_buf[5].as<int>();
    const int flag = n_gly * atoms_per_gly;
    sofia::launch_pdl(k_ptta_refresh, sofia::grid_for(np, 256), 256, 0, st, np,
                      (const float4 *)dpos, (const int *)dgid, flag, a);
    sofia::launch_pdl(k_cluster_centres, sofia::grid_for(n_gly, 64), 64, 0, st, a);
    sofia::launch_pdl(k_cluster_cells, 1, 1024, 0, st, a);
    sofia::launch_pdl(k_cluster_density, sofia::grid_for(n_gly, 4), 128, 0, st, a);
    sofia::launch_pdl(k_cluster_hook, sofia::grid_for(n_gly, 4), 128, 0, st, a);
    sofia::launch_pdl(k_cluster_result, 1, 1024, 0, st, a, (int)*greatest_belongsto);
    SOFIA_CUDA(ctx, cudaGetLastError());
    if ((rc = sofia::finish_out(ctx, o_ptta))) return rc;
    // size, cluster number and density-list overflows into pinned words
    int32_t *res = ctx->h_status;
    SOFIA_CUDA(ctx, cudaMemcpyAsync(res, a.result, sizeof(int32_t) * 3, cudaMemcpyDeviceToHost, st));
    for (const auto &o : {std::make_pair(denstrack, a.denstrack), std::make_pair(belongsto, a.label)}) {
        if (!o.first) continue;
        if (sofia::is_device_ptr(o.first))
            SOFIA_CUDA(ctx, cudaMemcpyAsync(o.first, o.second, sizeof(int) * n,
                                            cudaMemcpyDeviceToDevice, st));
        else if ((rc = copies.out(o.first, o.second, sizeof(int) * n)))
            return rc;
    }
    if ((rc = copies.sync())) return rc;
    if (res[2])
        return sofia::fail(ctx, SOFIA_EINVAL, "density list overflow (more than 256 entries)%s");
    *size_out = res[0];
    *greatest_belongsto = res[1];
    return SOFIA_OK;
}
