// The demagnetising potential as a dense matrix over the nodes.
//
// The direct sum phi_i = sum_s q_s / (4 pi |x_i - y_s|) + corrections is linear in the field: the
// charges of a tetrahedron are -Ms detJ w_g sum_a da_a . m_a, those of a triangle and its
// self-corrections dMs (...) n . m_k (Tet::charges, Tri::charges, Tri::correctionCharges and
// Tri::potential, src/tetra.cpp:347-359, src/triangle.cpp:45-125). With the geometry fixed,
// phi_i = sum_j B_ij . m_j with one 3-vector per pair of magnetic nodes. A context of the direct
// sum forms B once, in FP64 and in the order of the charges' own sums over Gauss points, and an
// evaluation is one pass over it for both fields: 24 bytes and 6 FP64 fused multiply-adds per pair
// of nodes instead of 26 (Gauss point, node) pairs of 15 operations' time each. Measured per evaluation
// of both fields: 9,261 nodes (48,000 tetrahedra, B 2.06 GB) 0.93 ms, of which the FP64 pipe (2 per
// clock and SM) needs 0.82 and HBM 0.30; the sum over Gauss points takes 59 ms on that pipe. 1,680
// nodes 0.061 ms, 180 nodes 0.013. Forming B costs about one such sum. Against quadruple
// precision the potentials are as exact as those sums (6e-16 for a smooth field of 1,680 nodes).
#include <algorithm>
#include <vector>

#include "fg_ds.cuh"
#include "fg_internal.h"

namespace fg {

namespace {

constexpr int ROWS = 32;  // nodes per build launch: one lane each

// G[e][r], e < nmt: sum_g w_g / |x_r - y_g| of a tetrahedron's Gauss points; e = nmt + 3 f + k:
// sum_g w_g a_k(g) / |x_r - y_g| of a triangle's. One warp per element, lane r = node row0 + r.
__global__ void __launch_bounds__(256) k_dense_geometry(int n, int row0, const int *__restrict__ nodes,
                                                        const double *__restrict__ xyz, int nmt, int nft,
                                                        const double *__restrict__ src, const DevTri *__restrict__ tc,
                                                        Rules R, double *__restrict__ G) {
    const int e = blockIdx.x * 8 + (threadIdx.x >> 5), lane = threadIdx.x & 31;
    if (e >= nmt + nft) return;
    const size_t i = 3 * (size_t)nodes[min(row0 + lane, n - 1)];
    const double x = xyz[i], y = xyz[i + 1], z = xyz[i + 2];
    const bool is_tet = e < nmt;
    const int f = e - nmt, np = is_tet ? R.npi_t : R.npi_f;
    const double *p = src + 3 * (is_tet ? (size_t)e * R.npi_t : (size_t)nmt * R.npi_t + (size_t)f * R.npi_f);
    double s[3] = {0.0, 0.0, 0.0};
    for (int g = 0; g < np; g++) {
        const double dx = x - p[3 * g], dy = y - p[3 * g + 1], dz = z - p[3 * g + 2];
        const double r = rsqrt(dx * dx + dy * dy + dz * dz);
        if (is_tet) {
            s[0] += R.tp[g] * r;
        } else {
            const double w = tc[f].w[g] * r;
            s[0] += w * R.fa[0][g];
            s[1] += w * R.fa[1][g];
            s[2] += w * R.fa[2][g];
        }
    }
    if (is_tet) {
        G[(size_t)e * ROWS + lane] = s[0];
    } else {
#pragma unroll
        for (int k = 0; k < 3; k++) G[((size_t)nmt + 3 * (size_t)f + k) * ROWS + lane] = s[k];
    }
}

// B of the rows row0 ..: one warp per column node, lane = row; the node's tetrahedra and triangles
// in the order of their incidence lists.
__global__ void __launch_bounds__(256) k_dense_rows(int n, int row0, const int *__restrict__ nodes, int nmt,
                                                    const double *__restrict__ da, const double *__restrict__ detJ,
                                                    const int *__restrict__ treg, const DevRegion *__restrict__ regs,
                                                    const int *__restrict__ inc_ptr, const int *__restrict__ inc,
                                                    const int4 *__restrict__ tri, const DevTri *__restrict__ tc,
                                                    const int *__restrict__ tinc_ptr, const int *__restrict__ tinc,
                                                    const double *__restrict__ G, double *__restrict__ B) {
    const int j = blockIdx.x * 8 + (threadIdx.x >> 5), lane = threadIdx.x & 31;
    if (j >= n) return;
    const int node = nodes[j], row = row0 + lane, me = row < n ? nodes[row] : -1;
    double b[3] = {0.0, 0.0, 0.0};
    for (int k = inc_ptr[node]; k < inc_ptr[node + 1]; k++) {
        const int t = inc[k] >> 2, a = inc[k] & 3;
        const double q = -regs[treg[t]].Ms * detJ[t] * G[(size_t)t * ROWS + lane];
#pragma unroll
        for (int c = 0; c < 3; c++) b[c] += q * da[(3 * a + c) * (size_t)nmt + t];
    }
    for (int k = tinc_ptr[node]; k < tinc_ptr[node + 1]; k++) {
        const int f = tinc[k] / 3, a = tinc[k] % 3;
        const DevTri &T = tc[f];
        const int4 v = tri[f];
        const int own = me == v.x ? 0 : me == v.y ? 1 : me == v.z ? 2 : -1;
        double q = G[((size_t)nmt + 3 * (size_t)f + a) * ROWS + lane];
        if (own >= 0) q += T.beta[3 * own + a];
        q *= T.dMs;
#pragma unroll
        for (int c = 0; c < 3; c++) b[c] += q * T.n[c];
    }
    if (row < n) {
        double *o = B + (size_t)row * 3 * n + 3 * (size_t)j;
#pragma unroll
        for (int c = 0; c < 3; c++) o[c] = b[c] / (4 * M_PI);
    }
}

// phi = B m for NQ fields: 16 rows per block (two per warp), the columns of the block's share in
// tiles staged with the fields in shared memory; partial sums [set][share][row], or the potentials
// themselves where there is one share.
constexpr int MV_ROWS = 16, MV_TILE = 128;  // rows per block, nodes per tile
template <int NQ>
__global__ void __launch_bounds__(256) k_dense_mv(int n, const int *__restrict__ nodes, const double *__restrict__ B,
                                                  const double *__restrict__ m0, const double *__restrict__ m1,
                                                  double *__restrict__ part, double *__restrict__ phi0,
                                                  double *__restrict__ phi1) {
    __shared__ double sm[3 * MV_TILE][NQ];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int r0 = blockIdx.x * MV_ROWS + 2 * warp, r1 = min(r0 + 1, n - 1);
    const int nshare = gridDim.y;
    const int c0 = (int)((long long)n * blockIdx.y / nshare), c1 = (int)((long long)n * (blockIdx.y + 1) / nshare);
    const double *b0 = B + (size_t)min(r0, n - 1) * 3 * n, *b1 = B + (size_t)r1 * 3 * n;
    double s[2][NQ];
#pragma unroll
    for (int q = 0; q < NQ; q++) s[0][q] = s[1][q] = 0.0;
    for (int base = c0; base < c1; base += MV_TILE) {
        const int len = 3 * min(MV_TILE, c1 - base);
        __syncthreads();
        for (int e = threadIdx.x; e < len; e += 256) {
            const size_t o = 3 * (size_t)nodes[base + e / 3] + e % 3;
            sm[e][0] = m0[o];
            if constexpr (NQ == 2) sm[e][1] = m1[o];
        }
        __syncthreads();
        const double *p0 = b0 + 3 * (size_t)base, *p1 = b1 + 3 * (size_t)base;
#pragma unroll 4
        for (int e = lane; e < len; e += 32) {
            const double x0 = __ldcs(p0 + e), x1 = __ldcs(p1 + e);
#pragma unroll
            for (int q = 0; q < NQ; q++) {
                s[0][q] = fma(x0, sm[e][q], s[0][q]);
                s[1][q] = fma(x1, sm[e][q], s[1][q]);
            }
        }
    }
#pragma unroll
    for (int h = 0; h < 2; h++)
#pragma unroll
        for (int q = 0; q < NQ; q++)
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) s[h][q] += __shfl_xor_sync(0xffffffffu, s[h][q], o);
    if (lane < 2 && r0 + lane < n) {
#pragma unroll
        for (int q = 0; q < NQ; q++) {
            const double v = lane ? s[1][q] : s[0][q];
            if (nshare > 1) part[((size_t)q * nshare + blockIdx.y) * n + r0 + lane] = v;
            else (q ? phi1 : phi0)[nodes[r0 + lane]] = v;
        }
    }
}

__global__ void k_dense_sum(int n, const int *__restrict__ nodes, int nshare, const double *__restrict__ part,
                            double *__restrict__ phi0, double *__restrict__ phi1) {
    const int k = blockIdx.x * blockDim.x + threadIdx.x;
    if (k >= n) return;
    const double *p = part + (size_t)blockIdx.y * nshare * n + k;
    double v = 0.0;
    for (int b = 0; b < nshare; b++) v += p[(size_t)b * n];
    (blockIdx.y ? phi1 : phi0)[nodes[k]] = v;
}

}  // namespace

// Forms B where it fits: at most 1/16 of the device's memory (12,000 nodes take 3.5 GB) and half of
// what is free, unless fg_opts.demag_blocks asks for it or against it. Without it (direct_mat null)
// the sum over Gauss points runs.
cudaError_t dense_build(Ctx &c, const Rules &R) {
    const int n = c.n_mag_nodes;
    size_t free_b = 0, total_b = 0;
    cudaError_t e = cudaMemGetInfo(&free_b, &total_b);
    if (e != cudaSuccess) return e;
    const size_t bytes = 24 * (size_t)n * n, ncol = (size_t)c.nmt + 3 * (size_t)c.nft;
    if (n == 0 || c.opts.demag_blocks == 1) return cudaSuccess;
    if (c.opts.demag_blocks == 0 && bytes > std::min(total_b / 16, free_b / 2)) return cudaSuccess;
    double *G = nullptr;
    // shares of the columns: 8 blocks per SM in all (the last wave costs little and the FP64 pipe of
    // every SM is busy), at least 32 nodes in each
    const int rows = (n + MV_ROWS - 1) / MV_ROWS;
    c.dense_nshare = std::max(1, std::min((8 * c.nsm + rows - 1) / rows, n / 32));
    if (cudaMalloc(&c.direct_mat, bytes) != cudaSuccess || cudaMalloc(&G, ncol * ROWS * sizeof(double)) != cudaSuccess ||
        cudaMalloc(&c.direct_part, 2 * (size_t)c.dense_nshare * n * sizeof(double)) != cudaSuccess) {
        cudaGetLastError();
        for (void *p : {(void *)c.direct_mat, (void *)G, (void *)c.direct_part})
            if (p) cudaFree(p);
        c.direct_mat = c.direct_part = nullptr;
        return cudaSuccess;
    }
    for (int row0 = 0; row0 < n; row0 += ROWS) {
        k_dense_geometry<<<(c.nmt + c.nft + 7) / 8, 256, 0, c.stream>>>(n, row0, c.mag_nodes, c.xyz, c.nmt, c.nft, c.src_xyz,
                                                                       c.tri_c, R, G);
        k_dense_rows<<<(n + 7) / 8, 256, 0, c.stream>>>(n, row0, c.mag_nodes, c.nmt, c.da, c.detJ, c.treg, c.regs, c.inc_ptr,
                                                       c.inc, c.tri, c.tri_c, c.tinc_ptr, c.tinc, G, c.direct_mat);
    }
    e = cudaGetLastError();
    if (e == cudaSuccess) e = cudaStreamSynchronize(c.stream);
    cudaFree(G);
    return e;
}

cudaError_t launch_dense(Ctx &c, const double *m0, const double *m1, double *phi0, double *phi1) {
    const int n = c.n_mag_nodes;
    const dim3 grid((n + MV_ROWS - 1) / MV_ROWS, c.dense_nshare);
    (m1 ? k_dense_mv<2> : k_dense_mv<1>)<<<grid, 256, 0, c.stream>>>(n, c.mag_nodes, c.direct_mat, m0, m1, c.direct_part,
                                                                    phi0, phi1);
    if (c.dense_nshare > 1)
        k_dense_sum<<<dim3((n + 127) / 128, m1 ? 2 : 1), 128, 0, c.stream>>>(n, c.mag_nodes, c.dense_nshare, c.direct_part,
                                                                            phi0, phi1);
    return cudaGetLastError();
}

}  // namespace fg

// ---------------------------------------------------------------------------------
// Near field of the FP64 FMM as dense blocks over the nodes.
//
// The same linearity holds leaf by leaf: the potentials of a leaf's target nodes from the Gauss
// points of its adjacent leaves, plus the triangles' self-corrections, are a block of
// [targets][3 column nodes], the columns being the nodes of every element with a Gauss point
// there (an element whose points lie in near and far leaves contributes its near points only).
// Formed once in FP64, stored as double-single pairs (48 bits, the arithmetic of the pair sum it
// replaces), 8 bytes per entry: film of 1.2M tets 4.1 GB, read once per evaluation of both fields.

namespace fg {

namespace {

constexpr int HASH = 8192;      // slots of a leaf's tables in shared memory
constexpr int MAX_NODE = 4096;  // column nodes and elements a leaf may have
constexpr int MAX_ELEM = 6144;
constexpr int MAX_OWN = 1024;   // elements with a Gauss point in one leaf (P2M)
constexpr int TG = 8;           // targets formed together
constexpr int NRM = 100;        // reals per expansion

__device__ __forceinline__ int hash_of(int key) { return (int)(((unsigned)key * 2654435761u) >> 19); }

// Adds key to the table unless it holds more than `most` keys (the caller then gives the leaf up).
__device__ __forceinline__ int hash_add(int *tab, int key, int *count, int most) {
    int h = hash_of(key);
    for (;;) {
        if (*(volatile int *)count > most) return -1;
        const int prev = atomicCAS(&tab[h], -1, key);
        if (prev == -1) atomicAdd(count, 1);
        if (prev == -1 || prev == key) return h;
        h = (h + 1) & (HASH - 1);
    }
}
__device__ __forceinline__ int hash_find(const int *tab, int key) {
    for (int h = hash_of(key);; h = (h + 1) & (HASH - 1)) {
        const int k = tab[h];
        if (k == key) return h;
        if (k == -1) return -1;
    }
}

struct NearArgs {
    int own;  // 1: the sources of the leaf itself only (P2M), 0: those of its adjacent leaves
    int nleaf, nmt, npi_t, npi_f;
    const int *leaf_src, *leaf_tgt, *tgt_node, *near_ptr, *near_leaf, *src_orig;
    const int4 *tet, *tri;
    const int *tinc_ptr, *tinc;
};

// f(element, Gauss point) for every source of the leaf's adjacent leaves (or its own); elements are
// the magnetic tetrahedra, then the triangles. Every thread of the block takes part.
template <typename Fn>
__device__ __forceinline__ void near_sources(const NearArgs &a, int leaf, Fn &&f) {
    const int e0 = a.own ? 0 : a.near_ptr[leaf], e1 = a.own ? 1 : a.near_ptr[leaf + 1];
    for (int e = e0; e < e1; e++) {
        const int nl = a.own ? leaf : a.near_leaf[e];
        for (int s = a.leaf_src[nl] + threadIdx.x; s < a.leaf_src[nl + 1]; s += blockDim.x) {
            const int o = a.src_orig[s], nt = a.nmt * a.npi_t;
            if (o < nt) f(o / a.npi_t, o % a.npi_t);
            else f(a.nmt + (o - nt) / a.npi_f, (o - nt) % a.npi_f);
        }
    }
}

// The column nodes of a leaf into the table `nodes`, its elements into `elems`.
__device__ __forceinline__ void near_tables(const NearArgs &a, int leaf, int *nodes, int *elems, int *nn, int *ne) {
    for (int k = threadIdx.x; k < HASH; k += blockDim.x) nodes[k] = elems[k] = -1;
    if (threadIdx.x == 0) *nn = *ne = 0;
    __syncthreads();
    near_sources(a, leaf, [&](int el, int) { hash_add(elems, el, ne, MAX_ELEM); });
    __syncthreads();
    auto add_tri = [&](int f) {
        const int4 v = a.tri[f];
        hash_add(nodes, v.x, nn, MAX_NODE);
        hash_add(nodes, v.y, nn, MAX_NODE);
        hash_add(nodes, v.z, nn, MAX_NODE);
    };
    for (int k = threadIdx.x; k < HASH; k += blockDim.x) {
        const int el = elems[k];
        if (el < 0) continue;
        if (el < a.nmt) {
            const int4 v = a.tet[el];
            hash_add(nodes, v.x, nn, MAX_NODE);
            hash_add(nodes, v.y, nn, MAX_NODE);
            hash_add(nodes, v.z, nn, MAX_NODE);
            hash_add(nodes, v.w, nn, MAX_NODE);
        } else {
            add_tri(el - a.nmt);
        }
    }
    // the self-corrections reach the nodes of every triangle of a target
    for (int t = a.leaf_tgt[leaf] + threadIdx.x; !a.own && t < a.leaf_tgt[leaf + 1]; t += blockDim.x) {
        const int i = a.tgt_node[t];
        for (int k = a.tinc_ptr[i]; k < a.tinc_ptr[i + 1]; k++) add_tri(a.tinc[k] / 3);
    }
    __syncthreads();
}

// Columns of every leaf, and the most elements of one (the largest int where a leaf has too many nodes).
__global__ void __launch_bounds__(256) k_near_count(NearArgs a, int *ncol, int *most) {
    extern __shared__ int tab[];
    __shared__ int nn, ne;
    const int leaf = blockIdx.x;
    const int *range = a.own ? a.leaf_src : a.leaf_tgt;
    if (range[leaf] == range[leaf + 1]) {
        if (threadIdx.x == 0) ncol[leaf] = 0;
        return;
    }
    near_tables(a, leaf, tab, tab + HASH, &nn, &ne);
    if (threadIdx.x == 0) {
        ncol[leaf] = nn;
        atomicMax(most, nn > MAX_NODE ? 0x7fffffff : ne);
    }
}

// The columns of every leaf in ascending order (cptr: first column, padded to an even number with -1).
__global__ void __launch_bounds__(256) k_near_cols(NearArgs a, const int *cptr, const int *ncol, int *col) {
    extern __shared__ int tab[];
    __shared__ int nn, ne, cnt;
    const int leaf = blockIdx.x, n = ncol[leaf];
    if (n == 0) return;
    near_tables(a, leaf, tab, tab + HASH, &nn, &ne);
    if (threadIdx.x == 0) cnt = 0;
    int *list = tab + HASH;
    int m = 1;
    while (m < n) m <<= 1;
    for (int k = threadIdx.x; k < m; k += 256) list[k] = 0x7fffffff;
    __syncthreads();
    for (int k = threadIdx.x; k < HASH; k += 256)
        if (tab[k] >= 0) list[atomicAdd(&cnt, 1)] = tab[k];
    for (int size = 2; size <= m; size <<= 1)
        for (int s = size >> 1; s > 0; s >>= 1) {
            __syncthreads();
            for (int k = threadIdx.x; k < m; k += 256) {
                const int p = k ^ s;
                if (p > k && (list[k] > list[p]) == ((k & size) == 0)) {
                    const int t = list[k];
                    list[k] = list[p];
                    list[p] = t;
                }
            }
        }
    __syncthreads();
    for (int k = threadIdx.x; k < cptr[leaf + 1] - cptr[leaf]; k += 256) col[cptr[leaf] + k] = k < n ? list[k] : -1;
}

// The entries of every leaf's block, 8 targets at a time: G[slot][target] = sum over a tetrahedron's
// near Gauss points of w_g / r, then a thread per column node gathers its tetrahedra (in the
// order of its incidence list) and triangles.
__global__ void __launch_bounds__(256) k_near_fill(NearArgs a, Rules R, const int *__restrict__ cptr,
                                                   const int *__restrict__ col, const size_t *__restrict__ boff,
                                                   const double *__restrict__ xyz, const double *__restrict__ src,
                                                   const double *__restrict__ da, const double *__restrict__ detJ,
                                                   const int *__restrict__ treg, const DevRegion *__restrict__ regs,
                                                   const int *__restrict__ inc_ptr, const int *__restrict__ inc,
                                                   const DevTri *__restrict__ tc, double *__restrict__ scratch,
                                                   float2 *__restrict__ B) {
    extern __shared__ int tab[];
    int *mask = tab + HASH;
    __shared__ double tx[TG][3];
    __shared__ int tn[TG], ne;
    double *G = scratch + (size_t)blockIdx.x * HASH * TG;
    for (int leaf = blockIdx.x; leaf < a.nleaf; leaf += gridDim.x) {
        const int t0 = a.leaf_tgt[leaf], t1 = a.leaf_tgt[leaf + 1], c0 = cptr[leaf], nc = cptr[leaf + 1] - c0;
        if (t0 == t1) continue;
        __syncthreads();
        for (int k = threadIdx.x; k < HASH; k += 256) {
            tab[k] = -1;
            mask[k] = 0;
        }
        if (threadIdx.x == 0) ne = 0;
        __syncthreads();
        near_sources(a, leaf, [&](int el, int g) {
            const int h = hash_add(tab, el, &ne, MAX_ELEM);
            if (h >= 0) atomicOr(&mask[h], 1 << g);
        });
        for (int tb = t0; tb < t1; tb += TG) {
            const int nt = min(TG, t1 - tb);
            __syncthreads();
            if (threadIdx.x < TG) {
                const int i = a.tgt_node[tb + min((int)threadIdx.x, nt - 1)];
                tn[threadIdx.x] = i;
                for (int d = 0; d < 3; d++) tx[threadIdx.x][d] = xyz[3 * (size_t)i + d];
            }
            __syncthreads();
            for (int k = threadIdx.x; k < HASH; k += 256) {
                const int el = tab[k], mk = mask[k];
                if (el < 0 || el >= a.nmt) continue;
                double s[TG];
#pragma unroll
                for (int t = 0; t < TG; t++) s[t] = 0.0;
                for (int g = 0; g < R.npi_t; g++) {
                    if (!(mk >> g & 1)) continue;
                    const double *p = src + 3 * ((size_t)el * R.npi_t + g);
                    const double px = p[0], py = p[1], pz = p[2], w = R.tp[g];
#pragma unroll
                    for (int t = 0; t < TG; t++) {
                        const double dx = tx[t][0] - px, dy = tx[t][1] - py, dz = tx[t][2] - pz;
                        s[t] += w * rsqrt(dx * dx + dy * dy + dz * dz);
                    }
                }
#pragma unroll
                for (int t = 0; t < TG; t++) G[(size_t)k * TG + t] = s[t];
            }
            __syncthreads();
            for (int j = threadIdx.x; j < nc; j += 256) {
                const int node = col[c0 + j];
                double b[TG][3];
#pragma unroll
                for (int t = 0; t < TG; t++) b[t][0] = b[t][1] = b[t][2] = 0.0;
                if (node >= 0) {
                    for (int q = inc_ptr[node]; q < inc_ptr[node + 1]; q++) {
                        const int el = inc[q] >> 2, v = inc[q] & 3, h = hash_find(tab, el);
                        if (h < 0) continue;
                        const double w = -regs[treg[el]].Ms * detJ[el];
                        double k[3];
#pragma unroll
                        for (int c = 0; c < 3; c++) k[c] = w * da[(3 * v + c) * (size_t)a.nmt + el];
#pragma unroll
                        for (int t = 0; t < TG; t++) {
                            const double g = G[(size_t)h * TG + t];
#pragma unroll
                            for (int c = 0; c < 3; c++) b[t][c] += k[c] * g;
                        }
                    }
                    for (int q = a.tinc_ptr[node]; q < a.tinc_ptr[node + 1]; q++) {
                        const int f = a.tinc[q] / 3, v = a.tinc[q] % 3, h = hash_find(tab, a.nmt + f);
                        const int mk = h >= 0 ? mask[h] : 0;
                        const DevTri &T = tc[f];
                        const int4 vt = a.tri[f];
#pragma unroll
                        for (int t = 0; t < TG; t++) {
                            double g = 0.0;
                            for (int p = 0; p < R.npi_f; p++) {
                                if (!(mk >> p & 1)) continue;
                                const double *y = src + 3 * ((size_t)a.nmt * R.npi_t + (size_t)f * R.npi_f + p);
                                const double dx = tx[t][0] - y[0], dy = tx[t][1] - y[1], dz = tx[t][2] - y[2];
                                g += T.w[p] * R.fa[v][p] * rsqrt(dx * dx + dy * dy + dz * dz);
                            }
                            const int own = tn[t] == vt.x ? 0 : tn[t] == vt.y ? 1 : tn[t] == vt.z ? 2 : -1;
                            if (own >= 0) g += T.beta[3 * own + v];
                            g *= T.dMs;
#pragma unroll
                            for (int c = 0; c < 3; c++) b[t][c] += g * T.n[c];
                        }
                    }
                }
#pragma unroll
                for (int t = 0; t < TG; t++) {
                    if (t >= nt) break;
                    float2 *o = B + boff[leaf] + (size_t)(tb + t - t0) * 3 * nc + 3 * j;
#pragma unroll
                    for (int c = 0; c < 3; c++) {
                        const double v = b[t][c] / (4 * M_PI);
                        const float h = (float)v;
                        o[c] = make_float2(h, (float)(v - (double)h));
                    }
                }
            }
        }
    }
}

// The multipoles of a leaf as a block [100][3 columns] over the nodes of its own sources' elements:
// W[slot][k] = sum over the element's Gauss points in the leaf of w_g conj(Ups_k)(y_g) (a triangle
// counts as three elements, one per shape function; a block's scratch holds `rows` of them), then a
// warp per column node gathers its elements, lanes = coefficients. One thread forms one harmonic
// column of one element.
__global__ void __launch_bounds__(256) k_p2m_fill(NearArgs a, Rules R, const int *__restrict__ cptr,
                                                  const int *__restrict__ col, const size_t *__restrict__ boff,
                                                  const int *__restrict__ src_pos, const double4 *__restrict__ sloc,
                                                  const double *__restrict__ da, const double *__restrict__ detJ,
                                                  const int *__restrict__ treg, const DevRegion *__restrict__ regs,
                                                  const int *__restrict__ inc_ptr, const int *__restrict__ inc,
                                                  const DevTri *__restrict__ tc, int rows,
                                                  double *__restrict__ scratch, float2 *__restrict__ B) {
    constexpr int P = 9;
    extern __shared__ int tab[];
    int *mask = tab + HASH, *list = mask + HASH;  // the table, its masks, the occupied slots
    __shared__ int ne, nl;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    double *W = scratch + (size_t)blockIdx.x * rows * NRM;
    for (int leaf = blockIdx.x; leaf < a.nleaf; leaf += gridDim.x) {
        const int c0 = cptr[leaf], nc = cptr[leaf + 1] - c0;
        if (nc == 0) continue;
        __syncthreads();
        for (int k = threadIdx.x; k < HASH; k += 256) {
            tab[k] = -1;
            mask[k] = 0;
        }
        if (threadIdx.x == 0) ne = nl = 0;
        __syncthreads();
        near_sources(a, leaf, [&](int el, int g) {
            const bool tet = el < a.nmt;
            for (int k = 0; k < (tet ? 1 : 3); k++) {
                const int h = hash_add(tab, tet ? el : a.nmt + 3 * (el - a.nmt) + k, &ne, 3 * MAX_OWN);
                if (h >= 0) atomicOr(&mask[h], 1 << g);
            }
        });
        __syncthreads();
        for (int k = threadIdx.x; k < HASH; k += 256)
            if (tab[k] >= 0) {
                const int n = atomicAdd(&nl, 1);
                list[n] = k;
                mask[k] |= n << 8;  // row of W
            }
        __syncthreads();
        for (int q = threadIdx.x; q < nl * (P + 1); q += 256) {
            const int k = list[q / (P + 1)], m = q % (P + 1), el = tab[k], mk = mask[k] & 255;
            const bool tet = el < a.nmt;
            const int f = (el - a.nmt) / 3, v = (el - a.nmt) % 3, np = tet ? R.npi_t : R.npi_f;
            double re[P + 1], im[P + 1];
#pragma unroll
            for (int n = 0; n <= P; n++) re[n] = im[n] = 0.0;
            for (int g = 0; g < np; g++) {
                if (!(mk >> g & 1)) continue;
                const size_t o = tet ? (size_t)el * R.npi_t + g : (size_t)a.nmt * R.npi_t + (size_t)f * R.npi_f + g;
                const double4 y = sloc[src_pos[o]];
                const double w = tet ? R.tp[g] : tc[f].w[g] * R.fa[v][g];
                double dr = w, di = 0.0;  // the column's diagonal, times the weight
                for (int i = 1; i <= m; i++) {
                    const double t = (y.x * dr - y.y * di) / (2 * i);
                    di = (y.x * di + y.y * dr) / (2 * i);
                    dr = t;
                }
                const double r2 = y.x * y.x + y.y * y.y + y.z * y.z;
                double p2r = 0.0, p2i = 0.0, p1r = dr, p1i = di;
#pragma unroll
                for (int n = 0; n <= P; n++) {  // degree n >= m
                    if (n < m) continue;
                    re[n] += p1r;
                    im[n] += p1i;
                    const int d = n + 1;
                    const double b = d == m + 1 ? 1.0 : 1.0 / double((d + m) * (d - m));
                    const double az = (d == m + 1 ? 1.0 : 2 * d - 1) * y.z;
                    const double nr = (az * p1r - r2 * p2r) * b, ni = (az * p1i - r2 * p2i) * b;
                    p2r = p1r; p2i = p1i;
                    p1r = nr; p1i = ni;
                }
            }
            double *w = W + (size_t)(mask[k] >> 8) * NRM;
#pragma unroll
            for (int n = 0; n <= P; n++) {
                if (n < m) continue;
                if (m == 0) w[n * n] = re[n];
                else {
                    w[n * n + 2 * m - 1] = re[n];
                    w[n * n + 2 * m] = -im[n];
                }
            }
        }
        __syncthreads();
        for (int j = warp; j < nc; j += 8) {
            const int node = col[c0 + j];
            double b[4][3];
#pragma unroll
            for (int i = 0; i < 4; i++) b[i][0] = b[i][1] = b[i][2] = 0.0;
            auto gather = [&](int key, double kx, double ky, double kz) {
                const int h = hash_find(tab, key);
                if (h < 0) return;
                const double *w = W + (size_t)(mask[h] >> 8) * NRM;
#pragma unroll
                for (int i = 0; i < 4; i++) {
                    const int k = lane + 32 * i;
                    const double x = k < NRM ? w[k] : 0.0;
                    b[i][0] += kx * x;
                    b[i][1] += ky * x;
                    b[i][2] += kz * x;
                }
            };
            if (node >= 0) {
                for (int q = inc_ptr[node]; q < inc_ptr[node + 1]; q++) {
                    const int el = inc[q] >> 2, v = inc[q] & 3;
                    const double w = -regs[treg[el]].Ms * detJ[el];
                    gather(el, w * da[(3 * v) * (size_t)a.nmt + el], w * da[(3 * v + 1) * (size_t)a.nmt + el],
                           w * da[(3 * v + 2) * (size_t)a.nmt + el]);
                }
                for (int q = a.tinc_ptr[node]; q < a.tinc_ptr[node + 1]; q++) {
                    const DevTri &T = tc[a.tinc[q] / 3];
                    gather(a.nmt + a.tinc[q], T.dMs * T.n[0], T.dMs * T.n[1], T.dMs * T.n[2]);
                }
            }
#pragma unroll
            for (int i = 0; i < 4; i++) {
                const int k = lane + 32 * i;
                if (k >= NRM) continue;
                float2 *o = B + boff[leaf] + (size_t)k * 3 * nc + 3 * j;
#pragma unroll
                for (int c = 0; c < 3; c++) {
                    const float h = (float)b[i][c];
                    o[c] = make_float2(h, (float)(b[i][c] - (double)h));
                }
            }
        }
    }
}

// The fields as double-single pairs: (u hi, u lo, v hi, v lo) per component.
__global__ void k_field_pairs(size_t n3, const double *__restrict__ u, const double *__restrict__ v,
                              float4 *__restrict__ m) {
    const size_t k = blockIdx.x * (size_t)blockDim.x + threadIdx.x;
    if (k >= n3) return;
    const double x = u[k], y = v ? v[k] : 0.0;
    const float xh = (float)x, yh = (float)y;
    m[k] = make_float4(xh, (float)(x - (double)xh), yh, (float)(y - (double)yh));
}

// Rows of the blocks times NQ fields: a block per task (some rows of a leaf), two rows per warp at a
// time, the column nodes' fields staged in shared memory in tiles of TILE entries (once where one
// tile holds them), two entries of a row per 16-byte load. 12 FP32 operations per entry and field
// (product with its rounding error and cross terms, two-sum), 8 bytes of the block: HBM bounds
// it. The next two steps' loads are issued before a step is used, the first ones before the staging,
// in 64 registers (near field and L2P of the film 0.93 -> 0.83 ms, wire 0.57 -> 0.50; the same in 80
// registers 0.90, the loop unrolled by four without it 0.86 but P2M 0.48 -> 0.53). Row r goes to out[rows ? rows[first + r] : first + r].
constexpr int TILE = 1536;
template <int NQ>
__global__ void __launch_bounds__(256, 4) k_block_mv(const int4 *__restrict__ task, const int *__restrict__ rows,
                                                  const int *__restrict__ cptr, const int *__restrict__ col,
                                                  const size_t *__restrict__ boff, const float2 *__restrict__ B,
                                                  const float4 *__restrict__ m, double *__restrict__ out0,
                                                  double *__restrict__ out1) {
    __shared__ float4 sm[TILE];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int4 t = task[blockIdx.x];  // leaf, first row of its block, rows, first output
    const int c0 = cptr[t.x], ne = 3 * (cptr[t.x + 1] - c0);
    auto add = [&](float &hi, float &lo, float bh, float bl, float mh, float ml) {
        const float p = bh * mh;
        const float e = fmaf(bl, mh, fmaf(bh, ml, fmaf(bh, mh, -p)));
        const float s = hi + p, x = s - hi;
        lo += ((hi - (s - x)) + (p - x)) + e;
        hi = s;
    };
    for (int r0 = 0; r0 < t.z; r0 += 16) {
        const int r = r0 + 2 * warp;
        const bool on0 = r < t.z, on1 = r + 1 < t.z;
        const float2 *b0 = B + boff[t.x] + (size_t)(t.y + (on0 ? r : 0)) * ne;
        const float2 *b1 = on1 ? b0 + ne : b0;
        float h[2][NQ], l[2][NQ];
#pragma unroll
        for (int q = 0; q < NQ; q++) h[0][q] = h[1][q] = l[0][q] = l[1][q] = 0.f;
        for (int base = 0; base < ne; base += TILE) {
            const int len = min(TILE, ne - base), n = on0 ? len / 2 : 0;
            const float4 *p0 = reinterpret_cast<const float4 *>(b0 + base), *p1 = reinterpret_cast<const float4 *>(b1 + base);
            // two steps of both rows in flight, the first ones while the fields are staged
            float4 x[2][2];
            auto load = [&](int e) {
#pragma unroll
                for (int k = 0; k < 2; k++)
                    if (e + 32 * k < n) {
                        x[k][0] = __ldcs(p0 + e + 32 * k);
                        x[k][1] = __ldcs(p1 + e + 32 * k);
                    }
            };
            load(lane);
            if (r0 == 0 || ne > TILE) {
                __syncthreads();
                for (int e = threadIdx.x; e < len; e += 256) {
                    const int node = col[c0 + (base + e) / 3];
                    sm[e] = node >= 0 ? m[3 * (size_t)node + (base + e) % 3] : make_float4(0.f, 0.f, 0.f, 0.f);
                }
                __syncthreads();
            }
            for (int e = lane; e < n; e += 64) {
                const float4 y[2][2] = {{x[0][0], x[0][1]}, {x[1][0], x[1][1]}};
                load(e + 64);
#pragma unroll
                for (int k = 0; k < 2; k++) {
                    if (e + 32 * k >= n) break;
                    const float4 x0 = y[k][0], x1 = y[k][1], ma = sm[2 * (e + 32 * k)], mb = sm[2 * (e + 32 * k) + 1];
                    add(h[0][0], l[0][0], x0.x, x0.y, ma.x, ma.y);
                    add(h[1][0], l[1][0], x1.x, x1.y, ma.x, ma.y);
                    add(h[0][0], l[0][0], x0.z, x0.w, mb.x, mb.y);
                    add(h[1][0], l[1][0], x1.z, x1.w, mb.x, mb.y);
                    if constexpr (NQ == 2) {
                        add(h[0][1], l[0][1], x0.x, x0.y, ma.z, ma.w);
                        add(h[1][1], l[1][1], x1.x, x1.y, ma.z, ma.w);
                        add(h[0][1], l[0][1], x0.z, x0.w, mb.z, mb.w);
                        add(h[1][1], l[1][1], x1.z, x1.w, mb.z, mb.w);
                    }
                }
            }
        }
        if (!on0) continue;
#pragma unroll
        for (int i = 0; i < 2; i++)
#pragma unroll
            for (int q = 0; q < NQ; q++) {
                dsf s = ds_quick(h[i][q], l[i][q]);
#pragma unroll
                for (int o = 16; o > 0; o >>= 1)
                    s = ds_add(s, dsf{__shfl_xor_sync(0xffffffffu, s.h, o), __shfl_xor_sync(0xffffffffu, s.l, o)});
                if (lane == 0 && (i == 0 || on1)) {
                    const size_t k = (size_t)t.w + r + i;
                    (q ? out1 : out0)[rows ? rows[k] : k] = ds_to(s);
                }
            }
    }
}

// Local expansions at the targets from a table of the harmonics: T[k][target] = Ups_k of the
// target (doubled for m > 0), one thread per target, so the FP64 pipe does 100 operations per field
// instead of forming the harmonics (film: L2P 0.37 ms). phi = sum_k F_k T_k scale / (4 pi) + near.
__global__ void __launch_bounds__(128) k_l2p_table(int ntgt, const double4 *__restrict__ tloc, double *__restrict__ T) {
    constexpr int P = 9;
    const int t = blockIdx.x * 128 + threadIdx.x;
    if (t >= ntgt) return;
    const double4 y = tloc[t];
    const double r2 = y.x * y.x + y.y * y.y + y.z * y.z;
    double dr = 1.0, di = 0.0;
    for (int m = 0; m <= P; m++) {
        if (m) {
            const double s = (y.x * dr - y.y * di) / (2 * m);
            di = (y.x * di + y.y * dr) / (2 * m);
            dr = s;
        }
        double p2r = 0.0, p2i = 0.0, p1r = dr, p1i = di;
        for (int n = m; n <= P; n++) {
            if (m == 0) T[(size_t)(n * n) * ntgt + t] = p1r;
            else {
                T[(size_t)(n * n + 2 * m - 1) * ntgt + t] = 2.0 * p1r;
                T[(size_t)(n * n + 2 * m) * ntgt + t] = 2.0 * p1i;
            }
            const int d = n + 1;
            const double b = d == m + 1 ? 1.0 : 1.0 / double((d + m) * (d - m)), az = (d == m + 1 ? 1.0 : 2 * d - 1) * y.z;
            const double nr = (az * p1r - r2 * p2r) * b, ni = (az * p1i - r2 * p2i) * b;
            p2r = p1r; p2i = p1i;
            p1r = nr; p1i = ni;
        }
    }
}
template <int NQ>
__global__ void __launch_bounds__(128) k_l2p_apply(int ntgt, const int *__restrict__ tgt_leaf,
                                                   const int *__restrict__ tgt_node, const double *__restrict__ T,
                                                   const double *__restrict__ leaf_scale, const double *__restrict__ F0,
                                                   const double *__restrict__ F1, const double *__restrict__ near0,
                                                   const double *__restrict__ near1, double *__restrict__ phi0,
                                                   double *__restrict__ phi1) {
    const int t = blockIdx.x * 128 + threadIdx.x;
    if (t >= ntgt) return;
    const int leaf = tgt_leaf[t], node = tgt_node[t];
    const double *a = F0 + (size_t)leaf * NRM, *b = NQ == 2 ? F1 + (size_t)leaf * NRM : nullptr;
    double s0 = 0.0, s1 = 0.0;
#pragma unroll 10
    for (int k = 0; k < NRM; k++) {
        const double x = __ldcs(T + (size_t)k * ntgt + t);
        s0 = fma(a[k], x, s0);
        if constexpr (NQ == 2) s1 = fma(b[k], x, s1);
    }
    const double f = leaf_scale[leaf] / (4 * M_PI);
    phi0[node] = fma(s0, f, near0[node]);
    if constexpr (NQ == 2) phi1[node] = fma(s1, f, near1[node]);
}

}  // namespace

// Forms the blocks of one kind (own: P2M, else near field) where they fit: MAX_NODE columns and
// MAX_ELEM (MAX_OWN) elements per leaf and, unless fg_opts.demag_blocks asks for them, at most 1/8 of
// the device's memory and half of what is free. Without them (N.B null) the sums over Gauss points
// run; N.why then tells whether memory (FG_ENOMEM) or a leaf (FG_EINVAL) was the reason.
static cudaError_t blocks_build(Ctx &c, const Rules &R, const NearTree &t, bool own, DenseBlocks &N) {
    size_t free_b = 0, total_b = 0;
    cudaError_t e = cudaMemGetInfo(&free_b, &total_b);
    if (e != cudaSuccess) return e;
    NearArgs a{own, t.nleaf, c.nmt, R.npi_t, R.npi_f, t.leaf_src, t.leaf_tgt, t.tgt_node, t.near_ptr, t.near_leaf, t.src_orig,
               c.tet, c.tri, c.tinc_ptr, c.tinc};
    int *ncol = nullptr;
    double *scratch = nullptr;
    const int smem = 2 * HASH * (int)sizeof(int), smem_own = 3 * HASH * (int)sizeof(int);
    const int blocks = std::min(t.nleaf, 2 * std::max(1, c.nsm));
    auto done = [&](cudaError_t r) {
        if (ncol) cudaFree(ncol);
        if (scratch) cudaFree(scratch);
        if (r != cudaSuccess || !N.B) {
            const int why = r == cudaErrorMemoryAllocation ? FG_ENOMEM : N.why;
            blocks_free(N);
            N.why = why;
        }
        cudaGetLastError();
        // what does not fit is no error: the sums over Gauss points need none of it
        return r == cudaErrorMemoryAllocation ? cudaSuccess : r;
    };
#define NCK(call)                               \
    do {                                        \
        const cudaError_t r_ = (call);          \
        if (r_ != cudaSuccess) return done(r_); \
    } while (0)
    NCK(cudaFuncSetAttribute(k_near_count, cudaFuncAttributeMaxDynamicSharedMemorySize, smem));
    NCK(cudaFuncSetAttribute(k_near_cols, cudaFuncAttributeMaxDynamicSharedMemorySize, smem));
    NCK(cudaFuncSetAttribute(k_near_fill, cudaFuncAttributeMaxDynamicSharedMemorySize, smem));
    NCK(cudaFuncSetAttribute(k_p2m_fill, cudaFuncAttributeMaxDynamicSharedMemorySize, smem_own));
    NCK(cudaMalloc(&ncol, sizeof(int) * (t.nleaf + 1)));
    NCK(cudaMemsetAsync(ncol, 0, sizeof(int) * (t.nleaf + 1), c.stream));
    k_near_count<<<t.nleaf, 256, smem, c.stream>>>(a, ncol, ncol + t.nleaf);
    std::vector<int> hn(t.nleaf + 1);
    NCK(cudaMemcpyAsync(hn.data(), ncol, sizeof(int) * (t.nleaf + 1), cudaMemcpyDeviceToHost, c.stream));
    NCK(cudaStreamSynchronize(c.stream));
    N.why = FG_EINVAL;
    if (hn[t.nleaf] > (own ? MAX_OWN : MAX_ELEM)) return done(cudaSuccess);
    const int rows = 3 * hn[t.nleaf];  // P2M: the most that a leaf's elements take, all triangles
    std::vector<int> cptr(t.nleaf + 1, 0);
    std::vector<size_t> boff(t.nleaf, 0);
    std::vector<int4> task;
    size_t entries = 0, cols = 0;
    for (int l = 0; l < t.nleaf; l++) {
        const int nc = (hn[l] + 1) & ~1, nt = own ? NRM : t.h_leaf_tgt[l + 1] - t.h_leaf_tgt[l];
        cols += nc;
        if (cols > 0x7fffffff || (own && (size_t)t.nleaf * NRM > 0x7fffffff)) return done(cudaSuccess);
        cptr[l + 1] = (int)cols;
        boff[l] = entries;  // a leaf without columns has tasks too: its rows are zero
        entries += (size_t)nt * 3 * nc;
        // near field: up to 16 rows; P2M: all rows of a leaf (few columns), or 16 where a tile of
        // columns does not hold them
        const int most = own && 3 * nc <= TILE ? NRM : 16, groups = (nt + most - 1) / most;
        for (int g = 0; g < groups; g++) {
            const int b = (int)((long)nt * g / groups), f = (int)((long)nt * (g + 1) / groups);
            task.push_back(make_int4(l, b, f - b, (own ? NRM * l : t.h_leaf_tgt[l]) + b));
        }
    }
    if (entries == 0) return done(cudaSuccess);
    N.why = FG_ENOMEM;
    N.bytes = entries * sizeof(float2);
    if (c.opts.demag_blocks == 0 && N.bytes > std::min(total_b / 8, free_b / 2)) return done(cudaSuccess);
    N.ntask = (int)task.size();
    NCK(cudaMalloc(&scratch, sizeof(double) * (own ? (size_t)rows * NRM : (size_t)HASH * TG) * blocks));
    NCK(cudaMalloc(&N.cptr, sizeof(int) * (t.nleaf + 1)));
    NCK(cudaMalloc(&N.boff, sizeof(size_t) * t.nleaf));
    NCK(cudaMalloc(&N.task, sizeof(int4) * N.ntask));
    NCK(cudaMalloc(&N.col, sizeof(int) * cols));
    NCK(cudaMalloc(&N.B, sizeof(float2) * entries));
    auto filled = [&]() -> cudaError_t {
        cudaError_t r = cudaMemcpyAsync(N.cptr, cptr.data(), sizeof(int) * (t.nleaf + 1), cudaMemcpyHostToDevice, c.stream);
        if (r == cudaSuccess)
            r = cudaMemcpyAsync(N.boff, boff.data(), sizeof(size_t) * t.nleaf, cudaMemcpyHostToDevice, c.stream);
        if (r == cudaSuccess)
            r = cudaMemcpyAsync(N.task, task.data(), sizeof(int4) * N.ntask, cudaMemcpyHostToDevice, c.stream);
        if (r != cudaSuccess) return r;
        k_near_cols<<<t.nleaf, 256, smem, c.stream>>>(a, N.cptr, ncol, N.col);
        if (own)
            k_p2m_fill<<<blocks, 256, smem_own, c.stream>>>(a, R, N.cptr, N.col, N.boff, t.src_pos, t.sloc, c.da, c.detJ,
                                                            c.treg, c.regs, c.inc_ptr, c.inc, c.tri_c, rows, scratch,
                                                            N.B);
        else
            k_near_fill<<<blocks, 256, smem, c.stream>>>(a, R, N.cptr, N.col, N.boff, c.xyz, c.src_xyz, c.da, c.detJ, c.treg,
                                                         c.regs, c.inc_ptr, c.inc, c.tri_c, scratch, N.B);
        r = cudaGetLastError();
        return r == cudaSuccess ? cudaStreamSynchronize(c.stream) : r;
    };
    const cudaError_t r = filled();
    if (r != cudaSuccess) {
        cudaFree(N.B);
        N.B = nullptr;
    }
#undef NCK
    return done(r);
}

// The near field's blocks, the P2M blocks beside them, the fields' pairs and the L2P table.
cudaError_t near_build(Ctx &c, const Rules &R, const NearTree &t, NearMat &N) {
    cudaError_t e = blocks_build(c, R, t, false, N.near);
    if (e != cudaSuccess || !N.near.B) return e;
    if (c.opts.demag_blocks != 2) e = blocks_build(c, R, t, true, N.p2m);
    if (e != cudaSuccess) return e;
    if (cudaMalloc(&N.field, sizeof(float4) * 3 * (size_t)c.nn) != cudaSuccess ||
        cudaMalloc(&N.l2p, sizeof(double) * NRM * (size_t)std::max(1, t.ntgt)) != cudaSuccess) {
        cudaGetLastError();
        near_free(N);
        N.near.why = FG_ENOMEM;
        return cudaSuccess;
    }
    if (t.ntgt > 0) k_l2p_table<<<(t.ntgt + 127) / 128, 128, 0, c.stream>>>(t.ntgt, t.tloc, N.l2p);
    return cudaGetLastError();
}

void blocks_free(DenseBlocks &N) {
    for (void *p : {(void *)N.cptr, (void *)N.boff, (void *)N.task, (void *)N.col, (void *)N.B})
        if (p) cudaFree(p);
    N = DenseBlocks();
}
void near_free(NearMat &N) {
    blocks_free(N.near);
    blocks_free(N.p2m);
    if (N.field) cudaFree(N.field);
    if (N.l2p) cudaFree(N.l2p);
    N = NearMat();
}

cudaError_t launch_field_pairs(Ctx &c, const NearMat &N, const double *m0, const double *m1) {
    const size_t n3 = 3 * (size_t)c.nn;
    k_field_pairs<<<(unsigned)((n3 + 255) / 256), 256, 0, c.stream>>>(n3, m0, m1, N.field);
    return cudaGetLastError();
}

cudaError_t launch_blocks(const DenseBlocks &N, const NearMat &M, cudaStream_t st, int nq, const int *rows, double *out0,
                          double *out1) {
    if (N.ntask == 0) return cudaSuccess;
    (nq == 2 ? k_block_mv<2> : k_block_mv<1>)<<<N.ntask, 256, 0, st>>>(N.task, rows, N.cptr, N.col, N.boff, N.B, M.field,
                                                                      out0, out1);
    return cudaGetLastError();
}

cudaError_t launch_l2p_table(Ctx &c, const NearTree &t, const NearMat &N, int nq, const double *F0, const double *F1,
                             const double *near0, const double *near1, double *phi0, double *phi1) {
    if (t.ntgt == 0) return cudaSuccess;
    (nq == 2 ? k_l2p_apply<2> : k_l2p_apply<1>)<<<(t.ntgt + 127) / 128, 128, 0, c.stream>>>(
        t.ntgt, t.tgt_leaf, t.tgt_node, N.l2p, t.leaf_scale, F0, F1, near0, near1, phi0, phi1);
    return cudaGetLastError();
}

}  // namespace fg
