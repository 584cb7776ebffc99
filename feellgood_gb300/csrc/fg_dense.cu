// The demagnetising potential as a dense matrix over the nodes.
//
// The direct sum phi_i = sum_s q_s / (4 pi |x_i - y_s|) + corrections is linear in the field: the
// charges of a tetrahedron are -Ms detJ w_g sum_a da_a . m_a, those of a triangle and its
// self-corrections dMs (...) n . m_k (Tet::charges, Tri::charges, Tri::correctionCharges and
// Tri::potential, src/tetra.cpp:347-359, src/triangle.cpp:45-125). With the geometry fixed,
// phi_i = sum_j B_ij . m_j with one 3-vector per pair of magnetic nodes. A context of the direct
// sum forms B once, in FP64 and in the order of the charges' own sums over Gauss points, and an
// evaluation is one pass over it for both fields: 24 bytes and 6 FP64 fused multiply-adds per pair
// of nodes instead of 26 (Gauss point, node) pairs of 13 operations each. Measured per evaluation
// of both fields: 9,261 nodes (48,000 tetrahedra, B 2.06 GB) 0.93 ms, of which the FP64 pipe (2 per
// clock and SM) needs 0.82 and HBM 0.30; the sum over Gauss points took 58 ms on that pipe. 1,680
// nodes 0.061 ms, 180 nodes 0.013. Forming B costs about one such sum. Against quadruple
// precision the potentials are as exact as those sums (6e-16 for a smooth field of 1,680 nodes).
#include <algorithm>

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
// what is free. Without it (direct_mat null) the sum over Gauss points runs.
cudaError_t dense_build(Ctx &c, const Rules &R) {
    const int n = c.n_mag_nodes;
    size_t free_b = 0, total_b = 0;
    cudaError_t e = cudaMemGetInfo(&free_b, &total_b);
    if (e != cudaSuccess) return e;
    const size_t bytes = 24 * (size_t)n * n, ncol = (size_t)c.nmt + 3 * (size_t)c.nft;
    if (n == 0 || bytes > std::min(total_b / 16, free_b / 2)) return cudaSuccess;
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
