// Fast multipole evaluation of the demagnetising potential on the GPU.
//
// Replaces the ScalFMM octree + rotation kernel that fmm::demag calls
// (src/fmm_demag.h:184-224: P2M, M2M, M2L, L2L, L2P of 1/r plus the P2P near field).
// The potential computed is the same sum pot_i = sum_s q_s / |x_i - y_s| over the
// Gauss-point sources; only the evaluator differs.
//
// Expansions use the scaled solid harmonics
//   Ups_n^m(r) = (-1)^m r^n P_n^m(cos t) e^{i m p} / (n+m)!        (regular)
//   The_n^m(r) = (-1)^m (n-m)! P_n^m(cos t) e^{i m p} / r^{n+1}     (irregular)
// (P_n^m with the Condon-Shortley phase), for which 1/|x-y| = sum Ups_n^m*(y) The_n^m(x),
// Ups(a+b) = sum_kl Ups_k^l(a) Ups_{n-k}^{m-l}(b) and The(x-y) = sum Ups_k^l*(y) The_{n+k}^{m+l}(x).
// Multipoles M_n^m = sum q Ups_n^m*(y - z); locals F_n^m with phi = sum F_n^m Ups_n^m*(x - z).
// For real charges X_n^-m = (-1)^m conj X_n^m, so each expansion is stored as (P+1)^2 reals:
// Re X_n^0, then Re/Im X_n^m for m = 1..n. Coefficients of a cell of width w are stored
// scaled (M/w^n, F*w^(n+1)), which makes every translation independent of the level.
//
// Every translation (M2L for each of the 316 cell offsets, M2M and L2L for the 8 child
// octants) is then a fixed real 100x100 matrix, built once on the host. One kernel applies
// them: a block owns 64 output cells, walks the operator codes, gathers the 64 input
// expansions of that code and accumulates a register-tiled 100x100 x 100x64 product in a
// fixed order (deterministic, no atomics).
//
// The octree is uniform (all leaves on one level) and built once per mesh on the host
// (geometry is static). Interaction lists follow the one-cell separation: M2L over the
// children of the parent's neighbours that are not adjacent, P2P over adjacent leaves.
#include <algorithm>
#include <chrono>
#include <cmath>
#include <complex>
#include <cstdint>
#include <cstring>
#include <unordered_map>
#include <queue>
#include <type_traits>
#include <vector>

#include "fg_ds.cuh"
#include "fg_f32x2.cuh"
#include "fg_internal.h"

namespace fg {

constexpr int FMM_P = 9;
constexpr int NR = (FMM_P + 1) * (FMM_P + 1);  // reals per expansion (100)
constexpr int NCODE_M2L = 343;                   // offsets in [-3,3]^3 (27 unused)
// CUDA-core translations: output cells per block and per thread. FP64 uses narrow blocks
// of 16 cells (the FP64 pipe bounds them, so operator reuse matters less than spreading
// the blocks evenly over the SMs, two per SM); FP32 blocks of 64 cells.
template <typename T> struct TrShape;
template <> struct TrShape<float> { static constexpr int TB = 64, CT = 4; };
template <> struct TrShape<double> { static constexpr int TB = 16, CT = 1; };
template <typename T> constexpr int tr_smem() { return (int)((100 * 100 + 100 * (TrShape<T>::TB + 4)) * sizeof(T)); }

__host__ __device__ constexpr int cidx(int n, int m) { return n * (n + 1) / 2 + m; }
// real layout: Re X_n^0 at n*n; Re/Im X_n^m (m>0) at n*n + 2m-1, n*n + 2m
__host__ __device__ constexpr int ridx(int n, int m, int part) { return m == 0 ? n * n : n * n + 2 * m - 1 + part; }

struct FmmTree {
    int L = 0, nleaf = 0, ncell = 0, leaf0 = 0, nsrc = 0;
    double s0 = 1, c0[3] = {0, 0, 0};
    std::vector<int> lev_begin;
    size_t n_m2l = 0, n_p2p_pairs = 0;
    bool fp32 = false;
    double eval_ms = 0;
    // profiling: two sets of stage events used in turn (recorded without synchronising); a
    // set is read back when it is about to be reused or when the timings are requested
    cudaEvent_t ev[2][6] = {};
    cudaEvent_t evn[2][2] = {};          // the near field on the second stream (overlapped evaluation)
    bool ev_pending[2] = {false, false};
    bool ev_split[2] = {false, false};  // the set timed an overlapped evaluation
    int ev_next = 0;
    double stage_sum[5] = {0, 0, 0, 0, 0};
    long long stage_n = 0;
    // device
    int *leaf_src = nullptr, *leaf_tgt = nullptr, *tgt_node = nullptr, *tgt_leaf = nullptr;
    int ntgt = 0;
    void *sloc = nullptr;  // 4 x nsrc: leaf-local source coordinates (T), w: charge of set 0
    void *tloc = nullptr;  // 4 x ntgt: leaf-local target coordinates (T)
    // FP64 path, near field in double-single arithmetic: every coordinate split as
    // hi (on a 2^-20 grid of leaf units) + lo, the charge as hi + lo; (x, y, z, q) per part
    bool ds = false;
    // The FP64 tree of an FP32 + refinement context (full evaluations, where CURRENT has no valid
    // potentials) keeps the arithmetic and the order of the sums that such runs have always started
    // from: the FP32 Krylov body turns a difference of 1e-13 in the first potentials into 3e-9 in
    // phiv two steps later (film). Other deterministic kernels would repeat bit for bit as well; these
    // also agree with the results of earlier versions to the last bit
    bool repeat = false;
    NearMat near;              // oz: P2M and near field as dense blocks, where they fit
    int4 *p2p_task = nullptr;  // leaf, first target, targets of a near-field task
    int n_p2p_task = 0;
    float4 *ds_src_hi = nullptr, *ds_src_lo = nullptr, *ds_tgt_hi = nullptr, *ds_tgt_lo = nullptr;
    int *leaf_ijk = nullptr;  // 3 x nleaf integer leaf coordinates (within the leaf's own tree)
    double *leaf_scale = nullptr;  // 1 / physical leaf width of the leaf's tree
    int *m2l_tab = nullptr;   // [ncell][343] source cell or -1
    int *m2m_tab = nullptr;   // [ncell][8] child per octant or -1
    int *l2l_tab = nullptr;   // [ncell][8] parent at the own octant, -1 elsewhere
    int *near_ptr = nullptr, *near_leaf = nullptr;
    void *M = nullptr, *F = nullptr;
    void *op_m2l = nullptr, *op_m2m = nullptr, *op_l2l = nullptr;  // [code][NR][NR] (out x in)
    // tensor-core translations (FP32 path): per launch, for each tile of 64 output cells,
    // the list of operator codes that bring any input to the tile
    bool tc = false;
    int *tc_code = nullptr;                      // codes per tile, all launches
    int4 *tc_units = nullptr, *tc_comb = nullptr;
    float *tc_scratch = nullptr;
    struct TcLaunch { int unit0 = 0, nunit = 0, comb0 = 0, ncomb = 0; };
    std::vector<TcLaunch> tc_m2m, tc_l2l;        // per level
    TcLaunch tc_m2l;
    // FP64 path: translations by exact digit products on the tensor cores (fg_fmm_oz.cu)
    bool oz = false;
    struct OzLaunch { int unit0 = 0, nunit = 0, tile0 = 0, ntile = 0, nsplit = 0; };
    std::vector<OzLaunch> oz_m2m, oz_l2l;        // per level
    OzLaunch oz_m2l;
    int *oz_cells = nullptr, *oz_codes = nullptr, *oz_wexp = nullptr, *oz_leaves = nullptr;
    int4 *oz_units = nullptr;
    int2 *oz_fin = nullptr;
    float2 *oz_scratch = nullptr;
    unsigned char *oz_digits = nullptr;          // of M up to M2L, of F from there
    float *oz_scale = nullptr;
    unsigned char *oz_img[3] = {nullptr, nullptr, nullptr};  // M2M, M2L, L2L
    float *oz_rows[3] = {nullptr, nullptr, nullptr};
    // repeat: the lists (oz_cells, oz_codes, oz_units) are those of k_translate_ds, the images its
    // split operators, M holds pairs hi + lo, and F_split those of the locals above the leaves
    void *F_split = nullptr;
    float *Mh = nullptr, *Ml = nullptr, *Fh = nullptr, *Fl = nullptr;  // hi/lo splits of M and F
    unsigned char *img_m2l = nullptr, *img_m2m = nullptr, *img_l2l = nullptr;  // operator images
    int *dst_keep = nullptr;
    // charge sets evaluated together (2: demag of m and of v in one pass): M, F, Mh, Ml, Fh,
    // Fl and tc_scratch hold nq sets one after the other; the second set's charges for the
    // near field are in sq2 (T) and, double-single, in ds_q2 (hi [nsrc] then lo [nsrc])
    int nq = 1;
    void *sq2 = nullptr;
    float *ds_q2 = nullptr;
    size_t nslot_floats = 0;  // floats of tc_scratch per set
};

// ---------------------------------------------------------------------------------
// host: complex operators (checked against a direct sum in the tests)

using cd = std::complex<double>;

static void ups_host(double x, double y, double z, int P, std::vector<cd> &U) {
    const double r2 = x * x + y * y + z * z;
    U.assign((P + 1) * (P + 2) / 2, 0.0);
    U[0] = 1.0;
    const cd w(x, y);
    for (int m = 0; m <= P; m++) {
        if (m > 0) U[cidx(m, m)] = w / (2.0 * m) * U[cidx(m - 1, m - 1)];
        if (m + 1 <= P) U[cidx(m + 1, m)] = z * U[cidx(m, m)];
        for (int n = m + 2; n <= P; n++)
            U[cidx(n, m)] = ((2.0 * n - 1) * z * U[cidx(n - 1, m)] - r2 * U[cidx(n - 2, m)]) / double((n + m) * (n - m));
    }
}
static void the_host(double x, double y, double z, int P, std::vector<cd> &T) {
    const double r2 = x * x + y * y + z * z, ir2 = 1.0 / r2;
    T.assign((P + 1) * (P + 2) / 2, 0.0);
    T[0] = 1.0 / std::sqrt(r2);
    const cd w(x, y);
    for (int m = 0; m <= P; m++) {
        if (m > 0) T[cidx(m, m)] = (2.0 * m - 1) * w * ir2 * T[cidx(m - 1, m - 1)];
        if (m + 1 <= P) T[cidx(m + 1, m)] = (2.0 * m + 1) * z * ir2 * T[cidx(m, m)];
        for (int n = m + 2; n <= P; n++)
            T[cidx(n, m)] = ((2.0 * n - 1) * z * T[cidx(n - 1, m)] - double((n + m - 1) * (n - m - 1)) * T[cidx(n - 2, m)]) * ir2;
    }
}
static inline cd getc(const std::vector<cd> &A, int n, int m) {
    if (m >= 0) return A[cidx(n, m)];
    const cd v = std::conj(A[cidx(n, -m)]);
    return (m & 1) ? -v : v;
}
static void to_complex(const double *r, int P, std::vector<cd> &A) {
    A.assign((P + 1) * (P + 2) / 2, 0.0);
    for (int n = 0; n <= P; n++)
        for (int m = 0; m <= n; m++) A[cidx(n, m)] = m == 0 ? cd(r[ridx(n, 0, 0)], 0) : cd(r[ridx(n, m, 0)], r[ridx(n, m, 1)]);
}
static void to_real(const std::vector<cd> &A, int P, double *r) {
    for (int n = 0; n <= P; n++)
        for (int m = 0; m <= n; m++) {
            r[ridx(n, m, 0)] = A[cidx(n, m)].real();
            if (m) r[ridx(n, m, 1)] = A[cidx(n, m)].imag();
        }
}
// F_n^m = (-1)^n sum_kl M_k^l The_{n+k}^{m+l}(t), t = target centre - source centre (cell units)
static void m2l_c(const std::vector<cd> &M, const std::vector<cd> &T, int P, std::vector<cd> &F) {
    F.assign((P + 1) * (P + 2) / 2, 0.0);
    for (int n = 0; n <= P; n++)
        for (int m = 0; m <= n; m++) {
            cd s = 0;
            for (int k = 0; k <= P; k++)
                for (int l = -k; l <= k; l++) s += getc(M, k, l) * getc(T, n + k, m + l);
            F[cidx(n, m)] = (n & 1) ? -s : s;
        }
}
// parent M from a child: M_n^m = sum conj(Ups_k^l(t)) 2^-(n-k) M_{n-k}^{m-l}, t = child - parent (parent units)
static void m2m_c(const std::vector<cd> &M, const std::vector<cd> &U, int P, std::vector<cd> &O) {
    O.assign((P + 1) * (P + 2) / 2, 0.0);
    for (int n = 0; n <= P; n++)
        for (int m = 0; m <= n; m++) {
            cd s = 0;
            for (int k = 0; k <= n; k++)
                for (int l = -k; l <= k; l++)
                    if (std::abs(m - l) <= n - k) s += std::conj(getc(U, k, l)) * std::ldexp(1.0, -(n - k)) * getc(M, n - k, m - l);
            O[cidx(n, m)] = s;
        }
}
// child F from the parent: F_k^l = sum_{n>=k} F_n^m 2^-(k+1) conj(Ups_{n-k}^{m-l}(t)), t = child - parent
static void l2l_c(const std::vector<cd> &F, const std::vector<cd> &U, int P, std::vector<cd> &O) {
    O.assign((P + 1) * (P + 2) / 2, 0.0);
    for (int k = 0; k <= P; k++)
        for (int l = 0; l <= k; l++) {
            cd s = 0;
            for (int n = k; n <= P; n++)
                for (int m = -n; m <= n; m++)
                    if (std::abs(m - l) <= n - k) s += getc(F, n, m) * std::conj(getc(U, n - k, m - l));
            O[cidx(k, l)] = s * std::ldexp(1.0, -(k + 1));
        }
}

// ---------------------------------------------------------------------------------
// device

template <typename T, int M, typename Fn>
__device__ __forceinline__ void ups_col(T x, T y, T z, T r2, T &dre, T &dim, Fn &f) {
    if constexpr (M > 0) {
        const T s = T(1) / T(2 * M);
        const T nre = (x * dre - y * dim) * s, nim = (x * dim + y * dre) * s;
        dre = nre;
        dim = nim;
    }
    f(M, M, dre, dim);
    if constexpr (M + 1 <= FMM_P) {
        T p2re = dre, p2im = dim;
        T p1re = z * dre, p1im = z * dim;
        f(M + 1, M, p1re, p1im);
#pragma unroll
        for (int n = M + 2; n <= FMM_P; n++) {
            const T a = T(2 * n - 1), b = T(1) / T((n + M) * (n - M));
            const T cre = (a * z * p1re - r2 * p2re) * b, cim = (a * z * p1im - r2 * p2im) * b;
            f(n, M, cre, cim);
            p2re = p1re; p2im = p1im;
            p1re = cre; p1im = cim;
        }
    }
    if constexpr (M < FMM_P) ups_col<T, M + 1>(x, y, z, r2, dre, dim, f);
}

// Every Ups_n^m(x, y, z), 0 <= m <= n <= P, passed to f(n, m, re, im) by the recurrences
// in m (diagonal) and n (columns); the column index m is a template parameter so that
// callers accumulating into register arrays see constant indices.
template <typename T, typename Fn>
__device__ __forceinline__ void ups_cols(T x, T y, T z, Fn &&f) {
    const T r2 = x * x + y * y + z * z;
    T dre = 1, dim = 0;
    ups_col<T, 0>(x, y, z, r2, dre, dim, f);
}


// P2M: one warp per leaf; each lane forms q*conj(Ups) of every 32nd source of the leaf into
// 100 register accumulators, which are then reduced over the warp in a fixed order (lane
// k mod 32 stores coefficient k). The charge is also stored for the near field (beside the
// source coordinates for the first set), and with the tensor-core translations the hi/lo
// split of M. Grid y selects the charge set.
template <typename T>
struct P2mSet {
    const double *q;        // charges (storage order)
    const float *qf;        // FP32 charges read instead of q (FP32 path, incremental demag), or nullptr
    T *M;                   // expansions of this set
    float *Mh, *Ml;         // their split (tensor-core translations) or nullptr
    T *qn;                  // charge for the near field, element s at qn[s * qn_stride]
    int qn_stride;
    float *qh, *ql;         // double-single charge for the FP64 near field (or nullptr)
    int qd_stride;
};

template <typename T>
__global__ void __launch_bounds__(128) k_p2m(int nleaf, const int *__restrict__ leaf_src, const T *__restrict__ sloc,
                                             int leaf0, P2mSet<T> set0, P2mSet<T> set1) {
    const P2mSet<T> st = blockIdx.y ? set1 : set0;
    const int lane = threadIdx.x & 31;
    const int leaf = blockIdx.x * 4 + (threadIdx.x >> 5);
    if (leaf >= nleaf) return;
    const int s0 = leaf_src[leaf], s1 = leaf_src[leaf + 1];
    const double *__restrict__ q = st.q;
    T acc[NR];
#pragma unroll
    for (int k = 0; k < NR; k++) acc[k] = 0;
    for (int s = s0 + lane; s < s1; s += 32) {
        const T x = sloc[4 * (size_t)s], y = sloc[4 * (size_t)s + 1], z = sloc[4 * (size_t)s + 2];
        const T qq = T(q[s]);
        st.qn[(size_t)s * st.qn_stride] = qq;
        ups_cols<T>(x, y, z, [&](int n, int m, T re, T im) {
            acc[ridx(n, m, 0)] += qq * re;
            if (m) acc[ridx(n, m, 1)] -= qq * im;
        });
    }
    const size_t base = (size_t)(leaf0 + leaf) * NR;
#pragma unroll
    for (int k = 0; k < NR; k++) {
        T v = acc[k];
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
        if ((k & 31) == lane) {
            st.M[base + k] = v;
            if (st.Mh) {  // split for the tensor-core translations: hi = tf32(x), lo = x - hi
                const float xf = (float)v;
                const float hi = __uint_as_float((__float_as_uint(xf) + 0x1000u) & 0xFFFFE000u);
                st.Mh[base + k] = hi;
                st.Ml[base + k] = xf - hi;
            }
        }
    }
}

// The same harmonics restricted to the columns M0..M1 (the diagonal recurrence still runs
// from m = 0): f(n, m, re, im) for M0 <= m <= M1 only, with the values and the order of
// operations of ups_cols.
template <typename T, int M, int M0, int M1, typename Fn>
__device__ __forceinline__ void ups_col_r(T x, T y, T z, T r2, T &dre, T &dim, Fn &f) {
    if constexpr (M > 0) {
        const T s = T(1) / T(2 * M);
        const T nre = (x * dre - y * dim) * s, nim = (x * dim + y * dre) * s;
        dre = nre;
        dim = nim;
    }
    if constexpr (M >= M0) {
        f(M, M, dre, dim);
        if constexpr (M + 1 <= FMM_P) {
            T p2re = dre, p2im = dim;
            T p1re = z * dre, p1im = z * dim;
            f(M + 1, M, p1re, p1im);
#pragma unroll
            for (int n = M + 2; n <= FMM_P; n++) {
                const T a = T(2 * n - 1), b = T(1) / T((n + M) * (n - M));
                const T cre = (a * z * p1re - r2 * p2re) * b, cim = (a * z * p1im - r2 * p2im) * b;
                f(n, M, cre, cim);
                p2re = p1re; p2im = p1im;
                p1re = cre; p1im = cim;
            }
        }
    }
    if constexpr (M < M1) ups_col_r<T, M + 1, M0, M1>(x, y, z, r2, dre, dim, f);
}

// Reals of harmonic column m (n = m..P; real and imaginary parts for m > 0).
__host__ __device__ constexpr int col_reals(int m) { return m == 0 ? FMM_P + 1 : 2 * (FMM_P + 1 - m); }
// Index of (n, m, part) among the reals of the columns M0.. (column-major).
__host__ __device__ constexpr int lidx(int M0, int n, int m, int part) {
    int k = 0;
    for (int c = M0; c < m; c++) k += col_reals(c);
    return k + (m == 0 ? n : 2 * (n - m) + part);
}

// One pass of k_p2m2 over the columns M0..M1 of the NS charge sets of a leaf's sources.
template <int NS, int M0, int M1>
__device__ __forceinline__ void p2m2_pass(int lane, int s0, int s1, const float *__restrict__ sloc, size_t base,
                                          const P2mSet<float> &a, const P2mSet<float> &b) {
    constexpr int NPR = lidx(M0, FMM_P, M1, 1) + 1;
    float acc0[NPR], acc1[NS == 2 ? NPR : 1];
#pragma unroll
    for (int k = 0; k < NPR; k++) acc0[k] = 0.f;
#pragma unroll
    for (int k = 0; k < (NS == 2 ? NPR : 1); k++) acc1[k] = 0.f;
    for (int s = s0 + lane; s < s1; s += 32) {
        const float x = sloc[4 * (size_t)s], y = sloc[4 * (size_t)s + 1], z = sloc[4 * (size_t)s + 2];
        const float qa = a.qf ? a.qf[s] : float(a.q[s]);
        const float qb = NS == 2 ? (b.qf ? b.qf[s] : float(b.q[s])) : 0.f;
        if constexpr (M0 == 0) {  // the charges for the near field, once
            a.qn[(size_t)s * a.qn_stride] = qa;
            if constexpr (NS == 2) b.qn[(size_t)s * b.qn_stride] = qb;
        }
        const float r2 = x * x + y * y + z * z;
        float dre = 1, dim = 0;
        auto f = [&](int n, int m, float re, float im) {
            const int k = lidx(M0, n, m, 0);
            acc0[k] += qa * re;
            if constexpr (NS == 2) acc1[k] += qb * re;
            if (m) {
                acc0[k + 1] -= qa * im;
                if constexpr (NS == 2) acc1[k + 1] -= qb * im;
            }
        };
        ups_col_r<float, 0, M0, M1>(x, y, z, r2, dre, dim, f);
    }
    auto put = [&](const P2mSet<float> &st, int g, float v) {
        st.M[base + g] = v;
        if (st.Mh) {  // split for the tensor-core translations: hi = tf32(x), lo = x - hi
            const float hi = __uint_as_float((__float_as_uint(v) + 0x1000u) & 0xFFFFE000u);
            st.Mh[base + g] = hi;
            st.Ml[base + g] = v - hi;
        }
    };
#pragma unroll
    for (int m = M0; m <= M1; m++)
#pragma unroll
        for (int n = m; n <= FMM_P; n++)
#pragma unroll
            for (int part = 0; part < (m ? 2 : 1); part++) {
                const int k = lidx(M0, n, m, part), g = ridx(n, m, part);
                float v0 = acc0[k], v1 = NS == 2 ? acc1[NS == 2 ? k : 0] : 0.f;
#pragma unroll
                for (int o = 16; o > 0; o >>= 1) {
                    v0 += __shfl_xor_sync(0xffffffffu, v0, o);
                    if constexpr (NS == 2) v1 += __shfl_xor_sync(0xffffffffu, v1, o);
                }
                if ((g & 31) == lane) {
                    put(a, g, v0);
                    if constexpr (NS == 2) put(b, g, v1);
                }
            }
}

// P2M of the FP32 path, the NS charge sets in one pass over the sources: the harmonics of a
// source are formed once for both sets (k_p2m forms them once per set), in three passes over
// the harmonic columns (0-2, 3-5, 6-9: 88, 72 and 40 register accumulators for two sets)
// that repeat the cheap diagonal recurrence. Each coefficient sums the terms of k_p2m in the
// same order; one set (fg_demag) and two (fg_compute_all) run the same code, so a set's
// expansion does not depend on whether the other is evaluated beside it.
template <int NS>
__global__ void __launch_bounds__(128) k_p2m2(int nleaf, const int *__restrict__ leaf_src,
                                              const float *__restrict__ sloc, int leaf0, P2mSet<float> set0,
                                              P2mSet<float> set1) {
    const int lane = threadIdx.x & 31;
    const int leaf = blockIdx.x * 4 + (threadIdx.x >> 5);
    if (leaf >= nleaf) return;
    const int s0 = leaf_src[leaf], s1 = leaf_src[leaf + 1];
    const size_t base = (size_t)(leaf0 + leaf) * NR;
    p2m2_pass<NS, 0, 2>(lane, s0, s1, sloc, base, set0, set1);
    p2m2_pass<NS, 3, 5>(lane, s0, s1, sloc, base, set0, set1);
    p2m2_pass<NS, 6, FMM_P>(lane, s0, s1, sloc, base, set0, set1);
}

// ---- P2M of the FP64 path in double-single arithmetic -------------------------------
// The harmonics and their sums on the FP32 pipes (GB300's FP64 pipe runs at 1/64 of their rate).
// A column m is formed without divisions as V_n = k_n Ups_n^m,
//   V_m = (x + i y)^m, V_{m+1} = z V_m, V_n = (2n-1) z V_{n-1} - g r^2 V_{n-2},
// g = 1 for n = m + 2 and (n-1+m)(n-1-m) above, k_m = k_{m+1} = 2^m m!, k_n = k_{n-1} (n+m)(n-m),
// and the leaf's sums are multiplied by 1 / k_n once.

__device__ __forceinline__ dsf dsc(double x) {  // a double constant as a double-single pair
    const float h = (float)x;
    return {h, (float)(x - (double)h)};
}

// A warp forms two columns of a leaf: (0, 5), (1, 9), (2, 8), (3, 7) or (4, 6), 20 reals every pair
// (80 registers of sums for two sets) and nearly the same work.
constexpr int P2M_COL[5][2] = {{0, 5}, {1, 9}, {2, 8}, {3, 7}, {4, 6}};
struct P2mTab {
    int idx[5][20];     // real index of each of a warp's 20 sums
    double fac[5][20];  // 1 / k_n, negative for imaginary parts (M = sum q conj(Ups))
};
constexpr P2mTab make_p2m_tab() {
    P2mTab t{};
    for (int w = 0; w < 5; w++) {
        int r = 0;
        for (int h = 0; h < 2; h++) {
            const int m = P2M_COL[w][h];
            double k = 1.0;
            for (int i = 1; i <= m; i++) k *= 2.0 * i;
            for (int n = m; n <= FMM_P; n++) {
                if (n >= m + 2) k *= double((n + m) * (n - m));
                for (int part = 0; part < (m ? 2 : 1); part++, r++) {
                    t.idx[w][r] = ridx(n, m, part);
                    t.fac[w][r] = (part ? -1.0 : 1.0) / k;
                }
            }
        }
    }
    return t;
}
__constant__ P2mTab c_p2m = make_p2m_tab();

// products and sums of normalised pairs; a product left unnormalised (hi, lo) keeps |lo| below
// 2^-22 |hi|
__device__ __forceinline__ dsf ds_prod(dsf x, dsf y) {
    const float p = x.h * y.h;
    return {p, fmaf(x.l, y.h, fmaf(x.h, y.l, fmaf(x.h, y.h, -p)))};
}
__device__ __forceinline__ dsf ds_diff(dsf x, dsf y) {  // of unnormalised products, normalised
    const dsf s = ds_two_sum_f(x.h, -y.h);
    return ds_quick(s.h, s.l + (x.l - y.l));
}
__device__ __forceinline__ dsf ds_sum(dsf x, dsf y) {
    const dsf s = ds_two_sum_f(x.h, y.h);
    return ds_quick(s.h, s.l + (x.l + y.l));
}
__device__ __forceinline__ dsf ds_scale(dsf x, float c) {  // times a small integer, unnormalised
    const float p = x.h * c;
    return {p, fmaf(x.l, c, fmaf(x.h, c, -p))};
}
struct dsc2 { dsf re, im; };
__device__ __forceinline__ dsc2 ds_cmul(dsc2 a, dsc2 b) {
    return {ds_diff(ds_prod(a.re, b.re), ds_prod(a.im, b.im)), ds_sum(ds_prod(a.re, b.im), ds_prod(a.im, b.re))};
}
template <int M>
__device__ __forceinline__ dsc2 ds_cpow(dsc2 w) {  // w^M, M >= 1
    if constexpr (M == 1) return w;
    else if constexpr (M % 2 == 0) {
        const dsc2 h = ds_cpow<M / 2>(w);
        return ds_cmul(h, h);
    } else return ds_cmul(ds_cpow<M - 1>(w), w);
}

// Column M of one source: f(n, V_n); the imaginary parts of column 0 are zero and unused.
template <int M, typename Fn>
__device__ __forceinline__ void p2m_column(dsc2 d, dsf z, dsf r2, Fn &&f) {
    f(M, d);
    if constexpr (M < FMM_P) {
        auto mul = [](dsf a, dsf b) {
            const dsf p = ds_prod(a, b);
            return ds_quick(p.h, p.l);
        };
        dsc2 p2 = d, p1;
        if constexpr (M == 0) p1 = {z, {0.f, 0.f}};
        else p1 = {mul(z, d.re), mul(z, d.im)};
        f(M + 1, p1);
#pragma unroll
        for (int n = M + 2; n <= FMM_P; n++) {
            const dsf az = ds_scale(z, float(2 * n - 1));
            const dsf gr = n == M + 2 ? r2 : ds_scale(r2, float((n - 1 + M) * (n - 1 - M)));
            dsc2 c;
            c.re = ds_diff(ds_prod(az, p1.re), ds_prod(gr, p2.re));
            if constexpr (M > 0) c.im = ds_diff(ds_prod(az, p1.im), ds_prod(gr, p2.im));
            else c.im = {0.f, 0.f};
            f(n, c);
            p2 = p1;
            p1 = c;
        }
    }
}

template <int NS, int W>
__device__ __forceinline__ void p2m_ds_warp(int lane, int s0, int s1, const float4 *__restrict__ shi,
                                            const float4 *__restrict__ slo, size_t base, const P2mSet<double> &a,
                                            const P2mSet<double> &b) {
    constexpr int MA = P2M_COL[W][0], MB = P2M_COL[W][1], NA = MA ? 2 * (FMM_P + 1 - MA) : FMM_P + 1;
    dsf acc[20 * NS];
#pragma unroll
    for (int k = 0; k < 20 * NS; k++) acc[k] = dsf{0.f, 0.f};
    int since = 0;
    for (int s = s0 + lane; s < s1; s += 32) {
        const float4 h = shi[s], l = slo[s];
        const dsf x = ds_two_sum_f(h.x, l.x), y = ds_two_sum_f(h.y, l.y), z = ds_two_sum_f(h.z, l.z);
        const double qa_d = a.q[s], qb_d = NS == 2 ? b.q[s] : 0.0;
        const dsf qa = dsc(qa_d), qb = dsc(qb_d);
        if constexpr (W == 0) {  // the charges for the near field, once
            a.qh[(size_t)s * a.qd_stride] = qa.h;
            a.ql[(size_t)s * a.qd_stride] = qa.l;
            if constexpr (NS == 2) {
                b.qh[(size_t)s * b.qd_stride] = qb.h;
                b.ql[(size_t)s * b.qd_stride] = qb.l;
            }
        }
        const dsf r2 = ds_sum(ds_sum(ds_prod(x, x), ds_prod(y, y)), ds_prod(z, z));
        auto add = [&](int k, dsf q, dsf v) {
            const dsf p = ds_prod(q, v), t = ds_two_sum_f(acc[k].h, p.h);
            acc[k].h = t.h;
            acc[k].l += t.l + p.l;
        };
        auto col = [&](int m, int k0, int n, dsc2 v) {
            const int k = k0 + (m ? 2 * (n - m) : n);
            add(k, qa, v.re);
            if (m) add(k + 1, qa, v.im);
            if constexpr (NS == 2) {
                add(20 + k, qb, v.re);
                if (m) add(20 + k + 1, qb, v.im);
            }
        };
        const dsc2 w{x, y};
        if constexpr (MA == 0) {
            p2m_column<0>({{1.f, 0.f}, {0.f, 0.f}}, z, r2, [&](int n, dsc2 v) { col(0, 0, n, v); });
            p2m_column<MB>(ds_cpow<MB>(w), z, r2, [&](int n, dsc2 v) { col(MB, NA, n, v); });
        } else {
            const dsc2 wa = ds_cpow<MA>(w);
            p2m_column<MA>(wa, z, r2, [&](int n, dsc2 v) { col(MA, 0, n, v); });
            // w^MB from w^MA: 9 = 8 + 1, 8 = 4 x 2, 7 = 4 + 3, 6 = 4 + 2
            dsc2 wb;
            if constexpr (MB == 9) wb = ds_cpow<9>(w);
            else if constexpr (MB == 8) wb = ds_cpow<4>(wa);
            else wb = ds_cmul(wa, ds_cpow<MB - MA>(w));
            p2m_column<MB>(wb, z, r2, [&](int n, dsc2 v) { col(MB, NA, n, v); });
        }
        if (++since == 16) {  // |lo| back to half an ulp of hi
            since = 0;
#pragma unroll
            for (int k = 0; k < 20 * NS; k++) acc[k] = ds_quick(acc[k].h, acc[k].l);
        }
    }
#pragma unroll
    for (int k = 0; k < 20 * NS; k++) acc[k] = ds_quick(acc[k].h, acc[k].l);
    // sums over the warp: the halves of the values are exchanged while their number is even (lane
    // bit 4 keeps the set of two), each value by the butterfly over lane bits 4 to 0
    int n = 20 * NS;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        const bool halve = n % 2 == 0, hi = lane & o;
        if (halve) n >>= 1;
#pragma unroll
        for (int k = 0; k < 10 * NS; k++)
            if (k < n) {
                const dsf keep = halve && hi ? acc[k + n] : acc[k], send = halve && !hi ? acc[k + n] : acc[k];
                acc[k] = ds_add(keep, dsf{__shfl_xor_sync(0xffffffffu, send.h, o), __shfl_xor_sync(0xffffffffu, send.l, o)});
            }
    }
    // five values left: of lanes that differ in bits 0 and 1 (two sets) or 0 to 2 the same ones
    const int sub = NS == 2 ? lane & 3 : lane & 7, set = NS == 2 ? lane >> 4 : 0;
    const int r0 = NS == 2 ? 10 * (lane >> 3 & 1) + 5 * (lane >> 2 & 1) : 10 * (lane >> 4) + 5 * (lane >> 3 & 1);
#pragma unroll
    for (int k = 0; k < 5; k++)
        if ((k & 3) == sub) (set ? b : a).M[base + c_p2m.idx[W][r0 + k]] = ds_to(acc[k]) * c_p2m.fac[W][r0 + k];
}

// P2M of the FP64 path: one warp per leaf and pair of columns (grid y) over the leaf's sources, the
// NS charge sets in one pass (the harmonics of a source are formed once for both; one set and two
// run the same arithmetic). About 5,400 FP32 operations per source for two sets. The loop bodies
// are straight-line code of some 20 KB each: the column pair is the slow grid index, so
// that an SM runs one of them at a time (with the five pairs side by side in a block, 18 of 20
// cycles went to instruction fetch: wire 2.77 ms).
template <int NS>
__global__ void __launch_bounds__(128, 4) k_p2m_ds(int nleaf, const int *__restrict__ leaf_src,
                                                   const float4 *__restrict__ shi, const float4 *__restrict__ slo,
                                                   int leaf0, P2mSet<double> set0, P2mSet<double> set1) {
    const int lane = threadIdx.x & 31, leaf = blockIdx.x * 4 + (threadIdx.x >> 5);
    if (leaf >= nleaf) return;
    const int s0 = leaf_src[leaf], s1 = leaf_src[leaf + 1];
    const size_t base = (size_t)(leaf0 + leaf) * NR;
    switch (blockIdx.y) {
        case 0: p2m_ds_warp<NS, 0>(lane, s0, s1, shi, slo, base, set0, set1); break;
        case 1: p2m_ds_warp<NS, 1>(lane, s0, s1, shi, slo, base, set0, set1); break;
        case 2: p2m_ds_warp<NS, 2>(lane, s0, s1, shi, slo, base, set0, set1); break;
        case 3: p2m_ds_warp<NS, 3>(lane, s0, s1, shi, slo, base, set0, set1); break;
        default: p2m_ds_warp<NS, 4>(lane, s0, s1, shi, slo, base, set0, set1); break;
    }
}

__device__ __forceinline__ float2 ds_split(double x) {
    const float h = (float)x;
    return make_float2(h, (float)(x - (double)h));
}

// ---- P2M of the full FP64 evaluation of the FP32 + refinement path (FmmTree::repeat) ----
// The recurrences of ups_cols with every operation a double-single one, the coordinates as the
// normalised pair of their stored hi + lo parts, the charge split once.
// The columns above 0 with real and imaginary parts as the lanes of packed pairs.
__device__ __forceinline__ ds2 ds2_dup(dsf a) { return {pk2(a.h, a.h), pk2(a.l, a.l)}; }
__device__ __forceinline__ ds2 ds2_neg(ds2 a) { return {neg2(a.h), neg2(a.l)}; }
__device__ __forceinline__ u64 swap2(u64 a) { return a >> 32 | a << 32; }

// Column 0 of one source: f(n, V_n), real.
template <typename Fn>
__device__ __forceinline__ void ups_col0_ds(dsf z, dsf r2, Fn &f) {
    dsf p2 = {1.f, 0.f}, p1 = ds_mul(z, p2);
    f(0, p2);
    f(1, p1);
#pragma unroll
    for (int n = 2; n <= FMM_P; n++) {
        const dsf az = ds_mul(dsf{(float)(2 * n - 1), 0.f}, z);
        const dsf c = ds_mul(ds_sub(ds_mul(az, p1), ds_mul(r2, p2)), dsc(1.0 / (n * n)));
        f(n, c);
        p2 = p1;
        p1 = c;
    }
}

// Columns M (1 first) to M1, f from column M0 on; d: the diagonal of column M - 1, X = (x, x),
// Y = (-y, y), Z = (z, z), R2 = (r2, r2).
template <int M, int M0, int M1, typename Fn>
__device__ __forceinline__ void ups_col_ds(ds2 X, ds2 Y, dsf z, ds2 Z, ds2 R2, ds2 d, Fn &f) {
    d = ds2_mul(ds2_add(ds2_mul(X, d), ds2_mul(Y, ds2{swap2(d.h), swap2(d.l)})), ds2_dup(dsc(1.0 / (2 * M))));
    if constexpr (M >= M0) {
        f(M, M, d);
        if constexpr (M + 1 <= FMM_P) {
            ds2 p2 = d, p1 = ds2_mul(Z, d);
            f(M + 1, M, p1);
#pragma unroll
            for (int n = M + 2; n <= FMM_P; n++) {
                const dsf az = ds_mul(dsf{(float)(2 * n - 1), 0.f}, z);
                const ds2 c = ds2_mul(ds2_add(ds2_mul(ds2_dup(az), p1), ds2_neg(ds2_mul(R2, p2))),
                                      ds2_dup(dsc(1.0 / ((n + M) * (n - M)))));
                f(n, M, c);
                p2 = p1;
                p1 = c;
            }
        }
    }
    if constexpr (M < M1) ups_col_ds<M + 1, M0, M1>(X, Y, z, Z, R2, d, f);
}

template <int NS, int M0, int M1>
__device__ __forceinline__ void p2m_ds_pass(int lane, int s0, int s1, int rounds, const float4 *__restrict__ shi,
                                            const float4 *__restrict__ slo, size_t base, const P2mSet<double> &a,
                                            const P2mSet<double> &b) {
    constexpr int NPR = lidx(M0, FMM_P, M1, 1) + 1, NV = M0 == 0 ? NPR : NPR / 2;  // column 0, or pairs
    using Acc = std::conditional_t<M0 == 0, dsf, ds2>;
    static_assert(M0 > 0 || M1 == 0, "column 0 alone");
    Acc acc0[NV] = {}, acc1[NS == 2 ? NV : 1] = {};
    for (int q = 0; q < rounds; q++) {
        __syncthreads();  // the block's warps in step, on the same instructions
        const int s = s0 + lane + 32 * q;
        if (s >= s1) continue;
        const float4 h = shi[s], l = slo[s];
        const dsf x = ds_two_sum_f(h.x, l.x), y = ds_two_sum_f(h.y, l.y), z = ds_two_sum_f(h.z, l.z);
        const double qa_d = a.q[s], qb_d = NS == 2 ? b.q[s] : 0.0;
        const dsf qa = dsc(qa_d), qb = dsc(qb_d);
        const dsf r2 = ds_add(ds_add(ds_mul(x, x), ds_mul(y, y)), ds_mul(z, z));
        if constexpr (M0 == 0) {
            a.qh[(size_t)s * a.qd_stride] = qa.h;  // the charges for the near field
            a.ql[(size_t)s * a.qd_stride] = qa.l;
            if constexpr (NS == 2) {
                b.qh[(size_t)s * b.qd_stride] = qb.h;
                b.ql[(size_t)s * b.qd_stride] = qb.l;
            }
            auto f = [&](int n, dsf re) {
                acc0[n] = ds_add(acc0[n], ds_mul(qa, re));
                if constexpr (NS == 2) acc1[n] = ds_add(acc1[n], ds_mul(qb, re));
            };
            ups_col0_ds(z, r2, f);
        } else {  // M = sum q conj(Ups): charges (q, -q)
            const ds2 QA = {pk2(qa.h, -qa.h), pk2(qa.l, -qa.l)}, QB = {pk2(qb.h, -qb.h), pk2(qb.l, -qb.l)};
            auto f = [&](int n, int m, ds2 v) {
                const int k = lidx(M0, n, m, 0) / 2;
                acc0[k] = ds2_add(acc0[k], ds2_mul(QA, v));
                if constexpr (NS == 2) acc1[k] = ds2_add(acc1[k], ds2_mul(QB, v));
            };
            const ds2 Y = {pk2(-y.h, y.h), pk2(-y.l, y.l)};
            ups_col_ds<1, M0, M1>(ds2_dup(x), Y, z, ds2_dup(z), ds2_dup(r2), ds2{pk2(1.f, 0.f), 0ull}, f);
        }
    }
    auto red = [&](Acc v) {
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) {
            const Acc w = {__shfl_xor_sync(0xffffffffu, v.h, o), __shfl_xor_sync(0xffffffffu, v.l, o)};
            if constexpr (M0 == 0) v = ds_add(v, w);
            else v = ds2_add(v, w);
        }
        return v;
    };
    // rounded to FP64, then the pair that the translations read
    auto put = [&](const P2mSet<double> &st, int g, dsf v) {
        if ((g & 31) == lane && s0 >= 0) reinterpret_cast<float2 *>(st.M)[base + g] = ds_split(ds_to(v));
    };
    auto store = [&](const P2mSet<double> &st, int n, int m, Acc v) {
        if constexpr (M0 == 0) put(st, ridx(n, m, 0), v);
        else {
            dsf re, im;
            upk2(v.h, re.h, im.h);
            upk2(v.l, re.l, im.l);
            put(st, ridx(n, m, 0), re);
            put(st, ridx(n, m, 1), im);
        }
    };
#pragma unroll
    for (int m = M0; m <= M1; m++)
#pragma unroll
        for (int n = m; n <= FMM_P; n++) {
            const int k = M0 == 0 ? n : lidx(M0, n, m, 0) / 2;
            store(a, n, m, red(acc0[k]));
            if constexpr (NS == 2) store(b, n, m, red(acc1[k]));
        }
}

// One warp per leaf and range of harmonic columns (0, 1, 2, 3, 4-5, 6-9: at most 22 reals, 88 floats
// of accumulators for two sets), the NS charge sets together (the FP64 tree's sources as hi/lo
// float4 pairs): the harmonics of a source are formed once for both sets; one set and two run the
// same code, so a set's expansion does not depend on whether the other is evaluated beside it. The
// range is the slow grid index and the block's warps keep in step: bound by fetching the unrolled
// instructions, which six passes by each warp at its own pace made worse (294k tets, two sets: six
// passes per warp 1.45 ms, a range per block 0.87, in step 0.73, real and imaginary parts as the lanes
// of packed FP32 operations 0.58).
template <int NS>
__global__ void __launch_bounds__(128, 3) k_p2m_ds_repeat(int nleaf, const int *__restrict__ leaf_src,
                                                const float4 *__restrict__ shi, const float4 *__restrict__ slo,
                                                int leaf0, P2mSet<double> set0, P2mSet<double> set1) {
    const int lane = threadIdx.x & 31;
    const int leaf = blockIdx.x * 4 + (threadIdx.x >> 5);
    const int s0 = leaf < nleaf ? leaf_src[leaf] : -1, s1 = leaf < nleaf ? leaf_src[leaf + 1] : -1;  // -1: no leaf
    int rounds = 0;  // of the block's longest leaf
    for (int k = blockIdx.x * 4; k < min(nleaf, (int)blockIdx.x * 4 + 4); k++)
        rounds = max(rounds, (leaf_src[k + 1] - leaf_src[k] + 31) / 32);
    const size_t base = (size_t)(leaf0 + leaf) * NR;
    switch (blockIdx.y) {
        case 0: p2m_ds_pass<NS, 6, FMM_P>(lane, s0, s1, rounds, shi, slo, base, set0, set1); break;
        case 1: p2m_ds_pass<NS, 4, 5>(lane, s0, s1, rounds, shi, slo, base, set0, set1); break;
        case 2: p2m_ds_pass<NS, 3, 3>(lane, s0, s1, rounds, shi, slo, base, set0, set1); break;
        case 3: p2m_ds_pass<NS, 2, 2>(lane, s0, s1, rounds, shi, slo, base, set0, set1); break;
        case 4: p2m_ds_pass<NS, 1, 1>(lane, s0, s1, rounds, shi, slo, base, set0, set1); break;
        default: p2m_ds_pass<NS, 0, 0>(lane, s0, s1, rounds, shi, slo, base, set0, set1); break;
    }
}

// Batched translation out[c] (+)= sum_code Op[code] in[tab[c][code]] for TB output cells
// per block. 160 threads: 10 row groups (10 rows each) x 16 column groups (CT cells each).
template <typename T>
__global__ void __launch_bounds__(160) k_translate(int n_out, int out0, int ncode, const int *__restrict__ tab,
                                                   const T *__restrict__ ops, const T *in, T *out,
                                                   int accumulate) {
    // in and out may be the same array (M2M, L2L): the cells read and written are disjoint.
    constexpr int TB = TrShape<T>::TB, CT = TrShape<T>::CT, RT = 10, BLD = TB + 4;
    extern __shared__ unsigned char smem_raw[];
    T *AT = reinterpret_cast<T *>(smem_raw);  // [NR][NR]: AT[k*NR + row] = Op[row][k]
    T *Bs = AT + NR * NR;                      // [NR][BLD]
    __shared__ int srcs[TB];
    const int tid = threadIdx.x, rg = tid / 16, cg = tid % 16;
    const int c_begin = blockIdx.x * TB;
    T acc[RT][CT];
#pragma unroll
    for (int i = 0; i < RT; i++)
#pragma unroll
        for (int j = 0; j < CT; j++) acc[i][j] = 0;
    for (int code = 0; code < ncode; code++) {
        int s = -1;
        if (tid < TB && c_begin + tid < n_out) s = tab[(size_t)(out0 + c_begin + tid) * ncode + code];
        if (tid < TB) srcs[tid] = s;
        if (!__syncthreads_or(s >= 0)) continue;
        for (int e = tid; e < NR * NR; e += blockDim.x) {
            const int row = e / NR, k = e % NR;
            AT[k * NR + row] = ops[(size_t)code * NR * NR + e];
        }
        for (int e = tid; e < NR * TB; e += blockDim.x) {
            const int col = e / NR, k = e % NR;
            const int sc = srcs[col];
            Bs[k * BLD + col] = sc >= 0 ? in[(size_t)sc * NR + k] : T(0);
        }
        __syncthreads();
#pragma unroll 4
        for (int k = 0; k < NR; k++) {
            T a[RT], b[CT];
#pragma unroll
            for (int i = 0; i < RT; i++) a[i] = AT[k * NR + rg * RT + i];
#pragma unroll
            for (int j = 0; j < CT; j++) b[j] = Bs[k * BLD + cg * CT + j];
#pragma unroll
            for (int i = 0; i < RT; i++)
#pragma unroll
                for (int j = 0; j < CT; j++) acc[i][j] += a[i] * b[j];
        }
        __syncthreads();
    }
#pragma unroll
    for (int j = 0; j < CT; j++) {
        const int c = c_begin + cg * CT + j;
        if (c >= n_out) continue;
        T *o = out + (size_t)(out0 + c) * NR + rg * RT;
#pragma unroll
        for (int i = 0; i < RT; i++) o[i] = accumulate ? o[i] + acc[i][j] : acc[i][j];
    }
}

// Translations in double-single arithmetic on the FP32 pipes (the full FP64 evaluation of the
// FP32 + refinement path, see FmmTree::repeat): per output and code the products in the order of
// k, every product exact through fma (Dekker's TwoProduct) and summed with Knuth's two-sum, the
// running sum renormalised once per code (about 44 significant bits), the result rounded to FP64
// once. 12 FP32 operations per product bound it.
//
// A block takes DS_ROWS rows of the operators for a tile of DS_TILE output cells that share their
// codes (the cells of one octant, in lists made with the tree), a lane per cell and DS_RT rows per
// warp; the tile's codes run one after the other, as the order of the sums is fixed. Operators
// (split when the tree is made, in the order in which the block reads them) and inputs (split by
// the kernel that forms them) come through a ring of DS_STAGE pieces of DS_KC columns by cp.async.
// Before, a block held all 100 rows of 16 neighbouring cells: most (cell, code) columns were zero,
// each block split 10,000 FP64 operator entries per code again, and 128 blocks left SMs idle (294k
// tets, two sets: M2L 6.24 -> 1.66 ms, FMA pipe busy 71% of the time; M2M 0.74 -> 0.12, L2L 0.66 -> 0.09).
constexpr int DS_TILE = 32, DS_RT = 5, DS_ROWS = 4 * DS_RT, DS_PARTS = NR / DS_ROWS, DS_KC = 20, DS_STAGE = 4;
constexpr int DS_CHUNKS = NR / DS_KC, DS_A4 = DS_ROWS * DS_KC / 2;  // float4 of operator per piece
constexpr int DS_B4 = DS_KC / 2 + 1;  // float4 per cell and piece, one of padding against bank conflicts
static_assert(DS_PARTS * DS_ROWS == NR && DS_CHUNKS * DS_KC == NR && DS_KC % 2 == 0);

// float4 of the operator image holding entries (row, k) and (row, k + 1), k even
__host__ __device__ constexpr size_t ds_image_at(int code, int row, int k) {
    return ((size_t)(code * DS_PARTS + row / DS_ROWS) * DS_CHUNKS + k / DS_KC) * DS_A4 + (k % DS_KC / 2) * DS_ROWS +
           row % DS_ROWS;
}
__global__ void k_ds_image(int ncode, const double *__restrict__ ops, float4 *__restrict__ img) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;  // (code, row, k / 2)
    if (i >= ncode * NR * NR / 2) return;
    const int k = i % (NR / 2) * 2, row = i / (NR / 2) % NR, code = i / (NR * NR / 2);
    const float2 a = ds_split(ops[2 * (size_t)i]), b = ds_split(ops[2 * (size_t)i + 1]);
    img[ds_image_at(code, row, k)] = make_float4(a.x, a.y, b.x, b.y);
}

__device__ __forceinline__ void ds_cp16(void *dst, const void *src, int bytes) {  // the rest of the 16 is zero
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"((unsigned)__cvta_generic_to_shared(dst)), "l"(src),
                 "r"(bytes) : "memory");
}

__global__ void __launch_bounds__(128, 5) k_translate_ds(const int4 *__restrict__ tiles, const int *__restrict__ cells,
                                                         const int *__restrict__ codes, int ncode,
                                                         const int *__restrict__ tab, const float4 *__restrict__ img,
                                                         const float2 *in, size_t in_stride, double *out,
                                                         size_t out_stride, float2 *split, size_t split_stride,
                                                         int nsplit, int accumulate) {
    // in and split may be the same array (M2M, L2L): the cells read and written are disjoint.
    __shared__ float4 As[DS_STAGE][DS_A4], Bs[DS_STAGE][DS_TILE][DS_B4];
    const int tid = threadIdx.x, lane = tid % 32, warp = tid / 32;
    const int4 t = tiles[blockIdx.x / DS_PARTS];  // first cell of the list, codes from and to
    const int part = blockIdx.x % DS_PARTS, set = blockIdx.y, nch = (t.z - t.y) * DS_CHUNKS;
    in += set * in_stride;
    // copies: thread 4 i + j brings 16-byte pieces j, j + 4, j + 8 of cell i; the source cell is
    // read one code, the code two codes ahead
    const int cc = tid / 4, cj = tid % 4, ccell = cells[t.x + cc];
    auto code_at = [&](int q) { return codes[min(q, t.z - 1)]; };
    auto src_at = [&](int code) { return ccell >= 0 ? tab[(size_t)ccell * ncode + code] : -1; };
    int iq = t.y, ich = 0, code0 = 0, code1 = 0, code2 = 0, src0 = -1, src1 = -1;
    if (nch) {
        code0 = code_at(iq);
        code1 = code_at(iq + 1);
        code2 = code_at(iq + 2);
        src0 = src_at(code0);
        src1 = src_at(code1);
    }
    auto issue = [&](int st) {
        if (iq < t.z) {
            const float4 *a = img + ((size_t)(code0 * DS_PARTS + part) * DS_CHUNKS + ich) * DS_A4;
            for (int i = tid; i < DS_A4; i += 128) ds_cp16(&As[st][i], a + i, 16);
            const float4 *b = reinterpret_cast<const float4 *>(in + (src0 >= 0 ? (size_t)src0 * NR + ich * DS_KC : 0));
#pragma unroll
            for (int j = cj; j < DS_KC / 2; j += 4) ds_cp16(&Bs[st][cc][j], b + (src0 >= 0 ? j : 0), src0 >= 0 ? 16 : 0);
            if (++ich == DS_CHUNKS) {
                ich = 0;
                iq++;
                code0 = code1;
                src0 = src1;
                code1 = code2;
                src1 = src_at(code1);
                code2 = code_at(iq + 2);
            }
        }
        asm volatile("cp.async.commit_group;" ::: "memory");
    };
    float ah[DS_RT], al[DS_RT];
#pragma unroll
    for (int i = 0; i < DS_RT; i++) ah[i] = al[i] = 0.f;
    for (int st = 0; st < DS_STAGE - 1; st++) issue(st);
    int ch = 0;
    for (int c = 0; c < nch; c++) {
        asm volatile("cp.async.wait_group %0;" ::"n"(DS_STAGE - 2) : "memory");
        __syncthreads();  // piece c is there, and every warp is done with piece c - 1
        issue((c + DS_STAGE - 1) % DS_STAGE);
        const float4 *A = As[c % DS_STAGE] + warp * DS_RT, *B = Bs[c % DS_STAGE][lane];
#pragma unroll 5
        for (int k = 0; k < DS_KC / 2; k++) {
            const float4 b2 = B[k];
            float4 a2[DS_RT];
#pragma unroll
            for (int i = 0; i < DS_RT; i++) a2[i] = A[k * DS_ROWS + i];
#pragma unroll
            for (int h = 0; h < 2; h++) {
                const float bx = h ? b2.z : b2.x, by = h ? b2.w : b2.y;
#pragma unroll
                for (int i = 0; i < DS_RT; i++) {
                    // (ah, al) += a b: exact leading product and cross terms, two-sum into hi
                    const float ax = h ? a2[i].z : a2[i].x, ay = h ? a2[i].w : a2[i].y;
                    const float p = __fmul_rn(ax, bx);
                    float e = fmaf(ax, bx, -p);
                    e = fmaf(ax, by, e);
                    e = fmaf(ay, bx, e);
                    const float s = __fadd_rn(ah[i], p);
                    const float bb = s - ah[i];
                    const float err = (ah[i] - (s - bb)) + (p - bb);
                    ah[i] = s;
                    al[i] += e + err;
                }
            }
        }
        if (++ch == DS_CHUNKS) {  // renormalise: |lo| back to half an ulp of hi
            ch = 0;
#pragma unroll
            for (int i = 0; i < DS_RT; i++) {
                const float s = ah[i] + al[i];
                al[i] = al[i] - (s - ah[i]);
                ah[i] = s;
            }
        }
    }
    asm volatile("cp.async.wait_all;" ::: "memory");
    const int cell = cells[t.x + lane];
    if (cell < 0) return;
    const size_t row0 = (size_t)cell * NR + part * DS_ROWS + warp * DS_RT;
#pragma unroll
    for (int i = 0; i < DS_RT; i++) {
        double v = (double)ah[i] + (double)al[i];
        if (out) {
            double *o = out + set * out_stride + row0 + i;
            if (accumulate) v = *o + v;
            *o = v;
        }
        if (cell < nsplit) split[set * split_stride + row0 + i] = ds_split(v);
    }
}

// 1/sqrt in the precision of the path.
template <typename T> __device__ __forceinline__ T rsqrt_p(T x);
template <> __device__ __forceinline__ float rsqrt_p<float>(float x) {
    float r;  // the SFU reciprocal square root (relative error below 2^-22), denormals flushed
    asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
    return r;
}
// FP64: CUDA's rsqrt (a single-precision-seeded Newton step written out here measured
// slower: the FP64 <-> FP32 conversions cost more than they save).
template <> __device__ __forceinline__ double rsqrt_p<double>(double x) { return rsqrt(x); }

template <typename T> struct Vec4;
template <> struct Vec4<float> { using type = float4; };
template <> struct Vec4<double> { using type = double4; };

// Charge sets of one near-field launch: the first set's charge rides in the w of the source
// coordinates, the second (demag of v beside that of m) in its own array; the local
// expansions and potentials of each set.
template <typename T>
struct NearSets {
    const T *q2;            // second set's charges (NQ = 2)
    const T *F[2];          // local expansions per set
    double *pot[2];         // potentials per set
    int near_only;          // 1: write the near-field sums only (k_l2p adds the far field later)
};

// One pass of the near field and L2P over up to NT targets tb.. of a leaf (nt of them real,
// the rest padding), for NQ charge sets at once (the pair geometry and the reciprocal
// distance are shared; each set keeps its own sums in the same order as alone): one warp;
// sources of the adjacent leaves spread over the lanes (x, y, z, q in one vector load; each
// lane takes two sources per step and already loads the next two); targets in registers;
// coordinates leaf-local (leaf units), so FP32 keeps the relative precision of close
// pairs. The per-lane sums are reduced over the warp in a fixed order, lane j then
// evaluates the local expansion(s) at target j.
template <typename T, int NT, int NQ>
__device__ __forceinline__ void l2p_p2p_pass(int leaf, int tb, int nt, int lane, int li, int lj, int lk,
                                             const int *__restrict__ leaf_src, const int *__restrict__ tgt_node,
                                             const T *__restrict__ tloc, const T *__restrict__ sloc,
                                             const int *__restrict__ leaf_ijk, const double *__restrict__ leaf_scale,
                                             const int *__restrict__ near_ptr, const int *__restrict__ near_leaf,
                                             size_t fbase, const NearSets<T> &sets) {
    using V4 = typename Vec4<T>::type;
    const V4 *__restrict__ src4 = reinterpret_cast<const V4 *>(sloc);
    const T *__restrict__ q2 = sets.q2;
    T tx[NT], ty[NT], tz[NT], ns[NQ][NT];
#pragma unroll
    for (int j = 0; j < NT; j++) {
        const int ti = tb + (j < nt ? j : 0);
        tx[j] = tloc[4 * (size_t)ti];
        ty[j] = tloc[4 * (size_t)ti + 1];
        tz[j] = tloc[4 * (size_t)ti + 2];
#pragma unroll
        for (int k = 0; k < NQ; k++) ns[k][j] = 0;
    }
    for (int e = near_ptr[leaf]; e < near_ptr[leaf + 1]; e++) {
        const int nl = near_leaf[e];
        // source coordinates relative to this leaf: own leaf-local + integer leaf offset
        const T ox = T(leaf_ijk[3 * nl] - li), oy = T(leaf_ijk[3 * nl + 1] - lj), oz = T(leaf_ijk[3 * nl + 2] - lk);
        const int s0 = leaf_src[nl], s1 = leaf_src[nl + 1];
        T acc[NQ][NT];
#pragma unroll
        for (int j = 0; j < NT; j++)
#pragma unroll
            for (int k = 0; k < NQ; k++) acc[k][j] = 0;
        // a missing source is a zero charge far away
        V4 far;
        far.x = far.y = far.z = T(1e4);
        far.w = T(0);
        int s = s0 + lane;
        V4 na = s < s1 ? src4[s] : far, nb = s + 32 < s1 ? src4[s + 32] : far;
        T na2 = 0, nb2 = 0;
        if constexpr (NQ == 2) {
            na2 = s < s1 ? q2[s] : T(0);
            nb2 = s + 32 < s1 ? q2[s + 32] : T(0);
        }
        for (; s < s1; s += 64) {
            const V4 sa = na, sb = nb;
            const T aq2 = na2, bq2 = nb2;
            na = s + 64 < s1 ? src4[s + 64] : far;
            nb = s + 96 < s1 ? src4[s + 96] : far;
            if constexpr (NQ == 2) {
                na2 = s + 64 < s1 ? q2[s + 64] : T(0);
                nb2 = s + 96 < s1 ? q2[s + 96] : T(0);
            }
            const T ax = sa.x + ox, ay = sa.y + oy, az = sa.z + oz, aq = sa.w;
            const T bx = sb.x + ox, by = sb.y + oy, bz = sb.z + oz, bq = sb.w;
#pragma unroll
            for (int j = 0; j < NT; j++) {
                const T dx = tx[j] - ax, dy = ty[j] - ay, dz = tz[j] - az;
                const T ex = tx[j] - bx, ey = ty[j] - by, ez = tz[j] - bz;
                const T ra = rsqrt_p<T>(dx * dx + dy * dy + dz * dz);
                const T rb = rsqrt_p<T>(ex * ex + ey * ey + ez * ez);
                acc[0][j] += aq * ra;
                acc[0][j] += bq * rb;
                if constexpr (NQ == 2) {
                    acc[1][j] += aq2 * ra;
                    acc[1][j] += bq2 * rb;
                }
            }
        }
#pragma unroll
        for (int j = 0; j < NT; j++)
#pragma unroll
            for (int k = 0; k < NQ; k++) ns[k][j] += acc[k][j];
    }
    // warp sums in the path's precision (fixed butterfly order), then FP64
    double near[NQ][NT];
#pragma unroll
    for (int k = 0; k < NQ; k++)
#pragma unroll
        for (int j = 0; j < NT; j++) {
            T v = ns[k][j];
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
            near[k][j] = double(v);
        }
    if (lane < nt) {
        T x = 0, y = 0, z = 0;
        double nr[NQ];
#pragma unroll
        for (int k = 0; k < NQ; k++) nr[k] = 0;
#pragma unroll
        for (int j = 0; j < NT; j++)
            if (j == lane) {
                x = tx[j]; y = ty[j]; z = tz[j];
#pragma unroll
                for (int k = 0; k < NQ; k++) nr[k] = near[k][j];
            }
        if (sets.near_only) {
            const int node = tgt_node[tb + lane];
#pragma unroll
            for (int k = 0; k < NQ; k++) sets.pot[k][node] = nr[k];
            return;
        }
        const T *__restrict__ Fa = sets.F[0] + fbase;
        const T *__restrict__ Fb = sets.F[NQ - 1] + fbase;
        T fa = 0, fb = 0;
        ups_cols<T>(x, y, z, [&](int n, int m, T re, T im) {
            if (m == 0) {
                fa += Fa[ridx(n, 0, 0)] * re;
                if constexpr (NQ == 2) fb += Fb[ridx(n, 0, 0)] * re;
            } else {
                fa += T(2) * (Fa[ridx(n, m, 0)] * re + Fa[ridx(n, m, 1)] * im);
                if constexpr (NQ == 2) fb += T(2) * (Fb[ridx(n, m, 0)] * re + Fb[ridx(n, m, 1)] * im);
            }
        });
        const double sc = leaf_scale[leaf];
        const int node = tgt_node[tb + lane];
        sets.pot[0][node] = (double(fa) + nr[0]) * sc;
        if constexpr (NQ == 2) sets.pot[1][node] = (double(fb) + nr[NQ - 1]) * sc;
    }
}

// The FP32 pass of l2p_p2p_pass with the pair arithmetic on packed target pairs: per two
// pairs 3 subtractions, 3 for r^2 (d_x^2, then + d_y^2, + d_z^2 as fused multiply-adds),
// two SFU reciprocal square roots and one fused multiply-add per charge set, the pair
// arithmetic of the scalar pass. The terms go straight into the pass sums (no per-leaf
// partial sums as in the scalar pass): 128 registers, so four blocks fit on an SM, or one
// beside a tensor-core translation CTA (1.61 -> 1.49 ms on the film, 1.26 with evenly shared
// tasks; the FP32 FMM's error against the FP64 FMM stays 4.7e-7 for the potential of m, 1.1e-6
// instead of 7e-7 for the potential of v).
template <int NT, int NQ>
__device__ __forceinline__ void l2p_p2p_pass_x2(int leaf, int tb, int nt, int lane, int li, int lj, int lk,
                                                const int *__restrict__ leaf_src, const int *__restrict__ tgt_node,
                                                const float *__restrict__ tloc, const float *__restrict__ sloc,
                                                const int *__restrict__ leaf_ijk,
                                                const double *__restrict__ leaf_scale,
                                                const int *__restrict__ near_ptr, const int *__restrict__ near_leaf,
                                                size_t fbase, const NearSets<float> &sets) {
    static_assert(NT % 2 == 0, "targets come in pairs");
    constexpr int NP = NT / 2;
    const float4 *__restrict__ src4 = reinterpret_cast<const float4 *>(sloc);
    const float *__restrict__ q2 = sets.q2;
    u64 TX[NP], TY[NP], TZ[NP], NS[NQ][NP];
#pragma unroll
    for (int p = 0; p < NP; p++) {
        const int t0 = tb + (2 * p < nt ? 2 * p : 0), t1 = tb + (2 * p + 1 < nt ? 2 * p + 1 : 0);
        TX[p] = pk2(tloc[4 * (size_t)t0], tloc[4 * (size_t)t1]);
        TY[p] = pk2(tloc[4 * (size_t)t0 + 1], tloc[4 * (size_t)t1 + 1]);
        TZ[p] = pk2(tloc[4 * (size_t)t0 + 2], tloc[4 * (size_t)t1 + 2]);
#pragma unroll
        for (int k = 0; k < NQ; k++) NS[k][p] = 0ull;
    }
    for (int e = near_ptr[leaf]; e < near_ptr[leaf + 1]; e++) {
        const int nl = near_leaf[e];
        const float ox = float(leaf_ijk[3 * nl] - li), oy = float(leaf_ijk[3 * nl + 1] - lj),
                    oz = float(leaf_ijk[3 * nl + 2] - lk);
        const int s0 = leaf_src[nl], s1 = leaf_src[nl + 1];
        const float4 far = make_float4(1e4f, 1e4f, 1e4f, 0.f);  // a missing source: zero charge far away
        int s = s0 + lane;
        float4 na = s < s1 ? src4[s] : far, nb = s + 32 < s1 ? src4[s + 32] : far;
        float na2 = 0.f, nb2 = 0.f;
        if constexpr (NQ == 2) {
            na2 = s < s1 ? q2[s] : 0.f;
            nb2 = s + 32 < s1 ? q2[s + 32] : 0.f;
        }
        for (; s < s1; s += 64) {
            const float4 sa = na, sb = nb;
            const float aq2 = na2, bq2 = nb2;
            na = s + 64 < s1 ? src4[s + 64] : far;
            nb = s + 96 < s1 ? src4[s + 96] : far;
            if constexpr (NQ == 2) {
                na2 = s + 64 < s1 ? q2[s + 64] : 0.f;
                nb2 = s + 96 < s1 ? q2[s + 96] : 0.f;
            }
            const float ax = sa.x + ox, ay = sa.y + oy, az = sa.z + oz;
            const float bx = sb.x + ox, by = sb.y + oy, bz = sb.z + oz;
            const u64 AX = pk2(ax, ax), AY = pk2(ay, ay), AZ = pk2(az, az), AQ = pk2(sa.w, sa.w);
            const u64 BX = pk2(bx, bx), BY = pk2(by, by), BZ = pk2(bz, bz), BQ = pk2(sb.w, sb.w);
            const u64 AQ2 = pk2(aq2, aq2), BQ2 = pk2(bq2, bq2);
#pragma unroll
            for (int p = 0; p < NP; p++) {
                const u64 dx = sub2(TX[p], AX), dy = sub2(TY[p], AY), dz = sub2(TZ[p], AZ);
                const u64 ex = sub2(TX[p], BX), ey = sub2(TY[p], BY), ez = sub2(TZ[p], BZ);
                const u64 da = fma2(dz, dz, fma2(dy, dy, mul2(dx, dx)));
                const u64 db = fma2(ez, ez, fma2(ey, ey, mul2(ex, ex)));
                float a0, a1, b0, b1;
                upk2(da, a0, a1);
                upk2(db, b0, b1);
                const u64 RA = pk2(rsqrt_p<float>(a0), rsqrt_p<float>(a1));
                const u64 RB = pk2(rsqrt_p<float>(b0), rsqrt_p<float>(b1));
                NS[0][p] = fma2(AQ, RA, NS[0][p]);
                NS[0][p] = fma2(BQ, RB, NS[0][p]);
                if constexpr (NQ == 2) {
                    NS[1][p] = fma2(AQ2, RA, NS[1][p]);
                    NS[1][p] = fma2(BQ2, RB, NS[1][p]);
                }
            }
        }
    }
    // warp sums (fixed butterfly order), then FP64
    double near[NQ][NT];
#pragma unroll
    for (int k = 0; k < NQ; k++)
#pragma unroll
        for (int p = 0; p < NP; p++) {
            float v0, v1;
            upk2(NS[k][p], v0, v1);
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) {
                v0 += __shfl_xor_sync(0xffffffffu, v0, o);
                v1 += __shfl_xor_sync(0xffffffffu, v1, o);
            }
            near[k][2 * p] = double(v0);
            near[k][2 * p + 1] = double(v1);
        }
    if (lane < nt) {
        float x = 0, y = 0, z = 0;
        double nr[NQ];
#pragma unroll
        for (int k = 0; k < NQ; k++) nr[k] = 0;
#pragma unroll
        for (int p = 0; p < NP; p++) {
            float x0, x1, y0, y1, z0, z1;
            upk2(TX[p], x0, x1);
            upk2(TY[p], y0, y1);
            upk2(TZ[p], z0, z1);
            if (2 * p == lane) {
                x = x0; y = y0; z = z0;
#pragma unroll
                for (int k = 0; k < NQ; k++) nr[k] = near[k][2 * p];
            }
            if (2 * p + 1 == lane) {
                x = x1; y = y1; z = z1;
#pragma unroll
                for (int k = 0; k < NQ; k++) nr[k] = near[k][2 * p + 1];
            }
        }
        if (sets.near_only) {
            const int node = tgt_node[tb + lane];
#pragma unroll
            for (int k = 0; k < NQ; k++) sets.pot[k][node] = nr[k];
            return;
        }
        const float *__restrict__ Fa = sets.F[0] + fbase;
        const float *__restrict__ Fb = sets.F[NQ - 1] + fbase;
        float fa = 0, fb = 0;
        ups_cols<float>(x, y, z, [&](int n, int m, float re, float im) {
            if (m == 0) {
                fa += Fa[ridx(n, 0, 0)] * re;
                if constexpr (NQ == 2) fb += Fb[ridx(n, 0, 0)] * re;
            } else {
                fa += 2.f * (Fa[ridx(n, m, 0)] * re + Fa[ridx(n, m, 1)] * im);
                if constexpr (NQ == 2) fb += 2.f * (Fb[ridx(n, m, 0)] * re + Fb[ridx(n, m, 1)] * im);
            }
        });
        const double sc = leaf_scale[leaf];
        const int node = tgt_node[tb + lane];
        sets.pot[0][node] = (double(fa) + nr[0]) * sc;
        if constexpr (NQ == 2) sets.pot[1][node] = (double(fb) + nr[NQ - 1]) * sc;
    }
}

// L2P + P2P of the FP32 path: one warp per task, up to 16 targets of a leaf (the leaf's targets
// shared out in pairs as evenly as they go, the pass instantiated for every number of pairs, so
// at most one target of a leaf is padding). Sources, lanes and sums are those of a warp that walks
// the whole leaf: the potentials do not depend on the tasks. Bound by the FP32 and SFU pipes, each
// at 16 pairs per clock and SM.
constexpr int P2P32_NT = 16;
template <int NQ>
__global__ void __launch_bounds__(128, 4)  // 128 registers, 4 blocks per SM
    k_l2p_p2p(int ntask, const int4 *__restrict__ task, const int *__restrict__ leaf_src,
              const int *__restrict__ tgt_node, const float *__restrict__ tloc, const float *__restrict__ sloc,
              const int *__restrict__ leaf_ijk, int leaf0, const double *__restrict__ leaf_scale,
              const int *__restrict__ near_ptr, const int *__restrict__ near_leaf, NearSets<float> sets) {
    const int lane = threadIdx.x & 31, k = blockIdx.x * 4 + (threadIdx.x >> 5);
    if (k >= ntask) return;
    const int4 t = task[k];  // leaf, first target, targets
    const int leaf = t.x, li = leaf_ijk[3 * leaf], lj = leaf_ijk[3 * leaf + 1], lk = leaf_ijk[3 * leaf + 2];
    const size_t fbase = (size_t)(leaf0 + leaf) * NR;
#define FG_PASS(N)                                                                                                  \
    case N:                                                                                                         \
        l2p_p2p_pass_x2<2 * N, NQ>(leaf, t.y, t.z, lane, li, lj, lk, leaf_src, tgt_node, tloc, sloc, leaf_ijk,      \
                                   leaf_scale, near_ptr, near_leaf, fbase, sets);                                   \
        break;
    switch ((t.z + 1) / 2) {
        FG_PASS(1) FG_PASS(2) FG_PASS(3) FG_PASS(4) FG_PASS(5) FG_PASS(6) FG_PASS(7) FG_PASS(8)
    }
#undef FG_PASS
}

// L2P + P2P on the FP64 pipe (fmm_native_fp64): one warp per target leaf, its targets in passes of 16
// and a tail pass of 8 or 4.
template <int NQ>
__global__ void __launch_bounds__(128, 2)
    k_l2p_p2p_fp64(int nleaf, const int *__restrict__ leaf_src, const int *__restrict__ leaf_tgt,
                   const int *__restrict__ tgt_node, const double *__restrict__ tloc, const double *__restrict__ sloc,
                   const int *__restrict__ leaf_ijk, int leaf0, const double *__restrict__ leaf_scale,
                   const int *__restrict__ near_ptr, const int *__restrict__ near_leaf, NearSets<double> sets) {
    const int lane = threadIdx.x & 31;
    const int leaf = blockIdx.x * 4 + (threadIdx.x >> 5);
    if (leaf >= nleaf) return;
    const int t0 = leaf_tgt[leaf], t1 = leaf_tgt[leaf + 1];
    if (t0 == t1) return;
    const int li = leaf_ijk[3 * leaf], lj = leaf_ijk[3 * leaf + 1], lk = leaf_ijk[3 * leaf + 2];
    const size_t fbase = (size_t)(leaf0 + leaf) * NR;
    for (int tb = t0; tb < t1;) {
        const int r = t1 - tb;
        const int nt = r > 8 ? 16 : r > 4 ? 8 : 4;
        if (nt == 16)
            l2p_p2p_pass<double, 16, NQ>(leaf, tb, min(16, r), lane, li, lj, lk, leaf_src, tgt_node, tloc, sloc,
                                         leaf_ijk, leaf_scale, near_ptr, near_leaf, fbase, sets);
        else if (nt == 8)
            l2p_p2p_pass<double, 8, NQ>(leaf, tb, r, lane, li, lj, lk, leaf_src, tgt_node, tloc, sloc, leaf_ijk,
                                        leaf_scale, near_ptr, near_leaf, fbase, sets);
        else
            l2p_p2p_pass<double, 4, NQ>(leaf, tb, r, lane, li, lj, lk, leaf_src, tgt_node, tloc, sloc, leaf_ijk,
                                        leaf_scale, near_ptr, near_leaf, fbase, sets);
        tb += nt;
    }
}

// Double-single arithmetic on the FP32 pipes: an FP64-accurate near field for the FP64
// path, whose FP64 pipe (2 DFMA per clock and SM on this GPU) would otherwise bound it.
// A value is hi + lo with |lo| <= ulp(hi)/2 (Dekker, "A floating-point technique for
// extending the available precision", 1971; Knuth's two-sum).
__device__ __forceinline__ void ds_two_sum(float a, float b, float &s, float &e) {
    s = a + b;
    const float bb = s - a;
    e = (a - (s - bb)) + (b - bb);
}

// Near field of the FP64 path in double-single arithmetic. Coordinates are leaf-local with hi
// parts on a 2^-20 grid (|x| < 4, so hi - hi' is exact in FP32) and lo = x - hi (|lo| <= 2^-21,
// held to 2^-45); per pair: d = (hi - hi') + (lo - lo'), r^2 as a double-single sum of the
// squares (the leading products exact through fma), 1/r from the SFU estimate y and
// y (1 + e/2 + 3 e^2/8), e = 1 - r^2 y^2 formed exactly to about 2^-46, q/r as a double-single
// product, summed with two-sum: 69 FP32 operations per pair for two charge sets, 45 of them for
// the geometry the sets share, so the FP32 pipe (128 lanes per clock and SM) bounds it.
//
// One block per task: up to 8 target nodes of one leaf (the leaf's targets shared out evenly),
// held in registers by every thread; the sources of all its adjacent leaves, one list, are
// spread over the 128 threads, so lanes idle only at the end of that list and a tree of a few
// hundred leaves still gives every SM work. Sums over the threads in FP64 in a fixed order.
constexpr int P2P_NT = 8;
template <int NT, int NQ>
__device__ __forceinline__ void p2p_ds_pass(int tb, int ntot, const int *seg_src, const int *seg_end,
                                            const float (*seg_off)[3], const float4 *__restrict__ th4,
                                            const float4 *__restrict__ tl4, const float4 *__restrict__ sh4,
                                            const float4 *__restrict__ sl4, const float *__restrict__ q2h,
                                            const float *__restrict__ q2l, double (&out)[NQ * P2P_NT]) {
    float thx[NT], thy[NT], thz[NT], tlx[NT], tly[NT], tlz[NT], ah[NQ][NT], al[NQ][NT];
#pragma unroll
    for (int j = 0; j < NT; j++) {
        const float4 h = __ldg(th4 + tb + j), l = __ldg(tl4 + tb + j);
        thx[j] = h.x; thy[j] = h.y; thz[j] = h.z;
        tlx[j] = l.x; tly[j] = l.y; tlz[j] = l.z;
#pragma unroll
        for (int k = 0; k < NQ; k++) ah[k][j] = al[k][j] = 0.f;
    }
    int e = 0;
    for (int i = threadIdx.x; i < ntot; i += 128) {
        while (i >= seg_end[e]) e++;
        const int s = seg_src[e] + i;
        const float4 h = sh4[s], l = sl4[s];
        // integer offset of the adjacent leaf, added exactly to the hi parts
        const float sx = h.x + seg_off[e][0], sy = h.y + seg_off[e][1], sz = h.z + seg_off[e][2];
        float qh[NQ], ql[NQ];
        qh[0] = h.w;
        ql[0] = l.w;
        if constexpr (NQ == 2) {
            qh[1] = q2h[s];
            ql[1] = q2l[s];
        }
#pragma unroll
        for (int j = 0; j < NT; j++) {
            const float d1x = thx[j] - sx, d1y = thy[j] - sy, d1z = thz[j] - sz;  // exact
            const float d2x = tlx[j] - l.x, d2y = tly[j] - l.y, d2z = tlz[j] - l.z;
            // squares: d^2 = d1^2 + d2 (2 d1 + d2), leading products exact
            const float px = d1x * d1x, py = d1y * d1y, pz = d1z * d1z;
            const float ex = fmaf(d2x, fmaf(2.f, d1x, d2x), fmaf(d1x, d1x, -px));
            const float ey = fmaf(d2y, fmaf(2.f, d1y, d2y), fmaf(d1y, d1y, -py));
            const float ez = fmaf(d2z, fmaf(2.f, d1z, d2z), fmaf(d1z, d1z, -pz));
            float s1_, e1, s2_, e2;
            ds_two_sum(px, py, s1_, e1);
            ds_two_sum(s1_, pz, s2_, e2);
            const float eps = (e1 + e2) + ((ex + ey) + ez);
            const float Sh = s2_ + eps, Sl = eps - (Sh - s2_);
            const float y = rsqrt_p<float>(Sh);
            const float p = Sh * y, pe = fmaf(Sl, y, fmaf(Sh, y, -p));  // r^2 y
            const float del = fmaf(-pe, y, fmaf(-p, y, 1.f));
            const float yl = (y * del) * fmaf(0.375f, del, 0.5f);
            // q / r = (qh + ql)(y + yl), accumulated with two-sum
#pragma unroll
            for (int k = 0; k < NQ; k++) {
                const float c1 = qh[k] * y;
                const float c2 = fmaf(ql[k], y, fmaf(qh[k], yl, fmaf(qh[k], y, -c1)));
                float sn, en;
                ds_two_sum(ah[k][j], c1, sn, en);
                ah[k][j] = sn;
                al[k][j] += en + c2;
            }
        }
    }
#pragma unroll
    for (int k = 0; k < NQ; k++)
#pragma unroll
        for (int j = 0; j < NT; j++) out[k * P2P_NT + j] = double(ah[k][j]) + double(al[k][j]);
}

template <int NQ>
__global__ void __launch_bounds__(128, 4) k_p2p_ds(const int4 *__restrict__ task, const int *__restrict__ leaf_src,
                                                   const int *__restrict__ tgt_node, const float4 *__restrict__ th4,
                                                   const float4 *__restrict__ tl4, const float4 *__restrict__ sh4,
                                                   const float4 *__restrict__ sl4, const float *__restrict__ q2h,
                                                   const float *__restrict__ q2l, const int *__restrict__ leaf_ijk,
                                                   const int *__restrict__ near_ptr, const int *__restrict__ near_leaf,
                                                   double *__restrict__ pot0, double *__restrict__ pot1) {
    // the adjacent leaves as one list of sources: source i of the list, seg_end[e - 1] <= i <
    // seg_end[e], is source seg_src[e] + i
    __shared__ int seg_src[28], seg_end[28];
    __shared__ float seg_off[28][3];
    constexpr int NV = NQ * P2P_NT;
    __shared__ double red[4][NV];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int4 t = task[blockIdx.x];
    const int leaf = t.x, tb = t.y, nt = t.z;
    const int e0 = near_ptr[leaf], ne = near_ptr[leaf + 1] - e0;
    if (warp == 0) {
        int s0 = 0, n = 0;
        if (lane < ne) {
            const int nl = near_leaf[e0 + lane];
            s0 = leaf_src[nl];
            n = leaf_src[nl + 1] - s0;
#pragma unroll
            for (int d = 0; d < 3; d++) seg_off[lane][d] = float(leaf_ijk[3 * nl + d] - leaf_ijk[3 * leaf + d]);
        }
        int end = n;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const int x = __shfl_up_sync(0xffffffffu, end, o);
            if (lane >= o) end += x;
        }
        if (lane < 28) {
            seg_src[lane] = s0 - (end - n);
            seg_end[lane] = end;
        }
    }
    __syncthreads();
    const int ntot = ne > 0 ? seg_end[ne - 1] : 0;
    double v[NV];
#pragma unroll
    for (int k = 0; k < NV; k++) v[k] = 0.0;
#define FG_P2P(N)                                                                                                  \
    case N:                                                                                                        \
        p2p_ds_pass<N, NQ>(tb, ntot, seg_src, seg_end, seg_off, th4, tl4, sh4, sl4, q2h, q2l, v);                  \
        break;
    switch (nt) {
        FG_P2P(1) FG_P2P(2) FG_P2P(3) FG_P2P(4) FG_P2P(5) FG_P2P(6) FG_P2P(7) FG_P2P(8)
    }
#undef FG_P2P
    // sums over the warp: the halves of the values are exchanged until each lane holds one, in the
    // order of a butterfly over lane bits 4 to 0 for every value
    int n = NV;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        if (n > 1) {
            n >>= 1;
            const bool hi = lane & o;
#pragma unroll
            for (int k = 0; k < NV / 2; k++)
                if (k < n) {
                    const double send = hi ? v[k] : v[k + n], keep = hi ? v[k + n] : v[k];
                    v[k] = keep + __shfl_xor_sync(0xffffffffu, send, o);
                }
        } else {
            v[0] += __shfl_xor_sync(0xffffffffu, v[0], o);
        }
    }
    constexpr int DUP = 32 / NV;  // lanes holding each value
    if (lane % DUP == 0) red[warp][lane / DUP] = v[0];
    __syncthreads();
    if (threadIdx.x < NV) {
        const int k = threadIdx.x / P2P_NT, j = threadIdx.x % P2P_NT;
        if (j < nt)
            (k ? pot1 : pot0)[tgt_node[tb + j]] =
                ((red[0][threadIdx.x] + red[1][threadIdx.x]) + red[2][threadIdx.x]) + red[3][threadIdx.x];
    }
}

// P2P in double-single arithmetic of the full FP64 evaluation of the FP32 + refinement path
// (FmmTree::repeat): the operations of k_p2p_ds but for 1/r (one Newton step evaluated in
// double-single, error ~1e-13) and the order of the sums: sources of each adjacent leaf spread over
// the lanes of one warp, per-lane sums reduced over the warp in FP64. A warp takes a task of up to 8
// targets of a leaf, the leaf's targets shared out evenly (a warp per leaf, in passes of 8 targets
// whatever was left, with the local expansions behind them, gave each SM a dozen unequal warps;
// 294k tets, two sets: 4.85 -> 2.23 ms and 0.09 for the local expansions; packed pairs of targets 2.14).
template <int NP, int NQ>
__device__ __forceinline__ void p2p_repeat_pass(int lane, int leaf, int tb, int nt, const int *__restrict__ leaf_src,
                                                const int *__restrict__ tgt_node, const float4 *__restrict__ th4,
                                                const float4 *__restrict__ tl4, const float4 *__restrict__ sh4,
                                                const float4 *__restrict__ sl4, const float *__restrict__ q2h,
                                                const float *__restrict__ q2l, const int *__restrict__ leaf_ijk,
                                                const int *__restrict__ near_ptr, const int *__restrict__ near_leaf,
                                                double *__restrict__ pot0, double *__restrict__ pot1) {
    const int li = leaf_ijk[3 * leaf], lj = leaf_ijk[3 * leaf + 1], lk = leaf_ijk[3 * leaf + 2];
    u64 thx[NP], thy[NP], thz[NP], tlx[NP], tly[NP], tlz[NP], ah[NQ][NP], al[NQ][NP];
#pragma unroll
    for (int j = 0; j < NP; j++) {
        const int t0 = tb + 2 * j, t1 = tb + min(2 * j + 1, nt - 1);
        const float4 h = th4[t0], l = tl4[t0], h1 = th4[t1], l1 = tl4[t1];
        thx[j] = pk2(h.x, h1.x); thy[j] = pk2(h.y, h1.y); thz[j] = pk2(h.z, h1.z);
        tlx[j] = pk2(l.x, l1.x); tly[j] = pk2(l.y, l1.y); tlz[j] = pk2(l.z, l1.z);
#pragma unroll
        for (int k = 0; k < NQ; k++) ah[k][j] = al[k][j] = 0ull;
    }
    const u64 two = pk2(2.f, 2.f), one = pk2(1.f, 1.f), half = pk2(0.5f, 0.5f);
    for (int e = near_ptr[leaf]; e < near_ptr[leaf + 1]; e++) {
        const int nl = near_leaf[e];
        // integer offset of the adjacent leaf, added exactly to the hi parts
        const float ox = float(leaf_ijk[3 * nl] - li), oy = float(leaf_ijk[3 * nl + 1] - lj),
                    oz = float(leaf_ijk[3 * nl + 2] - lk);
        const int s0 = leaf_src[nl], s1 = leaf_src[nl + 1];
        for (int s = s0 + lane; s < s1; s += 32) {
            const float4 h = sh4[s], l = sl4[s];
            const float sx = h.x + ox, sy = h.y + oy, sz = h.z + oz;
            const u64 SX = pk2(sx, sx), SY = pk2(sy, sy), SZ = pk2(sz, sz);
            const u64 LX = pk2(l.x, l.x), LY = pk2(l.y, l.y), LZ = pk2(l.z, l.z);
            u64 qh[NQ], ql[NQ];
            qh[0] = pk2(h.w, h.w);
            ql[0] = pk2(l.w, l.w);
            if constexpr (NQ == 2) {
                const float a = q2h[s], b = q2l[s];
                qh[1] = pk2(a, a);
                ql[1] = pk2(b, b);
            }
#pragma unroll
            for (int j = 0; j < NP; j++) {
                const u64 d1x = sub2(thx[j], SX), d1y = sub2(thy[j], SY), d1z = sub2(thz[j], SZ);  // exact
                const u64 d2x = sub2(tlx[j], LX), d2y = sub2(tly[j], LY), d2z = sub2(tlz[j], LZ);
                // squares: d^2 = d1^2 + d2 (2 d1 + d2), leading products exact
                const u64 px = mul2(d1x, d1x), py = mul2(d1y, d1y), pz = mul2(d1z, d1z);
                u64 ex = fma2(d1x, d1x, neg2(px)), ey = fma2(d1y, d1y, neg2(py)), ez = fma2(d1z, d1z, neg2(pz));
                ex = fma2(d2x, fma2(two, d1x, d2x), ex);
                ey = fma2(d2y, fma2(two, d1y, d2y), ey);
                ez = fma2(d2z, fma2(two, d1z, d2z), ez);
                const ds2 r1 = ds2_two_sum(px, py), r2 = ds2_two_sum(r1.h, pz);
                const u64 el = add2(add2(r1.l, r2.l), add2(add2(ex, ey), ez));
                const u64 Sh = add2(r2.h, el), Sl = sub2(el, sub2(Sh, r2.h));
                // 1/sqrt(S): SFU estimate y, then y (1 + (1 - S y^2) / 2) with S y^2 in
                // double-single (1 - S y^2 is small and exact to ~2^-46)
                float S0, S1;
                upk2(Sh, S0, S1);
                const u64 y = pk2(rsqrt_p<float>(S0), rsqrt_p<float>(S1));
                const u64 t1 = mul2(y, y), t2 = fma2(y, y, neg2(t1));
                const u64 u1 = mul2(Sh, t1);
                const u64 u2 = add2(fma2(Sh, t1, neg2(u1)), fma2(Sh, t2, mul2(Sl, t1)));
                const u64 delta = sub2(sub2(one, u1), u2);
                const u64 yl = mul2(mul2(half, y), delta);
                // q / r = (qh + ql)(y + yl), accumulated with two-sum
#pragma unroll
                for (int k = 0; k < NQ; k++) {
                    const u64 c1 = mul2(qh[k], y);
                    const u64 c2 = add2(fma2(qh[k], y, neg2(c1)), fma2(qh[k], yl, mul2(ql[k], y)));
                    const ds2 sn = ds2_two_sum(ah[k][j], c1);
                    ah[k][j] = sn.h;
                    al[k][j] = add2(al[k][j], add2(sn.l, c2));
                }
            }
        }
    }
#pragma unroll
    for (int k = 0; k < NQ; k++)
#pragma unroll
        for (int j = 0; j < 2 * NP; j++) {
            float h[2], l[2];
            upk2(ah[k][j / 2], h[0], h[1]);
            upk2(al[k][j / 2], l[0], l[1]);
            double v = double(h[j % 2]) + double(l[j % 2]);
            for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
            if (lane == j && j < nt) (k ? pot1 : pot0)[tgt_node[tb + j]] = v;
        }
}

template <int NQ>
__global__ void __launch_bounds__(128, 4)
    k_p2p_ds_repeat(int ntask, const int4 *__restrict__ task, const int *__restrict__ leaf_src,
                    const int *__restrict__ tgt_node, const float4 *__restrict__ th4, const float4 *__restrict__ tl4,
                    const float4 *__restrict__ sh4, const float4 *__restrict__ sl4, const float *__restrict__ q2h,
                    const float *__restrict__ q2l, const int *__restrict__ leaf_ijk, const int *__restrict__ near_ptr,
                    const int *__restrict__ near_leaf, double *__restrict__ pot0, double *__restrict__ pot1) {
    const int lane = threadIdx.x & 31, w = blockIdx.x * 4 + (threadIdx.x >> 5);
    if (w >= ntask) return;
    const int4 t = task[w];
#define FG_P2P(N)                                                                                                   \
    case N:                                                                                                         \
        p2p_repeat_pass<N, NQ>(lane, t.x, t.y, t.z, leaf_src, tgt_node, th4, tl4, sh4, sl4, q2h, q2l, leaf_ijk,      \
                               near_ptr, near_leaf, pot0, pot1);                                                    \
        break;
    switch ((t.z + 1) / 2) {
        FG_P2P(1) FG_P2P(2) FG_P2P(3) FG_P2P(4)
    }
#undef FG_P2P
}

// L2P after a near field that stored its sums: one thread per target evaluates its leaf's local
// expansion(s) and forms the potential from the stored near sum with the operations of the fused
// FP32 pass, pot = (far + near) * scale. Threads of a warp are targets of one or two leaves, so
// every lane works (one warp per leaf left lanes idle, which on the 1/64-rate FP64 pipe that
// bounds the FP64 form costs as much as work). The loads are volatile so that they stay beside
// their use: hoisted together they spilled.
__device__ __forceinline__ float ld_here(const float *p) {
    float v;
    asm volatile("ld.global.nc.f32 %0, [%1];" : "=f"(v) : "l"(p));
    return v;
}
__device__ __forceinline__ double ld_here(const double *p) {
    double v;
    asm volatile("ld.global.nc.f64 %0, [%1];" : "=d"(v) : "l"(p));
    return v;
}
template <typename T, int NQ>
__global__ void __launch_bounds__(128) k_l2p(int ntgt, const int *__restrict__ tgt_leaf,
                                             const int *__restrict__ tgt_node, const T *__restrict__ tloc, int leaf0,
                                             const double *__restrict__ leaf_scale, NearSets<T> sets) {
    const int ti = blockIdx.x * 128 + threadIdx.x;
    if (ti >= ntgt) return;
    const int leaf = tgt_leaf[ti];
    const size_t fbase = (size_t)(leaf0 + leaf) * NR;
    const double sc = leaf_scale[leaf];
    const T *Fa = sets.F[0] + fbase, *Fb = sets.F[NQ - 1] + fbase;
    const T x = tloc[4 * (size_t)ti], y = tloc[4 * (size_t)ti + 1], z = tloc[4 * (size_t)ti + 2];
    T fa = 0, fb = 0;
    ups_cols<T>(x, y, z, [&](int n, int m, T re, T im) {
        if (m == 0) {
            fa += ld_here(Fa + ridx(n, 0, 0)) * re;
            if constexpr (NQ == 2) fb += ld_here(Fb + ridx(n, 0, 0)) * re;
        } else {
            fa += T(2) * (ld_here(Fa + ridx(n, m, 0)) * re + ld_here(Fa + ridx(n, m, 1)) * im);
            if constexpr (NQ == 2) fb += T(2) * (ld_here(Fb + ridx(n, m, 0)) * re + ld_here(Fb + ridx(n, m, 1)) * im);
        }
    });
    const int node = tgt_node[ti];
    sets.pot[0][node] = (double(fa) + sets.pot[0][node]) * sc;
    if constexpr (NQ == 2) sets.pot[1][node] = (double(fb) + sets.pot[1][node]) * sc;
}

// ---------------------------------------------------------------------------------
// host: tree construction

static inline uint64_t spread3(uint64_t v) {
    v &= 0x1fffff;
    v = (v | v << 32) & 0x1f00000000ffffull;
    v = (v | v << 16) & 0x1f0000ff0000ffull;
    v = (v | v << 8) & 0x100f00f00f00f00full;
    v = (v | v << 4) & 0x10c30c30c30c30c3ull;
    v = (v | v << 2) & 0x1249249249249249ull;
    return v;
}
static inline uint64_t morton(int x, int y, int z) { return spread3(x) | (spread3(y) << 1) | (spread3(z) << 2); }
static void decode(uint64_t k, int *ijk) {
    ijk[0] = ijk[1] = ijk[2] = 0;
    for (int b = 0; b < 21; b++) {
        ijk[0] |= (int)((k >> (3 * b)) & 1) << b;
        ijk[1] |= (int)((k >> (3 * b + 1)) & 1) << b;
        ijk[2] |= (int)((k >> (3 * b + 2)) & 1) << b;
    }
}

template <typename T>
static cudaError_t up(T **p, const std::vector<T> &h) {
    cudaError_t e = cudaMalloc((void **)p, std::max<size_t>(1, h.size()) * sizeof(T));
    if (e != cudaSuccess) return e;
    if (!h.empty()) e = cudaMemcpy(*p, h.data(), h.size() * sizeof(T), cudaMemcpyHostToDevice);
    return e;
}
template <typename T>
static cudaError_t up_as(void **p, const std::vector<double> &h, bool fp32) {
    if (fp32) {
        std::vector<float> f(h.begin(), h.end());
        return up((float **)p, f);
    }
    return up((double **)p, h);
}

#define FCK(call)                                                                   \
    do {                                                                            \
        cudaError_t e_ = (call);                                                    \
        if (e_ != cudaSuccess) {                                                    \
            c.err = std::string("fmm: ") + #call + ": " + cudaGetErrorString(e_);   \
            return FG_ECUDA;                                                        \
        }                                                                           \
    } while (0)

// Operator matrices (level independent), [code][out][in], in the real layout.
struct FmmOps {
    std::vector<double> m2l, m2m, l2l;
};
static const FmmOps &fmm_ops() {
    static FmmOps ops;
    if (!ops.m2l.empty()) return ops;
    const int P = FMM_P;
    ops.m2l.assign((size_t)NCODE_M2L * NR * NR, 0.0);
    ops.m2m.assign((size_t)8 * NR * NR, 0.0);
    ops.l2l.assign((size_t)8 * NR * NR, 0.0);
    std::vector<cd> T, U, in, out;
    std::vector<double> e(NR), r(NR);
    for (int dx = -3; dx <= 3; dx++)
        for (int dy = -3; dy <= 3; dy++)
            for (int dz = -3; dz <= 3; dz++) {
                if (std::abs(dx) <= 1 && std::abs(dy) <= 1 && std::abs(dz) <= 1) continue;
                const int code = (dx + 3) * 49 + (dy + 3) * 7 + (dz + 3);
                the_host(dx, dy, dz, 2 * P, T);
                for (int j = 0; j < NR; j++) {
                    std::fill(e.begin(), e.end(), 0.0);
                    e[j] = 1.0;
                    to_complex(e.data(), P, in);
                    m2l_c(in, T, P, out);
                    to_real(out, P, r.data());
                    for (int i = 0; i < NR; i++) ops.m2l[(size_t)code * NR * NR + (size_t)i * NR + j] = r[i];
                }
            }
    for (int oc = 0; oc < 8; oc++) {
        ups_host((oc & 1) ? 0.25 : -0.25, (oc & 2) ? 0.25 : -0.25, (oc & 4) ? 0.25 : -0.25, P, U);
        for (int j = 0; j < NR; j++) {
            std::fill(e.begin(), e.end(), 0.0);
            e[j] = 1.0;
            to_complex(e.data(), P, in);
            m2m_c(in, U, P, out);
            to_real(out, P, r.data());
            for (int i = 0; i < NR; i++) ops.m2m[(size_t)oc * NR * NR + (size_t)i * NR + j] = r[i];
            l2l_c(in, U, P, out);
            to_real(out, P, r.data());
            for (int i = 0; i < NR; i++) ops.l2l[(size_t)oc * NR * NR + (size_t)i * NR + j] = r[i];
        }
    }
    return ops;
}

// Power-of-two weights of the coefficients for the digit products (fg_fmm_oz.cu): multipoles by
// the inverse of the rms of Ups_n^m over the cell times 0.6^-n, locals by the inverse of the
// rms of The_n^m over the M2L offsets times 2.5^n. The factors share the decay with the degree
// between the operator and the expansion (of 1, 0.8, 0.6, 0.5 and of 1, 1.5, 2, 3 the errors were
// smallest there: 2e-16 to 2e-14 against up to 1e-12 without).
static void oz_weights(int *wM, int *wF) {
    const int P = FMM_P, G = 8;
    std::vector<double> m2(NR, 0.0), f2(NR, 0.0);
    std::vector<cd> X;
    for (int a = 0; a < G * G * G; a++) {
        ups_host((a % G + 0.5) / G - 0.5, (a / G % G + 0.5) / G - 0.5, (a / G / G + 0.5) / G - 0.5, P, X);
        for (int n = 0; n <= P; n++)
            for (int m = 0; m <= n; m++) {
                const cd v = X[cidx(n, m)];
                m2[ridx(n, m, 0)] += v.real() * v.real() / (G * G * G);
                if (m) m2[ridx(n, m, 1)] += v.imag() * v.imag() / (G * G * G);
            }
    }
    for (int code = 0; code < NCODE_M2L; code++) {
        const int d[3] = {code / 49 - 3, code / 7 % 7 - 3, code % 7 - 3};
        if (std::abs(d[0]) <= 1 && std::abs(d[1]) <= 1 && std::abs(d[2]) <= 1) continue;
        the_host(d[0], d[1], d[2], P, X);
        for (int n = 0; n <= P; n++)
            for (int m = 0; m <= n; m++)
                for (int part = 0; part < (m ? 2 : 1); part++) f2[ridx(n, m, part)] += std::norm(X[cidx(n, m)]) / 316.0;
    }
    for (int n = 0; n <= P; n++)
        for (int k = n * n; k < (n + 1) * (n + 1); k++) {
            wM[k] = -(int)std::lrint(0.5 * std::log2(m2[k]) - n * std::log2(0.6));
            wF[k] = -(int)std::lrint(0.5 * std::log2(f2[k]) + n * std::log2(2.5));
        }
}

void fmm_free(Ctx &c);
static void harvest_set(FmmTree &t, int k);
static int fmm_build_forest(Ctx &c, int L);
template <typename T>
static cudaError_t fmm_eval_t(Ctx &c, FmmTree &t, int nq, const FmmFields &f);
static FmmFields tuning_fields(const Ctx &c) { return {{c.u[1], c.v[1]}, {c.pot, c.pot2}}; }
static NearTree near_tree(const FmmTree &t) {
    NearTree n{};
    n.nleaf = t.nleaf; n.ntgt = t.ntgt;
    n.leaf_src = t.leaf_src; n.leaf_tgt = t.leaf_tgt; n.tgt_node = t.tgt_node; n.tgt_leaf = t.tgt_leaf;
    n.near_ptr = t.near_ptr; n.near_leaf = t.near_leaf; n.leaf_scale = t.leaf_scale;
    n.tloc = (const double4 *)t.tloc;
    return n;
}

// Points of each sample (sources and target nodes) and the sample's root cube. A batch of
// independent meshes gets one octree per sample (a forest); a single mesh is one tree.
struct SamplePts {
    std::vector<int> src, tgt;  // source indices, target node ids
    double c0[3] = {0, 0, 0}, side = 1.0;
};

// Centre and side of every sample's root cube.
static std::vector<double4> sample_roots(const std::vector<SamplePts> &S) {
    std::vector<double4> r(S.size());
    for (size_t g = 0; g < S.size(); g++) r[g] = make_double4(S[g].c0[0], S[g].c0[1], S[g].c0[2], S[g].side);
    return r;
}

static std::vector<SamplePts> split_samples(const Ctx &c) {
    const int nseg = std::max(1, c.nseg);
    std::vector<SamplePts> S(nseg);
    for (int s = 0; s < c.nsrc; s++) S[c.h_src_seg.empty() ? 0 : c.h_src_seg[s]].src.push_back(s);
    for (int i = 0; i < c.nn; i++)
        if (c.h_mag[i]) S[c.h_node_seg.empty() ? 0 : c.h_node_seg[i]].tgt.push_back(i);
    for (auto &P : S) {
        double lo[3] = {1e300, 1e300, 1e300}, hi[3] = {-1e300, -1e300, -1e300};
        for (int s : P.src)
            for (int d = 0; d < 3; d++) {
                lo[d] = std::min(lo[d], c.h_src_xyz[3 * (size_t)s + d]);
                hi[d] = std::max(hi[d], c.h_src_xyz[3 * (size_t)s + d]);
            }
        for (int i : P.tgt)
            for (int d = 0; d < 3; d++) {
                lo[d] = std::min(lo[d], c.h_xyz[3 * (size_t)i + d]);
                hi[d] = std::max(hi[d], c.h_xyz[3 * (size_t)i + d]);
            }
        if (P.src.empty() && P.tgt.empty()) continue;
        // the root cube of the reference: the points scaled by 2 / max(l) about the centre
        // into a box of width 2.01 (src/fmm_demag.h:52-53, 72), i.e. 1.005 max(l)
        P.side = std::max(hi[0] - lo[0], std::max(hi[1] - lo[1], hi[2] - lo[2])) * (2.01 / 2.0);
        if (!(P.side > 0)) P.side = 1.0;
        for (int d = 0; d < 3; d++) P.c0[d] = 0.5 * (lo[d] + hi[d]);
    }
    return S;
}

// The tree has not the blocks that fg_opts.demag_blocks asks for: the reason, with c.err (else FG_OK).
static int blocks_missing(Ctx &c, const FmmTree &t) {
    const int want = t.oz ? c.opts.demag_blocks : 0;
    const DenseBlocks *none = want >= 2 && !t.near.near.B ? &t.near.near : want == 3 && !t.near.p2m.B ? &t.near.p2m : nullptr;
    if (!none) return FG_OK;
    c.err = none->why == FG_ENOMEM ? "fmm: the blocks of demag_blocks do not fit in the device's memory"
                                   : "fmm: demag_blocks: a leaf of the tree has too many elements for a block";
    return none->why == FG_ENOMEM ? FG_ENOMEM : FG_EINVAL;
}

// The tree of the fastest depth so far (and its source order) while others are tried.
struct KeptTree {
    Ctx &c;
    FmmTree *t = nullptr;
    int *src_dst = nullptr;
    explicit KeptTree(Ctx &ctx) : c(ctx) {}
    ~KeptTree() { drop(); }
    void drop() {
        if (!t) return;
        void *current = c.fmm;
        c.fmm = t;
        fmm_free(c);
        c.fmm = current;
        if (src_dst) cudaFree(src_dst);
        t = nullptr;
        src_dst = nullptr;
    }
    void take() {  // the context's tree
        drop();
        t = static_cast<FmmTree *>(c.fmm);
        src_dst = c.src_dst;
        c.fmm = nullptr;
        c.src_dst = nullptr;
    }
    void give() {  // back to the context
        if (c.src_dst) cudaFree(c.src_dst);
        c.fmm = t;
        c.src_dst = src_dst;
        t = nullptr;
        src_dst = nullptr;
    }
};

int fmm_build(Ctx &c) {
    const bool fp32 = (c.opts.precision == FG_PREC_FP32_REFINE);
    if (c.opts.fmm_order != 0 && c.opts.fmm_order != FMM_P) {
        c.err = "fmm: only expansion order P=9 is built";
        return FG_EINVAL;
    }
    const auto t_begin = std::chrono::steady_clock::now();
    c.tree_wall_ms = c.tree_sort_ms = 0.0;
    const std::vector<SamplePts> S = split_samples(c);
    if (!c.fmm_err) {
        FCK(cudaMalloc(&c.fmm_err, sizeof(int)));
        FCK(cudaMemset(c.fmm_err, 0, sizeof(int)));
    }
    // mean number of sources per occupied leaf at each depth, over all samples
    std::vector<double> occ(11, 0.0);
    {
        const auto t0 = std::chrono::steady_clock::now();
        std::vector<std::vector<uint64_t>> keys;
        if (c.opts.fmm_tree_host) {
            for (const SamplePts &P : S) {
                const int n10 = 1 << 10;
                keys.emplace_back();
                keys.back().reserve(P.src.size());
                for (int s : P.src) {
                    int ijk[3];
                    for (int d = 0; d < 3; d++)
                        ijk[d] = std::min(n10 - 1, std::max(0, (int)(((c.h_src_xyz[3 * (size_t)s + d] - P.c0[d]) / P.side + 0.5) * n10)));
                    keys.back().push_back(morton(ijk[0], ijk[1], ijk[2]));
                }
                std::sort(keys.back().begin(), keys.back().end());
            }
        } else {
            // one device sort of all samples' keys (the sample in the bits above the cell's):
            // the distinct prefixes of the sorted keys are the occupied cells of every sample
            keys.emplace_back();
            std::vector<int> idx;
            int *dseg = nullptr;
            cudaError_t e = c.h_src_seg.empty() ? cudaSuccess : up(&dseg, c.h_src_seg);
            if (e == cudaSuccess)
                e = morton_sort(c, c.nsrc, 10, (int)S.size(), c.src_xyz, dseg, sample_roots(S), nullptr, keys.back(),
                                idx, &c.tree_sort_ms);
            if (dseg) cudaFree(dseg);
            FCK(e);
        }
        for (const auto &K : keys)
            for (int l = 2; l <= 10; l++) {
                const int sh = 3 * (10 - l);
                uint64_t prev = ~0ull;
                for (uint64_t k : K)
                    if ((k >> sh) != prev) { occ[l] += 1; prev = k >> sh; }
            }
        c.tree_wall_ms += std::chrono::duration<double, std::milli>(std::chrono::steady_clock::now() - t0).count();
    }
    auto closest = [&](double target) {
        int best = 2;
        double bd = 1e300;
        for (int l = 2; l <= 10; l++) {
            const double mean = c.nsrc / std::max(1.0, occ[l]);
            const double d = std::fabs(std::log(mean / target));
            if (d < bd) { bd = d; best = l; }
        }
        return best;
    };
    std::vector<int> cands;
    if (c.opts.fmm_leaf < 0) cands.push_back(std::min(10, std::max(2, -c.opts.fmm_leaf)));  // fixed depth
    else if (c.opts.fmm_leaf > 0) cands.push_back(closest(c.opts.fmm_leaf));
    else {
        const int l0 = closest(fp32 ? 400.0 : 300.0);
        for (int l = std::max(2, l0 - 1); l <= std::min(10, l0 + 1); l++) cands.push_back(l);
    }
    cudaMemsetAsync(c.src_q, 0, sizeof(double) * std::max(1, c.nsrc), c.stream);
    if (c.src_q2) cudaMemsetAsync(c.src_q2, 0, sizeof(double) * std::max(1, c.nsrc), c.stream);
    int bestL = cands[0], missing = FG_OK;
    double bestms = 1e300;
    KeptTree best(c);
    for (size_t k = 0; k < cands.size(); k++) {
        fmm_free(c);
        size_t before = 0, after = 0, total = 0;
        FCK(cudaMemGetInfo(&before, &total));
        FmmTree *t = new FmmTree();
        c.fmm = t;
        t->fp32 = fp32;
        int s = fmm_build_forest(c, cands[k]);
        if (s != FG_OK) return s;
        FCK(cudaMemGetInfo(&after, &total));
        if (const int why = blocks_missing(c, *t)) {
            if (cands.size() == 1) return why;
            missing = why;
            continue;  // another depth may have them
        }
        if (cands.size() == 1) {
            c.fmm_setup_ms = std::chrono::duration<double, std::milli>(std::chrono::steady_clock::now() - t_begin).count();
            return FG_OK;
        }
        // autotune: time two evaluations (of all charge sets, as the steps run them) with
        // the current charges (values do not matter)
        cudaEvent_t a, b;
        FCK(cudaEventCreate(&a));
        FCK(cudaEventCreate(&b));
        FCK(fp32 ? fmm_eval_t<float>(c, *t, t->nq, tuning_fields(c)) : fmm_eval_t<double>(c, *t, t->nq, tuning_fields(c)));
        FCK(cudaEventRecord(a, c.stream));
        for (int r = 0; r < 2; r++)
            FCK(fp32 ? fmm_eval_t<float>(c, *t, t->nq, tuning_fields(c)) : fmm_eval_t<double>(c, *t, t->nq, tuning_fields(c)));
        FCK(cudaEventRecord(b, c.stream));
        FCK(cudaEventSynchronize(b));
        float ms = 0;
        cudaEventElapsedTime(&ms, a, b);
        cudaEventDestroy(a);
        cudaEventDestroy(b);
        if (c.opts.verbose) fprintf(stderr, "fmm autotune: L=%d %.3f ms/eval\n", cands[k], ms / 2);
        if (ms >= bestms) continue;
        bestms = ms;
        bestL = cands[k];
        // the fastest tree is kept rather than made again, which would be a quarter of the set-up,
        // unless the next one might want its memory
        best.drop();
        if (8 * (before - std::min(before, after)) < after) best.take();
    }
    if (bestms == 1e300) return missing;
    fmm_free(c);
    int s = FG_OK;
    if (best.t) {
        for (int k = 0; k < 2; k++) harvest_set(*best.t, k);  // the stage times of the trials do not count
        for (double &x : best.t->stage_sum) x = 0.0;
        best.t->stage_n = 0;
        best.give();
    } else {
        FmmTree *t = new FmmTree();
        c.fmm = t;
        t->fp32 = fp32;
        s = fmm_build_forest(c, bestL);
    }
    c.fmm_setup_ms = std::chrono::duration<double, std::milli>(std::chrono::steady_clock::now() - t_begin).count();
    return s;
}

// Per-sample octree of depth L (host vectors, sample-local indices).
struct TreeH {
    std::vector<uint64_t> leaf_keys;
    std::vector<std::vector<uint64_t>> keys;  // per level
    std::vector<std::pair<uint64_t, int>> sk, tk;  // (leaf key, source index / node id), sorted
    std::vector<int> leaf_src, leaf_tgt;           // CSR over sk / tk
};

static int fmm_build_forest(Ctx &c, int L) {
    const auto t_tree = std::chrono::steady_clock::now();
    FmmTree *t = static_cast<FmmTree *>(c.fmm);
    const bool fp32 = t->fp32;
    t->L = L;
    t->nsrc = c.nsrc;
    t->nq = (c.opts.first_order || !c.src_q2 || !c.pot2) ? 1 : 2;  // m, and v beside it
    const int nside = 1 << L;
    const std::vector<SamplePts> SP = split_samples(c);
    const int nseg = (int)SP.size();
    t->s0 = SP[0].side;
    for (int d = 0; d < 3; d++) t->c0[d] = SP[0].c0[d];
    std::vector<TreeH> T(nseg);
    if (!c.opts.fmm_tree_host) {
        // (leaf key, point) pairs of every sample in key order, from the device radix sort of
        // the sources and of the magnetic nodes
        const uint64_t cell_mask = (1ull << (3 * L)) - 1ull;
        std::vector<uint64_t> keys;
        std::vector<int> idx;
        int *dseg = nullptr;
        cudaError_t e = c.h_src_seg.empty() ? cudaSuccess : up(&dseg, c.h_src_seg);
        if (e == cudaSuccess)
            e = morton_sort(c, c.nsrc, L, nseg, c.src_xyz, dseg, sample_roots(SP), nullptr, keys, idx, &c.tree_sort_ms);
        if (dseg) cudaFree(dseg);
        FCK(e);
        for (size_t k = 0; k < keys.size(); k++) T[keys[k] >> (3 * L)].sk.push_back({keys[k] & cell_mask, idx[k]});
        FCK(morton_sort(c, c.nn, L, nseg, c.xyz, c.batch ? c.node_seg : nullptr, sample_roots(SP), c.mag, keys, idx,
                        &c.tree_sort_ms));
        for (size_t k = 0; k < keys.size(); k++) T[keys[k] >> (3 * L)].tk.push_back({keys[k] & cell_mask, idx[k]});
    }
    for (int g = 0; g < nseg; g++) {
        const SamplePts &P = SP[g];
        TreeH &H = T[g];
        if (c.opts.fmm_tree_host) {
            auto cell_of = [&](const double *p) {
                int ijk[3];
                for (int d = 0; d < 3; d++) ijk[d] = std::min(nside - 1, std::max(0, (int)(((p[d] - P.c0[d]) / P.side + 0.5) * nside)));
                return morton(ijk[0], ijk[1], ijk[2]);
            };
            for (int s : P.src) H.sk.push_back({cell_of(&c.h_src_xyz[3 * (size_t)s]), s});
            for (int i : P.tgt) H.tk.push_back({cell_of(&c.h_xyz[3 * (size_t)i]), i});
            std::sort(H.sk.begin(), H.sk.end());
            std::sort(H.tk.begin(), H.tk.end());
        }
        std::vector<uint64_t> a, b;
        for (auto &p : H.sk) if (a.empty() || a.back() != p.first) a.push_back(p.first);
        for (auto &p : H.tk) if (b.empty() || b.back() != p.first) b.push_back(p.first);
        std::set_union(a.begin(), a.end(), b.begin(), b.end(), std::back_inserter(H.leaf_keys));
        H.leaf_src.assign(H.leaf_keys.size() + 1, 0);
        H.leaf_tgt.assign(H.leaf_keys.size() + 1, 0);
        size_t ia = 0, ib = 0;
        for (size_t l = 0; l < H.leaf_keys.size(); l++) {
            H.leaf_src[l] = (int)ia;
            while (ia < H.sk.size() && H.sk[ia].first == H.leaf_keys[l]) ia++;
            H.leaf_tgt[l] = (int)ib;
            while (ib < H.tk.size() && H.tk[ib].first == H.leaf_keys[l]) ib++;
        }
        H.leaf_src.back() = (int)ia;
        H.leaf_tgt.back() = (int)ib;
        H.keys.assign(L + 1, {});
        H.keys[L] = H.leaf_keys;
        for (int l = L - 1; l >= 2; l--)
            for (uint64_t k : H.keys[l + 1])
                if (H.keys[l].empty() || H.keys[l].back() != (k >> 3)) H.keys[l].push_back(k >> 3);
    }
    // global numbering: level-major, then sample, then Morton order
    t->lev_begin.assign(L + 2, 0);
    std::vector<std::vector<int>> base(L + 1, std::vector<int>(nseg, 0));  // first global id of (level, sample)
    int next = 0;
    for (int l = 2; l <= L; l++) {
        t->lev_begin[l] = next;
        for (int g = 0; g < nseg; g++) {
            base[l][g] = next;
            next += (int)T[g].keys[l].size();
        }
    }
    t->lev_begin[L + 1] = next;
    const int ncell = next;
    t->ncell = ncell;
    t->leaf0 = t->lev_begin[L];
    int nleaf = ncell - t->leaf0;
    t->nleaf = nleaf;
    std::vector<int> leaf_src(nleaf + 1, 0), leaf_tgt(nleaf + 1, 0), leaf_ijk(3 * (size_t)nleaf, 0);
    std::vector<double> leaf_scale(nleaf, 0.0);
    std::vector<int> src_dst(c.nsrc, 0), tgt_node;
    std::vector<double> sloc(4 * (size_t)c.nsrc, 0.0), tloc;
    std::vector<int> nsub_src(ncell, 0), nsub_tgt(ncell, 0);
    std::vector<int> m2m_tab((size_t)ncell * 8, -1), l2l_tab((size_t)ncell * 8, -1);
    std::vector<int> m2l_tab((size_t)ncell * NCODE_M2L, -1);
    std::vector<unsigned char> octant(ncell, 0);  // within the parent
    std::vector<int> near_ptr(nleaf + 1, 0), near_leaf;
    size_t src_off = 0, tgt_off = 0, nm2l = 0, np2p = 0;
    int ijk[3];
    for (int g = 0; g < nseg; g++) {
        TreeH &H = T[g];
        const SamplePts &P = SP[g];
        const double w = P.side / nside;
        std::vector<std::unordered_map<uint64_t, int>> where(L + 1);
        for (int l = 2; l <= L; l++) {
            where[l].reserve(H.keys[l].size() * 2);
            for (size_t i = 0; i < H.keys[l].size(); i++) where[l][H.keys[l][i]] = base[l][g] + (int)i;
        }
        const int lf0 = base[L][g] - t->leaf0;  // first global leaf index of the sample
        for (size_t l = 0; l < H.leaf_keys.size(); l++) {
            const int gl = lf0 + (int)l;
            leaf_src[gl] = (int)src_off + H.leaf_src[l];
            leaf_tgt[gl] = (int)tgt_off + H.leaf_tgt[l];
            decode(H.leaf_keys[l], &leaf_ijk[3 * (size_t)gl]);
            leaf_scale[gl] = 1.0 / w;
            const int *q = &leaf_ijk[3 * (size_t)gl];
            double cc[3];
            for (int d = 0; d < 3; d++) cc[d] = P.c0[d] - 0.5 * P.side + (q[d] + 0.5) * w;
            for (int k = H.leaf_src[l]; k < H.leaf_src[l + 1]; k++) {
                const size_t gk = src_off + k;
                const int s = H.sk[k].second;
                src_dst[s] = (int)gk;
                for (int d = 0; d < 3; d++) sloc[4 * gk + d] = (c.h_src_xyz[3 * (size_t)s + d] - cc[d]) / w;
            }
            for (int k = H.leaf_tgt[l]; k < H.leaf_tgt[l + 1]; k++) {
                const int i = H.tk[k].second;
                tgt_node.push_back(i);
                for (int d = 0; d < 3; d++) tloc.push_back((c.h_xyz[3 * (size_t)i + d] - cc[d]) / w);
                tloc.push_back(0.0);
            }
            nsub_src[base[L][g] + (int)l] = H.leaf_src[l + 1] - H.leaf_src[l];
            nsub_tgt[base[L][g] + (int)l] = H.leaf_tgt[l + 1] - H.leaf_tgt[l];
        }
        for (int l = L; l >= 3; l--)
            for (size_t i = 0; i < H.keys[l].size(); i++) {
                const int gc = base[l][g] + (int)i;
                const int p = where[l - 1][H.keys[l][i] >> 3];
                const int oc = (int)(H.keys[l][i] & 7);
                nsub_src[p] += nsub_src[gc];
                nsub_tgt[p] += nsub_tgt[gc];
                if (nsub_src[gc] > 0) m2m_tab[(size_t)p * 8 + oc] = gc;
                l2l_tab[(size_t)gc * 8 + oc] = p;
            }
        for (int l = 2; l <= L; l++) {
            const int n = 1 << l;
            for (size_t i = 0; i < H.keys[l].size(); i++) {
                const int gc = base[l][g] + (int)i;
                octant[gc] = (unsigned char)(H.keys[l][i] & 7);
                if (nsub_tgt[gc] == 0) continue;
                decode(H.keys[l][i], ijk);
                const int px = ijk[0] >> 1, py = ijk[1] >> 1, pz = ijk[2] >> 1;
                for (int ax = 2 * (px - 1); ax <= 2 * (px + 1) + 1; ax++)
                    for (int ay = 2 * (py - 1); ay <= 2 * (py + 1) + 1; ay++)
                        for (int az = 2 * (pz - 1); az <= 2 * (pz + 1) + 1; az++) {
                            if (ax < 0 || ay < 0 || az < 0 || ax >= n || ay >= n || az >= n) continue;
                            const int dx = ijk[0] - ax, dy = ijk[1] - ay, dz = ijk[2] - az;
                            if (std::abs(dx) <= 1 && std::abs(dy) <= 1 && std::abs(dz) <= 1) continue;
                            auto it = where[l].find(morton(ax, ay, az));
                            if (it == where[l].end() || nsub_src[it->second] == 0) continue;
                            m2l_tab[(size_t)gc * NCODE_M2L + (dx + 3) * 49 + (dy + 3) * 7 + (dz + 3)] = it->second;
                            nm2l++;
                        }
            }
        }
        for (size_t l = 0; l < H.leaf_keys.size(); l++) {
            const int gl = lf0 + (int)l;
            std::vector<int> nb;
            if (H.leaf_tgt[l + 1] > H.leaf_tgt[l]) {
                const int *q = &leaf_ijk[3 * (size_t)gl];
                for (int dx = -1; dx <= 1; dx++)
                    for (int dy = -1; dy <= 1; dy++)
                        for (int dz = -1; dz <= 1; dz++) {
                            const int ax = q[0] + dx, ay = q[1] + dy, az = q[2] + dz;
                            if (ax < 0 || ay < 0 || az < 0 || ax >= nside || ay >= nside || az >= nside) continue;
                            auto it = where[L].find(morton(ax, ay, az));
                            if (it == where[L].end()) continue;
                            const int nl = it->second - t->leaf0;
                            const int ls = nl - lf0;
                            if (H.leaf_src[ls + 1] == H.leaf_src[ls]) continue;
                            nb.push_back(nl);
                            np2p += (size_t)(H.leaf_src[ls + 1] - H.leaf_src[ls]) * (H.leaf_tgt[l + 1] - H.leaf_tgt[l]);
                        }
            }
            near_leaf.insert(near_leaf.end(), nb.begin(), nb.end());
            near_ptr[gl + 1] = (int)near_leaf.size();
        }
        src_off += H.sk.size();
        tgt_off += H.tk.size();
    }
    leaf_src[nleaf] = (int)src_off;
    leaf_tgt[nleaf] = (int)tgt_off;
    t->n_m2l = nm2l;
    t->n_p2p_pairs = np2p;
    const FmmOps &ops = fmm_ops();
    t->tc = fp32 && c.opts.fmm_tensor != 0;
    if (t->tc) {
        std::vector<int> codes;
        std::vector<int4> units, comb;
        int nslot = 0;
        auto plan = [&](int n_out, int out0, int ncode, const std::vector<int> &tab, int max_codes) {
            FmmTree::TcLaunch l;
            l.unit0 = (int)units.size();
            l.comb0 = (int)comb.size();
            translate_tc_units(n_out, ncode, tab.data(), out0, max_codes, codes, units, comb, nslot);
            l.nunit = (int)units.size() - l.unit0;
            l.ncomb = (int)comb.size() - l.comb0;
            return l;
        };
        t->tc_m2m.assign(L + 1, FmmTree::TcLaunch());
        t->tc_l2l.assign(L + 1, FmmTree::TcLaunch());
        // M2M and L2L run level by level, each level a short launch: units of 2 codes keep
        // its critical path short. M2L has the whole tree in one launch; its unit size is
        // the one whose units, handed in launch order to the earliest free of the SMs' CTA
        // slots (one per SM), finish first: a unit costs its codes plus about 3 codes of
        // pipeline fill, drain and output, and a split tile adds a combine pass
        int m2l_codes = 48;
        {
            std::vector<int> cs;  // codes per tile: one unit per tile
            std::vector<int4> us, cb;
            int ns = 0;
            translate_tc_units(ncell, NCODE_M2L, m2l_tab.data(), 0, 1 << 30, cs, us, cb, ns);
            double best = 1e300;
            const int slots = std::max(1, c.nsm);
            for (int mc : {64, 48, 32, 24, 16, 12, 8}) {
                std::priority_queue<double, std::vector<double>, std::greater<double>> free_at;
                for (int k = 0; k < slots; k++) free_at.push(0.0);
                double span = 0.0;
                bool split = false;
                for (const int4 &u : us) {  // the split of translate_tc_units, unit by unit
                    const int n = u.z - u.y, nu = std::max(1, (n + mc - 1) / mc);
                    split = split || nu > 1;
                    for (int k = 0; k < nu; k++) {
                        const int cnt = (int)((long)n * (k + 1) / nu - (long)n * k / nu);
                        const double t0 = free_at.top();
                        free_at.pop();
                        const double t1 = t0 + 3.0 + cnt;
                        span = std::max(span, t1);
                        free_at.push(t1);
                    }
                }
                span += split ? 1.0 : 0.0;
                if (span < best) {
                    best = span;
                    m2l_codes = mc;
                }
            }
        }
        for (int l = L - 1; l >= 2; l--)
            t->tc_m2m[l] = plan(t->lev_begin[l + 1] - t->lev_begin[l], t->lev_begin[l], 8, m2m_tab, 2);
        t->tc_m2l = plan(ncell, 0, NCODE_M2L, m2l_tab, m2l_codes);
        for (int l = 3; l <= L; l++)
            t->tc_l2l[l] = plan(t->lev_begin[l + 1] - t->lev_begin[l], t->lev_begin[l], 8, l2l_tab, 2);
        FCK(up(&t->tc_code, codes));
        FCK(up(&t->tc_units, units));
        FCK(up(&t->tc_comb, comb));
        t->nslot_floats = (size_t)std::max(1, nslot) * translate_tc_tile() * NR;
        FCK(cudaMalloc(&t->tc_scratch, sizeof(float) * t->nslot_floats * t->nq));
        FCK(translate_tc_setup());
        const size_t nexp = (size_t)ncell * NR * t->nq;
        FCK(cudaMalloc(&t->Mh, nexp * sizeof(float)));
        FCK(cudaMalloc(&t->Ml, nexp * sizeof(float)));
        FCK(cudaMalloc(&t->Fh, nexp * sizeof(float)));
        FCK(cudaMalloc(&t->Fl, nexp * sizeof(float)));
        FCK(cudaMemset(t->Mh, 0, nexp * sizeof(float)));
        FCK(cudaMemset(t->Ml, 0, nexp * sizeof(float)));
        FCK(cudaMemset(t->Fh, 0, nexp * sizeof(float)));
        FCK(cudaMemset(t->Fl, 0, nexp * sizeof(float)));
        static const std::vector<float> im2l = translate_tc_images(ops.m2l, NCODE_M2L);
        static const std::vector<float> im2m = translate_tc_images(ops.m2m, 8);
        static const std::vector<float> il2l = translate_tc_images(ops.l2l, 8);
        FCK(up((float **)&t->img_m2l, im2l));
        FCK(up((float **)&t->img_m2m, im2m));
        FCK(up((float **)&t->img_l2l, il2l));
    }
    t->ds = !fp32 && c.opts.fmm_native_fp64 == 0;
    t->repeat = t->ds && c.opts.precision == FG_PREC_FP32_REFINE;
    t->oz = t->ds && !t->repeat;
    if (t->ds) {
        const int tile = t->oz ? OZ_TILE : DS_TILE;
        std::vector<int> cells, codes;
        std::vector<int4> units;
        std::vector<int2> fin;
        int nslot = 0;
        struct Tile { std::vector<int> cells, codes; };
        auto tiles_of = [&](const std::vector<int> &list, int ncode, const std::vector<int> &tab) {
            std::vector<Tile> T;
            for (size_t b = 0; b < list.size(); b += tile) {
                Tile x;
                x.cells.assign(list.begin() + b, list.begin() + std::min(list.size(), b + tile));
                for (int code = 0; code < ncode; code++)
                    for (int cc : x.cells)
                        if (tab[(size_t)cc * ncode + code] >= 0) {
                            x.codes.push_back(code);
                            break;
                        }
                x.cells.resize(tile, -1);
                T.push_back(std::move(x));
            }
            return T;
        };
        // tiles of a level: its cells in order, or the cells of each octant apart, whichever needs
        // fewer (tile, code) products (a tile costs about one more)
        auto level_tiles = [&](int l, int ncode, const std::vector<int> &tab) {
            std::vector<int> all;
            std::vector<std::vector<int>> oct(8);
            for (int k = t->lev_begin[l]; k < t->lev_begin[l + 1]; k++) {
                all.push_back(k);
                oct[octant[k]].push_back(k);
            }
            std::vector<Tile> A = tiles_of(all, ncode, tab), B;
            for (const auto &o : oct)
                for (auto &x : tiles_of(o, ncode, tab)) B.push_back(std::move(x));
            auto cost = [](const std::vector<Tile> &T) {
                size_t n = T.size();
                for (const auto &x : T) n += x.codes.size();
                return n;
            };
            return cost(B) < cost(A) ? B : A;
        };
        // units of at most mc codes: the size among the candidates whose units, handed in order to
        // the earliest free SM, finish first (a unit costs its codes plus about 2)
        auto plan_oz = [&](const std::vector<Tile> &T) {
            int mc = 64;
            double best = 1e300;
            for (int k : {64, 48, 32, 24, 16, 12, 8, 6, 4, 3, 2, 1}) {
                std::priority_queue<double, std::vector<double>, std::greater<double>> free_at;
                for (int q = 0; q < std::max(1, c.nsm); q++) free_at.push(0.0);
                double span = 0.0;
                for (const Tile &x : T) {
                    const int n = (int)x.codes.size(), nu = (n + k - 1) / k;
                    for (int q = 0; q < nu; q++) {
                        const double t1 = free_at.top() + 2.0 + ((long)n * (q + 1) / nu - (long)n * q / nu);
                        free_at.pop();
                        free_at.push(t1);
                        span = std::max(span, t1);
                    }
                }
                if (span < best) {
                    best = span;
                    mc = k;
                }
            }
            FmmTree::OzLaunch l;
            l.unit0 = (int)units.size();
            l.tile0 = (int)fin.size();
            int slot = 0;
            for (const Tile &x : T) {
                const int n = (int)x.codes.size(), nu = (n + mc - 1) / mc, first = (int)codes.size();
                for (int q = 0; q < nu; q++)
                    units.push_back(make_int4((int)fin.size(), first + (int)((long)n * q / nu),
                                              first + (int)((long)n * (q + 1) / nu), slot + q));
                fin.push_back(make_int2(slot, nu));
                slot += nu;
                codes.insert(codes.end(), x.codes.begin(), x.codes.end());
                cells.insert(cells.end(), x.cells.begin(), x.cells.end());
            }
            l.nunit = (int)units.size() - l.unit0;
            l.ntile = (int)fin.size() - l.tile0;
            nslot = std::max(nslot, slot);
            return l;
        };
        // double-single: one unit per tile (a sum's codes stay in order), the longest first
        auto plan_ds = [&](std::vector<Tile> T) {
            std::stable_sort(T.begin(), T.end(), [](const Tile &x, const Tile &y) { return x.codes.size() > y.codes.size(); });
            FmmTree::OzLaunch l;
            l.unit0 = (int)units.size();
            l.nunit = l.ntile = (int)T.size();
            for (const Tile &x : T) {
                const int first = (int)codes.size();
                units.push_back(make_int4((int)cells.size(), first, first + (int)x.codes.size(), 0));
                codes.insert(codes.end(), x.codes.begin(), x.codes.end());
                cells.insert(cells.end(), x.cells.begin(), x.cells.end());
            }
            return l;
        };
        auto plan = [&](const std::vector<Tile> &T) { return t->oz ? plan_oz(T) : plan_ds(T); };
        t->oz_m2m.assign(L + 1, FmmTree::OzLaunch());
        t->oz_l2l.assign(L + 1, FmmTree::OzLaunch());
        for (int l = L - 1; l >= 2; l--) t->oz_m2m[l] = plan(level_tiles(l, 8, m2m_tab));
        std::vector<Tile> all;
        int nsplit = 0;  // listed cells above the leaves: their locals are translated further
        for (int l = 2; l <= L; l++) {
            if (l == L) nsplit = tile * (int)all.size();
            for (auto &x : level_tiles(l, NCODE_M2L, m2l_tab)) all.push_back(std::move(x));
        }
        const size_t codes0 = codes.size();
        t->oz_m2l = plan(all);
        if (c.opts.verbose)
            fprintf(stderr, "fmm: m2l %zu (tile, code) products in %d tiles, %d units\n", codes.size() - codes0,
                    t->oz_m2l.ntile, t->oz_m2l.nunit);
        t->oz_m2l.nsplit = nsplit;
        for (int l = 3; l <= L; l++) t->oz_l2l[l] = plan(level_tiles(l, 8, l2l_tab));
        FCK(up(&t->oz_cells, cells));
        FCK(up(&t->oz_codes, codes));
        FCK(up(&t->oz_units, units));
        if (t->oz) {
            std::vector<int> wexp(2 * NR), leaves(nleaf);
            oz_weights(wexp.data(), wexp.data() + NR);
            for (int k = 0; k < nleaf; k++) leaves[k] = t->leaf0 + k;
            static const OzImages im[3] = {oz_images(ops.m2m, 8, wexp.data()), oz_images(ops.m2l, NCODE_M2L, wexp.data()),
                                           oz_images(ops.l2l, 8, wexp.data() + NR)};
            for (int k = 0; k < 3; k++) {
                FCK(up(&t->oz_img[k], im[k].img));
                FCK(up(&t->oz_rows[k], im[k].row_scale));
            }
            FCK(up(&t->oz_fin, fin));
            FCK(up(&t->oz_wexp, wexp));
            FCK(up(&t->oz_leaves, leaves));
            FCK(cudaMalloc(&t->oz_scratch, sizeof(float2) * std::max(1, nslot) * OZ_TILE * NR * t->nq));
            FCK(cudaMalloc(&t->oz_digits, (size_t)ncell * t->nq * OZ_CELL_BYTES));
            FCK(cudaMemset(t->oz_digits, 0, (size_t)ncell * t->nq * OZ_CELL_BYTES));
            FCK(cudaMalloc(&t->oz_scale, sizeof(float) * ncell * t->nq));
            FCK(cudaMemset(t->oz_scale, 0, sizeof(float) * ncell * t->nq));
            FCK(oz_setup());
        } else {
            const std::vector<double> *op[3] = {&ops.m2m, &ops.m2l, &ops.l2l};
            for (int k = 0; k < 3; k++) {
                const int n = k == 1 ? NCODE_M2L : 8;
                double *d = nullptr;
                FCK(cudaMalloc(&t->oz_img[k], (size_t)n * NR * NR * sizeof(float2)));
                FCK(up(&d, *op[k]));
                k_ds_image<<<(n * NR * NR / 2 + 255) / 256, 256, 0, c.stream>>>(n, d, (float4 *)t->oz_img[k]);
                const cudaError_t e = cudaStreamSynchronize(c.stream);
                cudaFree(d);
                FCK(e);
            }
            FCK(cudaMalloc(&t->F_split, sizeof(float2) * std::max(1, t->leaf0) * NR * t->nq));
        }
    }
    FCK(up(&t->leaf_src, leaf_src));
    FCK(up(&t->leaf_tgt, leaf_tgt));
    FCK(up(&t->tgt_node, tgt_node));
    t->ntgt = (int)tgt_node.size();
    std::vector<int> tgt_leaf(tgt_node.size());
    for (int l = 0; l < nleaf; l++) std::fill(tgt_leaf.begin() + leaf_tgt[l], tgt_leaf.begin() + leaf_tgt[l + 1], l);
    FCK(up(&t->tgt_leaf, tgt_leaf));
    FCK(up(&t->leaf_ijk, leaf_ijk));
    FCK(up(&t->leaf_scale, leaf_scale));
    FCK(up(&t->m2l_tab, m2l_tab));
    FCK(up(&t->m2m_tab, m2m_tab));
    FCK(up(&t->l2l_tab, l2l_tab));
    FCK(up(&t->near_ptr, near_ptr));
    FCK(up(&t->near_leaf, near_leaf));
    if (!t->ds) FCK(up_as<double>(&t->sloc, sloc, fp32));
    FCK(up_as<double>(&t->tloc, tloc, fp32));
    // near-field tasks of at most `most` targets: each leaf's targets shared out evenly, in multiples
    // of `step`. Where the sources (src_bytes each) fit in L2 the expensive tasks go first, which
    // evens out the last wave; else the leaf order keeps neighbouring tasks on the same sources
    auto near_tasks = [&](int most, int step, int src_bytes, bool warps) -> cudaError_t {
        std::vector<int4> task;
        std::vector<long> cost, leaf_near(nleaf, 0);
        long pairs = 0;
        for (int l = 0; l < nleaf; l++) {
            for (int e = near_ptr[l]; e < near_ptr[l + 1]; e++)
                leaf_near[l] += leaf_src[near_leaf[e] + 1] - leaf_src[near_leaf[e]];
            pairs += leaf_near[l] * (leaf_tgt[l + 1] - leaf_tgt[l]);
        }
        // a warp per task: none longer than what each resident warp (sixteen per SM) has to do on
        // average, else the longest task sets the time (24 uneven samples of up to 13k tets: near field
        // 210 -> 147 us; a cap of twice and of 0.7 times the average gave half of that)
        const double share = warps ? (double)pairs / (16.0 * std::max(1, c.nsm)) : 1e300;
        for (int l = 0; l < nleaf; l++) {
            const int n = leaf_tgt[l + 1] - leaf_tgt[l], units = (n + step - 1) / step;
            const long src = leaf_near[l];
            const int groups =
                std::min(units, std::max((n + most - 1) / most, (int)std::ceil((double)src * n / std::max(1.0, share))));
            for (int g = 0; g < groups; g++) {
                const int b = step * (int)((long)units * g / groups);
                const int e = std::min(n, step * (int)((long)units * (g + 1) / groups));
                task.push_back(make_int4(l, leaf_tgt[l] + b, e - b, 0));
                cost.push_back(src * (e - b));
            }
        }
        if ((size_t)c.nsrc * src_bytes < ((size_t)64 << 20)) {
            std::vector<int> order(task.size());
            for (size_t k = 0; k < order.size(); k++) order[k] = (int)k;
            std::stable_sort(order.begin(), order.end(), [&](int x, int y) { return cost[x] > cost[y]; });
            std::vector<int4> sorted;
            for (int k : order) sorted.push_back(task[k]);
            task.swap(sorted);
        }
        t->n_p2p_task = (int)task.size();
        return up(&t->p2p_task, task);
    };
    if (fp32) FCK(near_tasks(P2P32_NT, 2, 20, true));
    if (t->ds) {
        // x = hi + lo, hi on the 2^-20 grid (|x| < 4 leaf units: exact in FP32)
        auto split = [](const std::vector<double> &v, std::vector<float4> &hi, std::vector<float4> &lo) {
            const size_t n = v.size() / 4;
            hi.resize(n);
            lo.resize(n);
            for (size_t k = 0; k < n; k++) {
                float h[3], l[3];
                for (int d = 0; d < 3; d++) {
                    const double x = v[4 * k + d];
                    const double xh = std::nearbyint(x * 1048576.0) / 1048576.0;
                    h[d] = (float)xh;
                    l[d] = (float)(x - xh);
                }
                hi[k] = make_float4(h[0], h[1], h[2], 0.f);
                lo[k] = make_float4(l[0], l[1], l[2], 0.f);
            }
        };
        std::vector<float4> sh, sl, th, tl;
        split(sloc, sh, sl);
        split(tloc, th, tl);
        FCK(near_tasks(P2P_NT, t->repeat ? 2 : 1, 40, t->repeat));
        FCK(up(&t->ds_src_hi, sh));
        FCK(up(&t->ds_src_lo, sl));
        FCK(up(&t->ds_tgt_hi, th));
        FCK(up(&t->ds_tgt_lo, tl));
    }
    if (!t->ds) {
        FCK(up_as<double>(&t->op_m2l, ops.m2l, fp32));
        FCK(up_as<double>(&t->op_m2m, ops.m2m, fp32));
        FCK(up_as<double>(&t->op_l2l, ops.l2l, fp32));
    }
    if (c.src_dst) cudaFree(c.src_dst);
    c.src_dst = nullptr;
    FCK(up(&c.src_dst, src_dst));
    if (t->oz && c.opts.demag_blocks != 1) {
        std::vector<int> orig(c.nsrc);
        for (int k = 0; k < c.nsrc; k++) orig[src_dst[k]] = k;
        int *d_orig = nullptr;
        double *d_sloc = nullptr;
        cudaError_t e = up(&d_orig, orig);
        if (e == cudaSuccess) e = up(&d_sloc, sloc);
        if (e == cudaSuccess) {
            NearTree nt = near_tree(*t);
            nt.src_orig = d_orig;
            nt.src_pos = c.src_dst;
            nt.sloc = (const double4 *)d_sloc;
            nt.h_leaf_tgt = leaf_tgt.data();
            e = near_build(c, make_rules(c.opts.one_gauss_point != 0), nt, t->near);
        }
        if (d_orig) cudaFree(d_orig);
        if (d_sloc) cudaFree(d_sloc);
        FCK(e);
    }
    const size_t esz = fp32 ? sizeof(float) : sizeof(double);
    const size_t nexp_all = (size_t)ncell * NR * t->nq;
    FCK(cudaMalloc(&t->M, nexp_all * esz));
    FCK(cudaMalloc(&t->F, nexp_all * esz));
    FCK(cudaMemset(t->M, 0, nexp_all * esz));
    FCK(cudaMemset(t->F, 0, nexp_all * esz));
    if (t->nq == 2) {
        if (!t->ds) {
            FCK(cudaMalloc(&t->sq2, std::max(1, c.nsrc) * esz));
            FCK(cudaMemset(t->sq2, 0, std::max(1, c.nsrc) * esz));
        } else {
            FCK(cudaMalloc(&t->ds_q2, 2 * sizeof(float) * std::max(1, c.nsrc)));
            FCK(cudaMemset(t->ds_q2, 0, 2 * sizeof(float) * std::max(1, c.nsrc)));
        }
    }
    if (fp32) {
        FCK(cudaFuncSetAttribute(k_translate<float>, cudaFuncAttributeMaxDynamicSharedMemorySize, tr_smem<float>()));
    } else {
        FCK(cudaFuncSetAttribute(k_translate<double>, cudaFuncAttributeMaxDynamicSharedMemorySize, tr_smem<double>()));
    }
    if (c.opts.profile)
        for (auto &set : t->ev)
            for (auto &e : set) FCK(cudaEventCreate(&e));
    if (c.opts.profile)
        for (auto &set : t->evn)
            for (auto &e : set) FCK(cudaEventCreate(&e));
    if (c.opts.verbose)
        fprintf(stderr, "fmm: L=%d trees=%d leaves=%d cells=%d m2l=%zu p2p_pairs=%zu (%s)\n", L, nseg, nleaf, ncell,
                t->n_m2l, t->n_p2p_pairs, fp32 ? "fp32" : "fp64");
    c.tree_wall_ms += std::chrono::duration<double, std::milli>(std::chrono::steady_clock::now() - t_tree).count();
    return FG_OK;
}

void fmm_free(Ctx &c) {
    FmmTree *t = static_cast<FmmTree *>(c.fmm);
    if (!t) return;
    void *ptrs[] = {t->leaf_scale, t->leaf_src, t->leaf_tgt, t->tgt_node, t->tgt_leaf, t->sloc, t->tloc, t->leaf_ijk, t->m2l_tab, t->m2m_tab,
                    t->l2l_tab, t->near_ptr, t->near_leaf, t->M, t->F, t->op_m2l, t->op_m2m, t->op_l2l,
                    t->tc_code, t->tc_units, t->tc_comb, t->tc_scratch, t->Mh, t->Ml, t->Fh, t->Fl,
                    t->img_m2l, t->img_m2m, t->img_l2l, t->ds_src_hi, t->ds_src_lo, t->ds_tgt_hi, t->ds_tgt_lo,
                    t->sq2, t->ds_q2, t->p2p_task, t->oz_cells, t->oz_codes, t->oz_wexp, t->oz_leaves, t->oz_units, t->oz_fin,
                    t->oz_scratch, t->oz_digits, t->oz_scale, t->oz_img[0], t->oz_img[1], t->oz_img[2], t->oz_rows[0],
                    t->oz_rows[1], t->oz_rows[2], t->F_split};
    for (void *p : ptrs)
        if (p) cudaFree(p);
    near_free(t->near);
    for (auto &set : t->ev)
        for (auto &e : set)
            if (e) cudaEventDestroy(e);
    for (auto &set : t->evn)
        for (auto &e : set)
            if (e) cudaEventDestroy(e);
    delete t;
    c.fmm = nullptr;
}

template <typename T> static bool tc_path(const FmmTree &t);
template <> bool tc_path<float>(const FmmTree &t) { return t.tc; }
template <> bool tc_path<double>(const FmmTree &) { return false; }

// Adds the stage times of a recorded event set to the running sums (waits for its last event).
static void harvest_set(FmmTree &t, int k) {
    if (!t.ev_pending[k]) return;
    cudaEventSynchronize(t.ev[k][5]);
    for (int s = 0; s < 5; s++) {
        float ms = 0.f;
        if (s == 4 && t.ev_split[k]) cudaEventElapsedTime(&ms, t.evn[k][0], t.evn[k][1]);  // near field, own stream
        else cudaEventElapsedTime(&ms, t.ev[k][s], t.ev[k][s + 1]);
        t.stage_sum[s] += ms;
    }
    t.stage_n++;
    t.ev_pending[k] = false;
}

// One FMM evaluation of nq charge sets: set 0 from c.src_q into c.pot, set 1 (nq = 2) from
// c.src_q2 into c.pot2. The sets share every table, operator image and launch (grid y of
// P2M and of the tensor-core translations; one near-field pass computes both).
template <typename T>
static cudaError_t fmm_eval_t(Ctx &c, FmmTree &t, int nq, const FmmFields &f) {
    if (nq < 1 || nq > t.nq || (nq == 2 && (!c.src_q2 || !c.pot2))) return cudaErrorInvalidValue;
    const int L = t.L;
    T *M = (T *)t.M, *F = (T *)t.F;
    constexpr int TB = TrShape<T>::TB;
    const size_t sstride = (size_t)t.ncell * NR;  // elements between the sets' expansions
    const bool prof = c.opts.profile && t.ev[0][0];
    cudaEvent_t *ev = t.ev[t.ev_next];
    if (prof) {
        harvest_set(t, t.ev_next);
        cudaEventRecord(ev[0], c.stream);
    }
    const bool tc = tc_path<T>(t);
    P2mSet<T> ps[2];
    for (int k = 0; k < 2; k++) {
        const int q = k < nq ? k : 0;
        P2mSet<T> &p = ps[k];
        p.q = q ? c.src_q2 : c.src_q;
        p.qf = (sizeof(T) == 4 && c.charges32) ? (q ? c.src_q2f : c.src_qf) : nullptr;
        p.M = M + q * sstride;
        p.Mh = tc ? t.Mh + q * sstride : nullptr;
        p.Ml = tc ? t.Ml + q * sstride : nullptr;
        p.qn = t.ds ? nullptr : q ? (T *)t.sq2 : (T *)t.sloc + 3;
        p.qn_stride = q ? 1 : 4;
        p.qh = p.ql = nullptr;
        p.qd_stride = q ? 1 : 4;
        if (t.ds) {
            p.qh = q ? t.ds_q2 : (float *)t.ds_src_hi + 3;
            p.ql = q ? t.ds_q2 + t.nsrc : (float *)t.ds_src_lo + 3;
        }
    }
    // overlapped evaluation: after P2M (which stores the near field's charges) and M2M, the
    // near field runs on the second, lower-priority stream beside M2L and L2L: an FP32
    // near-field block (128 threads x 128 registers) fits on an SM beside a tensor-core
    // translation CTA (288 x 168), so the FP32 and SFU pipes work while the tensor pipe
    // does; L2P follows once both are done. (Forked before P2M, the near field's blocks took
    // every SM first and the short M2M launches waited behind them.)
    const bool split = c.opts.fmm_overlap != 0 && c.stream2 != nullptr;
    NearSets<T> ns;
    ns.q2 = nq == 2 ? (const T *)t.sq2 : nullptr;
    ns.F[0] = F;
    ns.F[1] = F + (nq == 2 ? sstride : 0);
    ns.pot[0] = c.pot;
    ns.pot[1] = nq == 2 ? c.pot2 : c.pot;
    ns.near_only = 0;
    const bool whole = t.near.near.B != nullptr;
    const int nb = (t.nleaf + 3) / 4;
    cudaError_t terr = cudaSuccess;  // first failed launch of a translation or of the near field
    auto note = [&](cudaError_t e) {
        if (e != cudaSuccess && terr == cudaSuccess) terr = e;
    };
    auto near_field = [&](cudaStream_t st) {
        if (whole) {
            note(launch_blocks(t.near.near, t.near, st, nq, t.tgt_node, c.pot, c.pot2));
            return;
        }
        if constexpr (sizeof(T) == 8) {
            if (t.repeat) {
                if (t.n_p2p_task > 0)
                    (nq == 2 ? k_p2p_ds_repeat<2> : k_p2p_ds_repeat<1>)<<<(t.n_p2p_task + 3) / 4, 128, 0, st>>>(
                        t.n_p2p_task, t.p2p_task, t.leaf_src, t.tgt_node, t.ds_tgt_hi, t.ds_tgt_lo, t.ds_src_hi,
                        t.ds_src_lo, t.ds_q2, t.ds_q2 ? t.ds_q2 + t.nsrc : nullptr, t.leaf_ijk, t.near_ptr,
                        t.near_leaf, ns.pot[0], ns.pot[1]);
            } else if (t.ds && t.n_p2p_task > 0)
                (nq == 2 ? k_p2p_ds<2> : k_p2p_ds<1>)<<<t.n_p2p_task, 128, 0, st>>>(
                    t.p2p_task, t.leaf_src, t.tgt_node, t.ds_tgt_hi, t.ds_tgt_lo, t.ds_src_hi, t.ds_src_lo, t.ds_q2,
                    t.ds_q2 ? t.ds_q2 + t.nsrc : nullptr, t.leaf_ijk, t.near_ptr, t.near_leaf, ns.pot[0], ns.pot[1]);
        }
        if constexpr (sizeof(T) == 4) {
            if (t.n_p2p_task > 0)
                (nq == 2 ? k_l2p_p2p<2> : k_l2p_p2p<1>)<<<(t.n_p2p_task + 3) / 4, 128, 0, st>>>(
                    t.n_p2p_task, t.p2p_task, t.leaf_src, t.tgt_node, (const float *)t.tloc, (const float *)t.sloc,
                    t.leaf_ijk, t.leaf0, t.leaf_scale, t.near_ptr, t.near_leaf, ns);
        } else if (!t.ds) {
            (nq == 2 ? k_l2p_p2p_fp64<2> : k_l2p_p2p_fp64<1>)<<<nb, 128, 0, st>>>(
                t.nleaf, t.leaf_src, t.leaf_tgt, t.tgt_node, (const double *)t.tloc, (const double *)t.sloc, t.leaf_ijk,
                t.leaf0, t.leaf_scale, t.near_ptr, t.near_leaf, ns);
        }
    };
    t.ev_split[t.ev_next] = split && prof;
    if (whole) note(launch_field_pairs(c, t.near, f.m[0], nq == 2 ? f.m[1] : nullptr));
    if constexpr (sizeof(T) == 4) {
        (nq == 2 ? k_p2m2<2> : k_p2m2<1>)<<<(t.nleaf + 3) / 4, 128, 0, c.stream>>>(
            t.nleaf, t.leaf_src, (const float *)t.sloc, t.leaf0, ps[0], ps[1]);
    } else if (t.near.p2m.B) {
        const size_t l0 = (size_t)t.leaf0 * NR;
        note(launch_blocks(t.near.p2m, t.near, c.stream, nq, nullptr, (double *)M + l0, (double *)M + l0 + sstride));
    } else if (t.oz) {
        (nq == 2 ? k_p2m_ds<2> : k_p2m_ds<1>)<<<dim3((t.nleaf + 3) / 4, 5), 128, 0, c.stream>>>(
            t.nleaf, t.leaf_src, (const float4 *)t.ds_src_hi, (const float4 *)t.ds_src_lo, t.leaf0, ps[0], ps[1]);
    } else if (t.ds) {
        (nq == 2 ? k_p2m_ds_repeat<2> : k_p2m_ds_repeat<1>)<<<dim3((t.nleaf + 3) / 4, 6), 128, 0, c.stream>>>(
            t.nleaf, t.leaf_src, (const float4 *)t.ds_src_hi, (const float4 *)t.ds_src_lo, t.leaf0, ps[0], ps[1]);
    } else {
        k_p2m<T><<<dim3((t.nleaf + 3) / 4, nq), 128, 0, c.stream>>>(t.nleaf, t.leaf_src, (const T *)t.sloc, t.leaf0,
                                                                     ps[0], ps[1]);
    }
    if (prof) cudaEventRecord(ev[1], c.stream);
    // out (+)= sum_code Op[code] in[tab[cell][code]] over n output cells from out0; the
    // tensor-core form reads the inputs' hi/lo split and writes the outputs' split
    enum { M2M, M2L, L2L };
    auto translate = [&](int kind, int n, int out0, const FmmTree::TcLaunch &tl) {
        if (!n) return;
        const int ncode = kind == M2L ? NCODE_M2L : 8;
        const int *tab = kind == M2M ? t.m2m_tab : kind == M2L ? t.m2l_tab : t.l2l_tab;
        if (tc) {
            TcArgs a{};
            a.n_out = n; a.out0 = out0; a.ncode = ncode; a.tab = tab;
            a.op_img = kind == M2M ? t.img_m2m : kind == M2L ? t.img_m2l : t.img_l2l;
            a.in_hi = kind == L2L ? t.Fh : t.Mh;
            a.in_lo = kind == L2L ? t.Fl : t.Ml;
            a.out = (float *)(kind == M2M ? M : F);
            a.out_hi = kind == M2M ? t.Mh : t.Fh;
            a.out_lo = kind == M2M ? t.Ml : t.Fl;
            a.accumulate = kind == L2L;
            a.tile_code = t.tc_code; a.err = c.fmm_err; a.terms = 7;
            a.units = t.tc_units + tl.unit0; a.nunits = tl.nunit;
            a.comb = t.tc_comb + tl.comb0; a.ncomb = tl.ncomb; a.scratch = t.tc_scratch;
            a.nset = nq; a.set_io = sstride; a.set_scratch = t.nslot_floats;
            const cudaError_t e = launch_translate_tc(c.stream, a);
            if (e != cudaSuccess && terr == cudaSuccess) terr = e;
        } else {
            const void *ops = kind == M2M ? t.op_m2m : kind == M2L ? t.op_m2l : t.op_l2l;
            for (int q = 0; q < nq; q++) {
                T *in = (kind == L2L ? F : M) + q * sstride, *out = (kind == M2M ? M : F) + q * sstride;
                k_translate<T><<<(n + TB - 1) / TB, 160, tr_smem<T>(), c.stream>>>(n, out0, ncode, tab,
                                                                                (const T *)ops, in, out, kind == L2L);
            }
        }
    };
    // FP64 path: exact digit products on the tensor cores, then the sums of the units' partial
    // results and the digits of the next translation's inputs
    OzFinish fa{};
    if (t.oz) {
        fa.ncell = t.ncell; fa.nset = nq; fa.scratch = t.oz_scratch; fa.digits = t.oz_digits; fa.scale = t.oz_scale;
        fa.io = (double *)M; fa.cells = t.oz_leaves; fa.nlist = t.nleaf; fa.accumulate = 1; fa.split = t.nleaf;
        fa.wexp = t.oz_wexp;
        note(launch_oz_finish(c.stream, fa));  // digits of the leaves' multipoles
    }
    auto translate_oz = [&](int kind, const FmmTree::OzLaunch &ol, int nsplit) {
        if (!ol.ntile) return;
        OzArgs a{};
        a.ncode = kind == M2L ? NCODE_M2L : 8; a.ncell = t.ncell; a.nset = nq;
        a.cells = t.oz_cells; a.codes = t.oz_codes;
        a.tab = kind == M2M ? t.m2m_tab : kind == M2L ? t.m2l_tab : t.l2l_tab;
        a.op_img = t.oz_img[kind]; a.row_scale = t.oz_rows[kind];
        a.in = t.oz_digits; a.in_scale = t.oz_scale;
        a.units = t.oz_units + ol.unit0; a.nunits = ol.nunit; a.scratch = t.oz_scratch; a.err = c.fmm_err;
        note(launch_translate_oz(c.stream, a));
        fa.io = (double *)(kind == M2M ? M : F);
        fa.cells = t.oz_cells + (size_t)ol.tile0 * OZ_TILE; fa.nlist = ol.ntile * OZ_TILE; fa.fin = t.oz_fin + ol.tile0;
        fa.accumulate = kind == L2L; fa.split = nsplit; fa.wexp = t.oz_wexp + (kind == M2M ? 0 : NR);
        note(launch_oz_finish(c.stream, fa));
    };
    // FP32 + refinement path's FP64 tree: double-single; M and the locals above the leaves as pairs
    auto translate_ds = [&](int kind, const FmmTree::OzLaunch &ol) {
        if (!ol.ntile) return;
        const size_t fstride = (size_t)t.leaf0 * NR;
        float2 *Ms = (float2 *)M, *Fs = (float2 *)t.F_split;
        k_translate_ds<<<dim3(ol.nunit * DS_PARTS, nq), 128, 0, c.stream>>>(
            t.oz_units + ol.unit0, t.oz_cells, t.oz_codes, kind == M2L ? NCODE_M2L : 8,
            kind == M2M ? t.m2m_tab : kind == M2L ? t.m2l_tab : t.l2l_tab, (const float4 *)t.oz_img[kind],
            kind == L2L ? Fs : Ms, kind == L2L ? fstride : sstride, kind == M2M ? nullptr : (double *)F, sstride,
            kind == M2M ? Ms : Fs, kind == M2M ? sstride : fstride, t.leaf0, kind == L2L);
    };
    const FmmTree::TcLaunch none;
    for (int l = L - 1; l >= 2; l--)
        if (t.repeat) translate_ds(M2M, t.oz_m2m[l]);
        else if (t.oz) translate_oz(M2M, t.oz_m2m[l], t.oz_m2m[l].ntile * OZ_TILE);
        else translate(M2M, t.lev_begin[l + 1] - t.lev_begin[l], t.lev_begin[l], t.tc ? t.tc_m2m[l] : none);
    if (prof) cudaEventRecord(ev[2], c.stream);
    if (split) {  // the near field beside M2L and L2L
        cudaEventRecord(c.ev_fork, c.stream);
        cudaStreamWaitEvent(c.stream2, c.ev_fork, 0);
        ns.near_only = 1;
        if (prof) cudaEventRecord(t.evn[t.ev_next][0], c.stream2);
        near_field(c.stream2);
        if (prof) cudaEventRecord(t.evn[t.ev_next][1], c.stream2);
        cudaEventRecord(c.ev_join, c.stream2);
        ns.near_only = 0;
    }
    if (t.repeat) translate_ds(M2L, t.oz_m2l);
    else if (t.oz) translate_oz(M2L, t.oz_m2l, t.oz_m2l.nsplit);
    else translate(M2L, t.ncell, 0, t.tc_m2l);
    if (prof) cudaEventRecord(ev[3], c.stream);
    for (int l = 3; l <= L; l++)
        if (t.repeat) translate_ds(L2L, t.oz_l2l[l]);
        else if (t.oz) translate_oz(L2L, t.oz_l2l[l], l < L ? t.oz_l2l[l].ntile * OZ_TILE : 0);
        else translate(L2L, t.lev_begin[l + 1] - t.lev_begin[l], t.lev_begin[l], t.tc ? t.tc_l2l[l] : none);
    if (prof) cudaEventRecord(ev[4], c.stream);
    if (split || t.ds) {  // L2P apart: the double-single near field stores its sums
        if (split) cudaStreamWaitEvent(c.stream, c.ev_join, 0);
        else near_field(c.stream);
        if (whole) {
            const double *Fl = (const double *)F + (size_t)t.leaf0 * NR;
            note(launch_l2p_table(c, near_tree(t), t.near, nq, Fl, Fl + sstride, c.pot, c.pot2, f.phi[0], f.phi[1]));
        }
        auto k = nq == 2 ? k_l2p<T, 2> : k_l2p<T, 1>;
        if (t.ntgt > 0 && !whole)
            k<<<(t.ntgt + 127) / 128, 128, 0, c.stream>>>(t.ntgt, t.tgt_leaf, t.tgt_node, (const T *)t.tloc, t.leaf0,
                                                          t.leaf_scale, ns);
    } else {
        near_field(c.stream);
    }
    if (prof) {
        cudaEventRecord(ev[5], c.stream);
        t.ev_pending[t.ev_next] = true;
        t.ev_next ^= 1;
    }
    const cudaError_t e = cudaGetLastError();
    return terr != cudaSuccess ? terr : e;
}

int fmm_blocks(const Ctx &c, size_t *bytes) {
    const FmmTree *t = static_cast<const FmmTree *>(c.fmm);
    *bytes = 0;
    if (!t || !t->oz) return 0;
    if (!t->near.near.B) return 1;
    *bytes = t->near.near.bytes + t->near.p2m.bytes;
    return t->near.p2m.B ? 3 : 2;
}

bool fmm_whole(const Ctx &c) {
    const FmmTree *t = static_cast<const FmmTree *>(c.fmm);
    return t && t->near.near.B;
}

bool fmm_charges(const Ctx &c) {
    const FmmTree *t = static_cast<const FmmTree *>(c.fmm);
    return !t || !t->near.near.B || !t->near.p2m.B;
}

cudaError_t fmm_eval(Ctx &c, int nq, const FmmFields &f) {
    FmmTree *t = static_cast<FmmTree *>(c.fmm);
    if (!t) return cudaErrorNotSupported;
    return t->fp32 ? fmm_eval_t<float>(c, *t, nq, f) : fmm_eval_t<double>(c, *t, nq, f);
}

int fmm_eval_fp64(Ctx &c, int nq) {
    FmmTree *t32 = static_cast<FmmTree *>(c.fmm);
    if (!t32 || !t32->fp32) {
        c.err = "fmm: no FP32 tree";
        return FG_EINVAL;
    }
    if (!c.fmm64) {
        // the same depth (and so the same source order, src_dst) as the FP32 tree
        FmmTree *t = new FmmTree();
        t->fp32 = false;
        c.fmm = t;
        const int s = fmm_build_forest(c, t32->L);
        if (s != FG_OK) {
            fmm_free(c);
            c.fmm = t32;
            return s;
        }
        c.fmm64 = t;
        c.fmm = t32;
    }
    FCK(fmm_eval_t<double>(c, *static_cast<FmmTree *>(c.fmm64), nq, FmmFields{}));
    return FG_OK;
}

void fmm64_free(Ctx &c) {
    if (!c.fmm64) return;
    void *keep = c.fmm;
    c.fmm = c.fmm64;
    fmm_free(c);
    c.fmm = keep;
    c.fmm64 = nullptr;
}

int fmm_stage_ms(const Ctx &c, double ms[5]) {
    FmmTree *t = static_cast<FmmTree *>(c.fmm);
    if (!t) return FG_EINVAL;
    harvest_set(*t, t->ev_next ^ 1);
    harvest_set(*t, t->ev_next);
    for (int k = 0; k < 5; k++) ms[k] = t->stage_n ? t->stage_sum[k] / t->stage_n : 0.0;
    for (double &x : t->stage_sum) x = 0.0;
    t->stage_n = 0;
    return FG_OK;
}

int fmm_launches_per_eval(const Ctx &c, int nq) {
    const FmmTree *t = static_cast<const FmmTree *>(c.fmm);
    if (!t) return 0;
    int n = 2;  // P2M, L2P + P2P (both sets in one launch each)
    if ((c.opts.fmm_overlap != 0 && c.stream2) || t->ds) n += 1;  // L2P apart from the near field
    if (t->near.near.B) n += 1;  // the fields as pairs
    if (t->oz) {  // digits of the leaves, then per translation the products and the sums
        n += 1;
        for (int l = 2; l <= t->L - 1; l++) n += (t->oz_m2m[l].nunit > 0) + (t->oz_m2m[l].ntile > 0);
        n += (t->oz_m2l.nunit > 0) + (t->oz_m2l.ntile > 0);
        for (int l = 3; l <= t->L; l++) n += (t->oz_l2l[l].nunit > 0) + (t->oz_l2l[l].ntile > 0);
        return n;
    }
    // tensor-core translations: both sets in one launch and one combine launch; the k_translate
    // form launches once per set
    const int per = t->tc || t->ds ? 1 : nq;
    for (int l = 2; l <= t->L - 1; l++) n += per + (t->tc && t->tc_m2m[l].ncomb > 0);
    n += per + (t->tc && t->tc_m2l.ncomb > 0);
    for (int l = 3; l <= t->L; l++) n += per + (t->tc && t->tc_l2l[l].ncomb > 0);
    return n;
}

int *fmm_error_flag(const Ctx &c) {
    return c.fmm_err;
}

int fmm_info(const Ctx &c, int *L, int *nleaf, double *n_m2l, double *n_p2p) {
    const FmmTree *t = static_cast<const FmmTree *>(c.fmm);
    if (!t) return FG_EINVAL;
    *L = t->L;
    *nleaf = t->nleaf;
    *n_m2l = (double)t->n_m2l;
    *n_p2p = (double)t->n_p2p_pairs;
    return FG_OK;
}

}  // namespace fg
