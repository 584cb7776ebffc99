// FMM translations of the FP64 path on the 5th-generation tensor cores (tcgen05).
//
// A translation applies a fixed 100x100 operator to 100-coefficient expansions held in FP64.
// The FP16 tensor pipe evaluates it by digits (the error-free splitting of Ozaki, Ogita,
// Oishi and Rump, "Error-free transformations of matrix multiplication by using fast routines of
// matrix multiplication and its applications", 2012): every operator row and every expansion is
// scaled by a power of two of its own and written as five signed digits of 10 bits,
//     a_ij = rs_i sum_s A_s[i][j] 2^-10s,    x_j = cs sum_t X_t[j] 2^-10t,
// |A_0| <= 512, |X_0| <= 1024 and |A_s|, |X_s| <= 512 for s >= 1: integers that FP16 holds. The
// digit products of equal weight s + t = l <= 4 are summed by MMAs with FP32 accumulation into one
// accumulator per l. A sum of integers is exact there while it stays below 2^24. For l = 0 the
// operators' scales see to it for every input; for l >= 1 nothing does, the sizes do: were all
// the lower digits' signs to agree, the worst rows (M2L) would reach 2.1, 3.0, 3.7 and 4.5 x 2^24
// for l = 1 to 4 (M2M at most 1.5, L2L 2.7), but digits spread over their range with the signs of
// a number's low digits add up to an rms of 0.12 to 0.15 x 2^24, so 2^24 is 8.5 standard
// deviations off for l = 1 and 6.6 for l = 4 (over all rows of the operators). A sum beyond it
// would be rounded to a multiple of 2 to 8 units of 2^-10l. The
// five accumulators of each operator are combined and added up in double-single arithmetic (about
// 48 bits). Neglected: digit products of weight 2^-50 and less of the largest ones. Before the
// splitting each coefficient is weighted by a power of two (and the operator column by its
// inverse) that makes typical coefficients of all degrees alike: the 50 bits of an expansion share
// one exponent, so a coefficient far below the largest weighted one keeps fewer significant bits
// (the pairs of FP32 before had 48 bits each), with an error relative to the largest. Against FP64 sums the
// potentials differ by 2e-16 to 2e-14, less than the double-single products on the FP32 pipes
// that this replaces (2e-14 to 7e-14, simulated on the same multipoles).
//
// GEMM of one operator code and a tile of 48 cells: D_l[128 x 48 ns] += A_s[128 x 112] X_t[112 x
// 48 ns] (ns = 1 or 2 charge sets; rows = output coefficients, 100 used; columns = the cells of
// each set), 15 digit products of 7 K-steps. 48 cells because five FP32 accumulators of 96
// columns are 480 of the 512 columns of tensor memory. A tile lists its cells: M2L and L2L tiles
// hold cells of the same octant of their parents where that needs fewer (tile, code) pairs,
// since such cells share one interaction list (189 of the 316 offsets) and one L2L code.
//
// One CTA of 16 warps per work unit (some codes of one tile), one CTA per SM, 7 stages of K = 16:
//   warps 0-2   fill a stage: one bulk copy of the operator's digits (16.6 KB, stored as the MMA
//               reads them: no-swizzle K-major core matrices), 16-byte cp.async of the digits of
//               the 48 ns expansions (160 contiguous bytes per expansion and stage);
//   warps 4-15  drain finished accumulators: warp w owns the coefficient rows 32 (w % 4).. and the
//               columns 32 (w / 4 - 1).., loads the five sums, combines them, scales by
//               rs_i cs and adds to its double-single sums; at the end the pairs to scratch (their
//               conversion to FP64 here, 1/64 of the FP32 rate, took a third of the short launches: M2M
//               and L2L of the wire 0.185 and 0.164 ms, converted in k_oz_finish 0.162 and 0.133);
//   warp 3      one lane issues the MMAs.
// Bound by shared-memory reads of the MMA operands (7 KB per MMA of 128x96x16) and the drain,
// which the single accumulator set puts in series with the next code's MMAs.
// k_oz_finish adds the units' partial sums, stores FP64 and splits the result for the next
// translation. Every wait is bounded (about 1 s) as in fg_fmm_tc.cu.
#include <cuda_fp16.h>

#include <algorithm>
#include <cmath>
#include <cstdint>
#include <cstring>
#include <vector>

#include "fg_f32x2.cuh"
#include "fg_internal.h"
#include "fg_tcgen05.cuh"

namespace fg {

namespace {

using namespace tc;

constexpr int NRC = 100;             // reals per expansion (P = 9)
constexpr int ND = 5;                // digits of 10 bits
constexpr int NCELL = OZ_TILE;       // output cells per tile
constexpr int NCOL = 2 * NCELL;      // columns of two charge sets
constexpr int KI = 16;               // K per pipeline item and MMA
constexpr int IPC = 7;               // items per code: K = 112
constexpr int NSTAGE = 7;
constexpr uint32_t LBO = 128, SBO = 256;        // core matrices along K, 8-row groups (K = 16)
constexpr int A_DIGIT = 13 * (int)SBO;          // operator rows 0..103 of one digit
constexpr int A_BYTES = ND * A_DIGIT;           // 16,640
constexpr int B_DIGIT = (NCOL / 8) * (int)SBO;  // 3,072
constexpr int B_BYTES = ND * B_DIGIT;
constexpr int STAGE_BYTES = A_BYTES + B_BYTES;  // 32,000 (the M = 128 MMA reads rows 104..127 of the
                                                // last digit from the X digits: their sums go unused)
constexpr int ITEM_BYTES = ND * KI * 2;         // digits of one expansion and item (160)
static_assert(OZ_CELL_BYTES == IPC * ITEM_BYTES, "digit layout");
constexpr int TMEM_COLS = 512;
constexpr int LAG = 3;  // items whose gathers are in flight; an item's arrival then waits for the MMAs of the
                        // fourth item before it only (M2L of the wire, LAG 3 / 4 / 5 / 6: 0.80 / 0.80 / 0.83 / 0.87 ms)
constexpr int NPROD = 96, NDRAIN = 384, NTHREAD = NPROD + 32 + NDRAIN;
constexpr int DCOL = 32;  // columns per drain warp

__device__ __forceinline__ uint64_t sdesc(uint32_t saddr) { return sdesc_kmajor(saddr, LBO, SBO); }

__global__ void __launch_bounds__(NTHREAD, 1) k_translate_oz(OzArgs a) {
    extern __shared__ unsigned char smem_raw[];
    unsigned char *sm = reinterpret_cast<unsigned char *>(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
    __shared__ __align__(8) uint64_t full[NSTAGE], bfull[NSTAGE], empty[NSTAGE], tfull, tfree, tdone;
    __shared__ uint32_t tmem_base;
    __shared__ volatile int bail;
    // per code (ring of 4: the producers are at most two codes ahead of the drain): scale of each
    // column's expansion, source cell of each tile cell
    __shared__ __align__(8) float colf[4][NCOL];
    __shared__ int scell[4][NCELL];
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int ns = a.nset > 1 ? 2 : 1;
    const int4 unit = a.units[blockIdx.x];
    const int *__restrict__ cells = a.cells + (size_t)unit.x * NCELL;
    const int *__restrict__ codes = a.codes + unit.y;
    const int ncodes = unit.z - unit.y, nitems = ncodes * IPC;
    int *err = a.err;
    if (tid == 0) {
        for (int s = 0; s < NSTAGE; s++) {
            mbar_init(&full[s], NPROD);
            mbar_init(&bfull[s], 1);
            mbar_init(&empty[s], 1);
        }
        mbar_init(&tfull, 1);
        mbar_init(&tfree, NDRAIN);
        mbar_init(&tdone, 1);
        bail = 0;
        fence_mbar_init();
    }
    if (warp == 3) tmem_alloc(&tmem_base, TMEM_COLS);
    fence_proxy_async();
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = tmem_base;

    if (warp < 3) {
        // lane pairs copy the two 16-byte halves of one column's digit, 16 columns per copy; warp w
        // copies columns 16 w .. 16 w + 15 of every set, all digits
        const int half = lane & 1, ccell = 16 * warp + (lane >> 1);
        const uint32_t dst = A_BYTES + (ccell >> 3) * SBO + half * LBO + (ccell & 7) * 16;
        const size_t set_bytes = (size_t)a.ncell * OZ_CELL_BYTES;
        bool live = true;
        const int pc = tid % NCELL, py = tid / NCELL;  // cell and set whose scale this thread reads
        const int mycell = py < ns ? cells[pc] : -1;
        auto src_of = [&](int ci) {
            return (mycell >= 0 && ci < ncodes) ? __ldg(a.tab + (size_t)mycell * a.ncode + codes[ci]) : -1;
        };
        auto scale_of = [&](int sc) { return sc >= 0 ? __ldg(a.in_scale + (size_t)py * a.ncell + sc) : 0.f; };
        int s_cur = src_of(0), s_next = src_of(1);
        float f_cur = scale_of(s_cur);
        const unsigned char *src = nullptr;
        uint32_t bytes = 0;
        int armed = 0;
        for (int it = 0; it < nitems + LAG; it++) {
            if (it >= LAG) {  // the copies of item it - LAG have landed
                cp_wait<LAG - 1>();
                fence_proxy_async();
                if (live) mbar_arrive(&full[(it - LAG) % NSTAGE]);
            }
            if (it < nitems) {
                const int ci = it / IPC, q = it % IPC, ring = ci & 3;
                if (q == 0) {
                    colf[ring][tid] = f_cur;  // 0 beyond the last set
                    if (py == 0) scell[ring][pc] = s_cur;
                    s_cur = s_next;
                    s_next = src_of(ci + 2);
                    f_cur = scale_of(s_cur);
                    asm volatile("bar.sync 1, %0;" ::"n"(NPROD) : "memory");
                    const int sc = scell[ring][ccell];
                    bytes = sc >= 0 ? 16u : 0u;  // 0: zero fill where the code brings the cell nothing
                    src = a.in + (sc >= 0 ? (size_t)sc * OZ_CELL_BYTES : 0) + half * 16;
                }
                const int s = it % NSTAGE;
                if (live && it >= NSTAGE && !mbar_wait(&empty[s], ((it / NSTAGE) - 1) & 1, err, &bail)) live = false;
                if (live) {
                    unsigned char *st = sm + s * STAGE_BYTES;
                    if (tid == 0) {
                        mbar_arrive_expect_tx(&bfull[s], A_BYTES);
                        bulk_g2s(st, a.op_img + ((size_t)codes[ci] * IPC + q) * A_BYTES, A_BYTES, &bfull[s]);
                        armed = it + 1;
                    }
                    const unsigned char *from = src + q * ITEM_BYTES;
                    unsigned char *to = st + dst;
                    for (int y = 0; y < ns; y++, from += set_bytes, to += (NCELL / 8) * SBO)
#pragma unroll
                        for (int d = 0; d < ND; d++) cp16(to + d * B_DIGIT, from + d * (KI * 2), bytes);
                }
            }
            cp_commit();
        }
        cp_wait<0>();
        if (tid == 0 && bail)
            for (int it = armed > NSTAGE ? armed - NSTAGE : 0; it < armed; it++)
                mbar_drain(&bfull[it % NSTAGE], (it / NSTAGE) & 1);
    } else if (warp == 3) {
        if (lane == 0) {
            const uint32_t idesc = idesc_f16(128, NCELL * ns);
            bool ok = true;
            for (int ci = 0; ci < ncodes && ok; ci++) {
                if (ci >= 1 && !mbar_wait(&tfree, (ci - 1) & 1, err, &bail)) break;
                tc_fence_after();
                for (int q = 0; q < IPC; q++) {
                    const int it = ci * IPC + q, s = it % NSTAGE;
                    if (!mbar_wait(&full[s], (it / NSTAGE) & 1, err, &bail) ||
                        !mbar_wait(&bfull[s], (it / NSTAGE) & 1, err, &bail)) {
                        ok = false;
                        break;
                    }
                    tc_fence_after();
                    // the address is the low field of the descriptor, in units of 16 bytes
                    const uint64_t da = sdesc(smem_u32(sm + s * STAGE_BYTES)), db = da + A_BYTES / 16;
#pragma unroll
                    for (int i = 0; i < ND; i++)
#pragma unroll
                        for (int j = 0; i + j < ND; j++)
                            mma_f16(tmem + (i + j) * NCOL, da + i * (A_DIGIT / 16), db + j * (B_DIGIT / 16), idesc,
                                    (q == 0 && i == 0) ? 0u : 1u);
                    mma_commit(&empty[s]);
                }
                mma_commit(&tfull);
            }
            mma_commit(&tdone);
            mbar_drain(&tdone, 0);
        }
    } else {
        const int c0 = DCOL * ((warp >> 2) - 1);
        const int ncol = min(DCOL, ns * NCELL - c0);  // 32, 16 or <= 0
        const int quarter = warp & 3, row = 32 * quarter + lane;
        const uint32_t lane_base = tmem + ((uint32_t)(32 * quarter) << 16) + c0;
        const u64 w1 = pk2(0x1p-10f, 0x1p-10f), w2 = pk2(0x1p-20f, 0x1p-20f), w3 = pk2(0x1p-30f, 0x1p-30f),
                  w4 = pk2(0x1p-40f, 0x1p-40f);
        u64 ah[DCOL / 2], al[DCOL / 2];
#pragma unroll
        for (int j = 0; j < DCOL / 2; j++) ah[j] = al[j] = 0ull;
        int drained = 0;
        for (int ci = 0; ci < ncodes; ci++) {
            const float rs = row < NRC ? __ldg(a.row_scale + (size_t)codes[ci] * NRC + row) : 0.f;
            const bool mine = mbar_wait(&tfull, ci & 1, err, &bail);
            if (!__all_sync(0xffffffffu, mine && !bail)) break;
            tc_fence_after();
            const u64 rs2 = pk2(rs, rs);
#pragma unroll
            for (int g = 0; g < DCOL / 8; g++) {
                if (8 * g >= ncol) break;
                uint32_t v[ND][8];
#pragma unroll
                for (int l = 0; l < ND; l++) tmem_ld8(lane_base + l * NCOL + 8 * g, v[l]);
                tmem_wait_ld();
#pragma unroll
                for (int k = 0; k < 4; k++) {
                    const int j = 4 * g + k;
                    auto val = [&](int l) { return pk2(__uint_as_float(v[l][2 * k]), __uint_as_float(v[l][2 * k + 1])); };
                    // h + lo = sum_l v_l 2^-10l: the first two additions with their exact errors
                    const u64 v0 = val(0), v1 = val(1), v2 = val(2);
                    const u64 h1 = fma2(v1, w1, v0), e1 = fma2(v1, w1, sub2(v0, h1));
                    const u64 h = fma2(v2, w2, h1), e2 = fma2(v2, w2, sub2(h1, h));
                    const u64 lo = fma2(val(4), w4, fma2(val(3), w3, add2(e1, e2)));
                    const u64 f = mul2(rs2, *reinterpret_cast<const u64 *>(&colf[ci & 3][c0 + 2 * j]));
                    // (ah, al) += f (h + lo): two-sum of the leading parts
                    const u64 x = mul2(h, f), s = add2(ah[j], x), bb = sub2(s, ah[j]);
                    const u64 er = add2(sub2(ah[j], sub2(s, bb)), sub2(x, bb));
                    const u64 t = add2(al[j], fma2(lo, f, er));
                    ah[j] = add2(s, t);  // renormalise
                    al[j] = sub2(t, sub2(ah[j], s));
                }
            }
            tc_fence_before();
            mbar_arrive(&tfree);
            drained++;
        }
        if (drained == ncodes && row < NRC) {
#pragma unroll
            for (int j = 0; j < DCOL; j++) {
                if (j >= ncol) break;
                const int col = c0 + j, y = col >= NCELL ? 1 : 0;
                float h0, h1, l0, l1;
                upk2(ah[j / 2], h0, h1);
                upk2(al[j / 2], l0, l1);
                a.scratch[(((size_t)unit.w * ns + y) * NCELL + col - NCELL * y) * NRC + row] =
                    (j & 1) ? make_float2(h1, l1) : make_float2(h0, l0);
            }
        }
    }
    tc_fence_before();
    __syncthreads();
    if (warp == 3) {
        tc_fence_after();
        tmem_dealloc(tmem, TMEM_COLS);
    }
}

// One warp per (listed cell, charge set): FP64 sum of the tile's partial results (in slot order),
// added to the expansion where accumulate, stored, and (the first `split` listed cells) cut into
// digits for the next translation: X = round(x 2^(50 - e + w)) with the coefficient weight 2^w and |x| 2^w < 2^e, cut into
// balanced 10-bit digits by integer arithmetic (FP64 arithmetic would run at 1/64 rate).
// A coefficient that is not finite becomes a NaN digit.
__global__ void __launch_bounds__(256) k_oz_finish(OzFinish a) {
    const int ns = a.nset > 1 ? 2 : 1;
    const int w = blockIdx.x * 8 + (threadIdx.x >> 5), lane = threadIdx.x & 31;
    const int k = w / ns, y = w % ns;
    if (k >= a.nlist) return;
    const int cell = a.cells[k];
    if (cell < 0) return;
    double *io = a.io + ((size_t)y * a.ncell + cell) * NRC;
    double v[4] = {0.0, 0.0, 0.0, 0.0};
    const int2 fin = a.fin ? a.fin[k / NCELL] : make_int2(0, 0);
#pragma unroll 4
    for (int s = 0; s < fin.y; s++) {
        const float2 *p = a.scratch + (((size_t)(fin.x + s) * ns + y) * NCELL + k % NCELL) * NRC;
#pragma unroll
        for (int m = 0; m < 4; m++) {
            const float2 x = lane + 32 * m < NRC ? p[lane + 32 * m] : make_float2(0.f, 0.f);
            v[m] += (double)x.x + (double)x.y;
        }
    }
#pragma unroll
    for (int m = 0; m < 4; m++) {
        const int r = lane + 32 * m;
        if (r < NRC) {
            if (a.accumulate) v[m] = fin.y ? io[r] + v[m] : io[r];
            if (a.fin && (fin.y || !a.accumulate)) io[r] = v[m];
        }
    }
    if (k >= a.split) return;
    int ex[4], e = -100000;
#pragma unroll
    for (int m = 0; m < 4; m++) {
        const int r = lane + 32 * m, field = (__double2hiint(v[m]) >> 20) & 0x7ff;
        ex[m] = (r < NRC && field > 0 && field < 2047) ? field - 1022 + a.wexp[r] : -100000;
        e = max(e, ex[m]);
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) e = max(e, __shfl_xor_sync(0xffffffffu, e, o));
    e = min(120, max(-110, e));
    __half *dig = reinterpret_cast<__half *>(a.digits + ((size_t)y * a.ncell + cell) * OZ_CELL_BYTES);
#pragma unroll
    for (int m = 0; m < 4; m++) {
        const int r = lane + 32 * m;
        if (r >= NRC) continue;
        const int sh = 50 - e + a.wexp[r];
        const bool bad = ((__double2hiint(v[m]) >> 20) & 0x7ff) == 2047;
        long long X = bad ? 0 : __double2ll_rn(v[m] * __hiloint2double((1023 + sh) << 20, 0));
        __half *o = dig + (r >> 4) * (ITEM_BYTES / 2) + (r & 15);
#pragma unroll
        for (int d = ND - 1; d >= 1; d--) {
            const int s = (int)((X + 512) & 1023) - 512;
            X = (X - s) >> 10;
            o[d * KI] = __int2half_rn(s);
        }
        o[0] = bad ? __ushort_as_half(0x7fff) : __int2half_rn((int)X);
    }
    if (lane == 0) a.scale[(size_t)y * a.ncell + cell] = __int_as_float((127 + e - 10) << 23);
}

int oz_smem() { return NSTAGE * STAGE_BYTES + 1024; }

}  // namespace

cudaError_t oz_setup() {
    return cudaFuncSetAttribute(k_translate_oz, cudaFuncAttributeMaxDynamicSharedMemorySize, oz_smem());
}

cudaError_t launch_translate_oz(cudaStream_t st, const OzArgs &a) {
    if (a.nunits <= 0) return cudaSuccess;
    k_translate_oz<<<a.nunits, NTHREAD, oz_smem(), st>>>(a);
    return cudaGetLastError();
}

cudaError_t launch_oz_finish(cudaStream_t st, const OzFinish &a) {
    if (a.nlist <= 0) return cudaSuccess;
    const int warps = a.nlist * (a.nset > 1 ? 2 : 1);
    k_oz_finish<<<(warps + 7) / 8, 256, 0, st>>>(a);
    return cudaGetLastError();
}

// Digits of the operators as the MMA reads them, and the scale of every row: column j carries the
// inverse 2^-wexp[j] of the weight of input coefficient j. The sum of a row's leading digits stays
// below 2^14, so that with |X_0| <= 1024 no sum of leading products (l = 0) reaches 2^24.
OzImages oz_images(const std::vector<double> &ops, int ncode, const int *wexp) {
    OzImages im;
    im.img.assign((size_t)ncode * IPC * A_BYTES, 0);
    im.row_scale.assign((size_t)ncode * NRC, 0.f);
    std::vector<long long> X(NRC);
    for (int code = 0; code < ncode; code++)
        for (int i = 0; i < NRC; i++) {
            const double *row = &ops[((size_t)code * NRC + i) * NRC];
            int e = -100000;
            for (int j = 0; j < NRC; j++)
                if (row[j] != 0.0) e = std::max(e, std::ilogb(row[j]) + 1 - wexp[j]);
            if (e == -100000) continue;
            for (;; e++) {
                long long lead = 0;
                for (int j = 0; j < NRC; j++) {
                    X[j] = std::llrint(std::ldexp(row[j], 49 - e - wexp[j]));
                    lead += std::llabs(X[j] >> 40) + 1;
                }
                if (lead <= 16384) break;
            }
            im.row_scale[(size_t)code * NRC + i] = std::ldexp(1.0f, e - 9);
            for (int j = 0; j < NRC; j++) {
                const int q = j / KI, kk = j % KI;
                long long x = X[j];
                for (int d = ND - 1; d >= 0; d--) {
                    const int s = d ? (int)((x + 512) & 1023) - 512 : (int)x;
                    x = (x - s) >> 10;
                    const __half h = __float2half((float)s);
                    std::memcpy(&im.img[((size_t)code * IPC + q) * A_BYTES + (size_t)d * A_DIGIT + (i >> 3) * SBO +
                                        (kk >> 3) * LBO + (i & 7) * 16 + (kk & 7) * 2],
                                &h, 2);
                }
            }
        }
    return im;
}

}  // namespace fg
