// quantize_prod_tc.cu -- Algorithm 2 (Prod) quantisation on the 5th-generation tensor cores:
//
//   u = x / ||x|| -> y = R u (tcgen05.mma) -> Lloyd-Max codes -> residual e = ||u|| y - c[codes], in rotated space
//   -> S R^T e (tcgen05.mma) -> signs, ||e||, bit planes                     (upstream reference.py:429-469)
//
// Codes are those of the float32 chain of quantize.cu: u is its unit vector to the bit; both operands of the rotation enter
// as two fp16 terms (22 bits, scaled by powers of two), three products summed in float32, low orders first; a coordinate
// closer to a decision boundary than the two can differ by (QP_CHAIN, QP_TERMS below) is computed again by that chain: one in
// 5,000 at two bits, in 1,100 at four.  (A zero row is zero on both sides: not again.)  A sign may fall the other way where the projection is zero to within
// float32 rounding, about 1e-7 of ||e||, as it may between any two float32 orders.
//
// What bounds it (d = 128, float32, 2 bits + sign; clocks of a 128-row tile on one SM): 2 x 1,536 on the tensor cores, 2,600
// issue slots for the exact divisions, 3,200 for code selection and residual terms, 1,300 of HBM: the phases of a tile
// depend on one another and shared memory (both matrices, 128 KB, and one tile's terms) holds no second tile, so the
// sixteen warps go through them together and only the loads run ahead.  Measured: 1 M rows 4.1 ms on the FFMA kernel, 0.71 ms
// here (53 tiles an SM, 13 us each, 1 of them for the coordinates computed again: issuing the projection before those instead
// of behind them cost more than it hid, 0.82 ms).
#include "common.cuh"
#include "pipe.cuh"
#include "tc.cuh"

namespace tqb {

constexpr int QP_TILE = 128, QP_WARPS = 16, QP_THREADS = QP_WARPS * 32, QP_RPW = QP_TILE / QP_WARPS;
constexpr int QP_LIST = 1024;                 // coordinates computed again in one go
// Bound of the difference between a coordinate and the float32 chain's, in units of ||row of R|| (sum |u_k R_jk| is at most
// that, ||u|| being one to within rounding; 2 % more covers it).  The chain: dim roundings of 2^-24.  The terms: either
// operand is off by 2^-22 of itself, the product of the low terms, 2^-22, is left out, and the accumulators round toward zero,
// up to 2^-22 after each of the dim / 16 MMAs of the leading product (the others are 2^-11 of it) and once more for their sum.
// Beside it sqrt(dim) 2^-25 of either operand's scale, for terms below fp16's normal range.
constexpr float QP_UNIT = 1.02f / 4194304.0f;                                    // 2^-22
__host__ __device__ constexpr float qp_guard(int dim) { return QP_UNIT * (0.25f * dim + 3.0f + dim / 16.0f + 1.0f); }

struct ProdArgs {
    const void* x; int64_t n, x_stride;
    const float* rot; const float* qjl_rot; const float* bnd; const float* cent;
    int dim;                                  // a multiple of 32, at most DP
    uint8_t* packed; uint8_t* signs; float* res_norms; float* norms;
    int* error;
};

template <int DP, int MB>
struct QpCfg {
    static constexpr int TERM = DP * DP * 2, ATERM = QP_TILE * DP * 2, W = DP / 32;
    static constexpr int OFF_R = 0, OFF_T = 2 * TERM, OFF_A = 4 * TERM, OFF_PLANES = OFF_A + 2 * ATERM;      // R hi lo, S R^T hi lo, rows hi lo
    static constexpr int OFF_SIGNS = OFF_PLANES + QP_TILE * MB * W * 4;
    static constexpr int OFF_LIST = OFF_SIGNS + QP_TILE * W * 4;
    static constexpr int OFF_ROW = OFF_LIST + QP_LIST * 4;                       // den, ||u||, 4 partial sums of e^2
    static constexpr int OFF_CB = OFF_ROW + 6 * QP_TILE * 4;                     // boundaries, centroids
    static constexpr int OFF_GUARD = OFF_CB + 128;                               // guard of every coordinate
    static constexpr int OFF_BAR = OFF_GUARD + DP * 4;
    static constexpr int TOTAL = OFF_BAR + 64 + 1024;                            // + slack for the 1024-byte alignment
    static constexpr int CG = DP / 4;                                            // columns of an epilogue thread
    static_assert(TOTAL <= 227 * 1024, "shared memory");
};

__device__ __forceinline__ void qp_sts128(uint32_t addr, uint32_t a, uint32_t b, uint32_t c, uint32_t d) {
    asm volatile("st.shared.v4.b32 [%0], {%1, %2, %3, %4};" ::"r"(addr), "r"(a), "r"(b), "r"(c), "r"(d) : "memory");
}
__device__ __forceinline__ void qp_split2(float a, float b, uint32_t& hi, uint32_t& lo) {
    const __half2 h = __floats2half2_rn(a, b);
    const float2 f = __half22float2(h);
    hi = *reinterpret_cast<const uint32_t*>(&h);
    lo = pack_half2(a - f.x, b - f.y);
}
// K-major, 128-byte-swizzled B operand of M (row n = output, column k = contraction), hi and lo terms; returns the scale.
// len (or null): the rows' lengths.
template <int DP>
__device__ __forceinline__ float qp_build(uint8_t* sm, int off_hi, int off_lo, const float* __restrict__ M, int dim, float* red, float* len) {
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    float mx = 0.0f;
    for (int n = warp; n < dim; n += QP_WARPS) {
        float ss = 0.0f;
        for (int k = lane; k < dim; k += 32) {
            const float v = __ldg(M + (int64_t)n * dim + k);
            mx = fmaxf(mx, fabsf(v));
            ss = fmaf(v, v, ss);
        }
        if (len) {
            ss = sqrtf(warp_sum(ss));
            if (lane == 0) len[n] = ss;
        }
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, o));
    if (lane == 0) red[warp] = mx;
    __syncthreads();
    mx = 0.0f;
    for (int w = 0; w < QP_WARPS; w++) mx = fmaxf(mx, red[w]);
    __syncthreads();
    const float sc = fp16_scale(mx);
#pragma unroll 4
    for (int e = threadIdx.x; e < DP * DP / 4; e += QP_THREADS) {
        const int n = e / (DP / 4), k = (e % (DP / 4)) * 4;
        const float4 v = n < dim && k < dim ? __ldg(reinterpret_cast<const float4*>(M + (int64_t)n * dim + k)) : make_float4(0.f, 0.f, 0.f, 0.f);
        uint32_t h0, l0, h1, l1;
        qp_split2(v.x * sc, v.y * sc, h0, l0);
        qp_split2(v.z * sc, v.w * sc, h1, l1);
        const uint32_t off = (uint32_t)(k >> 6) * (DP * 128) + sw128_offset(n, k & 63);
        *reinterpret_cast<uint2*>(sm + off_hi + off) = make_uint2(h0, h1);
        *reinterpret_cast<uint2*>(sm + off_lo + off) = make_uint2(l0, l1);
    }
    return sc;
}

template <typename T, int DP, int MB>
__global__ void __launch_bounds__(QP_THREADS, 1) quantize_prod_tc_kernel(const ProdArgs a) {
    using C = QpCfg<DP, MB>;
    constexpr int NB = (1 << MB) - 1, CG = C::CG, EPL = DP / 32;
    constexpr float USC = 256.0f;                          // scale of unit vectors and residuals
    extern __shared__ uint8_t smem_unaligned[];
    __shared__ float red[QP_WARPS];
    __shared__ int list_n;
    const uint32_t raw = smem_u32(smem_unaligned);
    const uint32_t base = (raw + 1023u) & ~1023u;
    uint8_t* const sm = smem_unaligned + (base - raw);
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const uint32_t bar = base + C::OFF_BAR, tmem_slot = bar + 16;
    if (threadIdx.x == 0) mbar_init(bar, 1);
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    if (warp == 0) tmem_alloc(tmem_slot, 2 * DP);
    float* const bnd_s = reinterpret_cast<float*>(sm + C::OFF_CB);
    float* const cent_s = bnd_s + 16;
    if (threadIdx.x < NB) bnd_s[threadIdx.x] = a.bnd[threadIdx.x];
    if (threadIdx.x <= NB) cent_s[threadIdx.x] = a.cent[threadIdx.x];
    float* const guard_s = reinterpret_cast<float*>(sm + C::OFF_GUARD);
    if (threadIdx.x < DP) guard_s[threadIdx.x] = -1.0f;    // (columns beyond dim: never)
    __syncthreads();
    const float rsc = qp_build<DP>(sm, C::OFF_R, C::OFF_R + C::TERM, a.rot, a.dim, red, guard_s);
    const float unscale = 1.0f / (USC * rsc);
    if (threadIdx.x < a.dim) guard_s[threadIdx.x] = fmaf(qp_guard(a.dim), guard_s[threadIdx.x], 12.0f * 2.9802322e-8f * (1.0f / rsc + guard_s[threadIdx.x] / USC));
    qp_build<DP>(sm, C::OFF_T, C::OFF_T + C::TERM, a.qjl_rot, a.dim, red, nullptr);      // (its product is used for its sign only)
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = lds32v(tmem_slot);
    float* const den_s = reinterpret_cast<float*>(sm + C::OFF_ROW);
    float* const n2_s = den_s + QP_TILE;
    float* const ee_s = n2_s + QP_TILE;                    // [4][128]
    uint32_t* const list = reinterpret_cast<uint32_t*>(sm + C::OFF_LIST);
    uint32_t* const planes = reinterpret_cast<uint32_t*>(sm + C::OFF_PLANES);
    uint32_t* const signw = reinterpret_cast<uint32_t*>(sm + C::OFF_SIGNS);
    const uint32_t ahi = base + C::OFF_A, alo = ahi + C::ATERM;
    const T* const x = reinterpret_cast<const T*>(a.x);
    const int per = a.dim >> 5, words = a.dim >> 5;        // consecutive elements of a lane; words of a plane
    const int64_t ntiles = (a.n + QP_TILE - 1) / QP_TILE;
    bool ok = true;
    uint32_t phase = 0;

    // Three products of the rows' terms with a matrix's, the small ones first.  The accumulator is rounded toward zero after
    // every MMA: the second half of the leading product goes to an accumulator of its own (d2), which halves that bias.
    auto multiply = [&](uint32_t d, uint32_t d2, int off_b) {
        constexpr uint32_t IDESC = (1u << 4) | ((uint32_t)(DP >> 3) << 17) | ((uint32_t)(QP_TILE >> 4) << 24);   // fp16 x fp16 -> f32
        tc_fence_after();
        uint32_t acc = 0;
#pragma unroll
        for (int t = 0; t < 3; t++) {
            const uint32_t am = t == 0 ? alo : ahi, bm = base + off_b + (t == 1 ? C::TERM : 0);
#pragma unroll
            for (int kb = 0; kb < DP / 64; kb++) {
                const uint64_t ad = umma_desc(am + kb * (QP_TILE * 128)), bd = umma_desc(bm + kb * (DP * 128));
#pragma unroll
                for (int k = 0; k < 4; k++) {
                    const int step = 4 * kb + k, half = DP / 32;
                    const bool second = t == 2 && step >= half;
                    umma_f16(second ? d2 : d, ad + 2 * k, bd + 2 * k, IDESC, t == 2 && step == half ? 0u : acc);
                    acc = 1;
                }
            }
        }
        umma_commit(bar);
    };
    auto finished = [&]() {                                // of the product: every thread
        ok = mbar_wait(bar, phase & 1) && ok;
        phase++;
        tc_fence_after();
    };
    // a lane's elements of a row
    auto load_row = [&](int64_t r, float (&v)[EPL]) {
        const T* p = x + r * a.x_stride + lane * per;
        if (per == 4) {
            const float4 f = load4(p);
            v[0] = f.x; v[1] = f.y; v[EPL - 2] = f.z; v[EPL - 1] = f.w;
        } else {
#pragma unroll
            for (int q = 0; q < EPL; q++) v[q] = q < per ? to_f32<T>(p[q]) : 0.0f;
        }
    };
    // the unit vector of quantize.cu (Prod): divided by its norm, then by the norm of the result
    auto unit = [&](float (&v)[EPL], float den, float den2) {
#pragma unroll
        for (int q = 0; q < EPL; q++) v[q] = v[q] / den / den2;
    };

    float nx[QP_RPW][EPL];
    auto request = [&](int64_t tile) {
#pragma unroll
        for (int i = 0; i < QP_RPW; i++) {
            const int64_t r = tile * QP_TILE + warp * QP_RPW + i;
            if (r < a.n) load_row(r, nx[i]);
            else
#pragma unroll
                for (int q = 0; q < EPL; q++) nx[i][q] = 0.0f;
        }
    };
    request(blockIdx.x);
    for (int64_t tile = blockIdx.x; tile < ntiles; tile += gridDim.x) {
        // ---- rows -> unit vectors -> terms ----
        {
            float ss[QP_RPW], s2[QP_RPW];
#pragma unroll
            for (int i = 0; i < QP_RPW; i++) {
                ss[i] = 0.0f;
#pragma unroll
                for (int q = 0; q < EPL; q++) ss[i] = fmaf(nx[i][q], nx[i][q], ss[i]);
            }
#pragma unroll
            for (int o = 16; o > 0; o >>= 1)
#pragma unroll
                for (int i = 0; i < QP_RPW; i++) ss[i] += __shfl_xor_sync(0xffffffffu, ss[i], o);
#pragma unroll
            for (int i = 0; i < QP_RPW; i++) {
                ss[i] = sqrtf(ss[i]);
                const float den = fmaxf(ss[i], 1e-10f);
                s2[i] = 0.0f;
#pragma unroll
                for (int q = 0; q < EPL; q++) { nx[i][q] = nx[i][q] / den; s2[i] = fmaf(nx[i][q], nx[i][q], s2[i]); }
            }
#pragma unroll
            for (int o = 16; o > 0; o >>= 1)
#pragma unroll
                for (int i = 0; i < QP_RPW; i++) s2[i] += __shfl_xor_sync(0xffffffffu, s2[i], o);
#pragma unroll
            for (int i = 0; i < QP_RPW; i++) {
                const int row = warp * QP_RPW + i;
                const int64_t r = tile * QP_TILE + row;
                s2[i] = sqrtf(s2[i]);
                const float den2 = fmaxf(s2[i], 1e-10f);
#pragma unroll
                for (int q = 0; q < EPL; q++) nx[i][q] = nx[i][q] / den2;
                if (lane == 0) {
                    den_s[row] = fmaxf(ss[i], 1e-10f);
                    n2_s[row] = s2[i];
                    if (r < a.n) a.norms[r] = ss[i];
                }
                if (per == EPL) {
                    uint32_t h[EPL / 2], l[EPL / 2];
#pragma unroll
                    for (int q = 0; q < EPL; q += 2) qp_split2(nx[i][q] * USC, nx[i][q + 1] * USC, h[q / 2], l[q / 2]);
                    const int k = lane * EPL;
                    const uint32_t off = (uint32_t)(k >> 6) * (QP_TILE * 128) + sw128_offset(row, k & 63);
#pragma unroll
                    for (int q = 0; q < EPL / 2; q++) {
                        *reinterpret_cast<uint32_t*>(sm + C::OFF_A + off + 4 * q) = h[q];
                        *reinterpret_cast<uint32_t*>(sm + C::OFF_A + C::ATERM + off + 4 * q) = l[q];
                    }
                } else {                                   // (96 dimensions: three elements a lane, zeros behind them)
#pragma unroll
                    for (int q = 0; q < EPL; q++) {
                        const int k = q < per ? lane * per + q : a.dim + lane + 32 * (q - per);
                        uint32_t h, l;
                        qp_split2(q < per ? nx[i][q] * USC : 0.0f, 0.0f, h, l);
                        const uint32_t off = (uint32_t)(k >> 6) * (QP_TILE * 128) + sw128_offset(row, k & 63);
                        *reinterpret_cast<uint16_t*>(sm + C::OFF_A + off) = (uint16_t)h;
                        *reinterpret_cast<uint16_t*>(sm + C::OFF_A + C::ATERM + off) = (uint16_t)l;
                    }
                }
            }
        }
        if (threadIdx.x == 0) list_n = 0;
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
        tc_fence_before();
        __syncthreads();
        if (threadIdx.x == 0) multiply(tmem, tmem + DP, C::OFF_R);
        if (tile + gridDim.x < ntiles) request(tile + gridDim.x);
        finished();
        // ---- codes and residuals: thread = a quarter of a row ----
        const int ew = warp & 3, cg = warp >> 2, row = ew * 32 + lane, col0 = cg * CG;
        const uint32_t src = tmem + ((uint32_t)(ew * 32) << 16) + col0;
        uint32_t plane[MB], guard = 0;
        {
            float bnd[NB], cent[NB + 1], ee = 0.0f;
#pragma unroll
            for (int i = 0; i < NB; i++) bnd[i] = bnd_s[i];
#pragma unroll
            for (int i = 0; i <= NB; i++) cent[i] = cent_s[i];
#pragma unroll
            for (int p = 0; p < MB; p++) plane[p] = 0;
            const float n2 = n2_s[row];
#pragma unroll
            for (int c = 0; c < CG; c += 8) {
                uint32_t v[8], v2[8], h[4], l[4];
                float e[8];
                const float4 ga = *reinterpret_cast<const float4*>(guard_s + col0 + c), gb = *reinterpret_cast<const float4*>(guard_s + col0 + c + 4);
                const float gd[8] = {ga.x, ga.y, ga.z, ga.w, gb.x, gb.y, gb.z, gb.w};
                tmem_ld8_async(src + c, v);
                tmem_ld8(src + DP + c, v2);                // (waits for both)
                tmem_wait8(v);
#pragma unroll
                for (int i = 0; i < 8; i++) {
                    const float y = (__uint_as_float(v[i]) + __uint_as_float(v2[i])) * unscale;
                    uint32_t code = 0;
                    float cv = cent[0], near = 1e30f;
#pragma unroll
                    for (int b = 0; b < NB; b++) {
                        const bool up = bnd[b] < y;
                        code += up ? 1u : 0u;
                        cv = up ? cent[b + 1] : cv;
                        near = fminf(near, fabsf(y - bnd[b]));
                    }
                    const bool in = col0 + c + i < a.dim;
                    if (near < gd[i]) guard |= 1u << (c + i);
                    e[i] = in ? fmaf(n2, y, -cv) : 0.0f;
                    ee = fmaf(e[i], e[i], ee);
                    const int bit = 8 * (c >> 3) + 7 - i;
#pragma unroll
                    for (int p = 0; p < MB; p++) plane[p] |= ((code >> p) & 1u) << bit;
                }
#pragma unroll
                for (int i = 0; i < 4; i++) qp_split2(e[2 * i] * USC, e[2 * i + 1] * USC, h[i], l[i]);
                const int k = col0 + c;
                const uint32_t off = (uint32_t)(k >> 6) * (QP_TILE * 128) + sw128_offset(row, k & 63);
                qp_sts128(ahi + off, h[0], h[1], h[2], h[3]);
                qp_sts128(alo + off, l[0], l[1], l[2], l[3]);
            }
            ee_s[cg * QP_TILE + row] = ee;
#pragma unroll
            for (int p = 0; p < MB; p++) {
                if (CG == 32) { if (cg < words) planes[(row * MB + p) * words + cg] = plane[p]; }
                else reinterpret_cast<uint16_t*>(planes)[(row * MB + p) * (2 * words) + cg] = (uint16_t)plane[p];
            }
        }
        if (tile * QP_TILE + row >= a.n || n2_s[row] == 0.0f) guard = 0;
        // ---- coordinates next to a boundary again, by the chain of quantize.cu: a warp per coordinate ----
        while (__syncthreads_or(guard != 0)) {
            while (guard) {
                const int pos = atomicAdd(&list_n, 1);
                if (pos >= QP_LIST) break;
                list[pos] = ((uint32_t)row << 8) | (uint32_t)(col0 + __ffs(guard) - 1);
                guard &= guard - 1;
            }
            __syncthreads();
            const int count = min(list_n, QP_LIST);
            for (int i = warp; i < count; i += QP_WARPS) {
                const int grow = (int)(list[i] >> 8), j = (int)(list[i] & 255u);
                const float n2 = n2_s[grow];
                float u[EPL], rr[EPL], y = 0.0f;
                load_row(tile * QP_TILE + grow, u);
                unit(u, den_s[grow], fmaxf(n2, 1e-10f));
#pragma unroll
                for (int q = 0; q < EPL; q++) rr[q] = q < per ? __ldg(a.rot + (int64_t)j * a.dim + lane * per + q) : 0.0f;
                for (int s = 0; s < 32; s++)
#pragma unroll
                    for (int q = 0; q < EPL; q++) {
                        const float us = __shfl_sync(0xffffffffu, u[q], s), rs = __shfl_sync(0xffffffffu, rr[q], s);
                        if (q < per) y = fmaf(us, rs, y);
                    }
                uint32_t code = 0;
                for (int b = 0; b < NB; b++) code += bnd_s[b] < y ? 1u : 0u;
                if (lane == 0) {
                    const uint32_t bit = 1u << (8 * ((j & 31) >> 3) + 7 - (j & 7));
#pragma unroll
                    for (int p = 0; p < MB; p++) {
                        uint32_t* w = &planes[(grow * MB + p) * words + (j >> 5)];
                        if ((code >> p) & 1u) atomicOr(w, bit);
                        else atomicAnd(w, ~bit);
                    }
                    const __half hi = __float2half_rn(fmaf(n2, y, -cent_s[code]) * USC);
                    const __half lo = __float2half_rn(fmaf(n2, y, -cent_s[code]) * USC - __half2float(hi));
                    const uint32_t off = (uint32_t)(j >> 6) * (QP_TILE * 128) + sw128_offset(grow, j & 63);
                    *reinterpret_cast<__half*>(sm + C::OFF_A + off) = hi;
                    *reinterpret_cast<__half*>(sm + C::OFF_A + C::ATERM + off) = lo;
                }
            }
            __syncthreads();
            if (threadIdx.x == 0) list_n = 0;
        }
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
        tc_fence_before();
        __syncthreads();
        if (threadIdx.x == 0) multiply(tmem, tmem + DP, C::OFF_T);
        // ---- codes and residual norms out, while the projection runs ----
        const int64_t r0 = tile * QP_TILE;
        const int rows = (int)min((int64_t)QP_TILE, a.n - r0);
        for (int i = threadIdx.x; i < rows * MB * words; i += QP_THREADS) reinterpret_cast<uint32_t*>(a.packed)[r0 * MB * words + i] = planes[i];
        if (threadIdx.x < rows) {
            const int r = threadIdx.x;
            a.res_norms[r0 + r] = sqrtf((ee_s[r] + ee_s[QP_TILE + r]) + (ee_s[2 * QP_TILE + r] + ee_s[3 * QP_TILE + r]));
        }
        finished();
        // ---- signs ----
        uint32_t sw = 0;
#pragma unroll
        for (int c = 0; c < CG; c += 8) {
            uint32_t v[8], v2[8];
            tmem_ld8_async(src + c, v);
            tmem_ld8(src + DP + c, v2);
            tmem_wait8(v);
#pragma unroll
            for (int i = 0; i < 8; i++) sw |= (__uint_as_float(v[i]) + __uint_as_float(v2[i]) >= 0.0f ? 1u : 0u) << (8 * (c >> 3) + 7 - i);
        }
        if (CG == 32) { if (cg < words) signw[row * words + cg] = sw; }
        else reinterpret_cast<uint16_t*>(signw)[row * (2 * words) + cg] = (uint16_t)sw;
        tc_fence_before();
        if (!__syncthreads_and(ok)) break;
        for (int i = threadIdx.x; i < rows * words; i += QP_THREADS) reinterpret_cast<uint32_t*>(a.signs)[r0 * words + i] = signw[i];
    }
    if (!ok && lane == 0) atomicExch(a.error, 1);
    tc_fence_before();
    __syncthreads();
    if (warp == 0) {
        tc_fence_after();
        tmem_dealloc(tmem, 2 * DP);
    }
}

template <typename T, int DP, int MB>
static int launch_qp(ProdArgs a, cudaStream_t st) {
    using C = QpCfg<DP, MB>;
    auto kern = quantize_prod_tc_kernel<T, DP, MB>;
    TQB_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, C::TOTAL));
    if (int e = tc_error_word(&a.error)) return e;
    const int grid = (int)std::min<int64_t>(sm_count(), (a.n + QP_TILE - 1) / QP_TILE);
    kern<<<grid, QP_THREADS, C::TOTAL, st>>>(a);
    return check_launch("quantize_prod_tc");
}
template <typename T, int DP>
static int qp_bits(int mb, const ProdArgs& a, cudaStream_t st) {
    switch (mb) {
        case 1: return launch_qp<T, DP, 1>(a, st);
        case 2: return launch_qp<T, DP, 2>(a, st);
        case 3: return launch_qp<T, DP, 3>(a, st);
        case 4: return launch_qp<T, DP, 4>(a, st);
    }
    return TQB_ERR_UNSUPPORTED;
}

// Tries the tensor-core path; TQB_ERR_UNSUPPORTED (without touching the last-error text) sends the call to the FFMA kernel.
int quantize_prod_tc_try(const void* x, int dtype, int64_t n, int dim, int64_t x_stride, const float* rot, const float* bnd, const float* cent,
                         const float* qjl_rot, int mse_bits, uint8_t* packed, uint8_t* signs, float* res_norms, float* norms, cudaStream_t st) {
    // (rows of 32 have too little work; the matrices' operands cost 10 us a call)
    if (dim % 32 || dim < 64 || dim > 128 || mse_bits < 1 || mse_bits > 4) return TQB_ERR_UNSUPPORTED;
    const size_t esz = dtype == TQB_F32 ? 4 : 2;
    if ((uintptr_t)x % 16 || (x_stride * esz) % 16 || ((uintptr_t)rot | (uintptr_t)qjl_rot) % 16) return TQB_ERR_UNSUPPORTED;
    if (((uintptr_t)packed | (uintptr_t)signs) % 4) return TQB_ERR_UNSUPPORTED;
    ProdArgs a{};
    a.x = x; a.n = n; a.x_stride = x_stride; a.rot = rot; a.qjl_rot = qjl_rot; a.bnd = bnd; a.cent = cent; a.dim = dim;
    a.packed = packed; a.signs = signs; a.res_norms = res_norms; a.norms = norms;
#define TQB_QP(T) (dim == 64 ? qp_bits<T, 64>(mse_bits, a, st) : qp_bits<T, 128>(mse_bits, a, st))
    switch (dtype) {
        case TQB_F32: return TQB_QP(float);
        case TQB_F16: return TQB_QP(__half);
        case TQB_BF16: return TQB_QP(__nv_bfloat16);
    }
#undef TQB_QP
    return TQB_ERR_UNSUPPORTED;
}

}  // namespace tqb
