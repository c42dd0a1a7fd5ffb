// scan_tc.cu -- the ranking pass of the index scan on the 5th-generation tensor cores, for calls with many queries and for
// Prod-mode rows.
//
// score[row][query] = norm * ( <c[codes], R q> [ + sqrt(pi/2)/d * ||r|| * <signs, S q> ] ).  Rows are the 128 rows of the MMA:
// their codes become fp16 centroids in a swizzled A tile (Prod rows: a second tile of +-fp16(sqrt(pi/2)/d ||r||)); up to 256
// queries (Prod: 128) lie in shared memory as the B operand.  The pass ranks only, like the passes of scan.cu: the merge
// re-scores the best k + 24 candidates in float32, and the scores it reports come from there.
//
// The list kernels rank Prod rows in float32, and MSE rows with queries of 22 bits where k > 24; here every operand has 11.
// Those calls' selections are PROVEN: with E a bound of |approximate - float32 score| (scan_tc_error), no row below the k-th
// best approximate score by more than 2 E can be among the best k, so everything above that is re-scored; where the buffer
// does not reach that far down (rows closer together than fp16 tells apart), the list kernels answer the query.  MSE calls of
// k <= 24 rank as they do there, on fp16 centroids and queries with the margin of 24.
//
// Candidates without lists: keeping sorted lists costs about k ln(rows) insertions per query and list, which bounds the other
// passes.  Here a first launch scores every `stride`-th tile and keeps only the largest score of each group of rows; the
// ksel-th largest of those maxima is not above the ksel-th best score of all rows (the maxima belong to distinct rows), and
// the main launch appends every row that is not below it, about ksel * stride of them, to the query's buffer.  A query
// whose buffer overflows (many rows tied with the bound), or would by what the sample shows, is scanned by the list kernels,
// which other queries skip; it gathers no further (32 queries, 28 of them zero, over 1 M rows: 17.5 ms with all tied rows
// counted, 0.46 ms now, 0.37 ms by the list kernels alone).
//
// What bounds it (d = 128, 256 queries, clocks of a 128-row tile): 1,024 on the tensor cores, about 1,400 issue slots per
// scheduler in the epilogue (a multiply-add, half a compare and a quarter of a shared load per score), 500 in the decoders.
// Two buffers of operands and of accumulators overlap them.
//   warps 0-7   decode: codes -> fp16 pairs through a table replicated per lane -> A tile
//   warps 8-15  epilogue: thread = row and half of the queries
//   warp 16     issues the MMAs (one lane)
// Every wait is bounded in time; one that expires sets the error word of tqb_quantize_status.
#include "scan_tc.cuh"
#include "pipe.cuh"
#include "tc.cuh"
#include "tiled_layout.cuh"

namespace tqb {

constexpr int ST_TILE = 128, ST_DEC = 8, ST_EPI = 8, ST_THREADS = (ST_DEC + ST_EPI + 1) * 32;
constexpr int ST_MAX_COLS = 256, ST_MAX_COLS_PROD = 128;
constexpr int ST_MAX_STRIDE = 16;
constexpr int ST_LOG = 96;                     // candidates an epilogue warp gathers before it takes places in the buffers
constexpr int ST_GROUPS = 512;                // group maxima per query, at least (four per wanted candidate where k is large)
constexpr float ST_NEG_INF = -__builtin_huge_valf();

template <int D, bool PROD>
struct StCfg {
    static constexpr int KBLK = D / 64 * (PROD ? 2 : 1);                  // 64-element blocks along K
    static constexpr int A_BUF = KBLK * ST_TILE * 128;
    static constexpr int COLS = PROD ? ST_MAX_COLS_PROD : ST_MAX_COLS;
    static constexpr int B_MAX = KBLK * COLS * 128;
    // an entry for each lane of a warp; 4-bit codes of Prod rows, for each half warp (shared memory is full)
    static constexpr int LUT_MAX = PROD ? 256 * 64 : 256 * 128;
    static constexpr int OFF_B = 0, OFF_A = B_MAX, OFF_LUT = OFF_A + 2 * A_BUF, OFF_THR = OFF_LUT + LUT_MAX, OFF_LOG = OFF_THR + ST_MAX_COLS * 4;
    static constexpr int OFF_BAR = OFF_LOG + ST_EPI * ST_LOG * 12;
    static constexpr int TOTAL = OFF_BAR + 128 + 1024;                    // + slack for the 1024-byte alignment
    static_assert(TOTAL <= 227 * 1024, "shared memory");
};

__device__ __forceinline__ void st_sts32(uint32_t addr, uint32_t a) { asm volatile("st.shared.b32 [%0], %1;" ::"r"(addr), "r"(a) : "memory"); }
__device__ __forceinline__ void st_sts128(uint32_t addr, uint32_t a, uint32_t b, uint32_t c, uint32_t d) {
    asm volatile("st.shared.v4.b32 [%0], {%1, %2, %3, %4};" ::"r"(addr), "r"(a), "r"(b), "r"(c), "r"(d) : "memory");
}
__device__ __forceinline__ float4 st_lds128(uint32_t addr) {
    float4 v;
    asm volatile("ld.shared.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "r"(addr));
    return v;
}
__device__ __forceinline__ void st_arrive(uint32_t bar) { asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(bar) : "memory"); }
__device__ __forceinline__ float st_warp_max(float v) {                  // (NaN is ignored)
    float r;
    asm volatile("redux.sync.max.f32 %0, %1, 0xffffffff;" : "=f"(r) : "f"(v));
    return r;
}
template <int NW>
__device__ __forceinline__ uint32_t st_field(const uint32_t (&w)[NW], int bit, int bits) {
    const int i = bit >> 5, s = bit & 31;
    if (bits == 8) return __byte_perm(w[i], 0, 0x4440u | (uint32_t)(s >> 3));
    uint32_t v = w[i] >> s;
    if (s + bits > 32) v = __funnelshift_r(w[i], w[i + 1 < NW ? i + 1 : i], s);
    return v & ((1u << bits) - 1u);
}

// ---- queries -> B operand images -------------------------------------------------------------------
// One block per column (padded columns are zero).  The scale is the query's own: scores of one query are only compared
// with one another.
__global__ void __launch_bounds__(128) scan_tc_image_kernel(const ScanTcArgs a) {
    __shared__ float red[4], sums[2][4];
    const int col = blockIdx.x, q = col, d = threadIdx.x;
    if (col == 0 && d < 3) a.limits[d] = 0;
    const bool prod = a.signs != nullptr, live = q < a.nq && d < a.dim;
    const float x = live ? a.qrot[(int64_t)q * a.dim + d] : 0.0f, y = live && prod ? a.qsign[(int64_t)q * a.dim + d] : 0.0f;
    float mx = fmaxf(fabsf(x), fabsf(y));
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, o));
    if ((d & 31) == 0) red[d >> 5] = mx;
    __syncthreads();
    const float sc = fp16_scale(fmaxf(fmaxf(red[0], red[1]), fmaxf(red[2], red[3])));
    if (d < a.dim) {
        const int kblk = a.dim / 64, blk = col / a.cols, n = col - blk * a.cols;
        uint8_t* img = a.images + (int64_t)blk * ((prod ? 2 : 1) * kblk * a.cols * 128);
        const uint32_t off = (uint32_t)(d >> 6) * (a.cols * 128) + sw128_offset(n, d & 63);
        *reinterpret_cast<__half*>(img + off) = __float2half_rn(x * sc);
        if (prod) *reinterpret_cast<__half*>(img + kblk * a.cols * 128 + off) = __float2half_rn(y * sc);
    }
    float sx = fabsf(x * sc), sy = fabsf(y * sc);
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) { sx += __shfl_xor_sync(0xffffffffu, sx, o); sy += __shfl_xor_sync(0xffffffffu, sy, o); }
    if ((d & 31) == 0) { sums[0][d >> 5] = sx; sums[1][d >> 5] = sy; }
    __syncthreads();
    if (d == 0 && q < a.nq)
        a.qsum[q] = make_float2((sums[0][0] + sums[0][1]) + (sums[0][2] + sums[0][3]), (sums[1][0] + sums[1][1]) + (sums[1][2] + sums[1][3]));
}

// ---- bound of every query from the sample's group maxima --------------------------------------------
// First the rank-th largest of the threads' own maxima, a lower bound that leaves few values; then the exact rank among those.
__global__ void __launch_bounds__(256) scan_tc_threshold_kernel(const ScanTcArgs a) {
    extern __shared__ float g[];
    __shared__ float top[256], bound, low;
    __shared__ int left, reach;                            // reach: maxima not below the bound
    const int q = blockIdx.x, t = threadIdx.x;
    if (t == 0) { bound = ST_NEG_INF; low = ST_NEG_INF; left = 0; reach = 0; }
    float v = ST_NEG_INF;
    for (int i = t; i < a.groups; i += 256) v = fmaxf(v, a.gmax[(int64_t)q * a.groups + i]);
    top[t] = v;
    __syncthreads();
    int rank = 0;
#pragma unroll 8
    for (int o = 0; o < 256; o++) rank += (top[o] > v || (top[o] == v && o < t)) ? 1 : 0;
    if (rank == a.rank - 1) low = v;                       // (never with more than 256 wanted: then all values are ranked)
    __syncthreads();
    for (int i = t; i < a.groups; i += 256) {
        const float x = a.gmax[(int64_t)q * a.groups + i];
        if (x >= low) g[atomicAdd(&left, 1)] = x;
    }
    __syncthreads();
    const int n = left;
    for (int i = t; i < n; i += 256) {
        const float x = g[i];
        int r = 0;
        for (int o = 0; o < n; o++) r += (g[o] > x || (g[o] == x && o < i)) ? 1 : 0;
        if (r == a.rank - 1) bound = x;                    // (ranks are distinct)
    }
    __syncthreads();
    for (int i = t; i < n; i += 256)
        if (g[i] >= bound) atomicAdd(&reach, 1);
    __syncthreads();
    if (t == 0) {
        // the main launch compares unrounded products with it: a little lower, so that the bound's own row stays (and finite,
        // so that infinite scores are not below it)
        a.thr[q] = fminf(bound, 3.4e38f) - fabsf(fminf(bound, 3.4e38f)) * 2e-6f;
        // The list kernels answer where the sample gave up, gave no bound (rows or queries that are not numbers), or tells that
        // the buffer will overflow: each maximum that reaches the bound stands for a.stride rows at least, and without ties
        // there are a.rank of them.
        a.count[q] = a.limits[2] || bound == ST_NEG_INF || (int64_t)reach * a.stride > a.cap ? a.cap + 1 : 0;
    }
}

// ---- largest norm of the records (proven MSE calls; inside the main launch it cost the calls that need none 5 %) ----
__global__ void __launch_bounds__(256) scan_tc_norms_kernel(const ScanTcArgs a) {
    const int norms = a.rec_bytes - 64;                    // key-only records end with their sixteen norms
    float top = 0.0f;
    for (int64_t i = (int64_t)blockIdx.x * 256 + threadIdx.x; i < a.rows / 4; i += (int64_t)gridDim.x * 256) {
        const float4 v = __ldg(reinterpret_cast<const float4*>(a.records + (i >> 2) * a.rec_bytes + norms) + (i & 3));
        top = fmaxf(fmaxf(top, fmaxf(fabsf(v.x), fabsf(v.y))), fmaxf(fabsf(v.z), fabsf(v.w)));     // (NaN: passed over)
    }
    top = st_warp_max(top);
    if ((threadIdx.x & 31) == 0) atomicMax(a.limits, __float_as_uint(top));
}

// ---- decoders ----------------------------------------------------------------------------------------
// Bit-plane rows: two-bit fields of the planes at the same position (dimensions 2u, 2u + 1 of a byte) concatenated to the
// index of the pair table; X[u] byte m = pair u of byte m.
__device__ __forceinline__ void st_pair_indices(const uint32_t (&w)[4], uint32_t (&X)[4]) {
    const uint32_t e01 = (w[0] & 0x33333333u) | ((w[1] & 0x33333333u) << 2), o01 = ((w[0] >> 2) & 0x33333333u) | (w[1] & 0xccccccccu);
    const uint32_t e23 = (w[2] & 0x33333333u) | ((w[3] & 0x33333333u) << 2), o23 = ((w[2] >> 2) & 0x33333333u) | (w[3] & 0xccccccccu);
    X[3] = (e01 & 0x0f0f0f0fu) | ((e23 & 0x0f0f0f0fu) << 4);
    X[1] = ((e01 >> 4) & 0x0f0f0f0fu) | (e23 & 0xf0f0f0f0u);
    X[2] = (o01 & 0x0f0f0f0fu) | ((o23 & 0x0f0f0f0fu) << 4);
    X[0] = ((o01 >> 4) & 0x0f0f0f0fu) | (o23 & 0xf0f0f0f0u);
}
// fp16 {+-h, +-h} for the sign pair u of byte m (bit set = +); `neg` = {-h, -h}
__device__ __forceinline__ uint32_t st_sign_pair(uint32_t w, int m, int u, uint32_t neg) {
    const int s = 8 * m + 6 - 2 * u;                       // bit s = dimension 2u + 1, bit s + 1 = dimension 2u
    const uint32_t hi = (w << (31 - s)) & 0x80000000u;
    const uint32_t lo = (s + 1 <= 15 ? w << (14 - s) : w >> (s - 14)) & 0x8000u;
    return neg ^ (hi | lo);
}

// ---- the kernel --------------------------------------------------------------------------------------
// grid (CTAs of a query block, query blocks).  SAMPLE: group maxima of every stride-th tile; else candidates of all tiles.
// BITS: of the records' codes; Prod rows take any (0 here).
template <int D, int BITS, bool PROD, bool SAMPLE>
__global__ void __launch_bounds__(ST_THREADS, 1) scan_tc_kernel(const ScanTcArgs a) {
    using C = StCfg<D, PROD>;
    constexpr int KBLK = C::KBLK;
    extern __shared__ uint8_t smem_unaligned[];
    const uint32_t raw = smem_u32(smem_unaligned);
    const uint32_t base = (raw + 1023u) & ~1023u;
    uint8_t* const sm = smem_unaligned + (base - raw);
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int q0 = blockIdx.y * a.cols;
    const int64_t ntiles = (a.rows + ST_TILE - 1) / ST_TILE;
    // (a block of queries that all go to the list kernels has nothing to gather)
    if (!SAMPLE && !__syncthreads_or(threadIdx.x < a.cols && q0 + (int)threadIdx.x < a.nq && a.count[q0 + threadIdx.x] <= a.cap)) return;
    const int64_t nwork = SAMPLE ? (ntiles + a.stride - 1) / a.stride : ntiles;
    auto tile_of = [&](int64_t u) { return SAMPLE ? u * a.stride : u; };

    const uint32_t bar0 = base + C::OFF_BAR;
    auto a_ready = [&](int b) { return bar0 + 8 * b; };
    auto a_free = [&](int b) { return bar0 + 8 * (2 + b); };
    auto acc_full = [&](int b) { return bar0 + 8 * (4 + b); };
    auto acc_free = [&](int b) { return bar0 + 8 * (6 + b); };
    const uint32_t b_full = bar0 + 64, tmem_slot = bar0 + 72;
    if (threadIdx.x == 0) {
        for (int b = 0; b < 2; b++) { mbar_init(a_ready(b), ST_DEC); mbar_init(a_free(b), 1); mbar_init(acc_full(b), 1); mbar_init(acc_free(b), ST_EPI); }
        mbar_init(b_full, 1);
    }
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    if (warp == ST_DEC + ST_EPI) tmem_alloc(tmem_slot, 512);
    // table of code pairs, an entry for each lane
    const int bits = PROD ? a.bits : BITS;
    float mxc = 0.0f;
    for (int i = 0; i < (1 << bits); i++) mxc = fmaxf(mxc, fabsf(__ldg(a.cent + i)));
    const float csc = fp16_scale(mxc);
    const int sh = PROD && bits == 4 ? 6 : 7;              // bytes of an entry's copies (power of two)
    for (int e = threadIdx.x; e < (1 << (2 * bits + sh - 2)); e += ST_THREADS) {
        const int x = e >> (sh - 2);
        int c0, c1;
        if (PROD) {                                        // plane by plane: bit 2p + 1 = first dimension, 2p = second
            c0 = c1 = 0;
            for (int p = 0; p < bits; p++) { c0 |= ((x >> (2 * p + 1)) & 1) << p; c1 |= ((x >> (2 * p)) & 1) << p; }
        } else {
            c0 = x & ((1 << bits) - 1); c1 = x >> bits;
        }
        *reinterpret_cast<uint32_t*>(sm + C::OFF_LUT + 4 * e) = pack_half2(__ldg(a.cent + c0) * csc, __ldg(a.cent + c1) * csc);
    }
    float* const thr_s = reinterpret_cast<float*>(sm + C::OFF_THR);
    if (!SAMPLE)
        for (int c = threadIdx.x; c < ST_MAX_COLS; c += ST_THREADS) thr_s[c] = c < a.cols && q0 + c < a.nq && a.count[q0 + c] <= a.cap ? a.thr[q0 + c] : -ST_NEG_INF;
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = lds32v(tmem_slot);
    bool ok = true;

    if (warp < ST_DEC) {
        // ================= decode =================
        const uint32_t tab = base + C::OFF_LUT + (lane & ((1 << (sh - 2)) - 1)) * 4;
        constexpr int NW = PROD ? 1 : D * BITS / 64;       // a lane's words of a record
        constexpr int HW = D / 64;                         // plane words of half a row
        const int half = lane >> 4, trow = warp * 16 + (lane & 15), bpp = D / 8;
        uint32_t w[PROD ? 1 : NW], wn[PROD ? 1 : NW], pw[HW][4], pn[HW][4], sg[HW], sn[HW];
        float res = 0.0f, resn = 0.0f, top_sign = 0.0f;    // (top_sign: largest magnitude of the sign operand)
        auto request = [&](int64_t tile) {
            if constexpr (PROD) {
                const int64_t r = tile * ST_TILE + trow;
                const bool have = r < a.rows;
                const uint8_t* row = a.packed + r * (int64_t)(bits * bpp);
#pragma unroll
                for (int i = 0; i < HW; i++) {
#pragma unroll
                    for (int p = 0; p < 4; p++) pn[i][p] = have && p < bits ? __ldg(reinterpret_cast<const uint32_t*>(row + p * bpp) + half * HW + i) : 0u;
                    sn[i] = have ? __ldg(reinterpret_cast<const uint32_t*>(a.signs + r * bpp) + half * HW + i) : 0u;
                }
                resn = have ? __ldg(a.res_norms + r) : 0.0f;
            } else {
                const int64_t rec = tile * (ST_TILE / 16) + warp;
                const bool have = rec * 16 < a.rows;
                const uint8_t* rp = a.records + rec * a.rec_bytes;
#pragma unroll
                for (int i = 0; i < NW; i++) {
                    const int off = NW == 8 ? (i >> 2) * 512 + lane * 16 + (i & 3) * 4 : lane * (NW * 4) + i * 4;      // (tl_key_piece_offset)
                    wn[i] = have ? __ldg(reinterpret_cast<const uint32_t*>(rp + off)) : 0u;
                }
            }
        };
        if ((int64_t)blockIdx.x < nwork) request(tile_of(blockIdx.x));
        uint32_t it = 0;
        for (int64_t u = blockIdx.x; u < nwork; u += gridDim.x, it++) {
            const int b = it & 1;
            if constexpr (PROD) {
#pragma unroll
                for (int i = 0; i < HW; i++) {
#pragma unroll
                    for (int p = 0; p < 4; p++) pw[i][p] = pn[i][p];
                    sg[i] = sn[i];
                }
                res = resn;
            } else {
#pragma unroll
                for (int i = 0; i < NW; i++) w[i] = wn[i];
            }
            if (u + gridDim.x < nwork) request(tile_of(u + gridDim.x));
            if (it >= 2) ok = mbar_wait(a_free(b), ((it >> 1) - 1) & 1);
            if (!__all_sync(0xffffffffu, ok)) { ok = false; break; }
            const uint32_t at = base + C::OFF_A + b * C::A_BUF;
            if constexpr (PROD) {
                const float mag = a.sign_coef * res * csc;
                if (!SAMPLE) top_sign = fmaxf(top_sign, fabsf(mag) > 60000.0f ? -ST_NEG_INF : fabsf(mag));  // (beyond fp16: no bound; NaN: no score)
                const uint32_t h = __half_as_ushort(__float2half_rn(mag > 60000.0f ? 60000.0f : mag)), neg = (h | (h << 16)) ^ 0x80008000u;
#pragma unroll
                for (int i = 0; i < HW; i++) {
                    uint32_t X[4];
                    st_pair_indices(pw[i], X);
#pragma unroll
                    for (int m = 0; m < 4; m++) {
                        uint32_t v[4];
#pragma unroll
                        for (int x = 0; x < 4; x++) v[x] = lds32(tab + (((X[x] >> (8 * m)) & 0xffu) << sh));
                        const int k = 32 * (half * HW + i) + 8 * m;
                        const uint32_t off = (uint32_t)(k >> 6) * (ST_TILE * 128) + sw128_offset(trow, k & 63);
                        st_sts128(at + off, v[0], v[1], v[2], v[3]);
                        st_sts128(at + (D / 64) * (ST_TILE * 128) + off, st_sign_pair(sg[i], m, 0, neg), st_sign_pair(sg[i], m, 1, neg),
                                  st_sign_pair(sg[i], m, 2, neg), st_sign_pair(sg[i], m, 3, neg));
                    }
                }
            } else {
                const int g = lane >> 2, t = lane & 3;
                const uint32_t lane_at = at + (16 * warp + g) * 128 + (g << 4) + 4 * t;
#pragma unroll
                for (int e = 0; e < D / 8; e++)
#pragma unroll
                    for (int second = 0; second < 2; second++) {
                        const uint32_t f = st_field(w, tl_key_field_bit(D, BITS, e >> 1, e & 1, second), 2 * BITS);
                        st_sts32((lane_at ^ ((uint32_t)(e & 7) << 4)) + (e >> 3) * (ST_TILE * 128) + second * 1024, lds32(tab + (f << 7)));
                    }
            }
            asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
            __syncwarp();
            if (lane == 0) st_arrive(a_ready(b));
        }
        if (PROD && !SAMPLE) {
            top_sign = st_warp_max(top_sign);
            if (lane == 0) atomicMax(a.limits + 1, __float_as_uint(top_sign));
        }
    } else if (warp < ST_DEC + ST_EPI) {
        // ================= epilogue: thread = row, half of the columns =================
        const int ew = warp & 3, half = (warp - ST_DEC) >> 2, row = ew * 32 + lane;
        const int hc = a.cols / 2, col0 = half * hc;       // (cols: a multiple of 32)
        const uint32_t thr_at = base + C::OFF_THR + col0 * 4;
        uint32_t it = 0;
        float mine[4] = {ST_NEG_INF, ST_NEG_INF, ST_NEG_INF, ST_NEG_INF};       // SAMPLE: group maxima of columns 32 i + lane
        float top_norm = 0.0f;                             // Prod: largest |norm| of the thread's rows
        int flush = 0;
        auto put_group = [&]() {
#pragma unroll
            for (int i = 0; i < 4; i++) {
                const int q = q0 + col0 + 32 * i + lane;
                if (32 * i + lane < hc && q < a.nq) a.gmax[(int64_t)q * a.groups + ((int)blockIdx.x * 4 + ew) * a.flushes + flush] = mine[i];
                mine[i] = ST_NEG_INF;
            }
            flush++;
        };
        // Candidates go through a log of the warp's own: a place in a query's buffer is an atomic's round trip, which up to 96
        // candidates pay together.  (With the rolled loop below: 1,000 queries over 4 M rows 2,136 -> 1,494 us.)
        uint32_t* const log = reinterpret_cast<uint32_t*>(sm + C::OFF_LOG) + (warp - ST_DEC) * (ST_LOG * 3);
        int logged = 0;
        auto take_places = [&]() {
            __syncwarp();
            for (int e = lane; e < logged; e += 32) {
                const int q = (int)log[3 * e], at = atomicAdd(a.count + q, 1);
                if (at < a.cap) {
                    a.buf_s[(int64_t)q * a.cap + at] = __uint_as_float(log[3 * e + 1]);
                    a.buf_i[(int64_t)q * a.cap + at] = (int)log[3 * e + 2];
                } else {
                    thr_s[q - q0] = -ST_NEG_INF;           // overflowed: no more of this query's rows
                }
            }
            __syncwarp();
            logged = 0;
        };
        for (int64_t u = blockIdx.x; u < nwork; u += gridDim.x, it++) {
            const int b = it & 1;
            const int64_t r = tile_of(u) * ST_TILE + row;
            float nrm = __int_as_float(0x7fffffff);        // (a row that is not there: NaN never wins a comparison)
            if (r < a.rows)
                nrm = PROD ? __ldg(a.norms + r)
                           : __ldg(reinterpret_cast<const float*>(a.records + (r >> 4) * a.rec_bytes + tl_key_section(D, BITS ? BITS : 4) + tl_norm_offset(0, 0, (int)(r & 15))));
            if (PROD && !SAMPLE) top_norm = fmaxf(top_norm, fabsf(nrm));   // (NaN: passed over)
            ok = mbar_wait(acc_full(b), (it >> 1) & 1);
            if (!__all_sync(0xffffffffu, ok)) { ok = false; break; }
            tc_fence_after();
            const uint32_t src = tmem + ((uint32_t)(ew * 32) << 16) + b * 256 + col0;
            if constexpr (SAMPLE) {
#pragma unroll
                for (int i = 0; i < 4; i++)
                    if (32 * i < hc)
#pragma unroll 1
                        for (int c = 0; c < 32 && 32 * i + c < hc; c += 8) {
                            uint32_t v[8];
                            tmem_ld8(src + 32 * i + c, v);
#pragma unroll
                            for (int e = 0; e < 8; e++) {
                                const float m = st_warp_max(__uint_as_float(v[e]) * nrm);
                                if (lane == c + e) mine[i] = fmaxf(mine[i], m);
                            }
                        }
            } else {
// sixteen columns a turn, the next sixteen in flight (hc: a multiple of 16)
                auto columns = [&](const uint32_t (&v)[16], int c) {
                    float d[4] = {ST_NEG_INF, ST_NEG_INF, ST_NEG_INF, ST_NEG_INF}, th[16];
#pragma unroll
                    for (int i = 0; i < 16; i += 4) {
                        const float4 t4 = st_lds128(thr_at + 4 * (c + i));
                        th[i] = t4.x; th[i + 1] = t4.y; th[i + 2] = t4.z; th[i + 3] = t4.w;
                    }
#pragma unroll
                    for (int i = 0; i < 16; i++) d[i & 3] = fmaxf(d[i & 3], fmaf(__uint_as_float(v[i]), nrm, -th[i]));
                    if (!__any_sync(0xffffffffu, fmaxf(fmaxf(d[0], d[1]), fmaxf(d[2], d[3])) >= 0.0f)) return;
                    uint32_t in = 0;                       // columns this row is a candidate of
#pragma unroll
                    for (int i = 0; i < 16; i++) in |= fmaf(__uint_as_float(v[i]), nrm, -th[i]) >= 0.0f ? 1u << i : 0u;
                    // (rare per warp but not per tile, and four roles share the instruction cache: a short rolled loop -- sixteen
                    // unrolled columns cost 1,000 clocks a visit)
#pragma unroll 1
                    for (uint32_t mask; (mask = __ballot_sync(0xffffffffu, in != 0)) != 0;) {
                        if (in) {
                            const int i = __ffs(in) - 1;
                            uint32_t x = v[0];
#pragma unroll
                            for (int k = 1; k < 16; k++) x = i == k ? v[k] : x;
                            uint32_t* const e = log + 3 * (logged + __popc(mask & ((1u << lane) - 1u)));
                            e[0] = (uint32_t)(q0 + col0 + c + i); e[1] = __float_as_uint(__uint_as_float(x) * nrm); e[2] = (uint32_t)r;
                            in &= in - 1;
                        }
                        logged += __popc(mask);
                        if (logged > ST_LOG - 32) take_places();
                    }
                };
                uint32_t va[16], vb[16];
                tmem_ld16_async(src, va);
#pragma unroll 1
                for (int c = 0; c < hc; c += 32) {
                    tmem_wait16(va);
                    if (c + 16 < hc) tmem_ld16_async(src + c + 16, vb);
                    columns(va, c);
                    if (c + 16 >= hc) break;
                    tmem_wait16(vb);
                    if (c + 32 < hc) tmem_ld16_async(src + c + 32, va);
                    columns(vb, c + 16);
                }
            }
            tc_fence_before();
            __syncwarp();
            if (lane == 0) st_arrive(acc_free(b));
            if (SAMPLE && (it + 1) % a.tiles_per_flush == 0) put_group();
        }
        if (SAMPLE) {
            while (flush < a.flushes) put_group();         // (what is left, then groups without rows)
        } else {
            take_places();
            if (PROD && half == 0) {                       // (every block sees every row)
                top_norm = st_warp_max(top_norm);
                if (lane == 0) atomicMax(a.limits, __float_as_uint(top_norm));
            }
        }
    } else if (lane == 0) {
        // ================= MMA issuer (one lane) =================
        const uint32_t bbytes = (uint32_t)(KBLK * a.cols * 128);
        mbar_expect_tx(b_full, bbytes);
        bulk_g2s(base + C::OFF_B, a.images + (int64_t)blockIdx.y * bbytes, bbytes, b_full);
        ok = mbar_wait(b_full, 0);
        const uint32_t idesc = (1u << 4) | ((uint32_t)(a.cols >> 3) << 17) | ((uint32_t)(ST_TILE >> 4) << 24);      // fp16 x fp16 -> f32
        uint32_t it = 0;
        for (int64_t u = blockIdx.x; ok && u < nwork; u += gridDim.x, it++) {
            const int b = it & 1;
            ok = mbar_wait(a_ready(b), (it >> 1) & 1);
            if (ok && it >= 2) ok = mbar_wait(acc_free(b), ((it >> 1) - 1) & 1);
            if (!ok) break;
            tc_fence_after();
            uint32_t acc = 0;
#pragma unroll
            for (int kb = 0; kb < KBLK; kb++) {
                const uint64_t ad = umma_desc(base + C::OFF_A + b * C::A_BUF + kb * (ST_TILE * 128)), bd = umma_desc(base + C::OFF_B + kb * (a.cols * 128));
#pragma unroll
                for (int k = 0; k < 4; k++) { umma_f16(tmem + b * 256, ad + 2 * k, bd + 2 * k, idesc, acc); acc = 1; }
            }
            umma_commit(a_free(b));
            umma_commit(acc_full(b));
        }
        // (an unfinished copy must not outlive the block: the wait above is bounded, and so is this one)
        if (!ok) mbar_wait(b_full, 0);
    }
    if (!ok && lane == 0) {
        atomicExch(a.error, 1);
        if (SAMPLE) atomicExch(a.limits + 2, 1u);
        else
            for (int q = q0; q < min(a.nq, q0 + a.cols); q++) atomicMax(a.count + q, a.cap + 1);      // the list kernels answer
    }
    __syncwarp();
    tc_fence_before();
    __syncthreads();
    if (warp == ST_DEC + ST_EPI) {
        tc_fence_after();
        tmem_dealloc(tmem, 512);
    }
}

static size_t st_align(size_t v) { return (v + 255) / 256 * 256; }

// Group maxima of a query at most, as scan_tc_run deals them.
static int st_groups(int ksel, int gx) { return std::max(ST_GROUPS, 4 * ksel) + 4 * gx; }

ScanTcPlan scan_tc_plan(int nq, int dim, bool prod, int ksel) {
    ScanTcPlan pl{};
    if (!prod && nq < SCAN_TC_MIN_QUERIES) return pl;
    const int most = prod ? ST_MAX_COLS_PROD : ST_MAX_COLS;
    pl.blocks = (int)ceil_div(nq, most);
    pl.cols = (int)ceil_div(ceil_div(nq, pl.blocks), 32) * 32;
    pl.blocks = (int)ceil_div(nq, pl.cols);
    pl.gx = std::max(1, sm_count() / pl.blocks);
    // about ksel * stride candidates are expected: room for six times as many
    pl.cap = 1024;
    while (pl.cap < 6 * ksel * ST_MAX_STRIDE) pl.cap *= 2;
    size_t off = 0;
    pl.off_images = off; off = st_align(off + (size_t)pl.blocks * pl.cols * dim * 2 * (prod ? 2 : 1));
    pl.off_gmax = off;   off = st_align(off + (size_t)nq * st_groups(ksel, pl.gx) * 4);
    pl.off_thr = off;    off = st_align(off + (size_t)nq * 4);
    pl.off_count = off;  off = st_align(off + (size_t)nq * 4);
    pl.off_limits = off; off = st_align(off + 3 * 4);
    pl.off_qsum = off;   off = st_align(off + (size_t)nq * sizeof(float2));
    pl.off_s = off;      off = st_align(off + (size_t)nq * pl.cap * 4);
    pl.off_i = off;      off = st_align(off + (size_t)nq * pl.cap * 4);
    pl.total = off;
    return pl;
}

// Sample stride: a sampled tile (four groups of rows) per wanted candidate, no more than ST_MAX_STRIDE apart; small indexes
// are sampled whole.
static int st_stride(int64_t rows, int ksel) { return (int)std::max<int64_t>(1, std::min<int64_t>(ST_MAX_STRIDE, rows / ST_TILE / ksel)); }

bool scan_tc_wanted(int nq, int64_t rows, int dim, int bits, bool prod, int ksel, bool proven) {
    if ((dim != 64 && dim != 128) || bits < (prod ? 1 : 2) || bits > 4) return false;
    // Two groups of rows per wanted candidate at least.  From nine queries (two passes of the list kernels) on: 9 queries over
    // 2,300, 5,000 and 20,000 x d128 rows 127, 111 and 133 us there, 65 here.  Five to eight (one pass) are left to the list
    // kernels although 8 queries over 1 M rows take 207 us there and 16 take 124 here.  Prod rows: the list kernel scores a row a
    // lane; one query over 2,176 rows 74 us there, 66 here, over 30,000 360 and 67.
    if (4 * (rows / ST_TILE) < 2 * ksel) return false;
    // (a proof wants room below the k-th best score: twice the groups where k is large against the margin)
    if (proven && ksel > 64 && 4 * (rows / ST_TILE) < 4 * ksel) return false;
    return prod || nq >= SCAN_TC_MIN_QUERIES;
}

template <int D, int BITS, bool PROD>
static int st_launch(const ScanTcArgs& a, cudaStream_t st) {
    using C = StCfg<D, PROD>;
    const int64_t tiles = ceil_div(a.rows, ST_TILE);
    const dim3 grid(a.gx, a.blocks), grid_main((unsigned)std::min<int64_t>(std::max(1, sm_count() / a.blocks), tiles), a.blocks);
    auto sample = scan_tc_kernel<D, BITS, PROD, true>;
    auto main_pass = scan_tc_kernel<D, BITS, PROD, false>;
    TQB_CUDA(cudaFuncSetAttribute(sample, cudaFuncAttributeMaxDynamicSharedMemorySize, C::TOTAL));
    TQB_CUDA(cudaFuncSetAttribute(main_pass, cudaFuncAttributeMaxDynamicSharedMemorySize, C::TOTAL));
    sample<<<grid, ST_THREADS, C::TOTAL, st>>>(a);
    if (int e = check_launch("scan_tc_sample")) return e;
    scan_tc_threshold_kernel<<<a.nq, 256, a.groups * sizeof(float), st>>>(a);
    if (int e = check_launch("scan_tc_threshold")) return e;
    if (!PROD && a.proven) {
        scan_tc_norms_kernel<<<(unsigned)std::min<int64_t>(8 * sm_count(), ceil_div(a.rows, 1024)), 256, 0, st>>>(a);
        if (int e = check_launch("scan_tc_norms")) return e;
    }
    main_pass<<<grid_main, ST_THREADS, C::TOTAL, st>>>(a);
    return check_launch("scan_tc");
}

int scan_tc_run(ScanTcArgs a, const ScanTcPlan& pl, uint8_t* ws, cudaStream_t st) {
    a.images = ws + pl.off_images; a.gmax = reinterpret_cast<float*>(ws + pl.off_gmax); a.thr = reinterpret_cast<float*>(ws + pl.off_thr);
    a.count = reinterpret_cast<int*>(ws + pl.off_count); a.buf_s = reinterpret_cast<float*>(ws + pl.off_s);
    a.buf_i = reinterpret_cast<int*>(ws + pl.off_i);
    a.limits = reinterpret_cast<uint32_t*>(ws + pl.off_limits); a.qsum = reinterpret_cast<float2*>(ws + pl.off_qsum);
    a.cap = pl.cap; a.cols = pl.cols; a.blocks = pl.blocks;
    a.stride = st_stride(a.rows, a.ksel);
    const int64_t sampled = ceil_div(ceil_div(a.rows, ST_TILE), a.stride);
    a.gx = (int)std::min<int64_t>(pl.gx, sampled);
    const int64_t per_cta = ceil_div(sampled, a.gx);       // sampled tiles of a CTA
    // four groups per CTA and flush: enough of them, no more than the buffer holds
    int64_t want = ceil_div(std::max(ST_GROUPS, 4 * a.ksel), 4 * a.gx);
    want = std::min<int64_t>(want, per_cta);
    a.tiles_per_flush = (int)ceil_div(per_cta, want);
    a.flushes = (int)ceil_div(per_cta, a.tiles_per_flush);
    a.groups = 4 * a.gx * a.flushes;
    // The bound's rank among the sample's maxima: small indexes, sampled densely, take it lower (the buffer expects the
    // candidates of a stride of 16), so that a selection finds room below the k-th best score.
    a.rank = a.proven ? std::max(a.ksel, std::min(a.groups / 2, a.ksel * std::max(1, 4 / a.stride))) : a.ksel;
    if (int e = tc_error_word(&a.error)) return e;
    scan_tc_image_kernel<<<a.cols * a.blocks, 128, 0, st>>>(a);
    if (int e = check_launch("scan_tc_image")) return e;
    if (a.signs) return a.dim == 64 ? st_launch<64, 0, true>(a, st) : st_launch<128, 0, true>(a, st);
#define TQB_CASE(d, b) if (a.dim == d && a.bits == b) return st_launch<d, b, false>(a, st);
    TQB_CASE(64, 2) TQB_CASE(64, 3) TQB_CASE(64, 4) TQB_CASE(128, 2) TQB_CASE(128, 3) TQB_CASE(128, 4)
#undef TQB_CASE
    return fail(TQB_ERR_UNSUPPORTED, "scan: unsupported shape");
}

}  // namespace tqb
