// dequantize_tc.cu -- the inverse of Algorithm 1 / 2 on the 5th-generation tensor cores:
//
//   x~ = norm * ( c[codes] @ R  [ + sqrt(pi/2)/d * ||r|| * (signs @ S) ] )      (reference.py:320-367, :472-533)
//
// for upstream bit-plane rows and for the 16-token records of the KV store (tiled_layout.cuh) alike; the records
// are read where they lie, into the caller's dense (unit, token, dim) tensors.
//
// Arithmetic: float32.  Centroids, rotation and QJL matrix enter the MMAs as two fp16 terms each, hi = fp16(v) and
// lo = fp16(v - hi), after scaling by a power of two that keeps the low terms out of the subnormal range: 22 bits
// against float32's 24.  The three products that matter (lo hi, hi lo, then hi hi) are accumulated in float32; the
// signs are exact in one term.  The accumulator is rounded toward zero after every MMA, a loss in proportion to the
// partial sum there, which the matrices' low terms give back (DQ_LOSS).  Relative error against 64-bit sums of
// codes of normal rows, dims 32 to 128, 1 to 4 bits: 0.6 to 1.6e-7 (records with outlier channels among them), the float32
// FMA chain of dequantize.cu 1.0 to 2.1e-7; without what DQ_LOSS gives back 0.9 to 2.9e-7.
//
// What bounds it: the shared-memory pipe.  A 128-row tile of d = 128 writes 64 KB of float32 (2,900 clocks of HBM at 22
// bytes per clock and SM); it takes 24 MMAs that read 8 KB of operands each (1,536 clocks), 256 table loads and 64 KB of
// operand stores (about 1,900 wavefronts) and the output's shuffles and stores (1,500): 5,000 clocks, measured 3.0 us.
// Three groups of warps of one persistent CTA per SM keep them overlapped, two buffers of operands and of accumulators
// apart.  Measured (d = 128, 4 bits, float32): 75,776 rows 163 us on the FFMA kernel, 22.7 us here; 909,312 rows 155 us =
// 3.4 TB/s of rows; Prod rows (2 bits + sign) 4.0 -> 0.25 ms per million.  A call costs 8 (d = 64) to 12 us (d = 128)
// before the first tile is out, most of it the B operand, against 10 us of the FFMA kernel, hence its threshold of rows.
//   warps 0-7   decode: codes -> fp16 pairs through a table of code PAIRS (one 8-byte load gives the hi and lo terms of
//               two centroids), written as the K-major, 128-byte-swizzled A operand
//   warps 8-15  epilogue: tcgen05.ld, times the norm, 32-byte stores (thread = row)
//   warp 16     issues the MMAs (one lane)
// The B operand -- the transposed matrix in two fp16 terms -- is built once per CTA.  Every wait is bounded in time.
#include "common.cuh"
#include "pipe.cuh"
#include "tc.cuh"
#include "tiled_layout.cuh"

namespace tqb {

constexpr int DQ_TILE = 128;                 // rows per tile = TMEM lanes
constexpr int DQ_DEC = 8, DQ_EPI = 8;        // decoder and epilogue warps
constexpr int DQ_THREADS = (DQ_DEC + DQ_EPI + 1) * 32;
// Mean loss of a truncation to 24 bits, relative to the number: half a unit of the last place, which is 2^-23 to 2^-24 of it
// (0.36 2^-23 where all leading digits are as frequent as in products; measured 0.32).  A product added in step s of the
// leading product's n is in n - s truncated sums, so its matrix element is scaled by 1 + DQ_LOSS (n - s).
constexpr float DQ_LOSS = 0.32f * 1.1920929e-7f;

struct DqSide {                              // one operand set: rows, or the keys or values of a record store
    const uint8_t* src;                      // packed rows, or the record store
    const float* norms;                      // rows only (records carry their norms)
    const float* rot; const float* cent;
    void* out;
    int bits;
    int values;                              // records: 0 = keys, 1 = values
};
struct DqArgs {
    DqSide side[2];                          // by blockIdx.y
    const uint8_t* signs; const float* res_norms; const float* qjl; float qjl_scale;    // Prod rows
    int64_t n;                               // rows, or records
    int dim;                                 // <= DP; columns beyond it are padding (zero in B)
    int out_dtype;
    // records: unit u starts at record u * unit_records, its first `tokens` tokens go to rows u * out_pitch + token
    int kb, vb, rec_bytes;
    int64_t unit_records, unit_used;         // records per unit in the store, and those that hold tokens < `tokens`
    int64_t tokens, out_pitch;
    int* error;
};

// ---- configuration ---------------------------------------------------------------------------------
template <int DP, bool PROD>
struct DqCfg {
    static constexpr int KBLK = DP / 64;
    static constexpr int B_TERM = DP * DP * 2, A_TERM = DQ_TILE * DP * 2;
    static constexpr int NB = PROD ? 4 : 2;                         // B terms: R hi, R lo (, S hi, S lo)
    static constexpr int ABUF = PROD && DP == 128 ? 1 : 2;          // operand buffers (shared memory has room for one)
    static constexpr int A_SET = 2 * A_TERM + (PROD ? A_TERM : 0);  // hi, lo (, signs)
    // Pair table: entries of 8 bytes {hi pair, lo pair}, REPL copies side by side so that the lanes of a warp spread
    // over the banks.  Prod rows of 128 leave room for 512 bytes: 2^(2 bits) entries x 4 or fewer copies.
    static constexpr int LUT = PROD && DP == 128 ? 512 : 16384;
    static constexpr int OFF_B = 0, OFF_A = NB * B_TERM, OFF_LUT = OFF_A + ABUF * A_SET, OFF_BAR = OFF_LUT + LUT;
    static constexpr int TOTAL = OFF_BAR + 256 + 1024;              // + slack for the 1024-byte alignment
    static constexpr int ACC_COLS = PROD ? 2 * DP : DP;             // accumulator columns of one buffer
    static constexpr int TMEM_COLS = 2 * ACC_COLS;
    static_assert(TOTAL <= 227 * 1024, "shared memory");
    static_assert(TMEM_COLS <= 512, "tensor memory");
};

__device__ __forceinline__ void st_global32(void* p, const uint32_t* v) {   // 32 bytes, 32-byte aligned
    asm volatile("st.global.v8.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8};"
                 ::"l"(p), "r"(v[0]), "r"(v[1]), "r"(v[2]), "r"(v[3]), "r"(v[4]), "r"(v[5]), "r"(v[6]), "r"(v[7]) : "memory");
}
__device__ __forceinline__ void sts128(uint32_t addr, uint32_t a, uint32_t b, uint32_t c, uint32_t d) {
    asm volatile("st.shared.v4.b32 [%0], {%1, %2, %3, %4};" ::"r"(addr), "r"(a), "r"(b), "r"(c), "r"(d) : "memory");
}
__device__ __forceinline__ void sts32(uint32_t addr, uint32_t a) {
    asm volatile("st.shared.b32 [%0], %1;" ::"r"(addr), "r"(a) : "memory");
}
__device__ __forceinline__ void arrive(uint32_t bar) {
    asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(bar) : "memory");
}
// Lane q of every four holds one row as four 32-byte pieces; afterwards piece i of lane q is piece q of lane i's row, so
// that the four lanes store 128 contiguous bytes of row i together.  (With a row per lane, a 32-byte store costs two
// wavefronts a lane: 4,300 clocks of a 128 x 128 float32 tile's 7,000; this way 1,500, shuffles included.)
__device__ __forceinline__ void transpose4(uint32_t (&v)[32], int lane) {
#pragma unroll
    for (int bit = 1; bit <= 2; bit <<= 1) {
        const bool up = lane & bit;
#pragma unroll
        for (int s = 0; s < 4; s++) {
            if (s & bit) continue;
#pragma unroll
            for (int i = 0; i < 8; i++) {
                const uint32_t give = up ? v[8 * s + i] : v[8 * (s + bit) + i];
                const uint32_t take = __shfl_xor_sync(0xffffffffu, give, bit);
                if (up) v[8 * s + i] = take;
                else v[8 * (s + bit) + i] = take;
            }
        }
    }
}
// v (1 + more) -> {hi, lo} fp16 terms
__device__ __forceinline__ void split_half(float v, uint32_t& hi, uint32_t& lo, float more = 0.0f) {
    const __half h = __float2half_rn(v);
    const __half l = __float2half_rn(fmaf(v, more, v - __half2float(h)));
    hi = __half_as_ushort(h); lo = __half_as_ushort(l);
}
// B operand of one matrix M (dim x dim, row j = contraction index): B[n][k = j] = M[j][n], K-major with 128-byte
// swizzle, hi and lo terms, scaled by 1 + gain.  All threads of the CTA; returns the scale.  red: 32 floats of scratch.
template <int DP>
__device__ __forceinline__ float build_b(uint8_t* sm, int off_hi, int off_lo, const float* __restrict__ M, int dim, float gain, float* red) {
    constexpr int BLOCKS = (DP / 2) * (DP / 4);            // 2 rows x 4 columns each
    constexpr int PER = (BLOCKS + DQ_THREADS - 1) / DQ_THREADS;
    float4 r0[PER], r1[PER];
    float mx = 0.0f;
    // A warp takes 8 rows x 32 columns: its reads are 128-byte lines, and its stores (rotated so that the eight lanes of
    // a column group write eight different swizzle rows) touch every bank once.
    auto place = [](int b, int& j, int& n) {
        const int l = b & 31, blk = b >> 5;
        j = 8 * (blk / (DP / 32)) + 2 * (l & 3);
        n = 32 * (blk % (DP / 32)) + 4 * (l >> 2);
    };
#pragma unroll
    for (int i = 0; i < PER; i++) {
        const int b = threadIdx.x + i * DQ_THREADS;
        int j, n;
        place(b, j, n);
        const bool ok = b < BLOCKS && j < dim && n < dim;  // (dim is a multiple of 8)
        const float4 z = make_float4(0.f, 0.f, 0.f, 0.f);
        r0[i] = ok ? __ldg(reinterpret_cast<const float4*>(M + (int64_t)j * dim + n)) : z;
        r1[i] = ok ? __ldg(reinterpret_cast<const float4*>(M + (int64_t)(j + 1) * dim + n)) : z;
    }
#pragma unroll
    for (int i = 0; i < PER; i++)
        mx = fmaxf(fmaxf(fmaxf(fmaxf(mx, fabsf(r0[i].x)), fmaxf(fabsf(r0[i].y), fabsf(r0[i].z))), fmaxf(fabsf(r0[i].w), fabsf(r1[i].x))),
                   fmaxf(fmaxf(fabsf(r1[i].y), fabsf(r1[i].z)), fabsf(r1[i].w)));
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, o));
    if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = mx;
    __syncthreads();
    mx = 0.0f;
    for (int w = 0; w < DQ_THREADS / 32; w++) mx = fmaxf(mx, red[w]);
    __syncthreads();                                       // (red may be written again)
    const float sc = fp16_scale(mx);
#pragma unroll
    for (int i = 0; i < PER; i++) {
        const int b = threadIdx.x + i * DQ_THREADS;
        if (b >= BLOCKS) continue;
        int j, n;
        place(b, j, n);
        const float more = fmaf(DQ_LOSS, (float)((dim + 15) / 16 - (j >> 4)), gain);      // (j and j + 1 are in one step of 16)
        const int turn = (b >> 3) & 3;                     // rotation of the four columns, by column group
#pragma unroll
        for (int cc = 0; cc < 4; cc++) {
            const int c = (cc + turn) & 3;
            const float v0 = c & 2 ? (c & 1 ? r0[i].w : r0[i].z) : (c & 1 ? r0[i].y : r0[i].x);
            const float v1 = c & 2 ? (c & 1 ? r1[i].w : r1[i].z) : (c & 1 ? r1[i].y : r1[i].x);
            uint32_t h0, l0, h1, l1;
            split_half(v0 * sc, h0, l0, more);
            split_half(v1 * sc, h1, l1, more);
            const uint32_t off = (uint32_t)(j >> 6) * (DP * 128) + sw128_offset(n + c, j & 63);
            *reinterpret_cast<uint32_t*>(sm + off_hi + off) = h0 | (h1 << 16);
            *reinterpret_cast<uint32_t*>(sm + off_lo + off) = l0 | (l1 << 16);
        }
    }
    return sc;
}

// ---- decoders --------------------------------------------------------------------------------------
// Bit-plane rows.  Thread = half a row; word i holds the planes of 32 dimensions.  Two-bit fields of the planes at the
// same position (dimensions 2u, 2u+1 of a byte) are concatenated to the index of the pair table: two rounds of masked
// merges turn four plane words into four words of index bytes, X[u] byte m = pair u of byte m.
__device__ __forceinline__ void pair_indices(const uint32_t (&w)[4], uint32_t (&X)[4]) {
    const uint32_t e01 = (w[0] & 0x33333333u) | ((w[1] & 0x33333333u) << 2), o01 = ((w[0] >> 2) & 0x33333333u) | (w[1] & 0xccccccccu);
    const uint32_t e23 = (w[2] & 0x33333333u) | ((w[3] & 0x33333333u) << 2), o23 = ((w[2] >> 2) & 0x33333333u) | (w[3] & 0xccccccccu);
    X[3] = (e01 & 0x0f0f0f0fu) | ((e23 & 0x0f0f0f0fu) << 4);
    X[1] = ((e01 >> 4) & 0x0f0f0f0fu) | (e23 & 0xf0f0f0f0u);
    X[2] = (o01 & 0x0f0f0f0fu) | ((o23 & 0x0f0f0f0fu) << 4);
    X[0] = ((o01 >> 4) & 0x0f0f0f0fu) | (o23 & 0xf0f0f0f0u);
}
// fp16 {+-1, +-1} of the sign pair u of byte m (bit set = +1)
__device__ __forceinline__ uint32_t sign_pair(uint32_t w, int m, int u) {
    const int s = 8 * m + 6 - 2 * u;                       // bit s = dimension 2u+1, bit s+1 = dimension 2u
    const uint32_t hi = (w << (31 - s)) & 0x80000000u;
    const uint32_t lo = (s + 1 <= 15 ? w << (14 - s) : w >> (s - 14)) & 0x8000u;
    return 0xbc00bc00u ^ (hi | lo);
}

// Records: one warp per record.  `E` table entries: fields are little-endian code | code << bits pairs.
template <int D, int BITS>
struct RecChunk {
    static constexpr int L = D * BITS / 16;                // bytes of a lane's chunk
};
template <int D, int BITS>
__device__ __forceinline__ void load_rec_key(const uint8_t* rec, int lane, uint32_t (&w)[D / 16]) {
    constexpr int L = RecChunk<D, BITS>::L;
    if (L == 32) {
        const uint4 a = __ldg(reinterpret_cast<const uint4*>(rec + lane * 16)), b = __ldg(reinterpret_cast<const uint4*>(rec + 512 + lane * 16));
        w[0] = a.x; w[1] = a.y; w[2 % (D / 16)] = a.z; w[3 % (D / 16)] = a.w;
        w[4 % (D / 16)] = b.x; w[5 % (D / 16)] = b.y; w[6 % (D / 16)] = b.z; w[7 % (D / 16)] = b.w;
    } else {
#pragma unroll
        for (int i = 0; i < L / 4; i++) w[i] = __ldg(reinterpret_cast<const uint32_t*>(rec + lane * L) + i);
    }
}
template <int D, int BITS>
__device__ __forceinline__ void load_rec_val(const uint8_t* vsec, int lane, uint32_t (&w)[D / 16]) {
    constexpr int L = RecChunk<D, BITS>::L;
#pragma unroll
    for (int i = 0; i < L / 4; i++) w[i] = __ldg(reinterpret_cast<const uint32_t*>(vsec + lane * L) + i);
}
template <int NW>
__device__ __forceinline__ uint32_t field_of(const uint32_t (&w)[NW], int bit, int bits) {
    const int i = bit >> 5, s = bit & 31;
    uint32_t v = w[i] >> s;
    if (s + bits > 32) v = __funnelshift_r(w[i], w[i + 1 < NW ? i + 1 : i], s);
    return v & ((1u << bits) - 1u);
}
// Writes record `w8` (0..7 of the tile) of a key section: token rows g, g+8, one pair of dimensions per field.
template <int D, int BITS>
__device__ __forceinline__ void decode_key(const uint32_t (&w)[D / 16], uint32_t lut, int shift, uint32_t ahi, uint32_t alo, int w8, int lane) {
    const int g = lane >> 2, t = lane & 3;
#pragma unroll
    for (int second = 0; second < 2; second++)
#pragma unroll
        for (int e = 0; e < D / 8; e++) {
            const uint32_t f = field_of(w, tl_key_field_bit(D, BITS, e >> 1, e & 1, second), 2 * BITS);
            const uint2 v = lds64(lut + (f << shift));
            const int k = 8 * e + 2 * t, row = 16 * w8 + g + 8 * second;
            const uint32_t off = (uint32_t)(k >> 6) * (DQ_TILE * 128) + sw128_offset(row, k & 63);
            sts32(ahi + off, v.x);
            sts32(alo + off, v.y);
        }
}
// A value section: fields are pairs of TOKENS (2t, 2t+1); an 8 x 8 transpose turns them into pairs of dimensions.
template <int D, int BITS>
__device__ __forceinline__ void decode_val(const uint32_t (&w)[D / 16], uint32_t lut, int shift, uint32_t ahi, uint32_t alo, int w8, int lane) {
    const int g = lane >> 2, t = lane & 3;
#pragma unroll
    for (int mt = 0; mt < D / 16; mt++)
#pragma unroll
        for (int half = 0; half < 2; half++)
#pragma unroll
            for (int rs = 0; rs < 2; rs++) {
                const int bit = BITS == 2 ? (2 * mt + half) * 8 + 4 * rs : tl_val_field_bit(BITS, mt, half, rs);
                const uint32_t f = field_of(w, bit, 2 * BITS);
                const uint2 v = lds64(lut + (f << shift));
                const uint32_t hi = movmatrix_trans(v.x), lo = movmatrix_trans(v.y);
                const int k = 16 * mt + 8 * rs + 2 * t, row = 16 * w8 + g + 8 * half;
                const uint32_t off = (uint32_t)(k >> 6) * (DQ_TILE * 128) + sw128_offset(row, k & 63);
                sts32(ahi + off, hi);
                sts32(alo + off, lo);
            }
}

// ---- the kernel ------------------------------------------------------------------------------------
template <int DP, bool RECORDS, bool PROD>
__global__ void __launch_bounds__(DQ_THREADS, 1) dequantize_tc_kernel(const DqArgs a) {
    using C = DqCfg<DP, PROD>;
    constexpr int KBLK = C::KBLK, ABUF = C::ABUF;
    extern __shared__ uint8_t smem_unaligned[];
    __shared__ float red[32];
    __shared__ uint32_t tmem_slot;
    const uint32_t raw = smem_u32(smem_unaligned);
    const uint32_t base = (raw + 1023u) & ~1023u;
    uint8_t* const sm = smem_unaligned + (base - raw);
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const DqSide& sd = a.side[RECORDS ? blockIdx.y : 0];
    const bool values = RECORDS && sd.values;
    const int bits = sd.bits;

    const uint32_t bar0 = base + C::OFF_BAR;
    auto a_ready = [&](int part, int b) { return bar0 + 8 * (part * 2 + b); };          // part 1: the signs
    auto a_free = [&](int part, int b) { return bar0 + 8 * (4 + part * 2 + b); };
    auto acc_full = [&](int b) { return bar0 + 8 * (8 + b); };
    auto acc_free = [&](int b) { return bar0 + 8 * (10 + b); };
    if (threadIdx.x == 0) {
        for (int part = 0; part < 2; part++)
            for (int b = 0; b < 2; b++) { mbar_init(a_ready(part, b), DQ_DEC); mbar_init(a_free(part, b), 1); }
        for (int b = 0; b < 2; b++) { mbar_init(acc_full(b), 1); mbar_init(acc_free(b), DQ_EPI); }
    }
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    if (warp == DQ_DEC + DQ_EPI) tmem_alloc(smem_u32(&tmem_slot), C::TMEM_COLS);

    // ---- constants: the B operands, the pair table ----
    // What the terms of the centroids leave is the same for every coordinate of a code: the matrix takes it back on average.
    float mx = 0.0f, left = 0.0f, square = 0.0f;
    for (int i = 0; i < (1 << bits); i++) mx = fmaxf(mx, fabsf(__ldg(sd.cent + i)));
    const float sc = fp16_scale(mx);
    for (int i = 0; i < (1 << bits); i++) {
        const float v = __ldg(sd.cent + i) * sc, h = __half2float(__float2half_rn(v)), l = __half2float(__float2half_rn(v - h));
        left = fmaf(v - h - l, v, left);
        square = fmaf(v, v, square);
    }
    const float gain = square > 0.0f && square < 1e30f ? left / square : 0.0f;
    float unscale = 1.0f / build_b<DP>(sm, C::OFF_B, C::OFF_B + C::B_TERM, sd.rot, a.dim, gain, red), unscale_s = 1.0f;
    if (PROD) unscale_s = 1.0f / build_b<DP>(sm, C::OFF_B + 2 * C::B_TERM, C::OFF_B + 3 * C::B_TERM, a.qjl, a.dim, 0.0f, red);
    unscale *= 1.0f / sc;
    const int entries = 1 << (2 * bits);
    int shift = 3;                                             // entry stride = 8 bytes x copies (up to 8)
    while (shift < 6 && (entries << (shift + 1)) <= C::LUT) shift++;
    {
        for (int e = threadIdx.x; e < (entries << (shift - 3)); e += DQ_THREADS) {
            const int x = e >> (shift - 3);
            int c0, c1;                                        // codes of the pair's first and second element
            if (RECORDS) {
                c0 = x & ((1 << bits) - 1); c1 = x >> bits;
            } else {
                c0 = c1 = 0;
                for (int p = 0; p < bits; p++) { c0 |= ((x >> (2 * p + 1)) & 1) << p; c1 |= ((x >> (2 * p)) & 1) << p; }
            }
            uint32_t h0, l0, h1, l1;
            split_half(__ldg(sd.cent + c0) * sc, h0, l0);
            split_half(__ldg(sd.cent + c1) * sc, h1, l1);
            *reinterpret_cast<uint2*>(sm + C::OFF_LUT + e * 8) = make_uint2(h0 | (h1 << 16), l0 | (l1 << 16));
        }
    }
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem_base = tmem_slot;
    const int64_t ntiles = RECORDS ? (a.n + 7) / 8 : (a.n + DQ_TILE - 1) / DQ_TILE;
    bool ok = true;

    if (warp < DQ_DEC) {
        // ================= decoders =================
        const uint32_t lut = base + C::OFF_LUT + (lane & ((1 << (shift - 3)) - 1)) * 8;
        const int bpp = a.dim >> 3, words = a.dim >> 5;
        constexpr int HW = DP / 64;                            // plane words of a half row
        const int half = lane >> 4, trow = warp * 16 + (lane & 15);
        uint32_t it = 0;
        uint32_t w[HW][4], sg[HW], kw[DP / 16], w_next[HW][4], sg_next[HW], kw_next[DP / 16];
        auto request = [&](int64_t tile, uint32_t (&w)[HW][4], uint32_t (&sg)[HW], uint32_t (&kw)[DP / 16]) {
            if (RECORDS) {
                const int64_t rec = tile * 8 + warp;
                const int64_t u = rec / a.unit_used;
                const uint8_t* rp = sd.src + (rec < a.n ? u * a.unit_records + (rec - u * a.unit_used) : 0) * a.rec_bytes;
                const uint8_t* vp = rp + tl_key_section(DP, a.kb);
#pragma unroll
                for (int i = 0; i < DP / 16; i++) kw[i] = 0;
                if (rec < a.n) {
                    switch (bits) {
                        case 2: values ? load_rec_val<DP, 2>(vp, lane, kw) : load_rec_key<DP, 2>(rp, lane, kw); break;
                        case 3: values ? load_rec_val<DP, 3>(vp, lane, kw) : load_rec_key<DP, 3>(rp, lane, kw); break;
                        default: values ? load_rec_val<DP, 4>(vp, lane, kw) : load_rec_key<DP, 4>(rp, lane, kw); break;
                    }
                }
            } else {
                const int64_t r = tile * DQ_TILE + trow;
                const uint8_t* row = sd.src + r * (int64_t)(bits * bpp);
                const uint8_t* srow = PROD ? a.signs + r * bpp : nullptr;
#pragma unroll
                for (int i = 0; i < HW; i++) {
                    const int wi = half * HW + i;              // 32-dimension word of the row
                    const bool have = r < a.n && wi < words;
#pragma unroll
                    for (int p = 0; p < 4; p++)
                        w[i][p] = have && p < bits ? __ldg(reinterpret_cast<const uint32_t*>(row + p * bpp) + wi) : 0u;
                    if (PROD) sg[i] = have ? __ldg(reinterpret_cast<const uint32_t*>(srow) + wi) : 0u;
                }
            }
        };
        request(blockIdx.x, w_next, sg_next, kw_next);
        for (int64_t tile = blockIdx.x; tile < ntiles; tile += gridDim.x, it++) {
            const int b = it % ABUF;
            const uint32_t set = base + C::OFF_A + b * C::A_SET, ahi = set, alo = set + C::A_TERM, asg = set + 2 * C::A_TERM;
            // this tile's codes have been requested a tile ago; the next one's go out now
#pragma unroll
            for (int i = 0; i < HW; i++) {
#pragma unroll
                for (int p = 0; p < 4; p++) w[i][p] = w_next[i][p];
                sg[i] = sg_next[i];
            }
#pragma unroll
            for (int i = 0; i < DP / 16; i++) kw[i] = kw_next[i];
            if (tile + gridDim.x < ntiles) request(tile + gridDim.x, w_next, sg_next, kw_next);
            if (it >= (uint32_t)ABUF) ok = mbar_wait_compact(a_free(0, b), ((it / ABUF) - 1) & 1);
            if (!__all_sync(0xffffffffu, ok)) { ok = false; break; }
            if (RECORDS) {
                switch (bits) {
                    case 2: values ? decode_val<DP, 2>(kw, lut, shift, ahi, alo, warp, lane) : decode_key<DP, 2>(kw, lut, shift, ahi, alo, warp, lane); break;
                    case 3: values ? decode_val<DP, 3>(kw, lut, shift, ahi, alo, warp, lane) : decode_key<DP, 3>(kw, lut, shift, ahi, alo, warp, lane); break;
                    default: values ? decode_val<DP, 4>(kw, lut, shift, ahi, alo, warp, lane) : decode_key<DP, 4>(kw, lut, shift, ahi, alo, warp, lane); break;
                }
            } else {
#pragma unroll
                for (int i = 0; i < HW; i++) {
                    uint32_t X[4];
                    pair_indices(w[i], X);
#pragma unroll
                    for (int m = 0; m < 4; m++) {
                        uint2 v[4];
#pragma unroll
                        for (int u = 0; u < 4; u++) v[u] = lds64(lut + (((X[u] >> (8 * m)) & 0xffu) << shift));
                        const int k = 32 * (half * HW + i) + 8 * m;
                        const uint32_t off = (uint32_t)(k >> 6) * (DQ_TILE * 128) + sw128_offset(trow, k & 63);
                        sts128(ahi + off, v[0].x, v[1].x, v[2].x, v[3].x);
                        sts128(alo + off, v[0].y, v[1].y, v[2].y, v[3].y);
                    }
                }
            }
            asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
            __syncwarp();
            if (lane == 0) arrive(a_ready(0, b));
            if (PROD) {
                if (it >= (uint32_t)ABUF) ok = mbar_wait_compact(a_free(1, b), ((it / ABUF) - 1) & 1);
                if (!__all_sync(0xffffffffu, ok)) { ok = false; break; }
#pragma unroll
                for (int i = 0; i < HW; i++)
#pragma unroll
                    for (int m = 0; m < 4; m++) {
                        const int k = 32 * (half * HW + i) + 8 * m;
                        const uint32_t off = (uint32_t)(k >> 6) * (DQ_TILE * 128) + sw128_offset(trow, k & 63);
                        sts128(asg + off, sign_pair(sg[i], m, 0), sign_pair(sg[i], m, 1), sign_pair(sg[i], m, 2), sign_pair(sg[i], m, 3));
                    }
                asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
                __syncwarp();
                if (lane == 0) arrive(a_ready(1, b));
            }
        }
    } else if (warp < DQ_DEC + DQ_EPI) {
        // ================= epilogue: thread = half a row =================
        const int ew = warp & 3, half = (warp - DQ_DEC) >> 2;
        const int row = ew * 32 + lane, col0 = half * (DP / 2);
        // 32 accumulator columns -> scaled float32
        float nrm = 0.0f;
        bool small = false;                                    // a row of the warp has so small a norm that f would lose digits
        auto load_cols = [&](uint32_t taddr, float f, float fs, uint32_t (&v)[32]) {
            tmem_ld32(taddr, v);
            if (PROD) {
                uint32_t s[32];
                tmem_ld32(taddr + DP, s);
#pragma unroll
                for (int i = 0; i < 32; i++) v[i] = __float_as_uint(fmaf(__uint_as_float(v[i]), f, fs * __uint_as_float(s[i])));
            } else {
#pragma unroll
                for (int i = 0; i < 32; i++) v[i] = __float_as_uint(__uint_as_float(v[i]) * f);
            }
            if (small) {
#pragma unroll
                for (int i = 0; i < 32; i++) v[i] = __float_as_uint(__uint_as_float(v[i]) * nrm);
            }
        };
        auto pack_cols = [&](uint32_t (&v)[32]) {
#pragma unroll
            for (int i = 0; i < 16; i++) {
                const float lo = __uint_as_float(v[2 * i]), hi = __uint_as_float(v[2 * i + 1]);
                if (a.out_dtype == TQB_F16) v[i] = pack_half2(lo, hi);
                else { __nv_bfloat162 h = __floats2bfloat162_rn(lo, hi); v[i] = *reinterpret_cast<uint32_t*>(&h); }
            }
        };
        uint32_t it = 0;
        for (int64_t tile = blockIdx.x; tile < ntiles; tile += gridDim.x, it++) {
            const int b = it & 1;
            float coef = 0.0f;
            int64_t orow = -1;
            nrm = 0.0f;
            if (RECORDS) {
                const int64_t rec = tile * 8 + (row >> 4);
                if (rec < a.n) {
                    const int64_t u = rec / a.unit_used, ru = rec - u * a.unit_used, tok = ru * 16 + (row & 15);
                    if (tok < a.tokens) {
                        orow = u * a.out_pitch + tok;
                        const uint8_t* nsec = sd.src + (u * a.unit_records + ru) * a.rec_bytes + tl_key_section(DP, a.kb) + tl_val_section(DP, a.vb);
                        nrm = __ldg(reinterpret_cast<const float*>(nsec + tl_norm_offset(a.vb, values ? 1 : 0, row & 15)));
                    }
                }
            } else {
                const int64_t r = tile * DQ_TILE + row;
                if (r < a.n) {
                    orow = r;
                    nrm = __ldg(sd.norms + r);
                    if (PROD) coef = a.qjl_scale * __ldg(a.res_norms + r) * unscale_s;
                }
            }
            ok = mbar_wait_compact(acc_full(b), (it >> 1) & 1);
            if (!__all_sync(0xffffffffu, ok)) { ok = false; break; }
            tc_fence_after();
            const uint32_t trow = tmem_base + ((uint32_t)(ew * 32) << 16) + b * C::ACC_COLS + col0;
            // rows of this group of four lanes (the stores below are dealt so that four lanes share a row)
            int64_t rows4[4];
#pragma unroll
            for (int i = 0; i < 4; i++) rows4[i] = __shfl_sync(0xffffffffu, orow, (lane & ~3) + i);
            small = __any_sync(0xffffffffu, nrm != 0.0f && fabsf(unscale * nrm) < 1e-30f);
            const float f = small ? unscale : unscale * nrm, fs = small ? coef : coef * nrm;
            // 32 columns of float32, or 64 of a 16-bit type: 128 bytes of every row a turn
            const bool half_out = a.out_dtype != TQB_F32;
            const int turn = half_out && DP / 2 >= 64 ? 64 : 32;
#pragma unroll 1
            for (int c = 0; c < DP / 2; c += turn) {
                uint32_t v[32];
                load_cols(trow + c, f, fs, v);
                if (half_out) {
                    pack_cols(v);
                    if (DP / 2 >= 64) {
                        uint32_t w[32];
                        load_cols(trow + c + 32, f, fs, w);
                        pack_cols(w);
#pragma unroll
                        for (int i = 0; i < 16; i++) v[16 + i] = w[i];
                    }
                }
                if (half_out && DP / 2 < 64) {
                    // 64 bytes of a row: two 32-byte pieces, the row's own lane stores them
                    if (orow >= 0 && col0 + c < a.dim) {
                        uint8_t* o = reinterpret_cast<uint8_t*>(sd.out) + (orow * a.dim + col0 + c) * 2;
                        st_global32(o, &v[0]);
                        st_global32(o + 32, &v[8]);
                    }
                } else {
                    transpose4(v, lane);
                    const int es = half_out ? 2 : 4, col = col0 + c + (lane & 3) * (32 / es);
#pragma unroll
                    for (int i = 0; i < 4; i++)
                        if (rows4[i] >= 0 && col < a.dim)
                            st_global32(reinterpret_cast<uint8_t*>(sd.out) + (rows4[i] * a.dim + col) * es, &v[8 * i]);
                }
                __syncwarp();                                  // (the next tensor-memory load is warp-collective)
            }
            tc_fence_before();
            __syncwarp();
            if (lane == 0) arrive(acc_free(b));
        }
    } else {
        // ================= MMA issuer =================
        constexpr uint32_t IDESC = (1u << 4) | ((uint32_t)(DP >> 3) << 17) | ((uint32_t)(DQ_TILE >> 4) << 24);   // fp16 x fp16 -> f32
        auto issue = [&](uint32_t d, uint32_t am, uint32_t bm, uint32_t& acc) {
#pragma unroll
            for (int kb = 0; kb < KBLK; kb++) {
                const uint64_t ad = umma_desc(am + kb * (DQ_TILE * 128)), bd = umma_desc(bm + kb * (DP * 128));
#pragma unroll
                for (int k = 0; k < 4; k++) { umma_f16(d, ad + 2 * k, bd + 2 * k, IDESC, acc); acc = 1; }
            }
        };
        uint32_t it = 0;
        for (int64_t tile = blockIdx.x; tile < ntiles; tile += gridDim.x, it++) {
            const int b = it & 1, ab = it % ABUF;
            if (lane == 0) {
                ok = mbar_wait_compact(a_ready(0, ab), (it / ABUF) & 1);
                if (ok && it >= 2) ok = mbar_wait_compact(acc_free(b), ((it >> 1) - 1) & 1);
            }
            ok = __shfl_sync(0xffffffffu, ok ? 1 : 0, 0) != 0;
            if (!ok) break;
            const uint32_t set = base + C::OFF_A + ab * C::A_SET, bm = base + C::OFF_B, d = tmem_base + b * C::ACC_COLS;
            if (lane == 0) {
                tc_fence_after();
                uint32_t acc = 0;                              // low-order products first: the accumulator is small then
                issue(d, set + C::A_TERM, bm, acc);
                issue(d, set, bm + C::B_TERM, acc);
                issue(d, set, bm, acc);
                umma_commit(a_free(0, ab));
                if (PROD) {
                    ok = mbar_wait_compact(a_ready(1, ab), (it / ABUF) & 1);
                    tc_fence_after();
                    if (ok) {
                        acc = 0;
                        issue(d + DP, set + 2 * C::A_TERM, bm + 3 * C::B_TERM, acc);
                        issue(d + DP, set + 2 * C::A_TERM, bm + 2 * C::B_TERM, acc);
                        umma_commit(a_free(1, ab));
                    }
                }
                umma_commit(acc_full(b));
            }
            ok = __shfl_sync(0xffffffffu, ok ? 1 : 0, 0) != 0;
            if (!ok) break;
        }
    }
    if (!ok && lane == 0) atomicExch(a.error, 1);
    tc_fence_before();
    __syncthreads();
    if (warp == DQ_DEC + DQ_EPI) {
        tc_fence_after();
        tmem_dealloc(tmem_base, C::TMEM_COLS);
    }
}

template <int DP, bool RECORDS, bool PROD>
static int launch_dq_tc(DqArgs& a, int sides, cudaStream_t st) {
    using C = DqCfg<DP, PROD>;
    auto kern = dequantize_tc_kernel<DP, RECORDS, PROD>;
    TQB_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, C::TOTAL));
    if (int e = tc_error_word(&a.error)) return e;
    const int64_t ntiles = RECORDS ? (a.n + 7) / 8 : (a.n + DQ_TILE - 1) / DQ_TILE;
    const int gx = (int)std::min<int64_t>(std::max(1, sm_count() / sides), ntiles);
    kern<<<dim3(gx, sides), DQ_THREADS, C::TOTAL, st>>>(a);
    return check_launch("dequantize_tc");
}

// Rows: tries the tensor-core kernel; TQB_ERR_UNSUPPORTED (without touching the last-error text) sends the call to the
// FFMA kernel.  qjl != null: Prod rows, mse_bits = bits - 1.
int dequantize_tc_try(const uint8_t* packed, const float* norms, const uint8_t* signs, const float* res_norms, int64_t n, int dim,
                      const float* rot, const float* cent, const float* qjl, int mse_bits, void* out, int out_dtype, cudaStream_t st) {
    if (dim > 128 || dim % 32 || n < 256) return TQB_ERR_UNSUPPORTED;
    if (qjl && mse_bits > 3) return TQB_ERR_UNSUPPORTED;             // (no room for the pair table)
    if (((uintptr_t)packed | (uintptr_t)signs) % 4 || ((uintptr_t)rot | (uintptr_t)qjl) % 16 || (uintptr_t)out % 32) return TQB_ERR_UNSUPPORTED;
    DqArgs a{};
    a.side[0] = DqSide{packed, norms, rot, cent, out, mse_bits, 0};
    a.signs = signs; a.res_norms = res_norms; a.qjl = qjl; a.qjl_scale = 1.2533141373155003f / (float)dim;
    a.n = n; a.dim = dim; a.out_dtype = out_dtype;
    if (out_dtype != TQB_F32 && out_dtype != TQB_F16 && out_dtype != TQB_BF16) return TQB_ERR_UNSUPPORTED;
    if (dim <= 64) return qjl ? launch_dq_tc<64, false, true>(a, 1, st) : launch_dq_tc<64, false, false>(a, 1, st);
    return qjl ? launch_dq_tc<128, false, true>(a, 1, st) : launch_dq_tc<128, false, false>(a, 1, st);
}

}  // namespace tqb

extern "C" int tqb_kv_dequantize(const uint8_t* store, int64_t units, int64_t unit_pitch, int64_t tokens, int dim, const float* rot_k,
                                 const float* cent_k, int kbits, const float* rot_v, const float* cent_v, int vbits, void* k_out,
                                 void* v_out, int64_t out_pitch, int out_dtype, void* stream) {
    using namespace tqb;
    TQB_REQUIRE(units >= 0 && tokens >= 0, "kv_dequantize: negative size");
    if (dim != 64 && dim != 128) return fail(TQB_ERR_UNSUPPORTED, "kv_dequantize: head_dim must be 64 or 128, got %d", dim);
    if (kbits < 2 || kbits > 4 || vbits < 2 || vbits > 4)
        return fail(TQB_ERR_UNSUPPORTED, "kv_dequantize: key and value bits must be 2..4, got %d/%d", kbits, vbits);
    TQB_REQUIRE(out_dtype == TQB_F32 || out_dtype == TQB_F16 || out_dtype == TQB_BF16, "kv_dequantize: unknown dtype %d", out_dtype);
    if (units == 0 || tokens == 0 || (!k_out && !v_out)) return TQB_OK;
    TQB_REQUIRE(store && (!k_out || (rot_k && cent_k)) && (!v_out || (rot_v && cent_v)), "kv_dequantize: null pointer");
    TQB_REQUIRE(unit_pitch % 16 == 0 && tokens <= unit_pitch && tokens <= out_pitch, "kv_dequantize: tokens (%lld) exceed a pitch (%lld, %lld)",
                (long long)tokens, (long long)unit_pitch, (long long)out_pitch);
    TQB_REQUIRE((uintptr_t)store % 16 == 0, "kv_dequantize: the record store must be 16-byte aligned");
    TQB_REQUIRE(((uintptr_t)k_out | (uintptr_t)v_out) % 32 == 0, "kv_dequantize: outputs must be 32-byte aligned");
    TQB_REQUIRE(((uintptr_t)rot_k | (uintptr_t)rot_v) % 16 == 0, "kv_dequantize: rotation matrices must be 16-byte aligned");
    DqArgs a{};
    int sides = 0;
    if (k_out) a.side[sides++] = DqSide{store, nullptr, rot_k, cent_k, k_out, kbits, 0};
    if (v_out) a.side[sides++] = DqSide{store, nullptr, rot_v, cent_v, v_out, vbits, 1};
    a.dim = dim; a.out_dtype = out_dtype; a.kb = kbits; a.vb = vbits; a.rec_bytes = tl_record_bytes(dim, kbits, vbits);
    a.unit_records = unit_pitch / 16; a.unit_used = (tokens + 15) / 16; a.tokens = tokens; a.out_pitch = out_pitch;
    a.n = units * a.unit_used;
    cudaStream_t st = (cudaStream_t)stream;
    return dim == 64 ? launch_dq_tc<64, true, false>(a, sides, st) : launch_dq_tc<128, true, false>(a, sides, st);
}
