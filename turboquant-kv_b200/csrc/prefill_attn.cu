// prefill_attn.cu -- attention of several new tokens per request over the packed, paged KV cache.
//
// Replaces "every query token is a decode sequence of its own" for requests with several new tokens (prompts, chunks
// behind an earlier context, speculative verification): the records of a request are decoded once per block of query
// tokens instead of once per token, and the products run on the 5th-generation tensor cores.
//
// Work item = (request, KV head, two tiles of 128 query rows).  A row is (token, query head of the group): a tile holds
// 128 / group tokens.  One persistent CTA per SM takes its items from a list sorted by cost, forwards and backwards in
// turn.  Roles (544 threads):
//   warps 0-3, 4-7   one query tile each, thread = row: bring the queries in (hi / lo fp16 terms for the rotation), run
//                    the online softmax on the scores in tensor memory and write P (fp16) back over them, rescale the
//                    accumulator when a row's maximum moved by more than the slack, and hand the result out.
//   warps 8-15       decode: a warp takes one 16-token record of a 128-token tile, requested one tile ahead.  Codes become
//                    fp16 pairs through a lookup table replicated per lane; K goes to a [token][dim] tile, V to a [dim][token]
//                    tile, both K-major with 128-byte swizzle, without a bank conflict.  Three tile buffers in a ring; the
//                    two fp16 terms of R_k and R_v pass through the same ring (bulk copies of ready images).
//   warp 16          one lane issues the MMAs: Q' = q R_k^T, S = Q' K^T, O += P V (P read from tensor memory), out = O R_v.
//
// Arithmetic as in decode_attn.cu: fp16 centroids, queries and probabilities, float32 sums; the token norms multiply the
// float32 scores and probabilities, not the operands.  The rotations keep float32's accuracy: a row is scaled by a power of
// two, split into two fp16 terms (one where its type has no more than 11 significant bits) and multiplied with the two
// terms of the matrix.
//
// What bounds it (d = 128, clocks of a pair of query tiles against one key tile): 2,048 on the tensor cores, 2,048 of ex2,
// about 2,400 issue slots per scheduler (softmax 4 instructions a score, decode 450 a warp); measured about 6,000, because a
// tile's chain scores -> P -> P V -> next scores is serial (tensor memory holds one S per tile beside O) and the two tiles
// overlap only in part.  Beside them an item costs 3 us for its queries and 3 us for its output.  Measured, 8 requests of
// about 1,024 tokens, 32 query / 8 KV heads, K4/V3: 12.1 ms with every token a decode sequence of its own, 285 us here
// (77 GFLOP: 270 TFLOP/s); d = 64, K4/V2: 2,690 -> 192 us.  One-pass softmax (P in registers until no score exceeds the
// slack) took it from 320 to 285 us; a chunk of 300 tokens behind 2,000, 8 requests: 334 -> 253 us.
//
// Every wait is bounded; one that expires sets TQB_DECODE_WAIT_EXPIRED in the caller's status word.
#include "common.cuh"
#include "pipe.cuh"
#include "tc.cuh"
#include "tiled_layout.cuh"

#include <type_traits>

namespace tqb {

constexpr int PF_ROWS = 128;                  // rows of a query tile = tensor-memory lanes
constexpr int PF_KV = 128;                    // tokens of a key / value tile
constexpr int PF_DEC = 8;                     // decode warps
constexpr int PF_THREADS = (8 + PF_DEC + 1) * 32;
constexpr int PF_RING = 3;
constexpr float PF_SLACK = 8.0f;              // lazy maximum: it moves when a score exceeds it by more than this (log2)
constexpr float PF_SAFE = 4.0f;               // P up to 2^4 fits fp16 with value norms up to 4,000 (the decode kernel's bound): beyond it, look
constexpr float PF_HALF_MAX = 60000.0f;       // P times value norm stays below fp16's largest number
constexpr float PF_LOG2E = 1.4426950408889634f;
constexpr float PF_NEG_INF = -__builtin_huge_valf();
constexpr int PF_BUCKETS = 256;               // cost classes of the item list

struct PrefillParams {
    const void* query; void* out;
    const uint8_t* store;
    const int32_t* qstart; const int32_t* seq_lens; const int32_t* block_tables;
    const float* cent_k; const float* cent_v; const float* rot_k; const float* rot_v;
    int64_t n_tokens, max_len;
    int num_reqs, q_heads, kv_heads, group, tpt;          // tpt: tokens per query tile
    int first_token;                                      // what query_start counts from
    int max_blocks, block_size, causal;
    float scale_log2;
    int* status;
    // workspace
    int* n_items; int2* items; int item_cap;              // (request, block of 2 tpt tokens)
    uint8_t* images; float* unscale;                      // R_k hi, lo, R_v^T hi, lo; 1 / scale of both matrices
};

struct PfReq { int q0, qlen, base, len; };                // first token, new tokens, tokens before them, attended in all
__device__ __forceinline__ PfReq pf_request(const PrefillParams& p, int r) {
    PfReq q;
    const int hi = (int)min(p.n_tokens, (int64_t)0x7fffffff);
    q.q0 = min(max(p.qstart[r] - p.first_token, 0), hi);
    q.qlen = max(0, min(p.qstart[r + 1] - p.first_token, hi) - q.q0);
    q.len = p.seq_lens[r];
    q.base = q.len - q.qlen;
    return q;
}
// Tokens that query token t of the request attends, inside the announced bound.
__device__ __forceinline__ int pf_limit(const PrefillParams& p, const PfReq& q, int t) {
    const int n = p.causal ? q.base + t + 1 : q.len;
    return min(max(n, 0), (int)min(p.max_len, (int64_t)0x3fffffff));
}

// ---- plan: operand images of the rotations, item list ------------------------------------------------
// Block 0 sorts the items by cost (tiles of keys; the order inside a class does not matter); the other blocks write the
// fp16 terms of R_k ([i][k]) and R_v^T ([k][j]) as the K-major, 128-byte-swizzled operands the kernel's MMAs read.
constexpr int PF_PLAN_THREADS = 512, PF_PLAN_PARTS = 8, PF_PLAN_BLOCKS = 1 + 2 * PF_PLAN_PARTS;
template <int D>
__global__ void __launch_bounds__(PF_PLAN_THREADS) prefill_plan_kernel(const PrefillParams p) {
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    pdl_trigger();                                          // the attention kernel sets itself up meanwhile
    if (blockIdx.x == 0) {
        __shared__ int hist[PF_BUCKETS], at[PF_BUCKETS];
        for (int i = threadIdx.x; i < PF_BUCKETS; i += blockDim.x) hist[i] = 0;
        __syncthreads();
        const int top = max(1, (int)((min(p.max_len, (int64_t)0x3fffffff) + PF_KV - 1) / PF_KV));
#pragma unroll 1
        for (int pass = 0; pass < 2; pass++) {
            for (int r = warp; r < p.num_reqs; r += PF_PLAN_THREADS / 32) {
                const PfReq q = pf_request(p, r);
                const int blocks = (q.qlen + 2 * p.tpt - 1) / (2 * p.tpt);
                for (int b = lane; b < blocks; b += 32) {
                    const int last = min(q.qlen, (b + 1) * 2 * p.tpt) - 1;
                    const int cost = min(top, (pf_limit(p, q, last) + PF_KV - 1) / PF_KV);
                    const int bucket = PF_BUCKETS - 1 - (int)((int64_t)cost * (PF_BUCKETS - 1) / top);    // dearest first
                    if (pass == 0) atomicAdd(&hist[bucket], 1);
                    else {
                        const int i = atomicAdd(&at[bucket], 1);
                        if (i < p.item_cap) p.items[i] = make_int2(r, b);
                    }
                }
                if (pass == 0 && lane == 0) {      // lengths beyond what the host announced are clamped, and reported
                    const int longest = p.causal ? q.base + q.qlen : q.len;
                    if (q.qlen > 0 && ((int64_t)longest > p.max_len || (p.causal ? q.base + 1 : q.len) < 0))
                        atomicOr(p.status, TQB_DECODE_LEN_CLAMPED);
                }
            }
            __syncthreads();
            if (pass == 0 && threadIdx.x == 0) {
                int s = 0;
                for (int i = 0; i < PF_BUCKETS; i++) { at[i] = s; s += hist[i]; }
                *p.n_items = min(s, p.item_cap);
            }
            __syncthreads();
        }
        return;
    }
    __shared__ float red[PF_PLAN_THREADS / 32];
    const int which = (blockIdx.x - 1) & 1, part = (blockIdx.x - 1) >> 1;           // K or V; a part of the rows
    const float* M = which ? p.rot_v : p.rot_k;
    float mx = 0.0f;
#pragma unroll
    for (int i = 0; i < D * D / 4 / PF_PLAN_THREADS; i++) {
        const float4 v = __ldg(reinterpret_cast<const float4*>(M) + i * PF_PLAN_THREADS + threadIdx.x);
        mx = fmaxf(fmaxf(fmaxf(mx, fabsf(v.x)), fmaxf(fabsf(v.y), fabsf(v.z))), fabsf(v.w));
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, o));
    if (lane == 0) red[warp] = mx;
    __syncthreads();
    mx = 0.0f;
    for (int w = 0; w < PF_PLAN_THREADS / 32; w++) mx = fmaxf(mx, red[w]);
    const float sc = fp16_scale(mx);
    if (part == 0 && threadIdx.x == 0) p.unscale[which] = 1.0f / sc;
    uint8_t* hi = p.images + which * (4 * D * D);
    uint8_t* lo = hi + 2 * D * D;
#pragma unroll
    for (int i = 0; i < D * D / PF_PLAN_PARTS / PF_PLAN_THREADS; i++) {
        const int e = i * PF_PLAN_THREADS + threadIdx.x;
        const int r = part * (D / PF_PLAN_PARTS) + e / D, c = e % D;                // element (r, c) of M
        const float v = __ldg(M + r * D + c) * sc;
        const int n = which ? c : r, k = which ? r : c;
        const uint32_t off = (uint32_t)(k >> 6) * (D * 128) + sw128_offset(n, k & 63);
        const __half h = __float2half_rn(v), l = __float2half_rn(v - __half2float(h));
        *reinterpret_cast<__half*>(hi + off) = h;
        *reinterpret_cast<__half*>(lo + off) = l;
    }
}

// ---- configuration -----------------------------------------------------------------------------------
template <int D, int KB, int VB>
struct PfCfg {
    static constexpr int REC = 2 * D * (KB + VB) + 128;
    static constexpr int KSEC = 2 * D * KB, VSEC = 2 * D * VB;
    static constexpr int QTILE = PF_ROWS * D * 2, BUF = PF_KV * D * 2;
    static constexpr int RTERM = D * D * 2;                                          // one term of a rotation (<= BUF)
    // tables of code pairs, replicated per lane (no bank conflict); 4 + 4 bits at D = 128 leave room for 16 copies of V's
    static constexpr int KSH = 7, VSH = (D == 128 && KB == 4 && VB == 4) ? 6 : 7;
    static constexpr int LUTK = (1 << (2 * KB)) << KSH, LUTV = (1 << (2 * VB)) << VSH;
    static constexpr int OFF_Q = 0, OFF_RING = 2 * QTILE, OFF_LUTK = OFF_RING + PF_RING * BUF, OFF_LUTV = OFF_LUTK + LUTK;
    static constexpr int OFF_NRM = OFF_LUTV + LUTV;                                  // 2 slots x {key, value} x 128 floats
    static constexpr int OFF_BAR = OFF_NRM + 2 * 2 * PF_KV * 4;
    static constexpr int TOTAL = OFF_BAR + 256 + 1024;                               // + slack for the 1024-byte alignment
    static constexpr int S_COL = 0, O_COL = 256;                                     // tensor memory: S0 S1 (P over them) O0 O1
    static_assert(TOTAL <= 227 * 1024, "shared memory");
};

__device__ __forceinline__ void pf_sts128(uint32_t addr, uint32_t a, uint32_t b, uint32_t c, uint32_t d) {
    asm volatile("st.shared.v4.b32 [%0], {%1, %2, %3, %4};" ::"r"(addr), "r"(a), "r"(b), "r"(c), "r"(d) : "memory");
}
__device__ __forceinline__ void pf_sts32(uint32_t addr, uint32_t a) {
    asm volatile("st.shared.b32 [%0], %1;" ::"r"(addr), "r"(a) : "memory");
}
__device__ __forceinline__ float4 pf_lds128(uint32_t addr) {
    float4 v;
    asm volatile("ld.shared.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "r"(addr));
    return v;
}
__device__ __forceinline__ void pf_arrive(uint32_t bar) {
    asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(bar) : "memory");
}
// Bounded wait on the critical chain (scores -> P -> product): polls without suspending the thread, which costs a few
// hundred clocks to resume.
__device__ __forceinline__ bool pf_wait_spin(uint32_t bar, uint32_t parity) {
    auto test = [&]() {
        uint32_t ok;
        asm volatile(
            "{\n\t.reg .pred p;\n\t"
            "mbarrier.test_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
            "selp.u32 %0, 1, 0, p;\n\t}"
            : "=r"(ok) : "r"(bar), "r"(parity) : "memory");
        return ok != 0;
    };
    if (test()) return true;
    const unsigned long long t0 = wall_ns();
    for (;;) {
#pragma unroll 1
        for (int i = 0; i < 64; i++)
            if (test()) return true;
        if (wall_ns() - t0 > WAIT_LIMIT_NS) return false;
    }
}
__device__ __forceinline__ float pf_ex2(float x) {
    float y;
    asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
}
// D[tmem] (+)= A[tmem] * B[smem]: A is fp16, two per 32-bit column.
__device__ __forceinline__ void umma_f16_ta(uint32_t tmem_d, uint32_t tmem_a, uint64_t bdesc, uint32_t idesc, uint32_t accumulate) {
    asm volatile(
        "{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %2, %3, p;\n\t}"
        ::"r"(tmem_d), "r"(tmem_a), "l"(bdesc), "r"(idesc), "r"(accumulate) : "memory");
}
__device__ __forceinline__ void tmem_st16(uint32_t taddr, const uint32_t (&v)[16]) {
    asm volatile(
        "tcgen05.st.sync.aligned.32x32b.x16.b32 [%0], "
        "{%1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, %16};"
        ::"r"(taddr), "r"(v[0]), "r"(v[1]), "r"(v[2]), "r"(v[3]), "r"(v[4]), "r"(v[5]), "r"(v[6]), "r"(v[7]),
          "r"(v[8]), "r"(v[9]), "r"(v[10]), "r"(v[11]), "r"(v[12]), "r"(v[13]), "r"(v[14]), "r"(v[15]) : "memory");
}
__device__ __forceinline__ void tmem_st32(uint32_t taddr, const uint32_t (&v)[32]) {
    asm volatile(
        "tcgen05.st.sync.aligned.32x32b.x32.b32 [%0], "
        "{%1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, %16, "
        "%17, %18, %19, %20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31, %32};"
        ::"r"(taddr), "r"(v[0]), "r"(v[1]), "r"(v[2]), "r"(v[3]), "r"(v[4]), "r"(v[5]), "r"(v[6]), "r"(v[7]),
          "r"(v[8]), "r"(v[9]), "r"(v[10]), "r"(v[11]), "r"(v[12]), "r"(v[13]), "r"(v[14]), "r"(v[15]),
          "r"(v[16]), "r"(v[17]), "r"(v[18]), "r"(v[19]), "r"(v[20]), "r"(v[21]), "r"(v[22]), "r"(v[23]),
          "r"(v[24]), "r"(v[25]), "r"(v[26]), "r"(v[27]), "r"(v[28]), "r"(v[29]), "r"(v[30]), "r"(v[31]) : "memory");
}
__device__ __forceinline__ void tmem_wait_st() { asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory"); }

// Eight consecutive elements of a query row as float32.
template <typename T>
__device__ __forceinline__ void pf_load8(const T* p, float (&v)[8]) {
    const float4 a = load4(p), b = load4(p + 4);
    v[0] = a.x; v[1] = a.y; v[2] = a.z; v[3] = a.w; v[4] = b.x; v[5] = b.y; v[6] = b.z; v[7] = b.w;
}
template <>
__device__ __forceinline__ void pf_load8<__nv_bfloat16>(const __nv_bfloat16* p, float (&v)[8]) {
    const uint4 w = *reinterpret_cast<const uint4*>(p);
    const uint32_t u[4] = {w.x, w.y, w.z, w.w};
#pragma unroll
    for (int i = 0; i < 4; i++) { v[2 * i] = __uint_as_float(u[i] << 16); v[2 * i + 1] = __uint_as_float(u[i] & 0xffff0000u); }
}
template <>
__device__ __forceinline__ void pf_load8<__half>(const __half* p, float (&v)[8]) {
    const uint4 w = *reinterpret_cast<const uint4*>(p);
    const uint32_t u[4] = {w.x, w.y, w.z, w.w};
#pragma unroll
    for (int i = 0; i < 4; i++) {
        const float2 f = __half22float2(*reinterpret_cast<const __half2*>(&u[i]));
        v[2 * i] = f.x; v[2 * i + 1] = f.y;
    }
}
__device__ __forceinline__ uint32_t pf_pack(float a, float b, __half*) { return pack_half2(a, b); }
__device__ __forceinline__ uint32_t pf_pack(float a, float b, __nv_bfloat16*) {
    const __nv_bfloat162 h = __floats2bfloat162_rn(a, b);
    return *reinterpret_cast<const uint32_t*>(&h);
}
// {a, b} -> fp16 pair: the leading term, or what it leaves
template <bool LOW>
__device__ __forceinline__ uint32_t pf_term(float a, float b) {
    const __half2 h = __floats2half2_rn(a, b);
    if (!LOW) return *reinterpret_cast<const uint32_t*>(&h);
    const float2 f = __half22float2(h);
    return pack_half2(a - f.x, b - f.y);
}
// Writes one row of an A operand (D fp16 elements) from f(k) -> 8 float32 values at k.
template <int D, bool LOW, typename F>
__device__ __forceinline__ void pf_write_row(uint32_t tile, int row, F f) {
#pragma unroll 4
    for (int k = 0; k < D; k += 8) {
        float v[8];
        f(k, v);
        pf_sts128(tile + (uint32_t)(k >> 6) * (PF_ROWS * 128) + sw128_offset(row, k & 63), pf_term<LOW>(v[0], v[1]), pf_term<LOW>(v[2], v[3]),
                  pf_term<LOW>(v[4], v[5]), pf_term<LOW>(v[6], v[7]));
    }
}

template <int NW>
__device__ __forceinline__ uint32_t pf_field(const uint32_t (&w)[NW], int bit, int bits) {
    const int i = bit >> 5, s = bit & 31;
    if (bits == 8) return __byte_perm(w[i], 0, 0x4440u | (uint32_t)(s >> 3));
    uint32_t v = w[i] >> s;
    if (s + bits > 32) v = __funnelshift_r(w[i], w[i + 1 < NW ? i + 1 : i], s);
    return v & ((1u << bits) - 1u);
}

// One record's codes and norms in a lane's registers.
template <int D, int KB, int VB>
struct PfRecord {
    uint32_t k[D * KB / 64], v[D * VB / 64], norm;
    __device__ __forceinline__ void load(const uint8_t* rec, int lane) {
        using C = PfCfg<D, KB, VB>;
        constexpr int KL = D * KB / 16, VL = D * VB / 16;
        if (rec) {
            if (KL == 32) {
                const uint4 a = __ldg(reinterpret_cast<const uint4*>(rec + lane * 16)), b = __ldg(reinterpret_cast<const uint4*>(rec + 512 + lane * 16));
                k[0] = a.x; k[1] = a.y; k[2 % (KL / 4)] = a.z; k[3 % (KL / 4)] = a.w;
                k[4 % (KL / 4)] = b.x; k[5 % (KL / 4)] = b.y; k[6 % (KL / 4)] = b.z; k[7 % (KL / 4)] = b.w;
            } else {
                get<KL>(rec + lane * KL, k);
            }
            get<VL>(rec + C::KSEC + lane * VL, v);
            norm = __ldg(reinterpret_cast<const uint32_t*>(rec + C::KSEC + C::VSEC) + lane);
        } else {
#pragma unroll
            for (int i = 0; i < KL / 4; i++) k[i] = 0;
#pragma unroll
            for (int i = 0; i < VL / 4; i++) v[i] = 0;
            norm = 0;
        }
    }
    template <int NB>
    __device__ __forceinline__ static void get(const uint8_t* p, uint32_t (&w)[NB / 4]) {
        if (NB % 16 == 0) {
#pragma unroll
            for (int i = 0; i < NB / 16; i++) {
                const uint4 a = __ldg(reinterpret_cast<const uint4*>(p) + i);
                w[4 * i] = a.x; w[4 * i + 1] = a.y; w[4 * i + 2] = a.z; w[4 * i + 3] = a.w;
            }
        } else if (NB % 8 == 0) {
#pragma unroll
            for (int i = 0; i < NB / 8; i++) {
                const uint2 a = __ldg(reinterpret_cast<const uint2*>(p) + i);
                w[2 * i] = a.x; w[2 * i + 1] = a.y;
            }
        } else {
#pragma unroll
            for (int i = 0; i < NB / 4; i++) w[i] = __ldg(reinterpret_cast<const uint32_t*>(p) + i);
        }
    }
};

// Largest score of a row over one key tile: scores in tensor memory times the tokens' key norms.  `room`: tokens the row
// attends (MASKED: may be less than the tile).
template <bool MASKED>
__device__ __forceinline__ float pf_row_max(uint32_t S, uint32_t nk, int room) {
    float mx = PF_NEG_INF;
#pragma unroll 1
    for (int c = 0; c < PF_KV; c += 32) {
        uint32_t v[32];
        tmem_ld32(S + c, v);
#pragma unroll
        for (int i = 0; i < 32; i += 4) {
            const float4 a = pf_lds128(nk + 4 * (c + i));
            const float s[4] = {__uint_as_float(v[i]) * a.x, __uint_as_float(v[i + 1]) * a.y, __uint_as_float(v[i + 2]) * a.z, __uint_as_float(v[i + 3]) * a.w};
#pragma unroll
            for (int e = 0; e < 4; e++) mx = fmaxf(mx, MASKED && c + i + e >= room ? PF_NEG_INF : s[e]);
        }
    }
    return mx;
}
// Two float32 operations in one instruction.
__device__ __forceinline__ uint64_t pf_two(float a, float b) {
    uint64_t r;
    asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(a), "f"(b));
    return r;
}
__device__ __forceinline__ void pf_split(uint64_t v, float& a, float& b) { asm("mov.b64 {%0, %1}, %2;" : "=f"(a), "=f"(b) : "l"(v)); }
__device__ __forceinline__ uint64_t pf_fma2(uint64_t a, uint64_t b, uint64_t c) {
    uint64_t r;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
    return r;
}
__device__ __forceinline__ uint64_t pf_mul2(uint64_t a, uint64_t b) {
    uint64_t r;
    asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
    return r;
}
__device__ __forceinline__ uint64_t pf_add2(uint64_t a, uint64_t b) {
    uint64_t r;
    asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
    return r;
}
// P = 2^(score * key norm - m) * value norm as fp16 pairs, its sum without the value norms, and the largest exponent.
template <bool MASKED>
__device__ __forceinline__ void pf_probabilities(uint32_t S, uint32_t nk, uint32_t nv, int room, float m, uint32_t (&P)[PF_KV / 32][16],
                                                 float& over, float& sum) {
    float mx = PF_NEG_INF;
    const uint64_t m2 = pf_two(-m, -m);
    uint64_t l2[2] = {0, 0};
#pragma unroll
    for (int c = 0; c < PF_KV; c += 16) {
        uint32_t v[16];
        tmem_ld16(S + c, v);
#pragma unroll
        for (int i = 0; i < 16; i += 4) {
            const float4 a = pf_lds128(nk + 4 * (c + i)), b = pf_lds128(nv + 4 * (c + i));
            const uint64_t an[2] = {pf_two(a.x, a.y), pf_two(a.z, a.w)}, bn[2] = {pf_two(b.x, b.y), pf_two(b.z, b.w)};
#pragma unroll
            for (int e = 0; e < 2; e++) {
                float x0, x1, q0, q1;
                pf_split(pf_fma2(pf_two(__uint_as_float(v[i + 2 * e]), __uint_as_float(v[i + 2 * e + 1])), an[e], m2), x0, x1);
                if (MASKED && c + i + 2 * e >= room) x0 = PF_NEG_INF;
                if (MASKED && c + i + 2 * e + 1 >= room) x1 = PF_NEG_INF;
                mx = fmaxf(mx, fmaxf(x0, x1));
                const uint64_t pr = pf_two(pf_ex2(x0), pf_ex2(x1));
                l2[e] = pf_add2(l2[e], pr);
                pf_split(pf_mul2(pr, bn[e]), q0, q1);
                if (MASKED && c + i + 2 * e >= room) q0 = 0.0f;              // (a slot behind the length may hold anything)
                if (MASKED && c + i + 2 * e + 1 >= room) q1 = 0.0f;
                P[c / 32][((c & 16) + i) / 2 + e] = pack_half2_sat(q0, q1);
            }
        }
    }
    over = mx;
    float s0, s1;
    pf_split(pf_add2(l2[0], l2[1]), s0, s1);
    sum = s0 + s1;
}

// ---- the kernel --------------------------------------------------------------------------------------
// Item number `round` of this CTA: forwards and backwards through the sorted list in turn.
struct PfItem {
    int r, h, t0, n[2], rows_tok[2], kvlen;               // n: key tiles of each query tile; rows_tok: its tokens
    PfReq q;
    __device__ __forceinline__ bool get(const PrefillParams& p, int total, int round) {
        const int64_t i = (int64_t)round * gridDim.x + ((round & 1) ? (int)gridDim.x - 1 - (int)blockIdx.x : (int)blockIdx.x);
        if (i >= total) return false;
        const int2 it = p.items[i / p.kv_heads];
        r = it.x; h = (int)(i % p.kv_heads);
        q = pf_request(p, r);
        t0 = it.y * 2 * p.tpt;
        kvlen = 0;
#pragma unroll
        for (int w = 0; w < 2; w++) {
            const int lo = t0 + w * p.tpt;
            rows_tok[w] = max(0, min(p.tpt, q.qlen - lo));
            const int limit = rows_tok[w] ? pf_limit(p, q, lo + rows_tok[w] - 1) : 0;
            n[w] = (limit + PF_KV - 1) / PF_KV;
            kvlen = max(kvlen, limit);
        }
        return true;
    }
    __device__ __forceinline__ int tiles() const { return max(n[0], n[1]); }
};

template <int D, int KB, int VB, typename T>
__global__ void __launch_bounds__(PF_THREADS, 1) prefill_kernel(const PrefillParams p) {
    using C = PfCfg<D, KB, VB>;
    constexpr bool TWO = sizeof(T) == 4;                  // float32 queries: two fp16 terms
    constexpr int KBLK = D / 64;
    extern __shared__ uint8_t smem_unaligned[];
    const uint32_t raw = smem_u32(smem_unaligned);
    const uint32_t base = (raw + 1023u) & ~1023u;
    uint8_t* const sm = smem_unaligned + (base - raw);
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;

    const uint32_t bar0 = base + C::OFF_BAR;
    auto full = [&](uint32_t b) { return bar0 + 8 * b; };                  // ring buffer written
    auto free_ = [&](uint32_t b) { return bar0 + 8 * (3 + b); };           // ring buffer read by the MMAs
    auto s_full = [&](int w) { return bar0 + 8 * (6 + w); };               // a product for the tile's warps is in S
    auto p_full = [&](int w) { return bar0 + 8 * (8 + w); };               // their operand (Q, P, O terms) is written
    auto o_done = [&](int w) { return bar0 + 8 * (10 + w); };              // P V of a key tile has been added
    auto nrm_full = [&](int s) { return bar0 + 8 * (12 + s); };            // norms of a key tile
    const uint32_t tmem_slot = bar0 + 128;
    if (threadIdx.x == 0) {
        for (int b = 0; b < PF_RING; b++) { mbar_init(full(b), PF_DEC); mbar_init(free_(b), 1); }
        for (int w = 0; w < 2; w++) { mbar_init(s_full(w), 1); mbar_init(p_full(w), 4); mbar_init(o_done(w), 1); mbar_init(nrm_full(w), PF_DEC); }
    }
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    if (warp == 8 + PF_DEC) tmem_alloc(tmem_slot, 512);

    // tables: entry x holds the fp16 centroids of codes (x mod 2^b, x >> b)
    for (int e = threadIdx.x; e < (C::LUTK >> 2); e += PF_THREADS) {
        const int x = e >> (C::KSH - 2);
        *reinterpret_cast<uint32_t*>(sm + C::OFF_LUTK + 4 * e) = pack_half2(__ldg(p.cent_k + (x & ((1 << KB) - 1))), __ldg(p.cent_k + (x >> KB)));
    }
    for (int e = threadIdx.x; e < (C::LUTV >> 2); e += PF_THREADS) {
        const int x = e >> (C::VSH - 2);
        *reinterpret_cast<uint32_t*>(sm + C::OFF_LUTV + 4 * e) = pack_half2(__ldg(p.cent_v + (x & ((1 << VB) - 1))), __ldg(p.cent_v + (x >> VB)));
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = lds32v(tmem_slot);
    pdl_wait();                                            // the plan and the step's new records
    const int total = *p.n_items * p.kv_heads;
    bool ok = true;

    if (warp < 8) {
        // ================= query tiles: thread = row =================
        // registers: 544 threads start with 96 each; 2 x 128 x 120 + 2 x 128 x 72 + 32 x 96 is exactly their sum
        asm volatile("setmaxnreg.inc.sync.aligned.u32 120;");
        const int w = warp >> 2, row = (warp & 3) * 32 + lane;
        const uint32_t qtile = base + C::OFF_Q + w * C::QTILE;
        const uint32_t lanes = (uint32_t)((warp & 3) * 32) << 16;
        const uint32_t S = tmem + lanes + C::S_COL + w * 128, O = tmem + lanes + C::O_COL + w * 128;
        const float unk = p.unscale[0], unv = p.unscale[1];
        uint32_t s_ph = 0, o_ph = 0, jt = 0;               // phases of s_full and o_done; key tiles so far
        auto wait = [&](uint32_t bar, uint32_t parity) {
            ok = __all_sync(0xffffffffu, mbar_wait(bar, parity)) && ok;
            tc_fence_after();
            return ok;
        };
        auto hand_over = [&]() {                           // operand written: generic and tensor-memory stores
            asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
            tc_fence_before();
            __syncwarp();
            if (lane == 0) pf_arrive(p_full(w));
        };
        PfItem it;
        for (int round = 0; ok && it.get(p, total, round); round++) {
            const int tok = row / p.group, head = row - tok * p.group;
            const bool live = tok < it.rows_tok[w];
            const int t = it.t0 + w * p.tpt + tok;
            const int64_t at = ((int64_t)(it.q.q0 + t) * p.q_heads + it.h * p.group + head) * D;
            const int limit = live ? pf_limit(p, it.q, t) : 0;
            const int n = it.n[w];
            if (n == 0) {                                  // nothing attended
                if (live)
                    for (int k = 0; k < D * (int)sizeof(T) / 16; k++) reinterpret_cast<uint4*>(reinterpret_cast<T*>(p.out) + at)[k] = make_uint4(0, 0, 0, 0);
                jt += it.tiles();
                continue;
            }
            // ---- Q' = R_k q, scaled ----
            {
                const T* qr = reinterpret_cast<const T*>(p.query) + at;
                float mx = 0.0f;
                if (live)
#pragma unroll 4
                    for (int k = 0; k < D; k += 8) {
                        float v[8];
                        pf_load8<T>(qr + k, v);
#pragma unroll
                        for (int i = 0; i < 8; i++) mx = fmaxf(mx, fabsf(v[i]));
                    }
                const float sc = fp16_scale(mx);
                auto src = [&](int k, float (&v)[8]) {
                    if (live) {
                        pf_load8<T>(qr + k, v);
#pragma unroll
                        for (int i = 0; i < 8; i++) v[i] *= sc;
                    } else {
#pragma unroll
                        for (int i = 0; i < 8; i++) v[i] = 0.0f;
                    }
                };
                if (TWO) {
                    pf_write_row<D, true>(qtile, row, src);
                    hand_over();
                    if (!wait(s_full(w), s_ph++ & 1)) break;
                }
                pf_write_row<D, false>(qtile, row, src);
                hand_over();
                if (!wait(s_full(w), s_ph++ & 1)) break;
                const float f = unk / sc * p.scale_log2;
#pragma unroll 1
                for (int c = 0; c < D; c += 32) {
                    uint32_t v[32];
                    tmem_ld32(S + c, v);
#pragma unroll
                    for (int i = 0; i < 32; i += 8) {
                        uint32_t h[4];
#pragma unroll
                        for (int e = 0; e < 4; e++) h[e] = pack_half2_sat(__uint_as_float(v[i + 2 * e]) * f, __uint_as_float(v[i + 2 * e + 1]) * f);
                        const int k = c + i;
                        pf_sts128(qtile + (uint32_t)(k >> 6) * (PF_ROWS * 128) + sw128_offset(row, k & 63), h[0], h[1], h[2], h[3]);
                    }
                }
                hand_over();
            }
            // ---- key tiles ----
            float m = 0.0f, l = 0.0f, move = 0.0f;         // move: of the maximum, due before the next tile
            int j = 0;
            auto rescale = [&](float f) {                  // of what tiles before j have accumulated
                l *= f;
                if (!wait(o_done(w), (o_ph + j - 1) & 1)) return;
#pragma unroll 1
                for (int c = 0; c < D; c += 32) {
                    uint32_t v[32];
                    tmem_ld32(O + c, v);
#pragma unroll
                    for (int i = 0; i < 32; i++) v[i] = __float_as_uint(__uint_as_float(v[i]) * f);
                    tmem_st32(O + c, v);
                }
            };
            const int low = __reduce_min_sync(0xffffffffu, live ? limit : 0x7fffffff);
#pragma unroll 1
            for (; j < n; j++) {
                if (!wait(s_full(w), s_ph++ & 1)) break;
                if (__any_sync(0xffffffffu, move > 0.0f)) {
                    m += move;
                    rescale(pf_ex2(-move));
                    if (!ok) break;
                }
                const uint32_t slot = (jt + j) & 1;
                if (!wait(nrm_full(slot), ((jt + j) >> 1) & 1)) break;
                const uint32_t nk = base + C::OFF_NRM + slot * (2 * PF_KV * 4), nv = nk + PF_KV * 4;
                const int room = limit - j * PF_KV;        // tokens of this tile that the row attends
                const bool masked = (j + 1) * PF_KV > low;
                if (j == 0) {                              // the first tile sets the maximum outright
                    const float mx = masked ? pf_row_max<true>(S, nk, room) : pf_row_max<false>(S, nk, room);
                    m = mx == PF_NEG_INF ? 0.0f : mx;
                }
                // One pass with the maximum so far.  Exponents above it do no harm while P stays a finite fp16 number: then the
                // maximum moves after the tile, and everything accumulated shrinks before the next one.  Otherwise (tokens far
                // above all before them) it moves at once and the tile's P, still in registers, is made again.
                uint32_t P[PF_KV / 32][16];
                float over, sum;
                if (masked) pf_probabilities<true>(S, nk, nv, room, m, P, over, sum);
                else pf_probabilities<false>(S, nk, nv, room, m, P, over, sum);
                move = 0.0f;
                if (j > 0 && __any_sync(0xffffffffu, over > PF_SAFE)) {
                    const float4 b = pf_lds128(nv + 16 * lane);
                    const int first = j * PF_KV + 4 * lane;                                      // (behind the length: anything)
                    float top = 0.0f;
                    if (first < it.kvlen) top = b.x;
                    if (first + 1 < it.kvlen) top = fmaxf(top, b.y);
                    if (first + 2 < it.kvlen) top = fmaxf(top, b.z);
                    if (first + 3 < it.kvlen) top = fmaxf(top, b.w);
                    top = __uint_as_float(__reduce_max_sync(0xffffffffu, __float_as_uint(top)));  // (norms are not negative)
                    if (__any_sync(0xffffffffu, !(pf_ex2(over) * top < PF_HALF_MAX))) {
                        const float d = fmaxf(over, 0.0f);
                        m += d;
                        rescale(pf_ex2(-d));
                        pf_probabilities<true>(S, nk, nv, room, m, P, over, sum);
                    } else {
                        move = over > PF_SLACK ? over : 0.0f;
                    }
                }
                l += sum;
                if (!ok) break;
#pragma unroll
                for (int c = 0; c < PF_KV / 32; c++) tmem_st16(S + 16 * c, P[c]);  // P takes the place of the scores
                tmem_wait_st();
                tc_fence_before();
                __syncwarp();
                if (lane == 0) pf_arrive(p_full(w));
            }
            if (!ok) break;
            jt += it.tiles();
            // ---- out = (O / l) R_v ----
            o_ph += n;
            if (!wait(o_done(w), (o_ph - 1) & 1)) break;
            const float inv = l > 0.0f ? 1.0f / l : 0.0f;
            float mx = 0.0f;
#pragma unroll 1
            for (int c = 0; c < D; c += 32) {
                uint32_t v[32];
                tmem_ld32(O + c, v);
#pragma unroll
                for (int i = 0; i < 32; i++) mx = fmaxf(mx, fabsf(__uint_as_float(v[i]) * inv));
            }
            const float sc = fp16_scale(mx);
            auto terms = [&](auto low_term) {
#pragma unroll 1
                for (int c = 0; c < D; c += 32) {
                    uint32_t v[32];
                    tmem_ld32(O + c, v);
#pragma unroll
                    for (int i = 0; i < 32; i += 8) {
                        uint32_t h[4];
#pragma unroll
                        for (int e = 0; e < 4; e++)
                            h[e] = pf_term<decltype(low_term)::value>(__uint_as_float(v[i + 2 * e]) * inv * sc, __uint_as_float(v[i + 2 * e + 1]) * inv * sc);
                        const int k = c + i;
                        pf_sts128(qtile + (uint32_t)(k >> 6) * (PF_ROWS * 128) + sw128_offset(row, k & 63), h[0], h[1], h[2], h[3]);
                    }
                }
                hand_over();
            };
            terms(std::true_type{});
            if (!wait(s_full(w), s_ph++ & 1)) break;
            terms(std::false_type{});
            if (!wait(s_full(w), s_ph++ & 1)) break;
            const float f = unv / sc;
            T* orow = reinterpret_cast<T*>(p.out) + at;
#pragma unroll 1
            for (int c = 0; c < D; c += 32) {
                uint32_t v[32];
                tmem_ld32(S + c, v);
                if (live) {
                    if constexpr (TWO) {
#pragma unroll
                        for (int i = 0; i < 32; i += 4)
                            *reinterpret_cast<float4*>(orow + c + i) = make_float4(__uint_as_float(v[i]) * f, __uint_as_float(v[i + 1]) * f,
                                                                                   __uint_as_float(v[i + 2]) * f, __uint_as_float(v[i + 3]) * f);
                    } else {
#pragma unroll
                        for (int i = 0; i < 32; i += 8) {
                            uint32_t h[4];
#pragma unroll
                            for (int e = 0; e < 4; e++)
                                h[e] = pf_pack(__uint_as_float(v[i + 2 * e]) * f, __uint_as_float(v[i + 2 * e + 1]) * f, (T*)nullptr);
                            *reinterpret_cast<uint4*>(orow + c + i) = make_uint4(h[0], h[1], h[2], h[3]);
                        }
                    }
                }
                __syncwarp();
            }
            tc_fence_before();
        }
    } else if (warp < 8 + PF_DEC) {
        // ================= decode =================
        asm volatile("setmaxnreg.dec.sync.aligned.u32 72;");
        const int dw = warp - 8, g = lane >> 2, t = lane & 3;
        const uint32_t tabk = base + C::OFF_LUTK + lane * 4, tabv = base + C::OFF_LUTV + (lane & ((1 << (C::VSH - 2)) - 1)) * 4;
        uint32_t seq = 0, jt = 0;                          // ring fills and key tiles so far
        auto claim = [&]() {                               // the next ring buffer, once the MMAs have read it
            const uint32_t b = seq % PF_RING;
            if (seq >= PF_RING) ok = __all_sync(0xffffffffu, mbar_wait(free_(b), ((seq / PF_RING) - 1) & 1)) && ok;
            return b;
        };
        auto put_rotation = [&](int which) {               // both terms of R_k or R_v^T: ready images, one bulk copy each
#pragma unroll 1
            for (int term = 0; term < 2; term++, seq++) {
                const uint32_t b = claim();
                if (!ok) return;
                if (lane == 0) {
                    if (dw == 0) {
                        mbar_expect_tx(full(b), C::RTERM);
                        bulk_g2s(base + C::OFF_RING + b * C::BUF, p.images + (2 * which + term) * C::RTERM, C::RTERM, full(b));
                    } else {
                        pf_arrive(full(b));
                    }
                }
                __syncwarp();
            }
        };
        const int page_recs = p.block_size / 16;
        PfItem it;
        for (int round = 0; ok && it.get(p, total, round); round++) {
            const int tiles = it.tiles();
            if (tiles == 0) continue;
            const int32_t* table = p.block_tables + (int64_t)it.r * p.max_blocks;
            auto record = [&](int j) -> const uint8_t* {   // this warp's record of key tile j, null behind the length
                const int rec = j * (PF_KV / 16) + dw;
                if (rec * 16 >= it.kvlen) return nullptr;
                const int blk = rec / page_recs;
                return p.store + (((int64_t)__ldg(table + blk) * p.kv_heads + it.h) * page_recs + (rec - blk * page_recs)) * C::REC;
            };
            PfRecord<D, KB, VB> now, next;
            now.load(record(0), lane);
            const uint8_t* ahead = tiles > 1 ? record(1) : nullptr;
            put_rotation(0);
#pragma unroll 1
            for (int j = 0; ok && j < tiles; j++, jt++) {
                next.load(ahead, lane);                    // (null: zeros)
                ahead = j + 2 < tiles ? record(j + 2) : nullptr;
                {
                    const uint32_t b = claim();
                    if (!ok) break;
                    // norm `lane` of the record: token g or g+8, key or value
                    const int r = (lane >> 2) + 8 * (lane & 1), vside = (lane >> 1) & 1;
                    pf_sts32(base + C::OFF_NRM + (jt & 1) * (2 * PF_KV * 4) + vside * (PF_KV * 4) + 4 * (16 * dw + r), now.norm);
                    const uint32_t at = base + C::OFF_RING + b * C::BUF + (16 * dw + g) * 128 + (g << 4) + 4 * t;
#pragma unroll
                    for (int e = 0; e < D / 8; e++)
#pragma unroll
                        for (int second = 0; second < 2; second++) {
                            const uint32_t f = pf_field(now.k, tl_key_field_bit(D, KB, e >> 1, e & 1, second), 2 * KB);
                            pf_sts32((at ^ ((uint32_t)(e & 7) << 4)) + (e >> 3) * (PF_KV * 128) + second * 1024, lds32(tabk + (f << C::KSH)));
                        }
                    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
                    __syncwarp();
                    if (lane == 0) { pf_arrive(nrm_full(jt & 1)); pf_arrive(full(b)); }
                    seq++;
                }
                {
                    const uint32_t b = claim();
                    if (!ok) break;
                    // V^T: rows = dims, 64 tokens per 128-byte line; this warp's 16 tokens are chunks 2 dw, 2 dw + 1
                    const uint32_t at = base + C::OFF_RING + b * C::BUF + (dw >> 2) * (D * 128) + g * 128 + 4 * t;
                    const uint32_t c0 = (uint32_t)(((2 * dw) ^ g) & 7) << 4, c1 = c0 ^ 16u;
#pragma unroll
                    for (int mt = 0; mt < D / 16; mt++)
#pragma unroll
                        for (int half = 0; half < 2; half++)
#pragma unroll
                            for (int rs = 0; rs < 2; rs++) {
                                const uint32_t f = pf_field(now.v, (2 * (2 * mt + half) + rs) * 2 * VB, 2 * VB);
                                pf_sts32(at + (half ? c1 : c0) + (16 * mt + 8 * rs) * 128, lds32(tabv + (f << C::VSH)));
                            }
                    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
                    __syncwarp();
                    if (lane == 0) pf_arrive(full(b));
                    seq++;
                }
                now = next;
            }
            if (ok) put_rotation(1);
        }
        // a bulk copy still in flight must not outlive the block: the waits are bounded here too
        if (!ok && dw == 0 && lane == 0)
            for (uint32_t i = seq > PF_RING ? seq - PF_RING : 0; i < seq; i++) (void)mbar_wait(full(i % PF_RING), (i / PF_RING) & 1);
        __syncwarp();
    } else if (lane == 0) {
        // ================= MMA issuer (one lane) =================
        constexpr uint32_t IDESC_M = (1u << 4) | ((uint32_t)(PF_ROWS >> 4) << 24);     // fp16 x fp16 -> f32, 128 rows
        constexpr uint32_t ID_S = IDESC_M | ((uint32_t)(PF_KV >> 3) << 17), ID_D = IDESC_M | ((uint32_t)(D >> 3) << 17);
        uint32_t seq = 0, p_ph[2] = {0, 0};
        auto wait = [&](uint32_t bar, uint32_t parity) {
            if (ok) ok = pf_wait_spin(bar, parity);
            tc_fence_after();
            return ok;
        };
        auto wait_full = [&](uint32_t s) { return wait(full(s % PF_RING), (s / PF_RING) & 1); };
        auto wait_p = [&](int w) { return wait(p_full(w), p_ph[w]++ & 1); };
        auto buf = [&](uint32_t s) { return base + C::OFF_RING + (s % PF_RING) * C::BUF; };
        auto qt = [&](int w) { return base + C::OFF_Q + w * C::QTILE; };
        // S[w] (+)= tile [128][D] times a [rows_b][D] operand
        auto product = [&](int w, uint32_t bm, int rows_b, uint32_t idesc, uint32_t acc) {
#pragma unroll
            for (int kb = 0; kb < KBLK; kb++) {
                const uint64_t ad = umma_desc(qt(w) + kb * (PF_ROWS * 128)), bd = umma_desc(bm + kb * (rows_b * 128));
#pragma unroll
                for (int k = 0; k < 4; k++) { umma_f16(tmem + C::S_COL + w * 128, ad + 2 * k, bd + 2 * k, idesc, acc); acc = 1; }
            }
        };
        // rotation of the tiles' rows: low term first, then the high one; S holds the result
        auto rotate = [&](const PfItem& it, bool two) {
            if (!wait_full(seq) || !wait_full(seq + 1)) return;
            if (two)
                for (int w = 0; w < 2; w++) {
                    if (!it.n[w]) continue;
                    if (!wait_p(w)) return;
                    product(w, buf(seq), D, ID_D, 0);
                    umma_commit(s_full(w));
                }
            for (int w = 0; w < 2; w++) {
                if (!it.n[w]) continue;
                if (!wait_p(w)) return;
                product(w, buf(seq + 1), D, ID_D, two ? 1 : 0);
                product(w, buf(seq), D, ID_D, 1);
                if (w == 1 || !it.n[1]) { umma_commit(free_(seq % PF_RING)); umma_commit(free_((seq + 1) % PF_RING)); }
                umma_commit(s_full(w));
            }
            seq += 2;
        };
        PfItem it;
        for (int round = 0; ok && it.get(p, total, round); round++) {
            const int tiles = it.tiles();
            if (tiles == 0) continue;
            // the last tile that takes part in key tile j frees the buffers
            auto last = [&](int w, int j) { return w == 1 || j >= it.n[1]; };
            rotate(it, TWO);
            if (!ok) break;
            for (int w = 0; w < 2; w++) {
                if (!it.n[w]) continue;
                if (!wait_p(w) || !wait_full(seq)) break;
                product(w, buf(seq), PF_KV, ID_S, 0);
                if (last(w, 0)) umma_commit(free_(seq % PF_RING));
                umma_commit(s_full(w));
            }
#pragma unroll 1
            for (int j = 0; ok && j < tiles; j++, seq += 2)
                for (int w = 0; w < 2; w++) {
                    if (j >= it.n[w]) continue;
                    if (!wait_p(w) || !wait_full(seq + 1)) break;
                    const uint32_t vb = buf(seq + 1);
#pragma unroll
                    for (int k = 0; k < PF_KV / 16; k++)
                        umma_f16_ta(tmem + C::O_COL + w * 128, tmem + C::S_COL + w * 128 + 8 * k, umma_desc(vb + (k >> 2) * (D * 128)) + 2 * (k & 3), ID_D,
                                    j > 0 || k > 0);
                    if (last(w, j)) umma_commit(free_((seq + 1) % PF_RING));
                    umma_commit(o_done(w));
                    if (j + 1 < it.n[w]) {
                        if (!wait_full(seq + 2)) break;
                        product(w, buf(seq + 2), PF_KV, ID_S, 0);
                        if (last(w, j + 1)) umma_commit(free_((seq + 2) % PF_RING));
                        umma_commit(s_full(w));
                    }
                }
            if (!ok) break;
            rotate(it, true);
        }
    }
    if (!ok && lane == 0) atomicOr(p.status, TQB_DECODE_WAIT_EXPIRED);
    __syncwarp();
    tc_fence_before();
    __syncthreads();
    if (warp == 8 + PF_DEC) {
        tc_fence_after();
        tmem_dealloc(tmem, 512);
    }
}

template <int D, int KB, int VB, typename T>
static int launch_prefill(const PrefillParams& p, cudaStream_t st) {
    using C = PfCfg<D, KB, VB>;
    auto kern = prefill_kernel<D, KB, VB, T>;
    TQB_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, C::TOTAL));
    prefill_plan_kernel<D><<<PF_PLAN_BLOCKS, PF_PLAN_THREADS, 0, st>>>(p);
    if (int e = check_launch("prefill_plan")) return e;
    const int grid = (int)std::min<int64_t>(sm_count(), (int64_t)p.item_cap * p.kv_heads);
    TQB_CUDA(launch_pdl(1, kern, dim3(grid), dim3(PF_THREADS), C::TOTAL, st, p));
    return check_launch("prefill");
}
template <int D, typename T>
static int prefill_bits(int kbits, int vbits, const PrefillParams& p, cudaStream_t st) {
#define TQB_CASE(kb, vb) if (kbits == kb && vbits == vb) return launch_prefill<D, kb, vb, T>(p, st);
    TQB_CASE(4, 2) TQB_CASE(4, 3) TQB_CASE(4, 4)
    TQB_CASE(3, 2) TQB_CASE(3, 3) TQB_CASE(3, 4)
    TQB_CASE(2, 2) TQB_CASE(2, 3) TQB_CASE(2, 4)
#undef TQB_CASE
    return fail(TQB_ERR_UNSUPPORTED, "prefill_attention: key/value bits must be 2..4, got %d/%d", kbits, vbits);
}

struct PrefillWorkspace { size_t off_scale, off_images, off_items, total; int item_cap; };
static PrefillWorkspace plan_prefill(int64_t n_tokens, int num_reqs, int group, int dim) {
    PrefillWorkspace w;
    const int64_t span = 2 * (PF_ROWS / group);
    w.item_cap = (int)std::min<int64_t>(n_tokens / span + num_reqs, 0x7fffffff);
    w.off_scale = 16;
    w.off_images = 256;
    w.off_items = w.off_images + (size_t)8 * dim * dim;
    w.total = w.off_items + (size_t)w.item_cap * sizeof(int2);
    return w;
}

}  // namespace tqb

extern "C" size_t tqb_prefill_attention_workspace_bytes(int64_t n_tokens, int num_reqs, int q_heads, int kv_heads, int dim) {
    if (n_tokens <= 0 || num_reqs <= 0 || kv_heads <= 0 || q_heads <= 0 || q_heads % kv_heads || q_heads / kv_heads > 8) return 0;
    if (dim != 64 && dim != 128) return 0;
    return tqb::plan_prefill(n_tokens, num_reqs, q_heads / kv_heads, dim).total;
}

extern "C" int tqb_prefill_attention(const void* query, int dtype, int64_t n_tokens, int num_reqs, int q_heads, int kv_heads, int dim,
                                     const uint8_t* store, const int32_t* query_start, int first_token, const int32_t* seq_lens, int64_t max_len,
                                     const int32_t* block_tables, int max_blocks, int block_size, int causal, const float* rot_k,
                                     const float* cent_k, int kbits, const float* rot_v, const float* cent_v, int vbits, float scale,
                                     int32_t* status, void* workspace, size_t workspace_bytes, void* out, void* stream) {
    using namespace tqb;
    TQB_REQUIRE(n_tokens >= 0 && num_reqs >= 0 && q_heads > 0 && kv_heads > 0, "prefill_attention: bad sizes");
    TQB_REQUIRE(q_heads % kv_heads == 0, "prefill_attention: q_heads (%d) must be a multiple of kv_heads (%d)", q_heads, kv_heads);
    const int group = q_heads / kv_heads;
    if (dim != 64 && dim != 128) return fail(TQB_ERR_UNSUPPORTED, "prefill_attention: head_dim must be 64 or 128, got %d", dim);
    if (group > 8) return fail(TQB_ERR_UNSUPPORTED, "prefill_attention: at most 8 query heads per KV head, got %d", group);
    if (kbits < 2 || kbits > 4 || vbits < 2 || vbits > 4)
        return fail(TQB_ERR_UNSUPPORTED, "prefill_attention: key/value bits must be 2..4, got %d/%d", kbits, vbits);
    TQB_REQUIRE(dtype == TQB_F32 || dtype == TQB_F16 || dtype == TQB_BF16, "prefill_attention: unknown dtype %d", dtype);
    TQB_REQUIRE(max_len >= 0, "prefill_attention: negative max_len");
    if (max_len > ((int64_t)1 << 30) - PF_KV || n_tokens > 0x7fffffff)
        return fail(TQB_ERR_UNSUPPORTED, "prefill_attention: too many tokens");
    if (n_tokens == 0 || num_reqs == 0) return TQB_OK;
    TQB_REQUIRE(query && store && query_start && seq_lens && block_tables && rot_k && cent_k && rot_v && cent_v && status && workspace && out,
                "prefill_attention: null pointer");
    TQB_REQUIRE(block_size > 0 && block_size % 16 == 0, "prefill_attention: block_size must be a multiple of 16, got %d", block_size);
    TQB_REQUIRE(max_blocks > 0 && (int64_t)max_blocks * block_size >= max_len, "prefill_attention: block table shorter than max_len");
    TQB_REQUIRE(((uintptr_t)store | (uintptr_t)query | (uintptr_t)out | (uintptr_t)rot_k | (uintptr_t)rot_v) % 16 == 0,
                "prefill_attention: store, query, out and the rotations must be 16-byte aligned");
    TQB_REQUIRE((uintptr_t)workspace % 256 == 0, "prefill_attention: workspace must be 256-byte aligned");
    const PrefillWorkspace w = plan_prefill(n_tokens, num_reqs, group, dim);
    if (workspace_bytes < w.total)
        return fail(TQB_ERR_WORKSPACE, "prefill_attention: workspace %zu bytes < required %zu", workspace_bytes, w.total);
    if ((int64_t)w.item_cap * kv_heads + sm_count() >= 0x7fffffff)
        return fail(TQB_ERR_UNSUPPORTED, "prefill_attention: too many (request, head, block) work items");
    uint8_t* ws = reinterpret_cast<uint8_t*>(workspace);
    PrefillParams p{};
    p.query = query; p.out = out; p.store = store; p.qstart = query_start; p.seq_lens = seq_lens; p.block_tables = block_tables;
    p.cent_k = cent_k; p.cent_v = cent_v; p.rot_k = rot_k; p.rot_v = rot_v; p.n_tokens = n_tokens; p.first_token = first_token; p.max_len = max_len;
    p.num_reqs = num_reqs; p.q_heads = q_heads; p.kv_heads = kv_heads; p.group = group; p.tpt = PF_ROWS / group;
    p.max_blocks = max_blocks; p.block_size = block_size; p.causal = causal; p.scale_log2 = scale * PF_LOG2E; p.status = status;
    p.n_items = reinterpret_cast<int*>(ws); p.unscale = reinterpret_cast<float*>(ws + w.off_scale);
    p.images = ws + w.off_images; p.items = reinterpret_cast<int2*>(ws + w.off_items); p.item_cap = w.item_cap;
    cudaStream_t st = (cudaStream_t)stream;
    if (dim == 64) {
        if (dtype == TQB_F32) return prefill_bits<64, float>(kbits, vbits, p, st);
        return dtype == TQB_F16 ? prefill_bits<64, __half>(kbits, vbits, p, st) : prefill_bits<64, __nv_bfloat16>(kbits, vbits, p, st);
    }
    if (dtype == TQB_F32) return prefill_bits<128, float>(kbits, vbits, p, st);
    return dtype == TQB_F16 ? prefill_bits<128, __half>(kbits, vbits, p, st) : prefill_bits<128, __nv_bfloat16>(kbits, vbits, p, st);
}
