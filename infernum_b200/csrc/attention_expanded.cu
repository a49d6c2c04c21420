// Prompt attention through a latent with the keys and values made (bf16, tcgen05), for a head of EX_D unrotated and
// EX_R rotated query/key dimensions and values of EX_V (-DEX_D=128 -DEX_R=64 -DEX_V=128).
//
// Over the cached latents themselves (attention_latent_mma.cu) a query and a key cost 2 (2 kv_rank + rot) multiply-adds
// a head, 1,088 at a latent of 512; with the head's key W_uk c and value W_uv c made once per cached vector - one product
// over the step's keys - they cost EX_D + EX_R + EX_V = 320.  A prompt has enough queries for every key to pay for it.
//
// A CTA owns 128 query rows of one head and walks the keys in tiles of 128:
//   producer warp   TMA: the queries once (unrotated part from the projection's rows, rotated part from its own
//                   array), then per tile the keys (unrotated part from the made keys, the rotated part, which
//                   all heads share, from the gathered latents) and the values
//   MMA warp        S = Q K^T into tensor memory (12 MMAs of 128 x 128 x 16), O += P V (8 of 128 x EX_V x 16, P from
//                   tensor memory)
//   4 softmax warps one thread a query row = TMEM lane, 128 scores in registers, exactly as in attention_tcgen05.cu
// Scores, keys and values are double-buffered: the scores of tile t + 1 are computed while the softmax warps work on
// tile t.  Key tiles of 128 because an MMA of 64 columns takes as long as one of 128 (107 cycles, attention_tcgen05.cu's
// measurement); they fill the SM's shared memory (213 KB) with one CTA.
// 2,048 tokens, 32 heads, one layer: 1,085 us over the latents -> 67 us here, and 32 us for the gathered
// latents and the product.
//
// Every wait is bounded.  The grid has the head on x, the request on y, the row tile on z, the last rows first.
#include "common.cuh"

#include <cuda.h>

using namespace ib;

namespace {

constexpr int D = EX_D, R = EX_R, VD = EX_V;
static_assert((D == 64 || D == 128) && R == 64 && (VD == 64 || VD == 128), "blocks of 64 elements");
constexpr int BM = 128;                 // query rows per CTA
constexpr int BN = 128;                 // keys per tile
constexpr int DB = D / 64, KB = DB + 1, VB = VD / 64;   // blocks of 64 elements of a key (the last one rotated), a value
constexpr int SOFTMAX_WARPS = 4;
constexpr int SOFTMAX_THREADS = SOFTMAX_WARPS * 32;
constexpr int PRODUCER_WARP = SOFTMAX_WARPS, MMA_WARP = SOFTMAX_WARPS + 1;
constexpr int NUM_THREADS = SOFTMAX_THREADS + 64;
constexpr int BLOCK_BYTES = 128 * 128;  // 128 rows of 64 elements
constexpr int Q_BYTES = KB * BLOCK_BYTES, K_BYTES = KB * BLOCK_BYTES, V_BYTES = VB * BLOCK_BYTES;
constexpr int TILE_BYTES = Q_BYTES + 2 * K_BYTES + 2 * V_BYTES;
constexpr int BAR_BYTES = 128;
constexpr int SMEM_BYTES = TILE_BYTES + BAR_BYTES + 1024;
static_assert(SMEM_BYTES <= 232448, "one CTA must fit an SM");
constexpr unsigned TMEM_COLS = 512;     // two score tiles in columns [0, 128) and [128, 256), output from 256
constexpr unsigned O_COL = 256;

struct Params {
    bf16* out;
    const int* cu_rows;
    const int* q_start;
    unsigned* err;
    const float* sink;   // optional [nh]
    const bf16* gate;    // optional: head h of row n is multiplied by sigmoid(gate[n * gate_stride + h])
    int gate_stride, out_stride, nh, window, v_col, r_col;   // where the values and the rotated keys begin in their rows
    float scale_log2;
};

// What a row's accumulated values are multiplied by at the end: 1 / l, or, with a sink (a learned
// logit of the head, not scaled, with no key and no value), 1 / (l + exp(sink - m)).  `m2` is the
// row's reference maximum in the exponent's units (score * scale * log2 e), `l` the sum of
// exp2(score - reference); nothing seen (l = 0, m2 = -inf or unused) gives 0.
__device__ __forceinline__ float inv_denominator(const float* sink, int head, float m2, float l) {
    if (!sink) return l > 0.f ? 1.f / l : 0.f;
    if (!(l > 0.f)) return 0.f;
    const float s2 = sink[head] * 1.4426950408889634f;
    const float top = fmaxf(m2, s2);
    const float c = exp2f(m2 - top);
    return c / (l * c + exp2f(s2 - top));
}

__device__ __forceinline__ unsigned smem_u32(const void* p) { return (unsigned)__cvta_generic_to_shared(p); }
__device__ __forceinline__ bool elect_one() {
    unsigned pred = 0;
    asm volatile("{\n\t.reg .pred p;\n\telect.sync _|p, 0xffffffff;\n\tselp.u32 %0, 1, 0, p;\n\t}\n" : "=r"(pred));
    return pred != 0;
}
__device__ __forceinline__ void mbar_init(void* bar, unsigned count) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;\n" ::"r"(smem_u32(bar)), "r"(count));
}
__device__ __forceinline__ void mbar_expect_tx(void* bar, unsigned bytes) {
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;\n" ::"r"(smem_u32(bar)), "r"(bytes) : "memory");
}
__device__ __forceinline__ void mbar_arrive(void* bar) {
    asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];\n" ::"r"(smem_u32(bar)) : "memory");
}
__device__ __forceinline__ bool mbar_wait(void* bar, unsigned parity) {
    return mbar_wait_bounded<false>(smem_u32(bar), parity);
}
__device__ __forceinline__ void tma_load_2d(void* dst, const CUtensorMap* map, void* bar, int x, int y) {
    asm volatile(
        "cp.async.bulk.tensor.2d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4}], [%2];\n"
        ::"r"(smem_u32(dst)), "l"(map), "r"(smem_u32(bar)), "r"(x), "r"(y) : "memory");
}
__device__ __forceinline__ void tma_load_3d(void* dst, const CUtensorMap* map, void* bar, int x, int y, int z) {
    asm volatile(
        "cp.async.bulk.tensor.3d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4, %5}], [%2];\n"
        ::"r"(smem_u32(dst)), "l"(map), "r"(smem_u32(bar)), "r"(x), "r"(y), "r"(z) : "memory");
}
__device__ __forceinline__ void tc_fence_before() { asm volatile("tcgen05.fence::before_thread_sync;\n" ::: "memory"); }
__device__ __forceinline__ void tc_fence_after() { asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory"); }
__device__ __forceinline__ void umma_bf16(unsigned tmem_d, uint64_t adesc, uint64_t bdesc, unsigned idesc,
                                          unsigned accumulate) {
    asm volatile(
        "{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}\n"
        ::"r"(tmem_d), "l"(adesc), "l"(bdesc), "r"(idesc), "r"(accumulate) : "memory");
}
// The same with the A operand in tensor memory: row i in lane i, two bf16 of
// consecutive k per 32-bit column (k even in the low half), 8 columns per MMA.
__device__ __forceinline__ void umma_bf16_a_tmem(unsigned tmem_d, unsigned tmem_a, uint64_t bdesc, unsigned idesc,
                                                 unsigned accumulate) {
    asm volatile(
        "{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %2, %3, p;\n\t}\n"
        ::"r"(tmem_d), "r"(tmem_a), "l"(bdesc), "r"(idesc), "r"(accumulate) : "memory");
}
__device__ __forceinline__ void umma_commit(void* bar) {
    asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];\n"
                 ::"r"(smem_u32(bar)) : "memory");
}
__device__ __forceinline__ void tmem_ld16(unsigned addr, unsigned (&r)[16]) {
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];\n"
        : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]),
          "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
        : "r"(addr));
}
__device__ __forceinline__ void tmem_st16(unsigned addr, const unsigned (&r)[16]) {
    asm volatile(
        "tcgen05.st.sync.aligned.32x32b.x16.b32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16};\n"
        ::"r"(addr), "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]),
          "r"(r[8]), "r"(r[9]), "r"(r[10]), "r"(r[11]), "r"(r[12]), "r"(r[13]), "r"(r[14]), "r"(r[15])
        : "memory");
}
// Sixty-four consecutive columns of this thread's lane and the wait for them, as
// one statement: the values may be used as soon as it returns, and the four
// loads are in flight together.
__device__ __forceinline__ void tmem_ld64_wait(unsigned addr, float (&r)[64]) {
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%64];\n\t"
        "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%16,%17,%18,%19,%20,%21,%22,%23,%24,%25,%26,%27,%28,%29,%30,%31}, [%65];\n\t"
        "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%32,%33,%34,%35,%36,%37,%38,%39,%40,%41,%42,%43,%44,%45,%46,%47}, [%66];\n\t"
        "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%48,%49,%50,%51,%52,%53,%54,%55,%56,%57,%58,%59,%60,%61,%62,%63}, [%67];\n\t"
        "tcgen05.wait::ld.sync.aligned;\n"
        : "=f"(r[0]), "=f"(r[1]), "=f"(r[2]), "=f"(r[3]), "=f"(r[4]), "=f"(r[5]), "=f"(r[6]), "=f"(r[7]),
          "=f"(r[8]), "=f"(r[9]), "=f"(r[10]), "=f"(r[11]), "=f"(r[12]), "=f"(r[13]), "=f"(r[14]), "=f"(r[15]),
          "=f"(r[16]), "=f"(r[17]), "=f"(r[18]), "=f"(r[19]), "=f"(r[20]), "=f"(r[21]), "=f"(r[22]), "=f"(r[23]),
          "=f"(r[24]), "=f"(r[25]), "=f"(r[26]), "=f"(r[27]), "=f"(r[28]), "=f"(r[29]), "=f"(r[30]), "=f"(r[31]),
          "=f"(r[32]), "=f"(r[33]), "=f"(r[34]), "=f"(r[35]), "=f"(r[36]), "=f"(r[37]), "=f"(r[38]), "=f"(r[39]),
          "=f"(r[40]), "=f"(r[41]), "=f"(r[42]), "=f"(r[43]), "=f"(r[44]), "=f"(r[45]), "=f"(r[46]), "=f"(r[47]),
          "=f"(r[48]), "=f"(r[49]), "=f"(r[50]), "=f"(r[51]), "=f"(r[52]), "=f"(r[53]), "=f"(r[54]), "=f"(r[55]),
          "=f"(r[56]), "=f"(r[57]), "=f"(r[58]), "=f"(r[59]), "=f"(r[60]), "=f"(r[61]), "=f"(r[62]), "=f"(r[63])
        : "r"(addr), "r"(addr + 16), "r"(addr + 32), "r"(addr + 48)
        : "memory");
}
__device__ __forceinline__ void tmem_ld_wait() { asm volatile("tcgen05.wait::ld.sync.aligned;\n" ::: "memory"); }
__device__ __forceinline__ void tmem_st_wait() { asm volatile("tcgen05.wait::st.sync.aligned;\n" ::: "memory"); }
__device__ __forceinline__ float fast_exp2(float x) {
    float y;
    asm("ex2.approx.ftz.f32 %0, %1;\n" : "=f"(y) : "f"(x));
    return y;
}
// Two float32 in one 64-bit register, for the packed arithmetic of sm_100 (one
// instruction, two results): the softmax warps are bound by the instructions
// they issue, not by any arithmetic unit.
__device__ __forceinline__ unsigned long long pack2(float lo, float hi) {
    unsigned long long r;
    asm("mov.b64 %0, {%1, %2};\n" : "=l"(r) : "f"(lo), "f"(hi));
    return r;
}
// (d0, d1) = (a0, a1) * b + c, b and c packed pairs
__device__ __forceinline__ void fma2(float& d0, float& d1, float a0, float a1, unsigned long long b,
                                     unsigned long long c) {
    asm("{\n\t.reg .b64 ra, rd;\n\tmov.b64 ra, {%2, %3};\n\tfma.rn.f32x2 rd, ra, %4, %5;\n\t"
        "mov.b64 {%0, %1}, rd;\n\t}\n"
        : "=f"(d0), "=f"(d1) : "f"(a0), "f"(a1), "l"(b), "l"(c));
}
// acc += (a0, a1), acc a packed pair
__device__ __forceinline__ void add2(unsigned long long& acc, float a0, float a1) {
    asm("{\n\t.reg .b64 ra;\n\tmov.b64 ra, {%1, %2};\n\tadd.rn.f32x2 %0, %0, ra;\n\t}\n"
        : "+l"(acc) : "f"(a0), "f"(a1));
}
__device__ __forceinline__ float sum2(unsigned long long v) {
    float lo, hi;
    asm("mov.b64 {%0, %1}, %2;\n" : "=f"(lo), "=f"(hi) : "l"(v));
    return lo + hi;
}
__device__ __forceinline__ float max3(float a, float b, float c) {
    float d;
    asm("max.f32 %0, %1, %2, %3;\n" : "=f"(d) : "f"(a), "f"(b), "f"(c));
    return d;
}

// K-major operand tile with 128-byte rows and the 128-byte swizzle: groups of 8
// rows are 1024 bytes apart.  (Addresses and offsets in units of 16 bytes;
// version 1; layout type 2 = SWIZZLE_128B.)
__device__ __forceinline__ uint64_t desc_k_major(const void* tile) {
    uint64_t d = 0;
    d |= (uint64_t)((smem_u32(tile) >> 4) & 0x3FFF);
    d |= (uint64_t)1 << 16;
    d |= (uint64_t)(1024 >> 4) << 32;
    d |= (uint64_t)1 << 46;
    d |= (uint64_t)2 << 61;
    return d;
}
// N-major operand (V as [key][dim] rows of 128 bytes, swizzled): along K, groups
// of 8 keys are 1024 bytes apart (stride byte offset); along N, the next block
// of 64 dims starts `block_bytes` further on (leading byte offset).
__device__ __forceinline__ uint64_t desc_n_major(const void* tile, unsigned block_bytes) {
    uint64_t d = 0;
    d |= (uint64_t)((smem_u32(tile) >> 4) & 0x3FFF);
    d |= (uint64_t)((block_bytes >> 4) & 0x3FFF) << 16;
    d |= (uint64_t)(1024 >> 4) << 32;
    d |= (uint64_t)1 << 46;
    d |= (uint64_t)2 << 61;
    return d;
}
// float32 accumulator, bf16 operands, A K-major; B K-major or N-major (bit 16).
__host__ __device__ constexpr unsigned make_idesc(int n, bool b_n_major) {
    return (1u << 4) | (1u << 7) | (1u << 10) | (b_n_major ? (1u << 16) : 0u) |
           ((unsigned)(n >> 3) << 17) | ((unsigned)(BM >> 4) << 24);
}

// The first key of entry e that the buffers hold (a multiple of 128; earlier ones lie behind every row's window), and
// in which row of the buffers it lies: the entries' keys follow one another.
__device__ __forceinline__ int first_key(int q_start, int window) {
    return window > 0 ? max(0, q_start - window + 1) / BN * BN : 0;
}
__device__ __forceinline__ int buffer_row(const int* cu_rows, const int* q_start, int e, int window) {
    int at = 0;
    for (int i = 0; i < e; ++i) {
        const int rows = cu_rows[i + 1] - cu_rows[i];
        if (rows > 0) at += q_start[i] + rows - first_key(q_start[i], window);
    }
    return at;
}

__global__ void __launch_bounds__(NUM_THREADS, 1)
attention_expanded_kernel(const __grid_constant__ CUtensorMap map_q, const __grid_constant__ CUtensorMap map_qr,
                          const __grid_constant__ CUtensorMap map_kv, const __grid_constant__ CUtensorMap map_c,
                          const Params p) {
    extern __shared__ unsigned char smem_dyn[];
    unsigned char* smem = (unsigned char*)(((uintptr_t)smem_dyn + 1023) & ~(uintptr_t)1023);
    unsigned char* q_s = smem;
    unsigned char* k_s = q_s + Q_BYTES;
    unsigned char* v_s = k_s + 2 * K_BYTES;
    unsigned long long* bars = reinterpret_cast<unsigned long long*>(v_s + 2 * V_BYTES);
    unsigned long long& q_full = bars[0];
    unsigned long long* k_full = bars + 1;
    unsigned long long* k_empty = bars + 3;
    unsigned long long* v_full = bars + 5;
    unsigned long long* v_empty = bars + 7;
    unsigned long long* s_full = bars + 9;
    unsigned long long& p_full = bars[11];   // P of tile t is written; every waiter follows every phase
    unsigned long long& o_done = bars[12];   // the output update of tile t is complete
    unsigned& tmem_slot = *reinterpret_cast<unsigned*>(bars + 13);

    pdl_trigger();
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int h = blockIdx.x, e = blockIdx.y;
    const int row0 = p.cu_rows[e];
    const int rows_e = p.cu_rows[e + 1] - row0;
    const int pos0 = p.q_start[e];
    const int r_begin = ((int)gridDim.z - 1 - (int)blockIdx.z) * BM;
    if (r_begin >= rows_e) {
        pdl_wait();  // a CTA without rows too: this grid is not complete before the ones before it are
        return;
    }
    const int r_count = min(BM, rows_e - r_begin);
    const int kv_hi = pos0 + r_begin + r_count;             // keys of this row tile end here
    const int lo = p.window > 0 ? max(0, pos0 + r_begin - p.window + 1) : 0;   // the first row's first key
    const int t_first = lo / BN;
    const int n_tiles = (kv_hi + BN - 1) / BN - t_first;
    const int base = buffer_row(p.cu_rows, p.q_start, e, p.window) - first_key(pos0, p.window);  // buffer row of key 0

    if (threadIdx.x == 0) {
        mbar_init(&q_full, 1);
        for (int i = 0; i < 2; ++i) {
            mbar_init(&k_full[i], 1);
            mbar_init(&k_empty[i], 1);
            mbar_init(&s_full[i], 1);
            mbar_init(&v_full[i], 1);
            mbar_init(&v_empty[i], 1);
        }
        mbar_init(&p_full, SOFTMAX_THREADS);
        mbar_init(&o_done, 1);
        asm volatile("fence.mbarrier_init.release.cluster;\n" ::: "memory");
    }
    if (warp == MMA_WARP) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;\n"
                     ::"r"(smem_u32(&tmem_slot)), "r"(TMEM_COLS));
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;\n" ::);
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const unsigned tmem = tmem_slot;
    pdl_wait();  // queries, keys and values come from the kernels before this one

    if (warp == PRODUCER_WARP) {
        if (elect_one()) {
            mbar_expect_tx(&q_full, Q_BYTES);
#pragma unroll
            for (int kb = 0; kb < DB; ++kb)
                tma_load_3d(q_s + kb * BLOCK_BYTES, &map_q, &q_full, kb * 64, h, row0 + r_begin);
            tma_load_3d(q_s + DB * BLOCK_BYTES, &map_qr, &q_full, 0, h, row0 + r_begin);
            bool ok = true;
            for (int t = 0; t < n_tiles + 1 && ok; ++t) {
                if (t < n_tiles) {   // keys run one tile ahead of the values
                    const int b = t & 1, y = base + (t_first + t) * BN;
                    if (t >= 2 && !mbar_wait(&k_empty[b], ((t - 2) >> 1) & 1)) { ok = false; break; }
                    mbar_expect_tx(&k_full[b], K_BYTES);
#pragma unroll
                    for (int kb = 0; kb < DB; ++kb)
                        tma_load_2d(k_s + b * K_BYTES + kb * BLOCK_BYTES, &map_kv, &k_full[b], h * D + kb * 64, y);
                    tma_load_2d(k_s + b * K_BYTES + DB * BLOCK_BYTES, &map_c, &k_full[b], p.r_col, y);
                }
                if (t >= 1) {
                    const int tv = t - 1, b = tv & 1, y = base + (t_first + tv) * BN;
                    if (tv >= 2 && !mbar_wait(&v_empty[b], ((tv - 2) >> 1) & 1)) { ok = false; break; }
                    mbar_expect_tx(&v_full[b], V_BYTES);
#pragma unroll
                    for (int vb = 0; vb < VB; ++vb)
                        tma_load_2d(v_s + b * V_BYTES + vb * BLOCK_BYTES, &map_kv, &v_full[b], p.v_col + h * VD + vb * 64, y);
                }
            }
            if (!ok) atomicOr(p.err, IB_TIMEOUT_AT(IB_SITE_EXPANDED_PRODUCER));
        }
    } else if (warp == MMA_WARP) {
        if (elect_one()) {
            constexpr unsigned idesc_s = make_idesc(BN, false);
            constexpr unsigned idesc_o = make_idesc(VD, true);
            bool ok = mbar_wait(&q_full, 0);
            auto issue_scores = [&](int t) -> bool {   // of tile t into score buffer t % 2
                const int b = t & 1;
                if (!mbar_wait(&k_full[b], (t >> 1) & 1)) return false;
                tc_fence_after();
#pragma unroll
                for (int kb = 0; kb < KB; ++kb) {
                    const uint64_t a = desc_k_major(q_s + kb * BLOCK_BYTES);
                    const uint64_t bd = desc_k_major(k_s + b * K_BYTES + kb * BLOCK_BYTES);
#pragma unroll
                    for (int kk = 0; kk < 4; ++kk)
                        umma_bf16(tmem + b * BN, a + 2 * kk, bd + 2 * kk, idesc_s, (kb > 0 || kk > 0) ? 1u : 0u);
                }
                umma_commit(&k_empty[b]);
                umma_commit(&s_full[b]);
                return true;
            };
            if (ok && n_tiles > 0) ok = issue_scores(0);
            for (int t = 0; t < n_tiles && ok; ++t) {
                // (the buffer of tile t + 1 held P of tile t - 1, which the update issued before reads; MMAs run in order)
                if (t + 1 < n_tiles && !issue_scores(t + 1)) { ok = false; break; }
                if (!mbar_wait(&p_full, t & 1) || !mbar_wait(&v_full[t & 1], (t >> 1) & 1)) { ok = false; break; }
                tc_fence_after();
                const unsigned a = tmem + (unsigned)((t & 1) * BN);   // P lies over its scores' first 64 columns
                const uint64_t b = desc_n_major(v_s + (t & 1) * V_BYTES, BLOCK_BYTES);
#pragma unroll
                for (int kk = 0; kk < BN / 16; ++kk)
                    umma_bf16_a_tmem(tmem + O_COL, a + 8 * kk, b + (uint64_t)(kk * ((16 * 128) >> 4)), idesc_o,
                                     (t > 0 || kk > 0) ? 1u : 0u);
                umma_commit(&v_empty[t & 1]);
                umma_commit(&o_done);
            }
            if (!ok) atomicOr(p.err, IB_TIMEOUT_AT(IB_SITE_EXPANDED_MMA));
        }
    } else {
        // ---- softmax: thread m owns query row m = TMEM lane m -------------------------
        const int m = threadIdx.x;
        const bool valid = m < r_count;
        const int my_pos = valid ? pos0 + r_begin + m : -1;
        const int my_lo = p.window > 0 ? my_pos - p.window + 1 : 0;
        const unsigned lane_addr = tmem + ((unsigned)(warp * 32) << 16);
        float m_run = -INFINITY, l_run = 0.f;   // the row's reference maximum and its sum
        bool ok = true;
        for (int t = 0; t < n_tiles; ++t) {
            if (ok && !mbar_wait(&s_full[t & 1], (t >> 1) & 1)) ok = false;
            tc_fence_after();
            float s[2][64];
            tmem_ld64_wait(lane_addr + (t & 1) * BN, s[0]);
            tmem_ld64_wait(lane_addr + (t & 1) * BN + 64, s[1]);
            const int key0 = (t_first + t) * BN;
            if (key0 + BN - 1 > pos0 + r_begin || !valid || (p.window > 0 && key0 <= kv_hi - 1 - p.window)) {
#pragma unroll
                for (int u = 0; u < 2; ++u)
#pragma unroll
                    for (int c = 0; c < 64; ++c) {
                        const int key = key0 + 64 * u + c;
                        s[u][c] = (key <= my_pos && key >= my_lo) ? s[u][c] : -INFINITY;
                    }
            }
            float ch[8];
#pragma unroll
            for (int q = 0; q < 8; ++q) {
                const float* v = &s[q >> 2][16 * (q & 3)];
                ch[q] = max3(v[0], v[1], v[2]);
#pragma unroll
                for (int i = 3; i < 15; i += 2) ch[q] = max3(ch[q], v[i], v[i + 1]);
                ch[q] = fmaxf(ch[q], v[15]);
            }
            float m_new = max3(max3(m_run, ch[0], ch[1]), ch[2], ch[3]);
            m_new = max3(max3(m_new, ch[4], ch[5]), ch[6], ch[7]);
            // (the reference follows the true maximum only when that rose by more than 2^8: attention_tcgen05.cu)
            float corr = 1.f;
            if (m_new > -INFINITY && (m_run == -INFINITY || (m_new - m_run) * p.scale_log2 > 8.f)) {
                corr = fast_exp2((m_run - m_new) * p.scale_log2);  // 0 from a reference of -inf
                m_run = m_new;
            }
            const float m_scaled = m_run == -INFINITY ? 0.f : m_run * p.scale_log2;
            const unsigned long long scale2 = pack2(p.scale_log2, p.scale_log2);
            const unsigned long long ref2 = pack2(-m_scaled, -m_scaled);
            unsigned long long acc[4] = {0ull, 0ull, 0ull, 0ull};
            // half of the keys at a time: the first half's P is on its way while the second's exponentials are made.
            // (P of this tile goes over its own scores, which are in registers.)
#pragma unroll
            for (int u = 0; u < 2; ++u) {
#pragma unroll
                for (int c = 0; c < 64; c += 2) {
                    fma2(s[u][c], s[u][c + 1], s[u][c], s[u][c + 1], scale2, ref2);
                    s[u][c] = fast_exp2(s[u][c]);
                    s[u][c + 1] = fast_exp2(s[u][c + 1]);
                    add2(acc[(c >> 1) & 3], s[u][c], s[u][c + 1]);
                }
#pragma unroll
                for (int i = 0; i < 2; ++i) {
                    unsigned pk[16];
#pragma unroll
                    for (int j = 0; j < 16; ++j) {
                        __nv_bfloat162 two = __floats2bfloat162_rn(s[u][32 * i + 2 * j], s[u][32 * i + 2 * j + 1]);
                        pk[j] = *reinterpret_cast<unsigned*>(&two);
                    }
                    tmem_st16(lane_addr + (t & 1) * BN + 32 * u + 16 * i, pk);
                }
            }
            l_run = l_run * corr + ((sum2(acc[0]) + sum2(acc[1])) + (sum2(acc[2]) + sum2(acc[3])));
            if (t > 0 && ok && !mbar_wait(&o_done, (t - 1) & 1)) ok = false;
            if (t > 0 && __any_sync(0xffffffffu, corr != 1.f)) {
                tc_fence_after();
#pragma unroll
                for (int c = 0; c < VD; c += 16) {
                    unsigned v[16];
                    tmem_ld16(lane_addr + O_COL + c, v);
                    tmem_ld_wait();
#pragma unroll
                    for (int j = 0; j < 16; ++j) v[j] = __float_as_uint(__uint_as_float(v[j]) * corr);
                    tmem_st16(lane_addr + O_COL + c, v);
                }
            }
            tmem_st_wait();
            if (t == n_tiles - 1 && key0 + BN > kv_hi) {
                // What lies behind the request's keys may be anything, and 0 x NaN is NaN in the product P V: the
                // values from key kv_hi on are cleared in shared memory once the tile has landed.
                if (ok && !mbar_wait(&v_full[t & 1], (t >> 1) & 1)) ok = false;
                const int first = kv_hi - key0;  // 1..127
                unsigned char* vt = v_s + (t & 1) * V_BYTES;
                for (int i = m; i < (BN - first) * VB * 8; i += SOFTMAX_THREADS) {
                    const int chunk = i & 7, row = first + (i >> 3) % (BN - first), vb = (i >> 3) / (BN - first);
                    *reinterpret_cast<uint4*>(vt + vb * BLOCK_BYTES + row * 128 + chunk * 16) = make_uint4(0, 0, 0, 0);
                }
                asm volatile("fence.proxy.async.shared::cta;\n" ::: "memory");
            }
            tc_fence_before();
            mbar_arrive(&p_full);
        }
        if (n_tiles > 0) {
            if (ok && !mbar_wait(&o_done, (n_tiles - 1) & 1)) ok = false;
            tc_fence_after();
        }
        if (!ok && lane == 0) atomicOr(p.err, IB_TIMEOUT_AT(IB_SITE_EXPANDED_SOFTMAX));
        float inv = inv_denominator(p.sink, h, m_run * p.scale_log2, l_run);
        if (p.gate && valid)
            inv *= 1.f / (1.f + expf(-load1(p.gate + (size_t)(row0 + r_begin + m) * p.gate_stride + h)));
        bf16* dst = valid ? p.out + (size_t)(row0 + r_begin + m) * p.out_stride + (size_t)h * VD : nullptr;
#pragma unroll
        for (int c = 0; c < VD; c += 16) {
            unsigned v[16];
            tmem_ld16(lane_addr + O_COL + c, v);
            tmem_ld_wait();
            if (valid && ok) {
                uint4 lo4, hi4;
                __nv_bfloat162* l2 = reinterpret_cast<__nv_bfloat162*>(&lo4);
                __nv_bfloat162* h2 = reinterpret_cast<__nv_bfloat162*>(&hi4);
#pragma unroll
                for (int j = 0; j < 4; ++j) {
                    l2[j] = __floats2bfloat162_rn(__uint_as_float(v[2 * j]) * inv, __uint_as_float(v[2 * j + 1]) * inv);
                    h2[j] = __floats2bfloat162_rn(__uint_as_float(v[8 + 2 * j]) * inv, __uint_as_float(v[8 + 2 * j + 1]) * inv);
                }
                *reinterpret_cast<uint4*>(dst + c) = lo4;
                *reinterpret_cast<uint4*>(dst + c + 8) = hi4;
            }
        }
        tc_fence_before();
    }
    __syncwarp();  // the elected lanes are back with their warps
    __syncthreads();
    if (warp == MMA_WARP) {
        tc_fence_after();
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;\n" ::"r"(tmem), "r"(TMEM_COLS));
    }
}

// The cached vectors of the entries' keys one after another: a warp a key, sixteen bytes a lane.  Keys behind the window
// of every row of the step are zeros (their pages may have been given back).
__global__ void __launch_bounds__(256)
gather_latents_kernel(const bf16* __restrict__ pool, bf16* __restrict__ out, const int* __restrict__ cu_rows,
                      const int* __restrict__ q_start, const int* __restrict__ tables, int max_blocks, int n_entries,
                      int page_size, int num_pages, int window, int width, int out_rows, unsigned* __restrict__ err) {
    pdl_trigger();
    pdl_wait();
    const int at = blockIdx.x * 8 + (threadIdx.x >> 5), lane = threadIdx.x & 31;
    if (at >= out_rows) return;
    // (keys without a row would be zeros to the attention, which reads nothing behind the buffer: reported)
    if (at == out_rows - 1 && lane == 0 && buffer_row(cu_rows, q_start, n_entries, window) > out_rows)
        atomicOr(err, IB_FLAG_KEYS_LOST);
    int e = 0, left = at, key = -1;
    for (; e < n_entries; ++e) {
        const int rows = cu_rows[e + 1] - cu_rows[e];
        if (rows <= 0) continue;
        const int first = first_key(q_start[e], window), n = q_start[e] + rows - first;
        if (left < n) {
            key = first + left;
            break;
        }
        left -= n;
    }
    if (key < 0) return;   // (behind the last key: nobody reads what is made of it)
    const bf16* src = nullptr;
    if (window <= 0 || key >= q_start[e] - window + 1) {
        const int b = key / page_size;
        const int page = b < max_blocks ? tables[(size_t)e * max_blocks + b] : -1;
        if (page < 0 || page >= num_pages) {
            if (lane == 0) atomicOr(err, IB_FLAG_BAD_PAGE);
        } else {
            src = pool + ((size_t)page * page_size + (key - b * page_size)) * width;
        }
    }
    bf16* dst = out + (size_t)at * width;
    for (int c = lane * 8; c < width; c += 256)
        *reinterpret_cast<uint4*>(dst + c) =
            src ? __ldcg(reinterpret_cast<const uint4*>(src + c)) : make_uint4(0u, 0u, 0u, 0u);
}

typedef CUresult (*EncodeTiledFn)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*,
                                  const cuuint64_t*, const cuuint32_t*, const cuuint32_t*,
                                  CUtensorMapInterleave, CUtensorMapSwizzle, CUtensorMapL2promotion,
                                  CUtensorMapFloatOOBfill);

EncodeTiledFn get_encode_fn() {
    static EncodeTiledFn fn = nullptr;
    if (!fn) {
        void* ptr = nullptr;
        cudaDriverEntryPointQueryResult qres;
        if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &ptr, cudaEnableDefault, &qres) == cudaSuccess &&
            qres == cudaDriverEntryPointSuccess)
            fn = (EncodeTiledFn)ptr;
    }
    return fn;
}

int make_map(CUtensorMap* map, const void* base, int dims, const cuuint64_t* size, const cuuint64_t* strides,
             const cuuint32_t* box) {
    EncodeTiledFn enc = get_encode_fn();
    if (!enc) return IB_ERR_UNSUPPORTED;
    const cuuint32_t es[3] = {1, 1, 1};
    return enc(map, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, dims, const_cast<void*>(base), size, strides, box, es,
               CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
               CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS ? IB_OK : IB_ERR_BAD_ARG;
}

}  // namespace

IB_EXPORT int ib_attention_expanded_sizes() { return D * 1000000 + R * 1000 + VD; }

// pool [num_pages][page_size][width] -> out [out_rows, width]: the keys of entry 0 that any of its rows sees (from the
// multiple of 128 before the first row's window on), then those of entry 1, ...; rows behind the last key are left as they
// are, and keys that find no row set IB_FLAG_KEYS_LOST.  width a multiple of 8.
IB_EXPORT int ib_gather_latents(const void* pool, void* out, const int* cu_rows, const int* q_start, const int* tables,
                                int max_blocks, int n_entries, int page_size, int num_pages, int window, int width,
                                int out_rows, unsigned* err, void* stream) {
    if (n_entries <= 0 || out_rows <= 0) return IB_OK;
    if (!pool || !out || !cu_rows || !q_start || !tables || !err || max_blocks <= 0 || page_size <= 0 || num_pages <= 0 ||
        width <= 0)
        return IB_ERR_BAD_ARG;
    if (width % 8 || ((uintptr_t)pool & 15) || ((uintptr_t)out & 15)) return IB_ERR_UNSUPPORTED;
    cudaError_t le = launch_kernel(gather_latents_kernel, dim3((out_rows + 7) / 8), dim3(256), 0, (cudaStream_t)stream,
                                   (const bf16*)pool, (bf16*)out, cu_rows, q_start, tables, max_blocks, n_entries, page_size,
                                   num_pages, window, width, out_rows, err);
    if (le != cudaSuccess) return (int)le;
    IB_LAUNCH_CHECK();
    return IB_OK;
}

// q: rows q_stride apart, head h at h * (EX_D + EX_R), of which the first EX_D elements are read; qr [n_rows][nh][EX_R]
// the rotated parts; c [key_rows, c_width] the gathered latents, whose rotated keys begin at column r_col; kv [key_rows,
// kv_stride]: head h's key at column h * EX_D, its value at v_col + h * EX_V.  out rows out_stride apart, head h at h * EX_V.
IB_EXPORT int ib_attention_expanded(const void* q, int q_stride, const void* qr, const void* c, int c_width, int r_col,
                                    const void* kv, int kv_stride, int v_col, int key_rows, void* out, int out_stride,
                                    const int* cu_rows, const int* q_start, int n_entries, int n_rows, int max_rows, int nh,
                                    int window, float scale, const float* sink, const void* gate, int gate_stride,
                                    unsigned* err, void* stream) {
    if (n_entries <= 0 || n_rows <= 0) return IB_OK;
    if (!q || !qr || !c || !kv || !out || !cu_rows || !q_start || !err || nh <= 0 || key_rows <= 0 || max_rows <= 0 ||
        r_col < 0 || r_col + R > c_width || v_col < nh * D || v_col + nh * VD > kv_stride || q_stride < nh * (D + R) ||
        out_stride < nh * VD || (gate && gate_stride < nh))
        return IB_ERR_BAD_ARG;
    if ((q_stride % 8) || (c_width % 8) || (r_col % 8) || (kv_stride % 8) || (v_col % 8) || (out_stride % 8) ||
        (((uintptr_t)q | (uintptr_t)qr | (uintptr_t)c | (uintptr_t)kv | (uintptr_t)out) & 15))
        return IB_ERR_UNSUPPORTED;
    const int row_tiles = (max_rows + BM - 1) / BM;
    if (n_entries > 65535 || row_tiles > 65535) return IB_ERR_TOO_LARGE;
    CUtensorMap mq, mqr, mkv, mc;
    const cuuint32_t box3[3] = {64, 1, BM}, box2[2] = {64, BN};
    const cuuint64_t q_size[3] = {(cuuint64_t)(D + R), (cuuint64_t)nh, (cuuint64_t)n_rows};
    const cuuint64_t q_step[2] = {(cuuint64_t)(D + R) * 2, (cuuint64_t)q_stride * 2};
    const cuuint64_t qr_size[3] = {(cuuint64_t)R, (cuuint64_t)nh, (cuuint64_t)n_rows};
    const cuuint64_t qr_step[2] = {(cuuint64_t)R * 2, (cuuint64_t)nh * R * 2};
    const cuuint64_t kv_size[2] = {(cuuint64_t)(v_col + nh * VD), (cuuint64_t)key_rows};
    const cuuint64_t kv_step[1] = {(cuuint64_t)kv_stride * 2};
    const cuuint64_t c_size[2] = {(cuuint64_t)c_width, (cuuint64_t)key_rows};
    const cuuint64_t c_step[1] = {(cuuint64_t)c_width * 2};
    int rc = make_map(&mq, q, 3, q_size, q_step, box3);
    if (rc == IB_OK) rc = make_map(&mqr, qr, 3, qr_size, qr_step, box3);
    if (rc == IB_OK) rc = make_map(&mkv, kv, 2, kv_size, kv_step, box2);
    if (rc == IB_OK) rc = make_map(&mc, c, 2, c_size, c_step, box2);
    if (rc != IB_OK) return rc;
    Params p;
    p.out = (bf16*)out;
    p.cu_rows = cu_rows;
    p.q_start = q_start;
    p.err = err;
    p.sink = sink;
    p.gate = (const bf16*)gate;
    p.gate_stride = gate_stride;
    p.out_stride = out_stride;
    p.nh = nh;
    p.window = window;
    p.v_col = v_col;
    p.r_col = r_col;
    p.scale_log2 = scale * 1.4426950408889634f;
    static bool attr_done = false;
    if (!attr_done) {
        cudaError_t e1 = cudaFuncSetAttribute(attention_expanded_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                              SMEM_BYTES);
        if (e1 != cudaSuccess) return (int)e1;
        attr_done = true;
    }
    cudaError_t le = launch_kernel(attention_expanded_kernel, dim3(nh, n_entries, row_tiles), dim3(NUM_THREADS),
                                   (size_t)SMEM_BYTES, (cudaStream_t)stream, mq, mqr, mkv, mc, p);
    if (le != cudaSuccess) return (int)le;
    IB_LAUNCH_CHECK();
    return IB_OK;
}
