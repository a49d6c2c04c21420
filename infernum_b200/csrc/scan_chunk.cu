// Recurrent scans of prompts in chunks of 64 tokens (state rows IB_ROWS, fixed when this file is compiled), 32-bit.
//
// scan.cu walks a request's tokens one after another, which leaves an SM eight warps that wait for one another.  Written
// for a chunk whose state at its begin is S0, a_t the decays, A_t their product up to token t and D[t][s] of those after s
// up to t, a state space layer is
//
//   y_t = A_t S0^T C_t + sum_{s<=t} D[t][s] (C_t.B_s) dt_s x_s + d x_t,      S <- A_L S0 + sum_s D[L][s] dt_s B_s x_s^T
//
// - matrix products of a chunk that need no other chunk, but for S0, which a short pass over the chunks hands on:
//
//   ssd_chunk_state   every chunk at once: sum_s D[L][s] dt_s B_s x_s^T per head, and C_t.B_s per group
//   ssd_chunk_pass    every state element walks its entry's chunks: S0 of each chunk, the state after the last
//   chunk_out         every chunk at once: y
//
// Decays are multiplied, never divided (a decay may be 0), and a token's result is made from what comes before it only:
// what a later token brings is left out of the sum, not multiplied by zero.  A chunk's tokens are counted from the entry's
// first row of the step: a prompt cut elsewhere rounds otherwise.
// Bound by the multiply-adds (as many as token by token).  2,048 tokens, 32 heads of 128 x 64: 414 us by scan.cu, 36 + 30 +
// 58 us here.
#include "common.cuh"

using namespace ib;

#ifndef IB_ROWS
#error "compile with -DIB_ROWS=<rows of the state matrix>"
#endif

namespace {

constexpr int ROWS = IB_ROWS;
static_assert(ROWS == 64 || ROWS == 128, "this file is built for states of 64 and 128 rows");
constexpr int L = 64;              // tokens of a chunk
constexpr int PT = 64;             // columns of the state a CTA takes
constexpr int PITCH = ROWS + 4;    // of rows read four elements at a time by neighbouring lanes

struct Chunk {
    int e, index, row, n;   // its entry, its place in it, its first row, its tokens
};
// Chunk `idx` of the step: the entries' chunks follow one another.  n = 0: there is none.
__device__ __forceinline__ Chunk find_chunk(const int* cu_rows, int n_entries, int idx) {
    for (int e = 0; e < n_entries; ++e) {
        const int first = cu_rows[e], n = cu_rows[e + 1] - first, c = n > 0 ? (n + L - 1) / L : 0;
        if (idx < c) return {e, idx, first + idx * L, min(L, n - idx * L)};
        idx -= c;
    }
    return {0, 0, 0, 0};
}

struct SsdParams {
    const float* x;        // [heads][rows][P]
    const float* bc;       // [groups][rows][2][ROWS]: B, then C
    const float* dd;       // ssd: float2 [heads][rows] (dt, decay); delta: float4 (beta, decay, unused, unused)
    const float* d_skip;
    const int* cu_rows;
    const int* slot_ids;
    float* state;          // slot s, head h: state + s * state_stride + h * P * ROWS, [P][ROWS]
    long long state_stride;
    float* carry;          // [heads][chunks][P][ROWS]: a chunk's own share of the state, then the state before it
    float* decay;          // [heads][chunks]: the product of the chunk's decays
    float* cb;             // [groups][chunks][L][L]: C_t.B_s
    float* out;            // [rows][heads * P]
    int n_rows, n_entries, chunks, heads, groups, P;
};

__device__ __forceinline__ float2 pfma(float a, float2 b, float2 c) {
    const float2 aa = make_float2(a, a);
    float2 d;
    asm("fma.rn.f32x2 %0, %1, %2, %3;"
        : "=l"(reinterpret_cast<unsigned long long&>(d))
        : "l"(reinterpret_cast<const unsigned long long&>(aa)), "l"(reinterpret_cast<const unsigned long long&>(b)),
          "l"(reinterpret_cast<const unsigned long long&>(c)));
    return d;
}

__device__ __forceinline__ void cp_async16(float* smem, const float* gmem, bool real) {   // zeros where not real
    const unsigned d = (unsigned)__cvta_generic_to_shared(smem);
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;\n" ::"r"(d), "l"(gmem), "r"(real ? 16 : 0) : "memory");
}
__device__ __forceinline__ void cp_async_land() {   // every thread's copies, for all
    asm volatile("cp.async.commit_group;\n\tcp.async.wait_group 0;\n" ::: "memory");
    __syncthreads();
}
// L rows of WIDTH floats, `stride` apart, to rows `pitch` apart; zeros behind row n.
template <int WIDTH>
__device__ __forceinline__ void fetch_rows(float* dst, int pitch, const float* src, size_t stride, int n) {
#pragma unroll 4
    for (int i = threadIdx.x; i < L * (WIDTH / 4); i += 128) {
        const int t = i / (WIDTH / 4), c = i % (WIDTH / 4) * 4;
        cp_async16(dst + t * pitch + c, src + (t < n ? t : 0) * stride + c, t < n);
    }
}

// Two products and sums at once: half the issue slots of fmaf, which leaves the loads between them room.
__device__ __forceinline__ void pfma2(float2& c, float ax, float ay, float bx, float by) {
    const float2 a = make_float2(ax, ay), b = make_float2(bx, by);
    asm("fma.rn.f32x2 %0, %1, %2, %0;"
        : "+l"(reinterpret_cast<unsigned long long&>(c))
        : "l"(reinterpret_cast<const unsigned long long&>(a)), "l"(reinterpret_cast<const unsigned long long&>(b)));
}

// acc[i][j] = sum_k a[i * 4 rows on][k] b[j * 8 rows on][k] over ROWS: both operands by rows of k, `pitch` apart
template <int M, int N>
__device__ __forceinline__ void dot_tile(const float* a, const float* b, int pitch, float (&acc)[M][N]) {
    float2 sum[M][N] = {};   // of the even and of the odd k
#pragma unroll 2
    for (int k = 0; k < ROWS; k += 4) {
        float4 u[M], v[N];
#pragma unroll
        for (int i = 0; i < M; ++i) u[i] = *reinterpret_cast<const float4*>(a + i * 4 * pitch + k);
#pragma unroll
        for (int j = 0; j < N; ++j) v[j] = *reinterpret_cast<const float4*>(b + j * 8 * pitch + k);
#pragma unroll
        for (int i = 0; i < M; ++i)
#pragma unroll
            for (int j = 0; j < N; ++j) pfma2(sum[i][j], u[i].x, u[i].y, v[j].x, v[j].y);
#pragma unroll
        for (int i = 0; i < M; ++i)
#pragma unroll
            for (int j = 0; j < N; ++j) pfma2(sum[i][j], u[i].z, u[i].w, v[j].z, v[j].w);
    }
#pragma unroll
    for (int i = 0; i < M; ++i)
#pragma unroll
        for (int j = 0; j < N; ++j) acc[i][j] = sum[i][j].x + sum[i][j].y;
}

constexpr int STATE_BYTES = 2 * L * PITCH * (int)sizeof(float);   // (C and B of the C.B product; B and x need less)
static_assert(L * ROWS + L * PT <= 2 * L * PITCH, "B and x fit where C and B do");

// blockIdx.y < heads * (P / PT): a head's columns of the chunk's share of the state; behind them, a group's C.B.
__global__ void __launch_bounds__(128) ssd_chunk_state_kernel(const SsdParams p) {
    pdl_wait();
    extern __shared__ __align__(16) float smem[];
    __shared__ float w[L];
    const Chunk at = find_chunk(p.cu_rows, p.n_entries, blockIdx.x);
    if (at.n == 0) return;
    const int tid = threadIdx.x, warp = tid / 32, lane = tid % 32, ly = lane / 8, lx = lane % 8;
    const int slices = p.P / PT;
    const int y = blockIdx.y;
    if (y >= p.heads * slices) {
        const int g = y - p.heads * slices;
        const float* src = p.bc + ((size_t)g * p.n_rows + at.row) * 2 * ROWS;
        float* cs = smem;
        float* bs = smem + L * PITCH;
        fetch_rows<ROWS>(bs, PITCH, src, 2 * ROWS, at.n);
        fetch_rows<ROWS>(cs, PITCH, src + ROWS, 2 * ROWS, at.n);
        cp_async_land();
        float acc[4][8];
        dot_tile(cs + (warp * 16 + ly) * PITCH, bs + lx * PITCH, PITCH, acc);
        float* out = p.cb + ((size_t)g * p.chunks + blockIdx.x) * L * L;
#pragma unroll
        for (int i = 0; i < 4; ++i)
#pragma unroll
            for (int j = 0; j < 8; ++j) out[(warp * 16 + i * 4 + ly) * L + lx + j * 8] = acc[i][j];
        return;
    }
    const int head = y / slices, p0 = y % slices * PT;
    const int grp = head / (p.heads / p.groups);
    const float2* dd = reinterpret_cast<const float2*>(p.dd) + (size_t)head * p.n_rows + at.row;
    float* bs = smem;                // [L][ROWS]
    float* xs = smem + L * ROWS;     // [L][PT]
    fetch_rows<ROWS>(bs, ROWS, p.bc + ((size_t)grp * p.n_rows + at.row) * 2 * ROWS, 2 * ROWS, at.n);
    fetch_rows<PT>(xs, PT, p.x + ((size_t)head * p.n_rows + at.row) * p.P + p0, p.P, at.n);
    if (warp == 0) {   // w_s = dt_s times the decays after s: products from the chunk's end on, two tokens a lane
        const float2 d0 = 2 * lane < at.n ? __ldcg(dd + 2 * lane) : make_float2(0.f, 1.f);
        const float2 d1 = 2 * lane + 1 < at.n ? __ldcg(dd + 2 * lane + 1) : make_float2(0.f, 1.f);
        float after = d0.y * d1.y;   // of this lane's tokens, then of all from this lane on
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const float v = __shfl_down_sync(0xffffffffu, after, o);
            if (lane + o < 32) after *= v;
        }
        float rest = __shfl_down_sync(0xffffffffu, after, 1);
        if (lane == 31) rest = 1.f;
        w[2 * lane + 1] = d1.x * rest;
        w[2 * lane] = d0.x * (d1.y * rest);
        if (lane == 0 && p0 == 0) p.decay[(size_t)head * p.chunks + blockIdx.x] = after;
    }
    cp_async_land();
#pragma unroll
    for (int k = 0; k < L * (PT / 4) / 128; ++k) {
        const int i = tid + k * 128;
        float4 v = reinterpret_cast<float4*>(xs)[i];
        const float f = w[i / (PT / 4)];
        reinterpret_cast<float4*>(xs)[i] = make_float4(v.x * f, v.y * f, v.z * f, v.w * f);
    }
    __syncthreads();
    // a thread: rows warp * 16 + ly * 4 .. + 3 (and, of 128, those 64 further on), columns lx * 4 .. + 3 and 32 further on
    constexpr int RB = ROWS / 64;
    float2 acc[RB][4][4] = {};
#pragma unroll 4
    for (int s = 0; s < L; ++s) {
        float4 b[RB];
#pragma unroll
        for (int r = 0; r < RB; ++r) b[r] = *reinterpret_cast<const float4*>(bs + s * ROWS + r * 64 + warp * 16 + ly * 4);
        const float4 v0 = *reinterpret_cast<const float4*>(xs + s * PT + lx * 4);
        const float4 v1 = *reinterpret_cast<const float4*>(xs + s * PT + 32 + lx * 4);
        const float2 v[4] = {make_float2(v0.x, v0.y), make_float2(v0.z, v0.w), make_float2(v1.x, v1.y), make_float2(v1.z, v1.w)};
#pragma unroll
        for (int r = 0; r < RB; ++r)
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                acc[r][0][j] = pfma(b[r].x, v[j], acc[r][0][j]);
                acc[r][1][j] = pfma(b[r].y, v[j], acc[r][1][j]);
                acc[r][2][j] = pfma(b[r].z, v[j], acc[r][2][j]);
                acc[r][3][j] = pfma(b[r].w, v[j], acc[r][3][j]);
            }
    }
    float* out = p.carry + (((size_t)head * p.chunks + blockIdx.x) * p.P + p0) * ROWS;
#pragma unroll
    for (int r = 0; r < RB; ++r)
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            const int col = (j / 2) * 32 + lx * 4 + (j % 2) * 2;
            float* o = out + (size_t)col * ROWS + r * 64 + warp * 16 + ly * 4;
            *reinterpret_cast<float4*>(o) = make_float4(acc[r][0][j].x, acc[r][1][j].x, acc[r][2][j].x, acc[r][3][j].x);
            *reinterpret_cast<float4*>(o + ROWS) = make_float4(acc[r][0][j].y, acc[r][1][j].y, acc[r][2][j].y, acc[r][3][j].y);
        }
}

// Four state elements a thread: the state before each of the entry's chunks takes the place of the chunk's own share.
__global__ void __launch_bounds__(128) ssd_chunk_pass_kernel(const SsdParams p) {
    pdl_trigger();
    pdl_wait();
    const int head = blockIdx.y, e = blockIdx.z;
    const int i = (blockIdx.x * 128 + threadIdx.x) * 4;
    const int n = p.cu_rows[e + 1] - p.cu_rows[e];
    if (n <= 0 || i >= p.P * ROWS) return;
    int first = 0;   // the entry's first chunk
    for (int q = 0; q < e; ++q) {
        const int m = p.cu_rows[q + 1] - p.cu_rows[q];
        if (m > 0) first += (m + L - 1) / L;
    }
    const int count = (n + L - 1) / L;
    float4* st = reinterpret_cast<float4*>(p.state + (long long)p.slot_ids[e] * p.state_stride + (size_t)head * p.P * ROWS + i);
    float* c = p.carry + ((size_t)head * p.chunks + first) * p.P * ROWS + i;
    const float* d = p.decay + (size_t)head * p.chunks + first;
    const size_t step = (size_t)p.P * ROWS;
    float4 S = __ldcg(st);
    constexpr int AHEAD = 8;
    for (int k0 = 0; k0 < count; k0 += AHEAD) {
        float4 u[AHEAD];
        float a[AHEAD];
#pragma unroll
        for (int k = 0; k < AHEAD; ++k)
            if (k0 + k < count) {
                u[k] = __ldcg(reinterpret_cast<const float4*>(c + (k0 + k) * step));
                a[k] = __ldcg(d + k0 + k);
            }
#pragma unroll
        for (int k = 0; k < AHEAD; ++k)
            if (k0 + k < count) {
                __stcg(reinterpret_cast<float4*>(c + (k0 + k) * step), S);
                S.x = fmaf(a[k], S.x, u[k].x);
                S.y = fmaf(a[k], S.y, u[k].y);
                S.z = fmaf(a[k], S.z, u[k].z);
                S.w = fmaf(a[k], S.w, u[k].w);
            }
    }
    *st = S;
}

constexpr int MP = L + 4;   // pitch of the chunk's own weights
constexpr int OUT_BYTES = (2 * L * PITCH + L * PT + L * MP) * (int)sizeof(float);

// DELTA: the same with k for B, q for C and the rule's u for dt x, without a share of x of its own.
template <bool DELTA>
__global__ void __launch_bounds__(128) chunk_out_kernel(const SsdParams p) {
    pdl_trigger();
    pdl_wait();
    extern __shared__ __align__(16) float smem[];
    float* cs = smem;                  // [L][PITCH] C
    float* ss = cs + L * PITCH;        // [PT][PITCH] the state before the chunk, column c at row c % 4 * 8 + c / 4 % 8 + c / 32 * 32
    float* xs = ss + PT * PITCH;       // [L][PT]
    float* ms = xs + L * PT;           // [L][MP] D[t][s] (C_t.B_s) dt_s
    __shared__ float dt[L], da[L], upto[L];
    const Chunk at = find_chunk(p.cu_rows, p.n_entries, blockIdx.x);
    if (at.n == 0) return;
    const int tid = threadIdx.x, warp = tid / 32, lane = tid % 32, ly = lane / 8, lx = lane % 8;
    const int head = blockIdx.y, p0 = blockIdx.z * PT;
    const int grp = head / (p.heads / p.groups);
    if (tid < L) {
        const float* d = p.dd + ((size_t)head * p.n_rows + at.row + tid) * (DELTA ? 4 : 2);
        dt[tid] = DELTA ? 1.f : tid < at.n ? __ldcg(d) : 0.f;
        da[tid] = tid < at.n ? __ldcg(d + 1) : 1.f;
    }
    fetch_rows<ROWS>(cs, PITCH, p.bc + (((size_t)grp * p.n_rows + at.row) * 2 + 1) * ROWS, 2 * ROWS, at.n);
    const float* st = p.carry + (((size_t)head * p.chunks + blockIdx.x) * p.P + p0) * ROWS;
#pragma unroll 4
    for (int i = tid; i < PT * (ROWS / 4); i += 128) {
        const int c = i / (ROWS / 4), r = i % (ROWS / 4) * 4;
        cp_async16(ss + (c % 4 * 8 + c / 4 % 8 + c / 32 * 32) * PITCH + r, st + (size_t)c * ROWS + r, true);
    }
    fetch_rows<PT>(xs, PT, p.x + ((size_t)head * p.n_rows + at.row) * p.P + p0, p.P, at.n);
    fetch_rows<L>(ms, MP, p.cb + ((size_t)grp * p.chunks + blockIdx.x) * L * L, L, L);
    cp_async_land();
    {   // a thread walks half of a column s of the weights downwards
        const int s = tid % L, half = tid / L;
        const int t1 = half ? L : L / 2, t0 = max(s, half ? L / 2 : 0);
        const float ds = dt[s];
        float d = 1.f;   // D[t][s]
        for (int t = s + 1; t <= t0 && t < L; ++t) d *= da[t];
#pragma unroll 8
        for (int t = t0; t < t1; ++t) {
            ms[t * MP + s] *= d * ds;
            d *= t + 1 < L ? da[t + 1] : 1.f;
        }
        if (warp == 0) {   // A_t: two tokens a lane
            const float d0 = da[2 * lane], d1 = da[2 * lane + 1];
            float before = d0 * d1;
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const float v = __shfl_up_sync(0xffffffffu, before, o);
                if (lane >= o) before *= v;
            }
            float prior = __shfl_up_sync(0xffffffffu, before, 1);
            if (lane == 0) prior = 1.f;
            upto[2 * lane] = prior * d0;
            upto[2 * lane + 1] = prior * d0 * d1;
        }
    }
    __syncthreads();
    // a thread: tokens warp * 16 + i * 4 + ly, columns (j / 4) * 32 + lx * 4 + j % 4 (row j * 8 + lx of `ss`)
    float acc[4][8];
    dot_tile(cs + (warp * 16 + ly) * PITCH, ss + lx * PITCH, PITCH, acc);
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        const float a = upto[warp * 16 + i * 4 + ly];
#pragma unroll
        for (int j = 0; j < 8; ++j) acc[i][j] *= a;
    }
    const float* mw = ms + (warp * 16 + ly) * MP;
    const float* xw = xs + lx * 4;
#pragma unroll 2
    for (int s = 0; s < warp * 16; s += 4) {
        float4 m[4];
#pragma unroll
        for (int i = 0; i < 4; ++i) m[i] = *reinterpret_cast<const float4*>(mw + i * 4 * MP + s);
#pragma unroll
        for (int u = 0; u < 4; ++u)
#pragma unroll
            for (int c = 0; c < 2; ++c) {
                const float4 v = *reinterpret_cast<const float4*>(xw + (s + u) * PT + c * 32);
#pragma unroll
                for (int i = 0; i < 4; ++i) {
                    const float q = u == 0 ? m[i].x : u == 1 ? m[i].y : u == 2 ? m[i].z : m[i].w;
                    acc[i][4 * c] = fmaf(q, v.x, acc[i][4 * c]);
                    acc[i][4 * c + 1] = fmaf(q, v.y, acc[i][4 * c + 1]);
                    acc[i][4 * c + 2] = fmaf(q, v.z, acc[i][4 * c + 2]);
                    acc[i][4 * c + 3] = fmaf(q, v.w, acc[i][4 * c + 3]);
                }
            }
    }
#pragma unroll 2
    for (int s = warp * 16; s < warp * 16 + 16; ++s) {   // the warp's own tokens: each takes those up to itself
        float4 v[2];
#pragma unroll
        for (int c = 0; c < 2; ++c) v[c] = *reinterpret_cast<const float4*>(xw + s * PT + c * 32);
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            if (s > warp * 16 + i * 4 + ly) continue;
            const float q = mw[i * 4 * MP + s];
#pragma unroll
            for (int c = 0; c < 2; ++c) {
                acc[i][4 * c] = fmaf(q, v[c].x, acc[i][4 * c]);
                acc[i][4 * c + 1] = fmaf(q, v[c].y, acc[i][4 * c + 1]);
                acc[i][4 * c + 2] = fmaf(q, v[c].z, acc[i][4 * c + 2]);
                acc[i][4 * c + 3] = fmaf(q, v[c].w, acc[i][4 * c + 3]);
            }
        }
    }
    const float skip = DELTA ? 0.f : p.d_skip[head];
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        const int t = warp * 16 + i * 4 + ly;
        if (t >= at.n) continue;
        float* o = p.out + (size_t)(at.row + t) * p.heads * p.P + (size_t)head * p.P + p0 + lx * 4;
#pragma unroll
        for (int c = 0; c < 2; ++c) {
            float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
            if (!DELTA) v = *reinterpret_cast<const float4*>(xw + t * PT + c * 32);
            *reinterpret_cast<float4*>(o + c * 32) =
                make_float4(fmaf(skip, v.x, acc[i][4 * c]), fmaf(skip, v.y, acc[i][4 * c + 1]),
                            fmaf(skip, v.z, acc[i][4 * c + 2]), fmaf(skip, v.w, acc[i][4 * c + 3]));
        }
    }
}

// ---- the gated delta rule ---------------------------------------------------------------------------------------
//   u_t = beta_t (v_t - A_t k_t.S0 - sum_{s<t} D[t][s] (k_t.k_s) u_s),   o_t = A_t q_t.S0 + sum_{s<=t} D[t][s] (q_t.k_s) u_s,
//   S <- A_L S0 + sum_s D[L][s] k_s u_s^T:
// with M[t][s] = beta_t D[t][s] (k_t.k_s) below the diagonal, (I + M) u = beta v - (beta A k) S0, so that
//   delta_chunk_dots    every chunk at once: k_t.k_s and q_t.k_s per key head
//   delta_chunk_solve   every chunk at once: U = (I + M)^-1 beta v and W = (I + M)^-1 beta A k, forward substitution
//                       in blocks of sixteen tokens, a thread two columns
//   delta_chunk_walk    an entry's chunks in turn: u = U - W S0 and the state after, 32 columns a CTA
//   chunk_out           every chunk at once: o
// The walk is the only part that waits for the chunk before: 32 columns a CTA, so that there are four for a head of 128,
// and the next chunk's operands come while one is worked on.  Two entries of 750 tokens, 16 heads of 128 x 128 on eight key
// heads: 376 us by scan.cu, 16 + 32 + 110 + 49 us here; the walk is bound by its chain of chunks, two small products between
// barriers each (a mapping of them with a third of the reads of shared memory: 113 -> 110 us).
struct DeltaParams {
    SsdParams o;           // what chunk_out reads: x is `u`, bc the k and q, cb the q_t.k_s, carry the states before the chunks
    const float* v;        // [heads][rows][P]
    float* u;              // [heads][rows][P]: U, then u
    float* w;              // [heads][rows][ROWS]
    float* kk;             // [groups][chunks][L][L]: k_t.k_s
};

__global__ void __launch_bounds__(128) delta_chunk_dots_kernel(const DeltaParams p) {
    pdl_wait();
    extern __shared__ __align__(16) float smem[];
    const Chunk at = find_chunk(p.o.cu_rows, p.o.n_entries, blockIdx.x);
    if (at.n == 0) return;
    const int tid = threadIdx.x, warp = tid / 32, lane = tid % 32, ly = lane / 8, lx = lane % 8, g = blockIdx.y;
    const float* src = p.o.bc + ((size_t)g * p.o.n_rows + at.row) * 2 * ROWS;
    float* ks = smem;
    float* qs = smem + L * PITCH;
    const bool which = blockIdx.z == 1;   // q_t.k_s
    fetch_rows<ROWS>(ks, PITCH, src, 2 * ROWS, at.n);
    if (which) fetch_rows<ROWS>(qs, PITCH, src + ROWS, 2 * ROWS, at.n);
    cp_async_land();
    float acc[4][8];
    dot_tile((which ? qs : ks) + (warp * 16 + ly) * PITCH, ks + lx * PITCH, PITCH, acc);
    float* dst = (which ? p.o.cb : p.kk) + ((size_t)g * p.o.chunks + blockIdx.x) * L * L;
#pragma unroll
    for (int i = 0; i < 4; ++i)
#pragma unroll
        for (int j = 0; j < 8; ++j) dst[(warp * 16 + i * 4 + ly) * L + lx + j * 8] = acc[i][j];
}

constexpr int SOLVE_COLS = 256, SB = 16;   // columns of a CTA, tokens of a block
constexpr int SOLVE_BYTES = (L * SOLVE_COLS + 2 * L * MP) * (int)sizeof(float);

__global__ void __launch_bounds__(128) delta_chunk_solve_kernel(const DeltaParams p) {
    pdl_trigger();
    pdl_wait();
    extern __shared__ __align__(16) float smem[];
    float* X = smem;                      // [L][SOLVE_COLS]: k | v, then W | U
    float* kks = X + L * SOLVE_COLS;      // [L][MP]
    float* mt = kks + L * MP;             // [L][MP]: M transposed, mt[s][t]
    __shared__ float beta[L], da[L], upto[L];
    const Chunk at = find_chunk(p.o.cu_rows, p.o.n_entries, blockIdx.x);
    if (at.n == 0) return;
    const int tid = threadIdx.x, warp = tid / 32, lane = tid % 32;
    const int head = blockIdx.y, P = p.o.P, col0 = blockIdx.z * SOLVE_COLS;
    const int cols = min(SOLVE_COLS, ROWS + P - col0);
    const int g = head / (p.o.heads / p.o.groups);
    const float* ksrc = p.o.bc + ((size_t)g * p.o.n_rows + at.row) * 2 * ROWS;
    const float* vsrc = p.v + ((size_t)head * p.o.n_rows + at.row) * P;
#pragma unroll 4
    for (int i = tid; i < L * (SOLVE_COLS / 4); i += 128) {
        const int t = i / (SOLVE_COLS / 4), c = i % (SOLVE_COLS / 4) * 4, col = col0 + c;
        if (c < cols)
            cp_async16(X + t * SOLVE_COLS + c, t >= at.n ? ksrc : col < ROWS ? ksrc + (size_t)t * 2 * ROWS + col
                                                                             : vsrc + (size_t)t * P + col - ROWS, t < at.n);
    }
    fetch_rows<L>(kks, MP, p.kk + ((size_t)g * p.o.chunks + blockIdx.x) * L * L, L, L);
    if (tid < L) {
        const float4 d = tid < at.n ? __ldcg(reinterpret_cast<const float4*>(p.o.dd) + (size_t)head * p.o.n_rows + at.row + tid)
                                    : make_float4(0.f, 1.f, 0.f, 0.f);
        beta[tid] = d.x;
        da[tid] = d.y;
    }
    cp_async_land();
    {
        const int s = tid % L, half = tid / L;
        const int t1 = half ? L : L / 2, t0 = max(s, half ? L / 2 : 0);
        float d = 1.f;   // D[t][s]
        for (int t = s + 1; t <= t0 && t < L; ++t) d *= da[t];
#pragma unroll 8
        for (int t = t0; t < t1; ++t) {
            mt[s * MP + t] = beta[t] * d * kks[t * MP + s];
            d *= t + 1 < L ? da[t + 1] : 1.f;
        }
        if (warp == 0) {   // A_t: two tokens a lane
            const float d0 = da[2 * lane], d1 = da[2 * lane + 1];
            float before = d0 * d1;
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const float v = __shfl_up_sync(0xffffffffu, before, o);
                if (lane >= o) before *= v;
            }
            float prior = __shfl_up_sync(0xffffffffu, before, 1);
            if (lane == 0) prior = 1.f;
            upto[2 * lane] = prior * d0;
            upto[2 * lane + 1] = prior * d0 * d1;
        }
    }
    __syncthreads();
    if (2 * tid >= cols) return;
    const bool is_k = col0 + 2 * tid < ROWS;
    float* xc = X + 2 * tid;   // (a thread reads and writes its own two columns only)
#pragma unroll 1
    for (int b = 0; b < L / SB; ++b) {
        float2 r[SB];
#pragma unroll
        for (int i = 0; i < SB; ++i) {
            const int t = b * SB + i;
            const float f = is_k ? beta[t] * upto[t] : beta[t];
            const float2 v = *reinterpret_cast<const float2*>(xc + t * SOLVE_COLS);
            r[i] = make_float2(v.x * f, v.y * f);
        }
#pragma unroll 2
        for (int s = 0; s < b * SB; ++s) {
            const float2 x = *reinterpret_cast<const float2*>(xc + s * SOLVE_COLS);
#pragma unroll
            for (int q = 0; q < SB / 4; ++q) {
                const float4 m = *reinterpret_cast<const float4*>(mt + s * MP + b * SB + 4 * q);
                r[4 * q] = pfma(-m.x, x, r[4 * q]);
                r[4 * q + 1] = pfma(-m.y, x, r[4 * q + 1]);
                r[4 * q + 2] = pfma(-m.z, x, r[4 * q + 2]);
                r[4 * q + 3] = pfma(-m.w, x, r[4 * q + 3]);
            }
        }
#pragma unroll
        for (int s = 0; s < SB; ++s) {
#pragma unroll
            for (int i = s + 1; i < SB; ++i) r[i] = pfma(-mt[(b * SB + s) * MP + b * SB + i], r[s], r[i]);
            *reinterpret_cast<float2*>(xc + (b * SB + s) * SOLVE_COLS) = r[s];
        }
    }
    const int col = col0 + 2 * tid;
    float* dst = is_k ? p.w + ((size_t)head * p.o.n_rows + at.row) * ROWS + col
                      : p.u + ((size_t)head * p.o.n_rows + at.row) * P + col - ROWS;
    const size_t step = is_k ? ROWS : P;
    for (int t = 0; t < at.n; ++t)
        *reinterpret_cast<float2*>(dst + t * step) = *reinterpret_cast<const float2*>(xc + t * SOLVE_COLS);
}

constexpr int WC = 32, UP = WC + 4;   // columns of a CTA that walks, pitch of its u
constexpr int WALK_STAGE = L * PITCH + L * ROWS + L * UP + L * 4;   // floats: W, k, U, gates
constexpr int WALK_BYTES = (2 * WALK_STAGE + WC * PITCH + L * UP) * (int)sizeof(float);

__global__ void __launch_bounds__(256) delta_chunk_walk_kernel(const DeltaParams p) {
    pdl_trigger();
    pdl_wait();
    extern __shared__ __align__(16) float smem[];
    float* ss = smem + 2 * WALK_STAGE;    // [WC][PITCH] the state, by columns
    float* us = ss + WC * PITCH;          // [L][UP] D[L][t] u_t
    const int e = blockIdx.x, head = blockIdx.y, P = p.o.P, p0 = blockIdx.z * WC;
    const int first = p.o.cu_rows[e], n = p.o.cu_rows[e + 1] - first;
    if (n <= 0) return;
    int chunk = 0;   // the entry's first
    for (int q = 0; q < e; ++q) {
        const int m = p.o.cu_rows[q + 1] - p.o.cu_rows[q];
        if (m > 0) chunk += (m + L - 1) / L;
    }
    const int count = (n + L - 1) / L;
    const int tid = threadIdx.x, warp = tid / 32, lane = tid % 32, ly = lane / 8, lx = lane % 8;
    const int g = head / (p.o.heads / p.o.groups);
    auto fetch = [&](int c) {
        float* st = smem + (c & 1) * WALK_STAGE;
        const size_t row = first + c * L;
        const int m = min(L, n - c * L);
        const float* w = p.w + ((size_t)head * p.o.n_rows + row) * ROWS;
        const float* k = p.o.bc + ((size_t)g * p.o.n_rows + row) * 2 * ROWS;
        const float* u = p.u + ((size_t)head * p.o.n_rows + row) * P + p0;
        const float* d = p.o.dd + ((size_t)head * p.o.n_rows + row) * 4;
#pragma unroll 4
        for (int i = tid; i < L * (ROWS / 4); i += 256) {
            const int t = i / (ROWS / 4), c4 = i % (ROWS / 4) * 4, from = t < m ? t : 0;
            cp_async16(st + t * PITCH + c4, w + (size_t)from * ROWS + c4, t < m);
            cp_async16(st + L * PITCH + t * ROWS + c4, k + (size_t)from * 2 * ROWS + c4, t < m);
        }
#pragma unroll
        for (int i = tid; i < L * (WC / 4); i += 256) {
            const int t = i / (WC / 4), c4 = i % (WC / 4) * 4, from = t < m ? t : 0;
            cp_async16(st + L * PITCH + L * ROWS + t * UP + c4, u + (size_t)from * P + c4, t < m);
        }
        if (tid < L) cp_async16(st + L * PITCH + L * ROWS + L * UP + tid * 4, d + (tid < m ? tid : 0) * 4, tid < m);
        asm volatile("cp.async.commit_group;\n" ::: "memory");
    };
    // a thread's part of the state: rows r4 .. + 3 of columns c0 .. + CPT - 1; a warp has 32 rows of 4 CPT columns, whose
    // factors it reads in one access each
    constexpr int CPT = WC * ROWS / 4 / 256;
    const int r4 = warp % (ROWS / 32) * 32 + lane % 8 * 4, c0 = warp / (ROWS / 32) * 4 * CPT + lane / 8 * CPT;
    float* state = p.o.state + (long long)p.o.slot_ids[e] * p.o.state_stride + ((size_t)head * P + p0 + c0) * ROWS + r4;
    float4 S[CPT];
#pragma unroll
    for (int j = 0; j < CPT; ++j) {
        S[j] = __ldcg(reinterpret_cast<const float4*>(state + (size_t)j * ROWS));
        *reinterpret_cast<float4*>(ss + (c0 + j) * PITCH + r4) = S[j];
    }
    fetch(0);
    for (int c = 0; c < count; ++c) {
        asm volatile("cp.async.wait_group 0;\n" ::: "memory");
        __syncthreads();   // the stage has come; the state is in shared memory; the other stage is read
        if (c + 1 < count) fetch(c + 1);
        const float* st = smem + (c & 1) * WALK_STAGE;
        const float* kc = st + L * PITCH;
        const float* uc = kc + L * ROWS;
        const float* dc = uc + L * UP;
        const int m = min(L, n - c * L);
        // D[L][t] of two tokens a lane, in every warp; the chunk's decay in lane 0
        const float g0 = 2 * lane < m ? dc[2 * lane * 4 + 1] : 1.f, g1 = 2 * lane + 1 < m ? dc[(2 * lane + 1) * 4 + 1] : 1.f;
        float after = g0 * g1;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const float v = __shfl_down_sync(0xffffffffu, after, o);
            if (lane + o < 32) after *= v;
        }
        float rest = __shfl_down_sync(0xffffffffu, after, 1);
        if (lane == 31) rest = 1.f;
        const float w1 = rest, w0 = g1 * rest, all = __shfl_sync(0xffffffffu, after, 0);
        // the state before the chunk, for the results
        float* carry = p.o.carry + (((size_t)head * p.o.chunks + chunk + c) * P + p0 + c0) * ROWS + r4;
#pragma unroll
        for (int j = 0; j < CPT; ++j) __stcg(reinterpret_cast<float4*>(carry + (size_t)j * ROWS), S[j]);
        // u = U - W S0: a thread tokens warp * 8 + ly and 4 further on, columns lx + 8 j
        float acc[2][4];
        dot_tile(st + (warp * 8 + ly) * PITCH, ss + lx * PITCH, PITCH, acc);
        float* ug = p.u + ((size_t)head * p.o.n_rows + first + c * L) * P + p0;
#pragma unroll
        for (int i = 0; i < 2; ++i) {
            const int t = warp * 8 + i * 4 + ly;
            const float even = __shfl_sync(0xffffffffu, w0, t / 2), odd = __shfl_sync(0xffffffffu, w1, t / 2);
            const float f = t & 1 ? odd : even;
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                const float v = uc[t * UP + lx + 8 * j] - acc[i][j];
                if (t < m) __stcg(ug + (size_t)t * P + lx + 8 * j, v);
                us[t * UP + lx + 8 * j] = t < m ? f * v : 0.f;
            }
        }
        __syncthreads();
        // S <- A_L S0 + sum_t k_t (D[L][t] u_t)^T
#pragma unroll
        for (int j = 0; j < CPT; ++j) S[j] = make_float4(S[j].x * all, S[j].y * all, S[j].z * all, S[j].w * all);
#pragma unroll 8
        for (int t = 0; t < L; ++t) {
            const float4 k = *reinterpret_cast<const float4*>(kc + t * ROWS + r4);
            float v[CPT];
            if (CPT == 4) *reinterpret_cast<float4*>(v) = *reinterpret_cast<const float4*>(us + t * UP + c0);
            else *reinterpret_cast<float2*>(v) = *reinterpret_cast<const float2*>(us + t * UP + c0);
#pragma unroll
            for (int j = 0; j < CPT; ++j) {
                float2* Sj = reinterpret_cast<float2*>(&S[j]);
                Sj[0] = pfma(v[j], make_float2(k.x, k.y), Sj[0]);
                Sj[1] = pfma(v[j], make_float2(k.z, k.w), Sj[1]);
            }
        }
#pragma unroll
        for (int j = 0; j < CPT; ++j) *reinterpret_cast<float4*>(ss + (c0 + j) * PITCH + r4) = S[j];
    }
#pragma unroll
    for (int j = 0; j < CPT; ++j) *reinterpret_cast<float4*>(state + (size_t)j * ROWS) = S[j];
}

}  // namespace

IB_EXPORT int ib_scan_chunk_rows() { return ROWS; }

// Floats of scratch a step of n_rows rows in n_entries entries takes.
IB_EXPORT long long ib_ssd_chunk_scratch(int n_rows, int n_entries, int heads, int groups, int P) {
    const long long chunks = n_rows / L + n_entries;
    return chunks * ((long long)heads * P * ROWS + (long long)groups * L * L + heads + 4);
}

// As ib_ssd_scan (scan.cu), bc float32 [groups][rows][2][ROWS] (B, then C); P a multiple of 64, x, bc, state, scratch and out 16-byte aligned, state_stride a multiple of 4.
IB_EXPORT int ib_ssd_chunk(const float* x, const void* bc, const void* dd, int n_rows, const float* d_skip, float* state,
                           long long state_stride, const int* cu_rows, const int* slot_ids, float* out, int n_entries,
                           int heads, int groups, int P, float* scratch, void* stream) {
    if (n_entries <= 0 || n_rows <= 0) return IB_OK;
    if (!x || !bc || !dd || !d_skip || !state || !cu_rows || !slot_ids || !out || !scratch || heads <= 0 || groups <= 0 ||
        heads % groups || P <= 0)
        return IB_ERR_BAD_ARG;
    if (P % PT || state_stride % 4 || ((uintptr_t)dd & 7) ||
        (((uintptr_t)x | (uintptr_t)bc | (uintptr_t)state | (uintptr_t)scratch | (uintptr_t)out) & 15))
        return IB_ERR_UNSUPPORTED;
    const int chunks = n_rows / L + n_entries;
    if ((long long)heads * (P / PT) + groups > 65535 || n_entries > 65535) return IB_ERR_TOO_LARGE;
    SsdParams p{x, (const float*)bc, (const float*)dd, d_skip, cu_rows, slot_ids, state, state_stride, scratch, nullptr,
                nullptr, out, n_rows, n_entries, chunks, heads, groups, P};
    p.cb = scratch + (size_t)chunks * heads * P * ROWS;
    p.decay = p.cb + (size_t)chunks * groups * L * L;
    static bool attr_done = false;
    if (!attr_done) {
        cudaError_t e = cudaFuncSetAttribute(ssd_chunk_state_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, STATE_BYTES);
        if (e == cudaSuccess)
            e = cudaFuncSetAttribute(chunk_out_kernel<false>, cudaFuncAttributeMaxDynamicSharedMemorySize, OUT_BYTES);
        if (e != cudaSuccess) return (int)e;
        attr_done = true;
    }
    cudaStream_t s = (cudaStream_t)stream;
    cudaError_t le = launch_kernel_in_order(ssd_chunk_state_kernel, dim3(chunks, heads * (P / PT) + groups), dim3(128),
                                            (size_t)STATE_BYTES, s, p);
    if (le == cudaSuccess)
        le = launch_kernel(ssd_chunk_pass_kernel, dim3((P * ROWS / 4 + 127) / 128, heads, n_entries), dim3(128), 0, s, p);
    if (le == cudaSuccess)
        le = launch_kernel(chunk_out_kernel<false>, dim3(chunks, heads, P / PT), dim3(128), (size_t)OUT_BYTES, s, p);
    if (le != cudaSuccess) return (int)le;
    IB_LAUNCH_CHECK();
    return IB_OK;
}

IB_EXPORT long long ib_delta_chunk_scratch(int n_rows, int n_entries, int heads, int groups, int P) {
    const long long chunks = n_rows / L + n_entries;
    return chunks * ((long long)heads * P * ROWS + 2LL * groups * L * L) + (long long)heads * n_rows * (P + ROWS);
}

// As ib_delta_scan (scan.cu), kq float32 [groups][rows][2][ROWS] (k, then q); P a multiple of 64, alignments as above, dd
// 16-byte aligned.
IB_EXPORT int ib_delta_chunk(const float* v, const void* kq, const void* dd, int n_rows, float* state,
                             long long state_stride, const int* cu_rows, const int* slot_ids, float* out, int n_entries,
                             int heads, int groups, int P, float* scratch, void* stream) {
    if (n_entries <= 0 || n_rows <= 0) return IB_OK;
    if (!v || !kq || !dd || !state || !cu_rows || !slot_ids || !out || !scratch || heads <= 0 || groups <= 0 ||
        heads % groups || P <= 0)
        return IB_ERR_BAD_ARG;
    if (P % PT || state_stride % 4 || (((uintptr_t)v | (uintptr_t)kq | (uintptr_t)dd | (uintptr_t)state | (uintptr_t)scratch |
                                        (uintptr_t)out) & 15))
        return IB_ERR_UNSUPPORTED;
    const int chunks = n_rows / L + n_entries;
    if (heads > 65535 || n_entries > 65535 || P / WC > 65535) return IB_ERR_TOO_LARGE;
    DeltaParams p;
    p.o = SsdParams{nullptr, (const float*)kq, (const float*)dd, nullptr, cu_rows, slot_ids, state, state_stride, scratch,
                    nullptr, nullptr, out, n_rows, n_entries, chunks, heads, groups, P};
    p.o.cb = scratch + (size_t)chunks * heads * P * ROWS;
    p.kk = p.o.cb + (size_t)chunks * groups * L * L;
    p.u = p.kk + (size_t)chunks * groups * L * L;
    p.w = p.u + (size_t)heads * n_rows * P;
    p.o.x = p.u;
    p.v = v;
    static bool attr_done = false;
    if (!attr_done) {
        cudaError_t e = cudaFuncSetAttribute(delta_chunk_dots_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, STATE_BYTES);
        if (e == cudaSuccess)
            e = cudaFuncSetAttribute(delta_chunk_solve_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, SOLVE_BYTES);
        if (e == cudaSuccess)
            e = cudaFuncSetAttribute(delta_chunk_walk_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, WALK_BYTES);
        if (e == cudaSuccess)
            e = cudaFuncSetAttribute(chunk_out_kernel<true>, cudaFuncAttributeMaxDynamicSharedMemorySize, OUT_BYTES);
        if (e != cudaSuccess) return (int)e;
        attr_done = true;
    }
    cudaStream_t s = (cudaStream_t)stream;
    cudaError_t le = launch_kernel_in_order(delta_chunk_dots_kernel, dim3(chunks, groups, 2), dim3(128), (size_t)STATE_BYTES, s, p);
    if (le == cudaSuccess)
        le = launch_kernel(delta_chunk_solve_kernel, dim3(chunks, heads, (ROWS + P + SOLVE_COLS - 1) / SOLVE_COLS), dim3(128),
                           (size_t)SOLVE_BYTES, s, p);
    if (le == cudaSuccess)
        le = launch_kernel(delta_chunk_walk_kernel, dim3(n_entries, heads, P / WC), dim3(256), (size_t)WALK_BYTES, s, p);
    if (le == cudaSuccess)
        le = launch_kernel(chunk_out_kernel<true>, dim3(chunks, heads, P / PT), dim3(128), (size_t)OUT_BYTES, s, p.o);
    if (le != cudaSuccess) return (int)le;
    IB_LAUNCH_CHECK();
    return IB_OK;
}
