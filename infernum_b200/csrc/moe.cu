// Routing of a mixture of experts.
//   z = router logits [N, E] (32-bit) + bias;  the `top` largest are chosen (the
//   lower index among equals), and their weights are the softmax over the chosen
//   logits only.  Written two ways: the lists ids[N, top] / weights[N, top] in
//   order of falling logit, and the dense row gate[N, E] that holds a chosen
//   expert's weight and 0 elsewhere.
// One warp per row; the row is kept in shared memory and a chosen logit is
// struck out there.
//
// A second way of scoring (ib_moe_route_scored): s_e = sigmoid(z_e); expert e belongs to
// group floor(e / (E / n_groups)); G_g = the sum of the `group_top` largest s_e of group g;
// the `keep` groups with the largest G_g stay open and the others' experts are struck out
// (n_groups <= 1: nothing is struck out); the `top` largest scores among those are
// chosen, the lower index among equals, and are the weights as they are - or,
// with `renorm`, divided by their sum.
#include "common.cuh"

using namespace ib;

// Router logits z[n, e] = sum_k x[n, k] w[e, k] in 32-bit: one warp per (row,
// expert), lanes stride over k, then a fixed tree over the lanes; a row's logits do
// not depend on the batch.  The product is skinny (a handful of experts, K in the
// thousands): a tiled product would leave one CTA walking all of K.
template <typename TX, typename TW>
__global__ void router_logits_kernel(const TX* __restrict__ x, int ldx, const TW* __restrict__ w, int ldw,
                                     float* __restrict__ z, int n_rows, int E, int K) {
    pdl_trigger();
    pdl_wait();
    const int warp = (blockIdx.x * blockDim.x + threadIdx.x) >> 5, lane = threadIdx.x & 31;
    if (warp >= n_rows * E) return;
    const int n = warp / E, e = warp % E;
    const TX* xr = x + (size_t)n * ldx;
    const TW* wr = w + (size_t)e * ldw;
    float acc = 0.f;
    for (int k = lane; k < K; k += 32) acc = fmaf(to_f32(xr[k]), to_f32(wr[k]), acc);
    acc = warp_sum(acc);
    if (lane == 0) z[(size_t)n * E + e] = acc;
}

// Eight neighbouring values of a row in 32-bit (16-byte aligned).
__device__ __forceinline__ void load8(const bf16* p, float (&v)[8]) {
    const uint4 r = __ldcg(reinterpret_cast<const uint4*>(p));
    const __nv_bfloat162* h = reinterpret_cast<const __nv_bfloat162*>(&r);
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        const float2 f = __bfloat1622float2(h[i]);
        v[2 * i] = f.x;
        v[2 * i + 1] = f.y;
    }
}
__device__ __forceinline__ void load8(const float* p, float (&v)[8]) {
    const float4 a = __ldcg(reinterpret_cast<const float4*>(p)), b = __ldcg(reinterpret_cast<const float4*>(p) + 1);
    v[0] = a.x; v[1] = a.y; v[2] = a.z; v[3] = a.w;
    v[4] = b.x; v[5] = b.y; v[6] = b.z; v[7] = b.w;
}

// The same for rows of eights: a CTA takes four rows by N experts (eight, where there are more than four), its four warps every fourth run of 256 k, a lane
// eight neighbouring k of a run.  An expert's values are converted once for four rows, a row's once for N experts.
// The lanes' sums meet by halves (31 shuffles for 32 logits) and the warps' in their order: a fixed order per logit,
// whatever the batch.  2,048 rows of 4,096, 16 experts: 64 us a warp a (row, expert) -> 17 us; eight rows 11 -> 5 us.
// N is 1, 2 or 4 where there are no more experts: one as eight took three times a warp a row (float32, 2,048 rows of
// 4,096: 22.6 us against 7.2; 8.1 as one, and 3.5 against 6.2 for eight rows).  Which N it is does not change a logit's order.
template <int N, typename TX, typename TW>
__global__ void __launch_bounds__(128) router_logits_tile_kernel(const TX* __restrict__ x, int ldx, const TW* __restrict__ w,
                                                                 int ldw, float* __restrict__ z, int n_rows, int E, int K) {
    pdl_trigger();
    pdl_wait();
    __shared__ float sums[4][32];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int row0 = blockIdx.x * 4, e0 = blockIdx.y * N;
    const TX* xr[4];
#pragma unroll
    for (int r = 0; r < 4; ++r) xr[r] = x + (size_t)min(row0 + r, n_rows - 1) * ldx;
    float v[32];   // [row][expert]
#pragma unroll
    for (int i = 0; i < 32; ++i) v[i] = 0.f;
    for (int k = warp * 256 + lane * 8; k < K; k += 1024) {
        float a[4][8];
#pragma unroll
        for (int r = 0; r < 4; ++r) load8(xr[r] + k, a[r]);
#pragma unroll
        for (int e = 0; e < N; ++e) {
            float b[8];
            load8(w + (size_t)min(e0 + e, E - 1) * ldw + k, b);
#pragma unroll
            for (int r = 0; r < 4; ++r)
#pragma unroll
                for (int i = 0; i < 8; ++i) v[r * 8 + e] = fmaf(a[r][i], b[i], v[r * 8 + e]);
        }
    }
    int o = 1;
#pragma unroll
    for (int n = 16; n >= 1; n >>= 1, o <<= 1) {
        const bool upper = lane & o;
#pragma unroll
        for (int i = 0; i < n; ++i) {
            const float give = upper ? v[i] : v[i + n], keep = upper ? v[i + n] : v[i];
            v[i] = keep + __shfl_xor_sync(0xffffffffu, give, o);
        }
    }
    sums[warp][__brev((unsigned)lane) >> 27] = v[0];   // (the logit a lane is left with: its bits reversed)
    __syncthreads();
    if (warp == 0) {
        const int row = row0 + lane / 8, e = e0 + lane % 8;
        if (row < n_rows && lane % 8 < N && e < E)
            z[(size_t)row * E + e] = ((sums[0][lane] + sums[1][lane]) + sums[2][lane]) + sums[3][lane];
    }
}

template <typename TX, typename TW>
static cudaError_t launch_router_tiles(const void* x, int ldx, const void* w, int ldw, float* z, int n_rows, int E, int K,
                                       cudaStream_t s) {
    const int n = E > 4 ? 8 : E > 2 ? 4 : E;
    const dim3 grid((n_rows + 3) / 4, (E + n - 1) / n);
    auto kernel = n == 8 ? router_logits_tile_kernel<8, TX, TW> : n == 4 ? router_logits_tile_kernel<4, TX, TW>
                : n == 2 ? router_logits_tile_kernel<2, TX, TW> : router_logits_tile_kernel<1, TX, TW>;
    return launch_kernel(kernel, grid, dim3(128), 0, s, (const TX*)x, ldx, (const TW*)w, ldw, z, n_rows, E, K);
}

template <typename TX, typename TW>
static bool rows_of_eights(const void* x, int ldx, const void* w, int ldw, int K) {
    return K % 8 == 0 && (size_t)ldx * sizeof(TX) % 16 == 0 && (size_t)ldw * sizeof(TW) % 16 == 0 && !((uintptr_t)x & 15) &&
           !((uintptr_t)w & 15);
}

IB_EXPORT int ib_router_logits(const void* x, int x_dtype, int ldx, const void* w, int w_dtype, int ldw, float* z,
                               int n_rows, int E, int K, void* stream) {
    if (n_rows <= 0) return IB_OK;
    if (!x || !w || !z || E <= 0 || K <= 0 || ldx < K || ldw < K) return IB_ERR_BAD_ARG;
    const long long warps = (long long)n_rows * E;
    const unsigned blocks = (unsigned)((warps + 7) / 8);
    cudaStream_t s = (cudaStream_t)stream;
    cudaError_t le;
    if (x_dtype == 0 && w_dtype == 0 && rows_of_eights<float, float>(x, ldx, w, ldw, K))
        le = launch_router_tiles<float, float>(x, ldx, w, ldw, z, n_rows, E, K, s);
    else if (x_dtype == 0 && w_dtype == 0)
        le = launch_kernel(router_logits_kernel<float, float>, dim3(blocks), dim3(256), 0, s, (const float*)x, ldx,
                           (const float*)w, ldw, z, n_rows, E, K);
    else if (x_dtype == 1 && w_dtype == 1 && rows_of_eights<bf16, bf16>(x, ldx, w, ldw, K))
        le = launch_router_tiles<bf16, bf16>(x, ldx, w, ldw, z, n_rows, E, K, s);
    else if (x_dtype == 1 && w_dtype == 1)
        le = launch_kernel(router_logits_kernel<bf16, bf16>, dim3(blocks), dim3(256), 0, s, (const bf16*)x, ldx,
                           (const bf16*)w, ldw, z, n_rows, E, K);
    else if (x_dtype == 1 && w_dtype == 0 && rows_of_eights<bf16, float>(x, ldx, w, ldw, K))
        le = launch_router_tiles<bf16, float>(x, ldx, w, ldw, z, n_rows, E, K, s);
    else if (x_dtype == 1 && w_dtype == 0)
        le = launch_kernel(router_logits_kernel<bf16, float>, dim3(blocks), dim3(256), 0, s, (const bf16*)x, ldx,
                           (const float*)w, ldw, z, n_rows, E, K);
    else
        return IB_ERR_UNSUPPORTED;
    if (le != cudaSuccess) return (int)le;
    IB_LAUNCH_CHECK();
    return IB_OK;
}

__global__ void moe_route_kernel(const float* __restrict__ logits, int ld, const float* __restrict__ bias, int E,
                                 int top, int* __restrict__ ids, float* __restrict__ weights,
                                 float* __restrict__ gate) {
    pdl_trigger();
    pdl_wait();
    extern __shared__ float z[];
    const int row = blockIdx.x, lane = threadIdx.x;
    const float* src = logits + (size_t)row * ld;
    for (int e = lane; e < E; e += 32) {
        z[e] = src[e] + (bias ? bias[e] : 0.f);
        if (gate) gate[(size_t)row * E + e] = 0.f;
    }
    __syncwarp();
    float zmax = 0.f, denom = 0.f;
    for (int k = 0; k < top; ++k) {
        float best = -INFINITY;
        int at = E;
        for (int e = lane; e < E; e += 32) {
            const float v = z[e];
            if (v > best || (v == best && e < at)) { best = v; at = e; }   // (NaN never wins)
        }
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) {
            const float ob = __shfl_xor_sync(0xffffffffu, best, o);
            const int oa = __shfl_xor_sync(0xffffffffu, at, o);
            if (ob > best || (ob == best && oa < at)) { best = ob; at = oa; }
        }
        if (at >= E) at = k < E ? k : 0;  // a row of NaN: any expert, weight NaN
        if (k == 0) zmax = best;
        const float p = expf(best - zmax);
        denom += p;
        if (lane == 0) {
            ids[(size_t)row * top + k] = at;
            weights[(size_t)row * top + k] = p;
            z[at] = -INFINITY;
        }
        __syncwarp();
    }
    if (lane == 0) {
        for (int k = 0; k < top; ++k) {
            const float w = weights[(size_t)row * top + k] / denom;
            weights[(size_t)row * top + k] = w;
            if (gate) gate[(size_t)row * E + ids[(size_t)row * top + k]] = w;
        }
    }
}

IB_EXPORT int ib_moe_route(const float* logits, int ld, const float* bias, int E, int top, int* ids,
                           float* weights, float* gate, int n_rows, void* stream) {
    if (n_rows <= 0) return IB_OK;
    if (!logits || !ids || !weights || E <= 0 || top <= 0 || top > E || ld < E) return IB_ERR_BAD_ARG;
    if ((size_t)E * sizeof(float) > 48 * 1024) return IB_ERR_TOO_LARGE;
    cudaError_t le = launch_kernel(moe_route_kernel, dim3(n_rows), dim3(32), (size_t)E * sizeof(float),
                                   (cudaStream_t)stream, logits, ld, bias, E, top, ids, weights, gate);
    if (le != cudaSuccess) return (int)le;
    IB_LAUNCH_CHECK();
    return IB_OK;
}

// Strikes out (-inf) the values z[E] of all but the `keep` best of `n_groups` equal groups of neighbours; a group's
// score, kept in gs[n_groups], is the sum of its `group_top` largest values, the lower index first among equals.
// By one warp; `group_top` > 1 needs groups of at most 64.
__device__ __forceinline__ void close_groups(float* z, float* gs, int E, int n_groups, int keep, int group_top,
                                             int lane) {
    const int per = E / n_groups;
    for (int g = lane; g < n_groups; g += 32) {
        float sum = 0.f;
        unsigned long long taken = 0ull;
        for (int k = 0; k < group_top && k < per; ++k) {
            float best = -INFINITY;
            int at = -1;
            for (int i = 0; i < per; ++i) {
                if (group_top > 1 && ((taken >> i) & 1ull)) continue;
                const float v = z[g * per + i];
                if (v > best) { best = v; at = i; }
            }
            if (at < 0) break;
            if (group_top > 1) taken |= 1ull << at;
            sum += best;
        }
        gs[g] = sum;
    }
    __syncwarp();
    // lane 0 picks the best groups; a chosen one is marked by -inf
    if (lane == 0) {
        for (int k = 0; k < keep; ++k) {
            float best = -INFINITY;
            int at = -1;
            for (int g = 0; g < n_groups; ++g)
                if (gs[g] > best) { best = gs[g]; at = g; }
            if (at < 0) break;
            gs[at] = -INFINITY;
        }
    }
    __syncwarp();
    for (int e = lane; e < E; e += 32)
        if (gs[e / per] != -INFINITY) z[e] = -INFINITY;
    __syncwarp();
}

__global__ void moe_route_scored_kernel(const float* __restrict__ logits, int ld, const float* __restrict__ bias,
                                        int E, int top, int n_groups, int keep, int group_top, int renorm,
                                        int* __restrict__ ids, float* __restrict__ weights,
                                        float* __restrict__ gate) {
    pdl_trigger();
    pdl_wait();
    extern __shared__ float z[];  // [E] scores, struck out as they are chosen; then [n_groups] group scores
    float* gs = z + E;
    const int row = blockIdx.x, lane = threadIdx.x;
    const float* src = logits + (size_t)row * ld;
    for (int e = lane; e < E; e += 32) {
        z[e] = 1.f / (1.f + expf(-(src[e] + (bias ? bias[e] : 0.f))));
        if (gate) gate[(size_t)row * E + e] = 0.f;
    }
    __syncwarp();
    if (n_groups > 1) close_groups(z, gs, E, n_groups, keep, group_top, lane);
    float denom = 0.f;
    for (int k = 0; k < top; ++k) {
        float best = -INFINITY;
        int at = E;
        for (int e = lane; e < E; e += 32) {
            const float v = z[e];
            if (v > best || (v == best && e < at)) { best = v; at = e; }
        }
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) {
            const float ob = __shfl_xor_sync(0xffffffffu, best, o);
            const int oa = __shfl_xor_sync(0xffffffffu, at, o);
            if (ob > best || (ob == best && oa < at)) { best = ob; at = oa; }
        }
        if (at >= E) { at = k < E ? k : 0; best = 0.f; }  // nothing left to choose (a row of NaN): weight 0
        denom += best;
        if (lane == 0) {
            ids[(size_t)row * top + k] = at;
            weights[(size_t)row * top + k] = best;
            z[at] = -INFINITY;
        }
        __syncwarp();
    }
    if (lane == 0) {
        for (int k = 0; k < top; ++k) {
            float w = weights[(size_t)row * top + k];
            if (renorm) {
                w = w / denom;
                weights[(size_t)row * top + k] = w;
            }
            if (gate) gate[(size_t)row * E + ids[(size_t)row * top + k]] = w;
        }
    }
}

IB_EXPORT int ib_moe_route_scored(const float* logits, int ld, const float* bias, int E, int top, int n_groups,
                                  int keep, int group_top, int renorm, int* ids, float* weights, float* gate,
                                  int n_rows, void* stream) {
    if (n_rows <= 0) return IB_OK;
    if (!logits || !ids || !weights || E <= 0 || top <= 0 || top > E || ld < E) return IB_ERR_BAD_ARG;
    if (n_groups > 1 && (E % n_groups || keep <= 0 || keep > n_groups || group_top <= 0 ||
                         (long long)keep * (E / n_groups) < top))
        return IB_ERR_BAD_ARG;
    if (n_groups > 1 && group_top > 1 && E / n_groups > 64) return IB_ERR_TOO_LARGE;
    const size_t smem = (size_t)(E + (n_groups > 1 ? n_groups : 0)) * sizeof(float);
    if (smem > 48 * 1024) return IB_ERR_TOO_LARGE;
    cudaError_t le = launch_kernel(moe_route_scored_kernel, dim3(n_rows), dim3(32), smem, (cudaStream_t)stream, logits,
                                   ld, bias, E, top, n_groups, keep, group_top, renorm, ids, weights, gate);
    if (le != cudaSuccess) return (int)le;
    IB_LAUNCH_CHECK();
    return IB_OK;
}

// A third way of scoring (ib_moe_route_softmax_all): s = softmax(z) over all E_all router
// outputs; the choice is made by s_e + correction_e (the lower index among equals), the
// weights are the chosen s_e (without the correction) over their sum + 1e-20, or - `renorm` 0 -
// as they are.  With n_groups > 1 only the experts of the `keep` best groups can be chosen,
// groups scored by the sum of their `group_top` largest choice values.  The last
// E_all - E outputs have no expert behind them: choosing one hands the token's input on
// with that weight.  Written: ids / weights [N, top]; the dense row gate[N, E] for the
// experts that exist; extra[N, 2] = (the sum of the weights that fell on the outputs
// without an expert, sigmoid(z[E_all]) when the logits carry one more column - the gate of
// an expert that every token uses - else 1).  With gate_cols > E the dense row is that wide and its
// columns from E on hold extra[n, 1]: the expert that every token uses, run as further columns of the
// experts' products.
__global__ void moe_route_softmax_all_kernel(const float* __restrict__ logits, int ld,
                                             const float* __restrict__ correction, int E_all, int E, int top,
                                             int with_gate, int* __restrict__ ids, float* __restrict__ weights,
                                             float* __restrict__ gate, float* __restrict__ extra, int gate_cols,
                                             int n_groups, int keep, int group_top, int renorm) {
    pdl_trigger();
    pdl_wait();
    extern __shared__ float sm[];
    float* s = sm;          // [E_all] the scores
    float* c = sm + E_all;  // [E_all] the choice values, struck out as they are chosen
    const int row = blockIdx.x, lane = threadIdx.x;
    const float* src = logits + (size_t)row * ld;
    float zmax = -INFINITY;
    for (int e = lane; e < E_all; e += 32) zmax = fmaxf(zmax, src[e]);
    zmax = warp_max(zmax);
    float part = 0.f;
    for (int e = lane; e < E_all; e += 32) {
        const float p = expf(src[e] - zmax);
        s[e] = p;
        part += p;
    }
    const float denom = warp_sum(part);
    __syncwarp();
    for (int e = lane; e < E_all; e += 32) {
        const float v = s[e] / denom;
        s[e] = v;
        c[e] = v + (correction ? correction[e] : 0.f);
        if (gate && e < E) gate[(size_t)row * gate_cols + e] = 0.f;
    }
    __syncwarp();
    if (n_groups > 1) close_groups(c, c + E_all, E_all, n_groups, keep, group_top, lane);
    float sum = 0.f;
    for (int k = 0; k < top; ++k) {
        float best = -INFINITY;
        int at = E_all;
        for (int e = lane; e < E_all; e += 32) {
            const float v = c[e];
            if (v > best || (v == best && e < at)) { best = v; at = e; }
        }
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) {
            const float ob = __shfl_xor_sync(0xffffffffu, best, o);
            const int oa = __shfl_xor_sync(0xffffffffu, at, o);
            if (ob > best || (ob == best && oa < at)) { best = ob; at = oa; }
        }
        if (at >= E_all) at = k < E_all ? k : 0;  // a row of NaN: any output
        sum += s[at];
        if (lane == 0) {
            ids[(size_t)row * top + k] = at;
            c[at] = -INFINITY;
        }
        __syncwarp();
    }
    if (lane == 0) {
        const float inv = renorm ? 1.f / (sum + 1e-20f) : 1.f;
        float passed = 0.f;
        for (int k = 0; k < top; ++k) {
            const int at = ids[(size_t)row * top + k];
            const float w = s[at] * inv;
            weights[(size_t)row * top + k] = w;
            if (at < E) {
                if (gate) gate[(size_t)row * gate_cols + at] = w;
            } else {
                passed += w;
            }
        }
        const float every = with_gate ? 1.f / (1.f + expf(-src[E_all])) : 1.f;
        if (extra) {
            extra[(size_t)row * 2] = passed;
            extra[(size_t)row * 2 + 1] = every;
        }
        if (gate)
            for (int e = E; e < gate_cols; ++e) gate[(size_t)row * gate_cols + e] = every;
    }
}

IB_EXPORT int ib_moe_route_softmax_all(const float* logits, int ld, const float* correction, int E_all, int E, int top,
                                       int with_gate, int* ids, float* weights, float* gate, float* extra,
                                       int gate_cols, int n_groups, int keep, int group_top, int renorm, int n_rows,
                                       void* stream) {
    if (n_rows <= 0) return IB_OK;
    if (!logits || !ids || !weights || E_all <= 0 || E < 0 || E > E_all || top <= 0 || top > E_all ||
        ld < E_all + (with_gate ? 1 : 0) || (gate && gate_cols < E))
        return IB_ERR_BAD_ARG;
    if (n_groups > 1 && (E_all % n_groups || keep <= 0 || keep > n_groups || group_top <= 0 ||
                         (long long)keep * (E_all / n_groups) < top))
        return IB_ERR_BAD_ARG;
    if (n_groups > 1 && group_top > 1 && E_all / n_groups > 64) return IB_ERR_TOO_LARGE;
    const size_t smem = (size_t)(E_all * 2 + (n_groups > 1 ? n_groups : 0)) * sizeof(float);
    if (smem > 48 * 1024) return IB_ERR_TOO_LARGE;
    cudaError_t le = launch_kernel(moe_route_softmax_all_kernel, dim3(n_rows), dim3(32), smem, (cudaStream_t)stream,
                                   logits, ld, correction, E_all, E, top, with_gate, ids, weights, gate, extra, gate_cols,
                                   n_groups, keep, group_top, renorm);
    if (le != cudaSuccess) return (int)le;
    IB_LAUNCH_CHECK();
    return IB_OK;
}

// out[n, :] = routed[n, :] + extra[n, 0] * h[n, :] + extra[n, 1] * shared[n, :]: the experts' weighted
// sum, the input handed on by the outputs without an expert, and the expert that every token uses behind
// its gate; `routed` and `shared` may be absent.  32-bit arithmetic, one rounding at the store.
template <typename T>
__global__ void moe_combine_kernel(const T* __restrict__ routed, const T* __restrict__ h, int h_stride,
                                   const T* __restrict__ shared, const float* __restrict__ extra,
                                   T* __restrict__ out, int n_rows, int W) {
    pdl_trigger();
    pdl_wait();
    const int row = blockIdx.x;
    const float passed = extra[(size_t)row * 2], g = extra[(size_t)row * 2 + 1];
    for (int i = blockIdx.y * blockDim.x + threadIdx.x; i < W; i += gridDim.y * blockDim.x) {
        float v = routed ? to_f32(routed[(size_t)row * W + i]) : 0.f;
        v = fmaf(passed, to_f32(h[(size_t)row * h_stride + i]), v);
        if (shared) v = fmaf(g, to_f32(shared[(size_t)row * W + i]), v);
        out[(size_t)row * W + i] = from_f32<T>(v);
    }
}

IB_EXPORT int ib_moe_combine(const void* routed, const void* h, int h_stride, const void* shared, const float* extra,
                             void* out, int dtype, int n_rows, int W, void* stream) {
    if (n_rows <= 0) return IB_OK;
    if (!h || !extra || !out || W <= 0 || h_stride < W) return IB_ERR_BAD_ARG;
    cudaStream_t s = (cudaStream_t)stream;
    const dim3 grid(n_rows, (W + 1023) / 1024), block(W >= 1024 ? 256 : 128);
    cudaError_t le;
    if (dtype == 0)
        le = launch_kernel(moe_combine_kernel<float>, grid, block, 0, s, (const float*)routed, (const float*)h, h_stride,
                           (const float*)shared, extra, (float*)out, n_rows, W);
    else if (dtype == 1)
        le = launch_kernel(moe_combine_kernel<bf16>, grid, block, 0, s, (const bf16*)routed, (const bf16*)h, h_stride,
                           (const bf16*)shared, extra, (bf16*)out, n_rows, W);
    else
        return IB_ERR_UNSUPPORTED;
    if (le != cudaSuccess) return (int)le;
    IB_LAUNCH_CHECK();
    return IB_OK;
}

// Who goes where: the (token, choice) pairs side by side expert by expert, in the order of the tokens.  By one CTA: a warp
// takes a run of tokens, counts its pairs per expert, and - once the counts before it are known - hands out places.
//   offsets[E + 3]    where each expert's rows begin, the last one's end; then 0 and N, the same for one expert of all rows
//   slot_of[N, top]   a pair's row, -1 where there is none (an output without an expert; an expert named again later in
//                     the row, whose last weight counts, as in the dense row of weights)
//   slot_scale[...]   a row's weight
constexpr int SORT_WARPS = 32;
__global__ void __launch_bounds__(SORT_WARPS * 32)
moe_sort_kernel(const int* __restrict__ ids, const float* __restrict__ weights, int n_rows, int top, int E,
                int* __restrict__ offsets, int* __restrict__ slot_of, float* __restrict__ slot_scale) {
    pdl_trigger();
    pdl_wait();
    extern __shared__ int place[];   // [SORT_WARPS][E]: a warp's pairs of an expert, then its next free row
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    int* mine = place + warp * E;
    for (int e = lane; e < E; e += 32) mine[e] = 0;
    __syncwarp();
    const int groups = (n_rows + 31) / 32, per = (groups + SORT_WARPS - 1) / SORT_WARPS;
    const int g0 = warp * per, g1 = min(groups, g0 + per);
    // Up to eight choices a token are read together; more one by one.  A pair's expert (E for none) waits in slot_of
    // until its place is known.
    constexpr int FIRST = 8;
    for (int g = g0; g < g1; ++g) {
        const int row = g * 32 + lane;
        const int* r = ids + (size_t)row * top;
        int first[FIRST];
#pragma unroll
        for (int j = 0; j < FIRST; ++j) first[j] = row < n_rows && j < top ? __ldcg(r + j) : -1;
        auto count = [&](int k, int e, bool again) {
            if (row >= n_rows || e < 0 || e >= E || again) e = E;
            if (row < n_rows) slot_of[(size_t)row * top + k] = e;
            const unsigned same = __match_any_sync(0xffffffffu, e);
            if (e < E && lane == __ffs(same) - 1) mine[e] += __popc(same);
            __syncwarp();
        };
#pragma unroll
        for (int k = 0; k < FIRST; ++k) {
            if (k >= top) break;
            bool again = false;
#pragma unroll
            for (int j = k + 1; j < FIRST; ++j) again |= first[j] == first[k];
            if (row < n_rows)
                for (int j = FIRST; j < top; ++j) again |= __ldcg(r + j) == first[k];
            count(k, first[k], again);
        }
        for (int k = FIRST; k < top; ++k) {
            const int e = row < n_rows ? __ldcg(r + k) : E;
            bool again = false;
            if (row < n_rows)
                for (int j = k + 1; j < top; ++j) again |= __ldcg(r + j) == e;
            count(k, e, again);
        }
    }
    __syncthreads();
    if (warp == 0) {
        int before = 0;
        for (int e0 = 0; e0 < E; e0 += 32) {
            const int e = e0 + lane;
            int total = 0;
            if (e < E) {
#pragma unroll
                for (int w = 0; w < SORT_WARPS; ++w) total += place[w * E + e];
            }
            int sum = total;
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const int up = __shfl_up_sync(0xffffffffu, sum, o);
                if (lane >= o) sum += up;
            }
            int at = before + sum - total;
            if (e < E) {
                offsets[e] = at;
                for (int w = 0; w < SORT_WARPS; ++w) {
                    const int n = place[w * E + e];
                    place[w * E + e] = at;
                    at += n;
                }
            }
            before += __shfl_sync(0xffffffffu, sum, 31);
        }
        if (lane == 0) {
            offsets[E] = before;
            offsets[E + 1] = 0;
            offsets[E + 2] = n_rows;
        }
    }
    __syncthreads();
    for (int g = g0; g < g1; ++g) {
        const int row = g * 32 + lane;
#pragma unroll 4
        for (int k = 0; k < top; ++k) {
            const int e = row < n_rows ? slot_of[(size_t)row * top + k] : E;   // (this thread's own)
            const float wt = row < n_rows ? __ldcg(weights + (size_t)row * top + k) : 0.f;
            const unsigned same = __match_any_sync(0xffffffffu, e);
            const int rank = __popc(same & ((1u << lane) - 1u));
            const int at = e < E ? mine[e] + rank : -1;
            __syncwarp();
            if (e < E && rank == 0) mine[e] += __popc(same);
            __syncwarp();
            if (row < n_rows) {
                slot_of[(size_t)row * top + k] = at;
                if (at >= 0) slot_scale[at] = wt;
            }
        }
    }
}

IB_EXPORT int ib_moe_sort(const int* ids, const float* weights, int n_rows, int top, int E, int* offsets, int* slot_of,
                          float* slot_scale, void* stream) {
    if (n_rows <= 0) return IB_OK;
    if (!ids || !weights || !offsets || !slot_of || !slot_scale || top <= 0 || E <= 0) return IB_ERR_BAD_ARG;
    if (E > 256) return IB_ERR_TOO_LARGE;
    cudaError_t le = launch_kernel(moe_sort_kernel, dim3(1), dim3(SORT_WARPS * 32), (size_t)SORT_WARPS * E * sizeof(int),
                                   (cudaStream_t)stream, ids, weights, n_rows, top, E, offsets, slot_of, slot_scale);
    if (le != cudaSuccess) return (int)le;
    IB_LAUNCH_CHECK();
    return IB_OK;
}

// Every token's row to the places of its pairs: xs[slot_of[n, k], :] = x[n, :], bf16, sixteen bytes a thread.
__global__ void moe_scatter_rows_kernel(const bf16* __restrict__ x, int ldx, const int* __restrict__ slot_of, int top,
                                        bf16* __restrict__ xs, int W) {
    pdl_trigger();
    pdl_wait();
    const int row = blockIdx.x;
    const int* to = slot_of + (size_t)row * top;
    for (int c = threadIdx.x * 8; c < W; c += blockDim.x * 8) {
        const uint4 v = __ldcg(reinterpret_cast<const uint4*>(x + (size_t)row * ldx + c));
        for (int k = 0; k < top; ++k) {
            const int s = __ldcg(to + k);
            if (s >= 0) *reinterpret_cast<uint4*>(xs + (size_t)s * W + c) = v;
        }
    }
}

IB_EXPORT int ib_moe_scatter_rows(const void* x, int ldx, const int* slot_of, int top, void* xs, int n_rows, int W,
                                  void* stream) {
    if (n_rows <= 0) return IB_OK;
    if (!x || !slot_of || !xs || top <= 0 || W <= 0 || ldx < W) return IB_ERR_BAD_ARG;
    if (W % 8 || ldx % 8 || ((uintptr_t)x & 15) || ((uintptr_t)xs & 15)) return IB_ERR_UNSUPPORTED;
    cudaError_t le = launch_kernel(moe_scatter_rows_kernel, dim3(n_rows), dim3(W >= 4096 ? 512 : W >= 2048 ? 256 : 128), 0,
                                   (cudaStream_t)stream, (const bf16*)x, ldx, slot_of, top, (bf16*)xs, W);
    if (le != cudaSuccess) return (int)le;
    IB_LAUNCH_CHECK();
    return IB_OK;
}

// out[n, :] = sum_k parts[slot_of[n, k], :] (+ shared[n, :]), the float32 results of a token's experts in the order of
// its choices, one rounding to bf16 at the store.
__global__ void moe_gather_sum_kernel(const float* __restrict__ parts, const int* __restrict__ slot_of, int top,
                                      const float* __restrict__ shared, bf16* __restrict__ out, int W) {
    pdl_trigger();
    pdl_wait();
    const int row = blockIdx.x;
    const int* from = slot_of + (size_t)row * top;
    for (int c = threadIdx.x * 4; c < W; c += blockDim.x * 4) {
        float4 a = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll 4
        for (int k = 0; k < top; ++k) {
            const int s = __ldcg(from + k);
            if (s < 0) continue;
            const float4 v = __ldcg(reinterpret_cast<const float4*>(parts + (size_t)s * W + c));
            a.x += v.x; a.y += v.y; a.z += v.z; a.w += v.w;
        }
        if (shared) {
            const float4 v = __ldcg(reinterpret_cast<const float4*>(shared + (size_t)row * W + c));
            a.x += v.x; a.y += v.y; a.z += v.z; a.w += v.w;
        }
        __nv_bfloat162 lo = __floats2bfloat162_rn(a.x, a.y), hi = __floats2bfloat162_rn(a.z, a.w);
        uint2 packed;
        packed.x = *reinterpret_cast<unsigned*>(&lo);
        packed.y = *reinterpret_cast<unsigned*>(&hi);
        *reinterpret_cast<uint2*>(out + (size_t)row * W + c) = packed;
    }
}

IB_EXPORT int ib_moe_gather_sum(const float* parts, const int* slot_of, int top, const float* shared, void* out, int n_rows,
                                int W, void* stream) {
    if (n_rows <= 0) return IB_OK;
    if (!parts || !slot_of || !out || top <= 0 || W <= 0) return IB_ERR_BAD_ARG;
    if (W % 4 || ((uintptr_t)parts & 15) || ((uintptr_t)shared & 15) || ((uintptr_t)out & 7)) return IB_ERR_UNSUPPORTED;
    cudaError_t le = launch_kernel(moe_gather_sum_kernel, dim3(n_rows), dim3(W >= 4096 ? 512 : W >= 2048 ? 256 : 128), 0,
                                   (cudaStream_t)stream, parts, slot_of, top, shared, (bf16*)out, W);
    if (le != cudaSuccess) return (int)le;
    IB_LAUNCH_CHECK();
    return IB_OK;
}
