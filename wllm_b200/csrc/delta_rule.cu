// The gated delta rule: a matrix state per (request, head) that every token first decays, then corrects towards its value
// along its key, then reads with its query:
//
//     S <- g_t S;    u_t = beta_t (v_t - S^T k_t);    S <- S + k_t u_t^T;    o_t = S^T q_t        S: [dim, vdim], 32-bit
//
// g_t in (0, 1) is one decay per head and token, or one per head, key channel and token (then it multiplies the rows of S one by
// one), beta_t in (0, 1) one step size per head and token.  q, k and v are each
// filtered along the sequence, channel by channel, by `taps` taps that look back only (the last tap weighs the token itself,
// inputs in front of the sequence count as zero) and pass SiLU; q and k are then scaled to unit length head by head.  Query and key heads may be
// fewer than value heads (head h reads q/k head h / (H / G)).  The state and the convolutions' last taps - 1 inputs live in
// the cache manager's state slots and are carried from step to step, so a whole prompt, a portion and a single decoded token
// are one case and, token by token, give the same bits (wllm_delta_blocks adds in another order).
//
//   wllm_delta_prepare      from a fused projection row (q | k | v | ... | b | a in one matrix product, possibly still in split-K
//                           slabs): convolution and SiLU of q, k and v, the unit norms x / sqrt(sum(x^2) + eps) (q also times
//                           q_scale), beta = sigmoid(b), g = exp(-exp(A_log) softplus(a + dt_bias)), all 32-bit.  A warp a head.
//                           Decays per key channel come from elsewhere (a low-rank map, linear_attention.cu): then beta alone.
//                           In a step of single tokens it also shifts the slots' inputs: the lane that read a channel's writes them.
//   wllm_delta_conv_update  the slots' last taps - 1 inputs after this step's tokens (a thread a channel, read first, written after).
//   wllm_delta_scan         the recurrence.  The columns of S do not meet: column j needs S[:, j] alone.  Eight or sixteen lanes
//                           hold a column (runs of four key channels each), a CTA of eight warps 32 or 16 columns of one
//                           (request, head); tokens arrive in tiles through a cp.async ring and are walked in order.  With
//                           a = S^T k and b = S^T q taken from the decayed state in one pass (two sums over a column's lanes),
//                           u = beta (v - g a) and o = g b + u (k . q), which is S^T q of the state that already holds the token's update.
//                           Decays per key channel come as g - 1 (a channel that forgets slowly has g close to one, and the rounding of g
//                           itself would grow with its memory): the lane's channels are decayed first, S + (g - 1) S, then summed.
//   wllm_delta_blocks       the same recurrence for portions of a bfloat16 model, eight tokens at a time (see delta_block_prepare_kernel).
#include "common.cuh"

__device__ __forceinline__ float dr_any(const void* p, int dtype, size_t i) {
    return dtype == WLLM_BF16 ? __bfloat162float(reinterpret_cast<const bf16*>(p)[i]) : reinterpret_cast<const float*>(p)[i];
}
// element i of a row that may come as `parts` 32-bit slabs `stride` elements apart, added in slab order
// An input from a tensor (AT_ONCE 0) or, where parts > 1, from slabs: part 0 + part 1 + ..., AT_ONCE loads in flight, the additions a chain.
template <int AT_ONCE>
__device__ __forceinline__ float dr_in(const void* p, int dtype, int parts, size_t stride, size_t i) {
    if (AT_ONCE == 0 || parts == 1) return dr_any(p, dtype, i);
    const float* f = reinterpret_cast<const float*>(p) + i;
    if (AT_ONCE == 1) {
        float v = f[0];
        for (int s = 1; s < parts; ++s) v += f[(size_t)s * stride];
        return v;
    }
    float v = 0.f;
    for (int s0 = 0; s0 < parts; s0 += AT_ONCE) {
        float part[AT_ONCE ? AT_ONCE : 1];
#pragma unroll
        for (int u = 0; u < AT_ONCE; ++u) part[u] = s0 + u < parts ? f[(size_t)(s0 + u) * stride] : 0.f;
#pragma unroll
        for (int u = 0; u < AT_ONCE; ++u)
            if (s0 + u < parts) v = s0 + u == 0 ? part[u] : v + part[u];
    }
    return v;
}
__device__ __forceinline__ float dr_silu(float z) { return z / (1.0f + expf(-z)); }
__device__ __forceinline__ float dr_softplus(float z) { return z > 20.f ? z : log1pf(expf(z)); }

constexpr int DR_MAX_TAPS = 16;
constexpr int DR_MAX_PER_LANE = 8;       // key or value channels a lane holds of a head in the prepare kernel: heads up to 256

// grid (tokens, ceil(units / 4)), 128 threads; unit < G: a query head, < 2G: a key head, < 2G + H: a value head, 2G + H: the
// token's beta and decay of every head.
// AT_ONCE: slabs with eight loads in flight take registers that leave five CTAs an SM, one after the other nine, as a tensor's tokens.  48 heads of
// 128 in five slabs, us with sixteen, eight and one at once: 24 tokens (312 CTAs) 14.9, 10.7, 11.3; 64 (832) 20.8, 16.9, 13.5.  A tensor, 64 tokens:
// 12.7 with the registers, 8.0 without.
constexpr int DR_PREPARE_CTAS = 5 * 148;
template <int AT_ONCE>
__global__ void __launch_bounds__(128, AT_ONCE > 1 ? 5 : 9)
delta_prepare_kernel(const void* __restrict__ fused, int in_dtype, int row_stride, int parts, size_t part_stride, int q_off,
                     int k_off, int v_off, int b_off, int a_off, int n, int H, int G, int D, int V, int taps,
                     const void* __restrict__ conv_q, const void* __restrict__ conv_k, const void* __restrict__ conv_v,
                     const void* __restrict__ a_log, const void* __restrict__ dt_bias, int w_dtype,
                     const int* __restrict__ token_req, const int* __restrict__ req_q_start, const int* __restrict__ req_q_len,
                     const int* __restrict__ req_slot, float* __restrict__ conv_state, float unit_eps, float q_scale, float* __restrict__ q,
                     float* __restrict__ k, float* __restrict__ v, float* __restrict__ beta, float* __restrict__ decay, int shift) {
    pdl_begin();
    auto in = [&](size_t at) { return dr_in<AT_ONCE>(fused, in_dtype, parts, part_stride, at); };
    const int t = blockIdx.x, warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int unit = blockIdx.y * 4 + warp;
    if (unit > 2 * G + H) return;
    if (unit == 2 * G + H) {
        for (int h = lane; h < H; h += 32) {
            const float bz = in((size_t)t * row_stride + b_off + h);
            beta[(size_t)t * H + h] = 1.0f / (1.0f + expf(-bz));
            if (a_off < 0) continue;                        // decays per key channel: worked out elsewhere
            const float az = in((size_t)t * row_stride + a_off + h);
            decay[(size_t)t * H + h] = expf(-expf(dr_any(a_log, w_dtype, h)) * dr_softplus(az + dr_any(dt_bias, w_dtype, h)));
        }
        return;
    }
    const int r = token_req[t];
    const int i = t - req_q_start[r], slot = req_slot[r];       // the token's place in its request's portion
    const int C = 2 * G * D + H * V;
    const bool keep = shift && slot >= 0 && req_q_len[r] > 0;   // (a row that stands for no token leaves the state alone)
    int col0, chan0, size, head;
    const void* w;
    if (unit < G) { head = unit; size = D; col0 = q_off + head * D; chan0 = head * D; w = conv_q; }
    else if (unit < 2 * G) { head = unit - G; size = D; col0 = k_off + head * D; chan0 = G * D + head * D; w = conv_k; }
    else { head = unit - 2 * G; size = V; col0 = v_off + head * V; chan0 = 2 * G * D + head * V; w = conv_v; }
    float y[DR_MAX_PER_LANE];
    float ss = 0.f;
#pragma unroll
    for (int e = 0; e < DR_MAX_PER_LANE; ++e) {
        const int c = lane + 32 * e;
        y[e] = 0.f;
        if (c < size) {
            float acc = 0.f;
            for (int j = taps - 1; j >= 0; --j) {            // the oldest input first: one order for every way of cutting
                float x;
                if (i - j >= 0) x = in((size_t)(t - j) * row_stride + col0 + c);
                else x = slot >= 0 ? conv_state[((size_t)slot * (taps - 1) + (taps - 1 + i - j)) * C + chan0 + c] : 0.f;
                acc = fmaf(dr_any(w, w_dtype, (size_t)(head * size + c) * taps + (taps - 1 - j)), x, acc);
                // every request brings one token: input j tokens back becomes input j + 1 back of the next one
                if (keep && j < taps - 1) conv_state[((size_t)slot * (taps - 1) + (taps - 2 - j)) * C + chan0 + c] = x;
            }
            y[e] = dr_silu(acc);
            ss = fmaf(y[e], y[e], ss);
        }
    }
    if (unit < 2 * G) {
        ss = warp_sum(ss);
        const float inv = (1.0f / sqrtf(ss + unit_eps)) * (unit < G ? q_scale : 1.0f);
        float* dst = (unit < G ? q : k) + ((size_t)t * G + head) * D;
#pragma unroll
        for (int e = 0; e < DR_MAX_PER_LANE; ++e)
            if (lane + 32 * e < size) dst[lane + 32 * e] = y[e] * inv;
    } else {
        float* dst = v + ((size_t)t * H + head) * V;
#pragma unroll
        for (int e = 0; e < DR_MAX_PER_LANE; ++e)
            if (lane + 32 * e < size) dst[lane + 32 * e] = y[e];
    }
}

// The same for many tokens, inputs in one tensor, convolutions of four taps: a warp takes a head of DR_RUN neighbouring tokens, so that a channel's
// taps and every input are read once a run instead of once a token and tap (a request that begins inside the run reads its first inputs'
// predecessors from the state as above).  Lanes, sums and their order are those of the kernel above: the bits are the same.
// Measured: 2,048 tokens, 48 heads of 128 channels, 166 us alone before; the whole step 1,704 -> 1,620 us (2,041 tokens, 24 heads: 1,792 -> 1,735).
constexpr int DR_RUN = 8, DR_RUN_TAPS = 4;
template <typename TI, int PER>
__global__ void __launch_bounds__(128)
delta_prepare_run_kernel(const TI* __restrict__ fused, int row_stride, int q_off, int k_off, int v_off, int b_off, int a_off, int n, int H, int G,
                         int D, int V, const void* __restrict__ conv_q, const void* __restrict__ conv_k, const void* __restrict__ conv_v,
                         const void* __restrict__ a_log, const void* __restrict__ dt_bias, int w_dtype, const int* __restrict__ token_req,
                         const int* __restrict__ req_q_start, const int* __restrict__ req_slot, const float* __restrict__ conv_state,
                         float unit_eps, float q_scale, float* __restrict__ q, float* __restrict__ k, float* __restrict__ v,
                         float* __restrict__ beta, float* __restrict__ decay) {
    constexpr int TAPS = DR_RUN_TAPS;
    pdl_launch_dependents();
    const int first = blockIdx.x * DR_RUN, count = min(DR_RUN, n - first), warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int unit = blockIdx.y * 4 + warp;
    if (unit > 2 * G + H) return;
    if (unit == 2 * G + H) {
        pdl_wait();
        for (int i = lane; i < count * H; i += 32) {
            const int t = first + i / H, h = i % H;
            beta[(size_t)t * H + h] = 1.0f / (1.0f + expf(-to_f32(fused[(size_t)t * row_stride + b_off + h])));
            if (a_off < 0) continue;
            const float az = to_f32(fused[(size_t)t * row_stride + a_off + h]);
            decay[(size_t)t * H + h] = expf(-expf(dr_any(a_log, w_dtype, h)) * dr_softplus(az + dr_any(dt_bias, w_dtype, h)));
        }
        return;
    }
    const int C = 2 * G * D + H * V;
    int col0, chan0, size, head;
    const void* w;
    if (unit < G) { head = unit; size = D; col0 = q_off + head * D; chan0 = head * D; w = conv_q; }
    else if (unit < 2 * G) { head = unit - G; size = D; col0 = k_off + head * D; chan0 = G * D + head * D; w = conv_k; }
    else { head = unit - 2 * G; size = V; col0 = v_off + head * V; chan0 = 2 * G * D + head * V; w = conv_v; }
    float taps[PER][TAPS];                       // written by no kernel: read while the predecessor still runs
#pragma unroll
    for (int e = 0; e < PER; ++e)
#pragma unroll
        for (int j = 0; j < TAPS; ++j)
            taps[e][j] = lane + 32 * e < size ? dr_any(w, w_dtype, (size_t)(head * size + lane + 32 * e) * TAPS + j) : 0.f;
    pdl_wait();
    float x[DR_RUN][PER];
#pragma unroll
    for (int i = 0; i < DR_RUN; ++i)
#pragma unroll
        for (int e = 0; e < PER; ++e)
            x[i][e] = i < count && lane + 32 * e < size ? to_f32(fused[(size_t)(first + i) * row_stride + col0 + lane + 32 * e]) : 0.f;
    float* dst = unit < G ? q + (size_t)head * D : (unit < 2 * G ? k + (size_t)head * D : v + (size_t)head * V);
    const size_t pitch = unit < 2 * G ? (size_t)G * D : (size_t)H * V;
    float back[TAPS - 1][PER];                   // the inputs of the TAPS - 1 tokens in front, the oldest first
    int r_before = -1;
#pragma unroll
    for (int i = 0; i < DR_RUN; ++i) {
        if (i >= count) break;
        const int t = first + i, r = token_req[t];
        if (r != r_before) {                     // the run's first token, or a request's
            const int at = t - req_q_start[r], slot = req_slot[r];
#pragma unroll
            for (int j = 1; j < TAPS; ++j)
#pragma unroll
                for (int e = 0; e < PER; ++e) {
                    const int c = lane + 32 * e;
                    float y = 0.f;
                    if (c < size) {
                        if (at - j >= 0) y = to_f32(fused[(size_t)(t - j) * row_stride + col0 + c]);
                        else if (slot >= 0) y = conv_state[((size_t)slot * (TAPS - 1) + (TAPS - 1 + at - j)) * C + chan0 + c];
                    }
                    back[TAPS - 1 - j][e] = y;
                }
            r_before = r;
        }
        float y[PER], ss = 0.f;
#pragma unroll
        for (int e = 0; e < PER; ++e) {
            float acc = 0.f;
#pragma unroll
            for (int j = 0; j < TAPS - 1; ++j) acc = fmaf(taps[e][j], back[j][e], acc);
            acc = fmaf(taps[e][TAPS - 1], x[i][e], acc);
            y[e] = lane + 32 * e < size ? dr_silu(acc) : 0.f;
            ss = fmaf(y[e], y[e], ss);
#pragma unroll
            for (int j = 0; j + 1 < TAPS - 1; ++j) back[j][e] = back[j + 1][e];
            back[TAPS - 2][e] = x[i][e];
        }
        float inv = 1.f;
        if (unit < 2 * G) inv = (1.0f / sqrtf(warp_sum(ss) + unit_eps)) * (unit < G ? q_scale : 1.0f);
#pragma unroll
        for (int e = 0; e < PER; ++e)
            if (lane + 32 * e < size) dst[(size_t)t * pitch + lane + 32 * e] = unit < 2 * G ? y[e] * inv : y[e];
    }
}

// The same for a step of single tokens and convolutions of four taps.  The kernel above takes a channel's inputs one after the other, and its writes of the
// slot's inputs keep the next channel's loads behind them; here a lane asks for everything it reads at once and writes at the end.  Same sums, same order.
// 32 requests, 24 heads of 128 in eight slabs or so: 16.3 -> 5.3 us; 8 requests, 48 heads: 10.4 -> 4.6 us (with the lone token's low-rank columns at once,
// linear_attention.cu, the decode steps 413 -> 400 and 309 -> 298 us).
template <int PER>
__global__ void __launch_bounds__(128)
delta_prepare_single_kernel(const void* __restrict__ fused, int in_dtype, int row_stride, int parts, size_t part_stride, int q_off, int k_off, int v_off,
                            int b_off, int a_off, int H, int G, int D, int V, const void* __restrict__ conv_q, const void* __restrict__ conv_k,
                            const void* __restrict__ conv_v, const void* __restrict__ a_log, const void* __restrict__ dt_bias, int w_dtype,
                            const int* __restrict__ token_req, const int* __restrict__ req_q_len, const int* __restrict__ req_slot,
                            float* __restrict__ conv_state, float unit_eps, float q_scale, float* __restrict__ q, float* __restrict__ k,
                            float* __restrict__ v, float* __restrict__ beta, float* __restrict__ decay) {
    constexpr int TAPS = DR_RUN_TAPS;
    pdl_launch_dependents();
    const int t = blockIdx.x, warp = threadIdx.x >> 5, lane = threadIdx.x & 31, unit = blockIdx.y * 4 + warp;
    if (unit > 2 * G + H) return;
    if (unit == 2 * G + H) {
        pdl_wait();
        for (int h = lane; h < H; h += 32) {
            const float bz = dr_in<16>(fused, in_dtype, parts, part_stride, (size_t)t * row_stride + b_off + h);
            beta[(size_t)t * H + h] = 1.0f / (1.0f + expf(-bz));
            if (a_off < 0) continue;
            const float az = dr_in<16>(fused, in_dtype, parts, part_stride, (size_t)t * row_stride + a_off + h);
            decay[(size_t)t * H + h] = expf(-expf(dr_any(a_log, w_dtype, h)) * dr_softplus(az + dr_any(dt_bias, w_dtype, h)));
        }
        return;
    }
    const int C = 2 * G * D + H * V;
    int col0, chan0, size, head;
    const void* w;
    if (unit < G) { head = unit; size = D; col0 = q_off + head * D; chan0 = head * D; w = conv_q; }
    else if (unit < 2 * G) { head = unit - G; size = D; col0 = k_off + head * D; chan0 = G * D + head * D; w = conv_k; }
    else { head = unit - 2 * G; size = V; col0 = v_off + head * V; chan0 = 2 * G * D + head * V; w = conv_v; }
    float taps[PER][TAPS];                       // written by no kernel: read while the predecessor still runs
#pragma unroll
    for (int e = 0; e < PER; ++e)
#pragma unroll
        for (int j = 0; j < TAPS; ++j)
            taps[e][j] = lane + 32 * e < size ? dr_any(w, w_dtype, (size_t)(head * size + lane + 32 * e) * TAPS + j) : 0.f;
    pdl_wait();
    const int r = token_req[t], slot = req_slot[r];
    const bool keep = slot >= 0 && req_q_len[r] > 0;
    float* st = conv_state + (size_t)(slot >= 0 ? slot : 0) * (TAPS - 1) * C + chan0;
    float x[PER][TAPS];                          // the oldest input first
#pragma unroll
    for (int e = 0; e < PER; ++e) {
        const int c = lane + 32 * e;
#pragma unroll
        for (int j = 0; j < TAPS - 1; ++j) x[e][j] = c < size && slot >= 0 ? st[(size_t)j * C + c] : 0.f;
        x[e][TAPS - 1] = c < size ? dr_in<16>(fused, in_dtype, parts, part_stride, (size_t)t * row_stride + col0 + c) : 0.f;
    }
    float y[PER], ss = 0.f;
#pragma unroll
    for (int e = 0; e < PER; ++e) {
        const int c = lane + 32 * e;
        float acc = 0.f;
#pragma unroll
        for (int j = 0; j < TAPS; ++j) acc = fmaf(taps[e][j], x[e][j], acc);
        y[e] = c < size ? dr_silu(acc) : 0.f;
        ss = fmaf(y[e], y[e], ss);
        if (keep && c < size) {
#pragma unroll
            for (int j = 0; j < TAPS - 1; ++j) st[(size_t)j * C + c] = x[e][j + 1];
        }
    }
    float inv = 1.f;
    if (unit < 2 * G) inv = (1.0f / sqrtf(warp_sum(ss) + unit_eps)) * (unit < G ? q_scale : 1.0f);
    float* dst = unit < G ? q + ((size_t)t * G + head) * D : (unit < 2 * G ? k + ((size_t)t * G + head) * D : v + ((size_t)t * H + head) * V);
#pragma unroll
    for (int e = 0; e < PER; ++e)
        if (lane + 32 * e < size) dst[lane + 32 * e] = unit < 2 * G ? y[e] * inv : y[e];
}

// grid (requests, ceil(C / 256)): a thread a channel; the taps - 1 inputs that end at the request's last token of this step.  AT_ONCE: as above (6,144
// channels, us with sixteen, eight and one at once: a tensor, 48 requests 5.8 with the registers, 3.9 without; eight slabs, 1 request 3.6, 3.1, 4.6, 64 9.5,
// 7.7, 6.5)
template <int AT_ONCE>
__global__ void __launch_bounds__(256)
delta_conv_update_kernel(const void* __restrict__ fused, int in_dtype, int row_stride, int parts, size_t part_stride, int q_off,
                         int k_off, int v_off, int H, int G, int D, int V, int taps, const int* __restrict__ req_q_start,
                         const int* __restrict__ req_q_len, const int* __restrict__ req_slot, float* __restrict__ conv_state) {
    pdl_begin();
    const int r = blockIdx.x, len = req_q_len[r], slot = req_slot[r];
    if (len <= 0 || slot < 0) return;
    const int C = 2 * G * D + H * V, ch = blockIdx.y * blockDim.x + threadIdx.x;
    if (ch >= C) return;
    const int col = ch < G * D ? q_off + ch : (ch < 2 * G * D ? k_off + ch - G * D : v_off + ch - 2 * G * D);
    const int keep = taps - 1, t0 = req_q_start[r];
    float* st = conv_state + (size_t)slot * keep * C + ch;
    float vals[DR_MAX_TAPS];
#pragma unroll
    for (int s = 0; s < DR_MAX_TAPS; ++s) {
        if (s < keep) {
            const int src = len - keep + s;               // place among this step's tokens; negative: an input kept from before
            vals[s] = src >= 0 ? dr_in<AT_ONCE>(fused, in_dtype, parts, part_stride, (size_t)(t0 + src) * row_stride + col)
                               : st[(size_t)(s + len) * C];
        }
    }
#pragma unroll
    for (int s = 0; s < DR_MAX_TAPS; ++s)
        if (s < keep) st[(size_t)s * C] = vals[s];
}

constexpr int DR_TT = 16;          // tokens of a tile
constexpr int DR_THREADS = 256;    // eight warps; with LPC lanes a column a warp holds 32 / LPC columns, a CTA 256 / LPC

__device__ __forceinline__ void dr_cp4(float* smem_dst, const float* src) {
    const unsigned dst = (unsigned)__cvta_generic_to_shared(smem_dst);
    asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"(dst), "l"(src) : "memory");
}
__device__ __forceinline__ void dr_cp16(float* smem_dst, const float* src) {      // both 16-byte aligned
    const unsigned dst = (unsigned)__cvta_generic_to_shared(smem_dst);
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dst), "l"(src) : "memory");
}

// One token of the walk for the lane's NE key channels of its column (see the kernel below).  CHANNEL: er holds g - 1 of every
// key channel, gt is not used.
template <int NE, int LPC, bool CHANNEL>
__device__ __forceinline__ void delta_token(float (&S)[NE], const float* __restrict__ kr, const float* __restrict__ qr,
                                            const float* __restrict__ er, int sub, float gt, float bt, float vt, float kq, float& o) {
    // the lane's channels: 4 sub + 4 LPC j + e (j < NE / 4, e < 4): a column's lanes read runs of 128 contiguous bytes a load
    float kv[NE], a4[4] = {0.f, 0.f, 0.f, 0.f}, b4[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
    for (int j = 0; j < NE / 4; ++j) {
        const float4 k4 = *reinterpret_cast<const float4*>(kr + 4 * sub + 4 * LPC * j);
        const float4 q4 = *reinterpret_cast<const float4*>(qr + 4 * sub + 4 * LPC * j);
        kv[4 * j] = k4.x; kv[4 * j + 1] = k4.y; kv[4 * j + 2] = k4.z; kv[4 * j + 3] = k4.w;
        if (CHANNEL) {
            const float4 e4 = *reinterpret_cast<const float4*>(er + 4 * sub + 4 * LPC * j);
            S[4 * j] = fmaf(e4.x, S[4 * j], S[4 * j]); S[4 * j + 1] = fmaf(e4.y, S[4 * j + 1], S[4 * j + 1]);
            S[4 * j + 2] = fmaf(e4.z, S[4 * j + 2], S[4 * j + 2]); S[4 * j + 3] = fmaf(e4.w, S[4 * j + 3], S[4 * j + 3]);
        }
        a4[0] = fmaf(S[4 * j], k4.x, a4[0]); a4[1] = fmaf(S[4 * j + 1], k4.y, a4[1]);
        a4[2] = fmaf(S[4 * j + 2], k4.z, a4[2]); a4[3] = fmaf(S[4 * j + 3], k4.w, a4[3]);
        b4[0] = fmaf(S[4 * j], q4.x, b4[0]); b4[1] = fmaf(S[4 * j + 1], q4.y, b4[1]);
        b4[2] = fmaf(S[4 * j + 2], q4.z, b4[2]); b4[3] = fmaf(S[4 * j + 3], q4.w, b4[3]);
    }
    float a = (a4[0] + a4[1]) + (a4[2] + a4[3]), b = (b4[0] + b4[1]) + (b4[2] + b4[3]);
#pragma unroll
    for (int off = 1; off < LPC; off <<= 1) {
        a += __shfl_xor_sync(0xffffffffu, a, off);
        b += __shfl_xor_sync(0xffffffffu, b, off);
    }
    const float u = CHANNEL ? bt * (vt - a) : bt * (vt - gt * a);
#pragma unroll
    for (int i = 0; i < NE; ++i) S[i] = CHANNEL ? fmaf(kv[i], u, S[i]) : fmaf(kv[i], u, gt * S[i]);
    o = CHANNEL ? fmaf(u, kq, b) : fmaf(u, kq, gt * b);
}

// LPC lanes hold a column, NE key channels each (dim <= LPC * NE, in runs of four).  grid (ceil(V / (256 / LPC)), H, requests),
// 256 threads.  The walk is one dependent chain a token (two sums over a column's lanes, the step, the update); a warp alone on
// its scheduler waits out every link of it, so heads of 64 channels and more spread a column over sixteen lanes: half the
// instructions a warp and token, twice the warps (one warp a scheduler issued a third of the time; profiles/delta_scan_2048.txt).
// Tiles of DR_TT tokens come through a ring of two cp.async stages, so that the
// next tile's rows are on their way while this one is walked; a key's and a query's rows are padded with zeros to 32 NE / 4
// channels in shared memory, so the walk carries no guards.  k . q of a tile's tokens is worked out once a tile by the
// warps together (it is the same for every column).
template <int NE, int LPC, int THREADS, bool CHANNEL>
__global__ void __launch_bounds__(THREADS)
delta_scan_kernel(const float* __restrict__ q, const float* __restrict__ k, const float* __restrict__ v,
                  const float* __restrict__ beta, const float* __restrict__ decay, float* __restrict__ state,
                  float* __restrict__ out, const int* __restrict__ req_q_start, const int* __restrict__ req_q_len,
                  const int* __restrict__ req_slot, int H, int G, int D, int V, int below) {
    constexpr int DP = LPC * NE;                        // channels of a row in shared memory
    constexpr int DR_COLS = THREADS / LPC;              // value columns of the CTA
    // two stages of [TT][DP] q, [TT][DP] k, (CHANNEL: [TT][DP] decay,) [TT][16] v, [TT] beta, [TT] decay; [TT] k.q
    extern __shared__ __align__(16) float dr_smem[];
    constexpr int ROWS = CHANNEL ? 3 : 2;
    pdl_begin();
    const int r = blockIdx.z, h = blockIdx.y;
    const int len = req_q_len[r], slot = req_slot[r];
    if (len <= 0 || slot < 0 || len >= below) return;      // a request that brings no token, or one that is walked in blocks
    const int g = h / (H / G), t0 = req_q_start[r];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, sub = lane & (LPC - 1);
    const int col0 = blockIdx.x * DR_COLS, mine = threadIdx.x / LPC, col = col0 + mine;
    const bool live = col < V;
    constexpr int per_stage = DR_TT * (ROWS * DP + DR_COLS + 2);
    float* kq = dr_smem + 2 * per_stage;
    const bool wide = (D & 3) == 0 && (V & 3) == 0 && ((((uintptr_t)q | (uintptr_t)k | (uintptr_t)v | (CHANNEL ? (uintptr_t)decay : 0)) & 15) == 0);
    if (D < DP)          // the channels behind the head's own stay zero in both stages
        for (int idx = threadIdx.x; idx < 2 * ROWS * DR_TT * (DP - D); idx += blockDim.x) {
            const int row = idx / (DP - D), c = D + idx % (DP - D);
            dr_smem[(row / (ROWS * DR_TT)) * per_stage + (row % (ROWS * DR_TT)) * DP + c] = 0.f;
        }
    auto load_tile = [&](int tile, int stage) {
        float* qs = dr_smem + stage * per_stage;
        float* ks = qs + DR_TT * DP;
        float* es = ks + DR_TT * DP;                       // CHANNEL alone
        float* vs = qs + ROWS * DR_TT * DP;
        float* bs = vs + DR_TT * DR_COLS;
        float* gs = bs + DR_TT;
        const int first = t0 + tile * DR_TT, count = min(DR_TT, len - tile * DR_TT);
        if (wide) {
            const int per_row = D >> 2;
            for (int idx = threadIdx.x; idx < count * per_row; idx += blockDim.x) {
                const int tt = idx / per_row, c = (idx - tt * per_row) * 4;
                const size_t at = ((size_t)(first + tt) * G + g) * D + c;
                dr_cp16(qs + tt * DP + c, q + at);
                dr_cp16(ks + tt * DP + c, k + at);
                if (CHANNEL) dr_cp16(es + tt * DP + c, decay + ((size_t)(first + tt) * H + h) * D + c);
            }
            for (int idx = threadIdx.x; idx < count * (DR_COLS / 4); idx += blockDim.x) {
                const int tt = idx / (DR_COLS / 4), cc = (idx % (DR_COLS / 4)) * 4;
                const float* vrow = v + ((size_t)(first + tt) * H + h) * V;
                if (col0 + cc + 3 < V) dr_cp16(vs + tt * DR_COLS + cc, vrow + col0 + cc);
                else
                    for (int e = 0; e < 4; ++e) dr_cp4(vs + tt * DR_COLS + cc + e, vrow + min(col0 + cc + e, V - 1));
            }
        } else {
            for (int idx = threadIdx.x; idx < count * D; idx += blockDim.x) {
                const int tt = idx / D, c = idx - tt * D;
                const size_t at = ((size_t)(first + tt) * G + g) * D + c;
                dr_cp4(qs + tt * DP + c, q + at);
                dr_cp4(ks + tt * DP + c, k + at);
                if (CHANNEL) dr_cp4(es + tt * DP + c, decay + ((size_t)(first + tt) * H + h) * D + c);
            }
            for (int idx = threadIdx.x; idx < count * DR_COLS; idx += blockDim.x) {
                const int tt = idx / DR_COLS, cc = idx % DR_COLS;
                dr_cp4(vs + idx, v + ((size_t)(first + tt) * H + h) * V + min(col0 + cc, V - 1));
            }
        }
        if (threadIdx.x < count) {
            dr_cp4(bs + threadIdx.x, beta + (size_t)(first + threadIdx.x) * H + h);
            if (!CHANNEL) dr_cp4(gs + threadIdx.x, decay + (size_t)(first + threadIdx.x) * H + h);
        }
        asm volatile("cp.async.commit_group;" ::: "memory");
    };
    float S[NE];
    float* Sg = state + (((size_t)slot * H + h) * D) * V;
#pragma unroll
    for (int i = 0; i < NE; ++i) {
        const int c = 4 * sub + 4 * LPC * (i >> 2) + (i & 3);
        S[i] = (live && c < D) ? Sg[(size_t)c * V + col] : 0.f;
    }
    const int tiles = (len + DR_TT - 1) / DR_TT;
    load_tile(0, 0);
    for (int tile = 0; tile < tiles; ++tile) {
        const int stage = tile & 1;
        if (tile + 1 < tiles) {
            load_tile(tile + 1, stage ^ 1);
            asm volatile("cp.async.wait_group 1;" ::: "memory");
        } else {
            asm volatile("cp.async.wait_group 0;" ::: "memory");
        }
        __syncthreads();                                   // the tile is here for everyone (and the zeros behind the heads, the first time)
        const float* qs = dr_smem + stage * per_stage;
        const float* ks = qs + DR_TT * DP;
        const float* es = CHANNEL ? ks + DR_TT * DP : ks;
        const float* vs = qs + ROWS * DR_TT * DP;
        const float* bs = vs + DR_TT * DR_COLS;
        const float* gs = bs + DR_TT;
        const int count = min(DR_TT, len - tile * DR_TT);
        for (int tt = warp; tt < count; tt += THREADS / 32) {     // k . q: a lane's strided chain, the warp's tree
            float acc = 0.f;
            for (int c = lane; c < D; c += 32) acc = fmaf(ks[tt * DP + c], qs[tt * DP + c], acc);
            acc = warp_sum(acc);
            if (lane == 0) kq[tt] = acc;
        }
        __syncthreads();
        float* orow = out + ((size_t)(t0 + tile * DR_TT) * H + h) * V + col;
        if (count == DR_TT) {
#pragma unroll 4
            for (int tt = 0; tt < DR_TT; ++tt) {
                float o;
                delta_token<NE, LPC, CHANNEL>(S, ks + tt * DP, qs + tt * DP, es + tt * DP, sub, CHANNEL ? 0.f : gs[tt], bs[tt],
                                              vs[tt * DR_COLS + mine], kq[tt], o);
                if (live && sub == 0) orow[(size_t)tt * H * V] = o;
            }
        } else {
            for (int tt = 0; tt < count; ++tt) {
                float o;
                delta_token<NE, LPC, CHANNEL>(S, ks + tt * DP, qs + tt * DP, es + tt * DP, sub, CHANNEL ? 0.f : gs[tt], bs[tt],
                                              vs[tt * DR_COLS + mine], kq[tt], o);
                if (live && sub == 0) orow[(size_t)tt * H * V] = o;
            }
        }
        __syncthreads();                                   // the stage and k . q are read to their end before the next tile overwrites them
    }
    if (live) {
#pragma unroll
        for (int i = 0; i < NE; ++i) {
            const int c = 4 * sub + 4 * LPC * (i >> 2) + (i & 3);
            if (c < D) Sg[(size_t)c * V + col] = S[i];
        }
    }
}

// The walk of a step whose requests bring one token each.  It is bound by reading and writing the states, and the layout above, made for long
// walks, reads them two neighbouring elements a row and instruction.  Here a warp has 32 neighbouring columns (128 contiguous bytes a row and
// instruction) and a quarter of the key channels; the four quarters' sums meet in shared memory.  A thread keeps, for each of the four lanes of the
// walk above that it stands for, that lane's chains, and adds them up in the order of that walk's exchanges: the bits are the same.
// 32 requests, 16 heads of 128 x 128 (67 MB there and back): 48.3 -> 18.4 us, the decode step 463 -> 430 us; 8 requests 14.0 -> 5.2 us, 315 -> 309 us.
// The walk and this, launches back to back: heads of 48, 32 requests 11.4 and 4.8 us, of 64 14.6 and 5.0, of 160 118 and 32; of 256 (a CTA's registers fill an
// SM) 180 and 71, 8 requests 45.8 and 14.4, one 7.9 and 4.4; a decay per channel as a decay per head within a tenth.
constexpr int DS_COLS = 64, DS_THREADS = 256;        // two column groups of a warp each, four quarters of the channels
template <int NE, bool CHANNEL>
__global__ void __launch_bounds__(DS_THREADS)
delta_single_kernel(const float* __restrict__ q, const float* __restrict__ k, const float* __restrict__ v, const float* __restrict__ beta,
                    const float* __restrict__ decay, float* __restrict__ state, float* __restrict__ out, const int* __restrict__ req_q_start,
                    const int* __restrict__ req_q_len, const int* __restrict__ req_slot, int H, int G, int D, int V) {
    constexpr int DP = 16 * NE;
    __shared__ __align__(16) float ks[DP], qs[DP], es[CHANNEL ? DP : 4];
    __shared__ float part[2][4][DS_COLS], kq_s;
    pdl_begin();
    const int r = blockIdx.z, h = blockIdx.y;
    const int len = req_q_len[r], slot = req_slot[r];
    if (len <= 0 || slot < 0) return;
    const int g = h / (H / G), t = req_q_start[r];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, quarter = warp >> 1;
    const int mine = (warp & 1) * 32 + lane, col = blockIdx.x * DS_COLS + mine;
    const bool live = col < V;
    float* Sg = state + (((size_t)slot * H + h) * D) * V + col;
    // channel of lane 4 quarter + u of the walk above, run j, element e
    auto channel = [&](int u, int j, int e) { return 4 * (4 * quarter + u) + 64 * j + e; };
    float S[4][NE];
#pragma unroll
    for (int u = 0; u < 4; ++u)
#pragma unroll
        for (int i = 0; i < NE; ++i) {
            const int c = channel(u, i >> 2, i & 3);
            S[u][i] = live && c < D ? Sg[(size_t)c * V] : 0.f;
        }
    for (int c = threadIdx.x; c < DP; c += DS_THREADS) {
        ks[c] = c < D ? k[((size_t)t * G + g) * D + c] : 0.f;
        qs[c] = c < D ? q[((size_t)t * G + g) * D + c] : 0.f;
        if (CHANNEL) es[c] = c < D ? decay[((size_t)t * H + h) * D + c] : 0.f;
    }
    const float bt = beta[(size_t)t * H + h], gt = CHANNEL ? 0.f : decay[(size_t)t * H + h];
    const float vt = live ? v[((size_t)t * H + h) * V + col] : 0.f;
    __syncthreads();
    if (warp == 0) {                                 // k . q, as the walk above adds it up
        float acc = 0.f;
        for (int c = lane; c < D; c += 32) acc = fmaf(ks[c], qs[c], acc);
        acc = warp_sum(acc);
        if (lane == 0) kq_s = acc;
    }
    float a[4], b[4];
#pragma unroll
    for (int u = 0; u < 4; ++u) {
        float a4[4] = {0.f, 0.f, 0.f, 0.f}, b4[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
        for (int j = 0; j < NE / 4; ++j) {
            float kv[4], qv[4], ev[4];
            *reinterpret_cast<float4*>(kv) = *reinterpret_cast<const float4*>(ks + channel(u, j, 0));
            *reinterpret_cast<float4*>(qv) = *reinterpret_cast<const float4*>(qs + channel(u, j, 0));
            if (CHANNEL) *reinterpret_cast<float4*>(ev) = *reinterpret_cast<const float4*>(es + channel(u, j, 0));
#pragma unroll
            for (int e = 0; e < 4; ++e) {
                float& x = S[u][4 * j + e];
                if (CHANNEL) x = fmaf(ev[e], x, x);
                a4[e] = fmaf(x, kv[e], a4[e]);
                b4[e] = fmaf(x, qv[e], b4[e]);
            }
        }
        a[u] = (a4[0] + a4[1]) + (a4[2] + a4[3]);
        b[u] = (b4[0] + b4[1]) + (b4[2] + b4[3]);
    }
    part[0][quarter][mine] = (a[0] + a[1]) + (a[2] + a[3]);
    part[1][quarter][mine] = (b[0] + b[1]) + (b[2] + b[3]);
    __syncthreads();
    const float sa = (part[0][0][mine] + part[0][1][mine]) + (part[0][2][mine] + part[0][3][mine]);
    const float u = CHANNEL ? bt * (vt - sa) : bt * (vt - gt * sa);
    if (quarter == 0 && live) {
        const float sb = (part[1][0][mine] + part[1][1][mine]) + (part[1][2][mine] + part[1][3][mine]);
        out[((size_t)t * H + h) * V + col] = CHANNEL ? fmaf(u, kq_s, sb) : fmaf(u, kq_s, gt * sb);
    }
    if (!live) return;
#pragma unroll
    for (int w = 0; w < 4; ++w)
#pragma unroll
        for (int i = 0; i < NE; ++i) {
            const int c = channel(w, i >> 2, i & 3);
            const float kc = ks[c];
            if (c < D) Sg[(size_t)c * V] = CHANNEL ? fmaf(kc, u, S[w][i]) : fmaf(kc, u, gt * S[w][i]);
        }
}

// fused [n, W] (or `parts` 32-bit slabs): q at q_off [G * D], k at k_off [G * D], v at v_off [H * V], b at b_off [H], a at a_off [H]
// (a_off < 0: the decays are worked out elsewhere; a_log, dt_bias and decay are not touched); shift: every request of the step brings at
// most one token, and conv_state is brought up to date here;
// conv_q, conv_k [G * D, taps], conv_v [H * V, taps], a_log, dt_bias [H] in one element type; conv_state [slots, taps - 1, 2 G D + H V];
// q, k [n, G, D], v [n, H, V], beta, decay [n, H], all 32-bit.
WLLM_API int wllm_delta_prepare(const void* fused, int in_dtype, int row_stride, int parts, long long part_stride, int q_off,
                                int k_off, int v_off, int b_off, int a_off, int n, int H, int G, int D, int V, int taps,
                                const void* conv_q, const void* conv_k, const void* conv_v, const void* a_log, const void* dt_bias,
                                int w_dtype, const int* token_req, const int* req_q_start, const int* req_q_len, const int* req_slot,
                                float* conv_state, float unit_eps, float q_scale, float* q, float* k, float* v, float* beta,
                                float* decay, int shift, cudaStream_t stream) {
    if (n <= 0) return WLLM_OK;
    if (H <= 0 || G <= 0 || H % G != 0 || D <= 0 || D > 32 * DR_MAX_PER_LANE || V <= 0 || V > 32 * DR_MAX_PER_LANE || taps < 1 ||
        taps > DR_MAX_TAPS || parts < 1 || (taps > 1 && conv_state == nullptr))
        return WLLM_BAD_SIZE;
    if ((in_dtype != WLLM_BF16 && in_dtype != WLLM_F32) || (w_dtype != WLLM_BF16 && w_dtype != WLLM_F32)) return WLLM_BAD_DTYPE;
    const int units = 2 * G + H + 1;
    if ((units + 3) / 4 > 65535) return WLLM_BAD_SIZE;
    // Runs where the CTAs of a token (and four heads) each would not be on the SMs at once, nine an SM: until then a run's eight tokens one after the
    // other are the longer chain.  48 heads of 128, 104 tokens (1,352 CTAs) 8.1 us a token each and 9.9 in runs, 128 (1,664) 12.6 and 9.9, 512 31 and 19;
    // 24 heads, 192 tokens 8.0 and 9.9, 224 (1,568) 12.1 and 9.9; heads of 64, 1,568 CTAs 7.7 and 8.3, 2,400 8.7 and 8.4.  Runs of heads over
    // 128 hold twice the registers and take twice the time: from a third round on (256, 2,048 CTAs 22.4 and 24.1).
    const bool few = D <= 128 && V <= 128;
    if ((long long)n * ((units + 3) / 4) > (few ? 1400 : 2700) && parts == 1 && taps == DR_RUN_TAPS && !shift) {
        const dim3 rgrid((n + DR_RUN - 1) / DR_RUN, (units + 3) / 4);
#define RUN(TI, PER) wllm_launch(delta_prepare_run_kernel<TI, PER>, rgrid, 128, 0, stream, (const TI*)fused, row_stride, q_off, k_off, v_off, b_off, \
                                 a_off, n, H, G, D, V, conv_q, conv_k, conv_v, a_log, dt_bias, w_dtype, token_req, req_q_start, req_slot, \
                                 (const float*)conv_state, unit_eps, q_scale, q, k, v, beta, decay)
        if (in_dtype == WLLM_BF16) return few ? RUN(bf16, 4) : RUN(bf16, 8);
        return few ? RUN(float, 4) : RUN(float, 8);
#undef RUN
    }
    if (shift && taps == DR_RUN_TAPS) {
#define ONE(PER) wllm_launch(delta_prepare_single_kernel<PER>, dim3(n, (units + 3) / 4), 128, 0, stream, fused, in_dtype, row_stride, parts, \
                             (size_t)part_stride, q_off, k_off, v_off, b_off, a_off, H, G, D, V, conv_q, conv_k, conv_v, a_log, dt_bias, w_dtype, \
                             token_req, req_q_len, req_slot, conv_state, unit_eps, q_scale, q, k, v, beta, decay)
        return few ? ONE(4) : ONE(8);
#undef ONE
    }
    const bool many = (long long)n * ((units + 3) / 4) > DR_PREPARE_CTAS;
    return wllm_launch(parts == 1 ? delta_prepare_kernel<0> : many ? delta_prepare_kernel<1> : delta_prepare_kernel<8>, dim3(n, (units + 3) / 4), 128, 0, stream, fused, in_dtype,
                       row_stride, parts, (size_t)part_stride, q_off, k_off, v_off, b_off, a_off, n, H, G, D, V, taps, conv_q, conv_k, conv_v, a_log,
                       dt_bias, w_dtype, token_req, req_q_start, req_q_len, req_slot, conv_state, unit_eps, q_scale, q, k, v, beta, decay, shift);
}

WLLM_API int wllm_delta_conv_update(const void* fused, int in_dtype, int row_stride, int parts, long long part_stride, int q_off,
                                    int k_off, int v_off, int H, int G, int D, int V, int taps, const int* req_q_start,
                                    const int* req_q_len, const int* req_slot, int requests, float* conv_state, cudaStream_t stream) {
    if (requests <= 0 || taps <= 1) return WLLM_OK;
    if (H <= 0 || G <= 0 || D <= 0 || V <= 0 || taps > DR_MAX_TAPS || parts < 1 || conv_state == nullptr) return WLLM_BAD_SIZE;
    if (in_dtype != WLLM_BF16 && in_dtype != WLLM_F32) return WLLM_BAD_DTYPE;
    const int C = 2 * G * D + H * V;
    if ((C + 255) / 256 > 65535) return WLLM_BAD_SIZE;
    const bool many = (long long)requests * ((C + 255) / 256) > 4 * 148;
    return wllm_launch(parts == 1 ? delta_conv_update_kernel<0> : many ? delta_conv_update_kernel<1> : delta_conv_update_kernel<8>,
                       dim3(requests, (C + 255) / 256), 256, 0, stream, fused, in_dtype, row_stride, parts, (size_t)part_stride, q_off, k_off, v_off, H, G, D, V, taps, req_q_start, req_q_len, req_slot, conv_state);
}

// state [slots, H, D, V]; out [n, H, V].  Requests by start, length and state slot; a length of 0 or a slot of -1 is passed by.
// decay [n, H], or (channel) [n, H, D] as g - 1.  Requests of `below` tokens or more are passed by (wllm_delta_blocks takes them).
// single: no request brings more than one token.
WLLM_API int wllm_delta_scan(const float* q, const float* k, const float* v, const float* beta, const float* decay, int channel, float* state,
                             float* out, const int* req_q_start, const int* req_q_len, const int* req_slot, int requests, int H,
                             int G, int D, int V, int below, int single, cudaStream_t stream) {
    if (requests <= 0) return WLLM_OK;
    if (H <= 0 || H > 65535 || G <= 0 || H % G != 0 || requests > 65535 || D <= 0 || D > 256 || V <= 0) return WLLM_BAD_SIZE;
    if (single && D > 32) {
        const dim3 sgrid((V + DS_COLS - 1) / DS_COLS, H, requests);
#define SINGLE2(NE, C) wllm_launch(delta_single_kernel<NE, C>, sgrid, DS_THREADS, 0, stream, q, k, v, beta, decay, state, out, req_q_start, req_q_len, \
                                   req_slot, H, G, D, V)
#define SINGLE(NE) (channel ? SINGLE2(NE, true) : SINGLE2(NE, false))
        return D <= 64 ? SINGLE(4) : (D <= 128 ? SINGLE(8) : SINGLE(16));
#undef SINGLE
#undef SINGLE2
    }
    // heads of up to 32 channels: eight lanes a column, four channels each; above: sixteen lanes, 4, 8 or 16 channels each
    const int lpc = D <= 32 ? 8 : 16, ne = D <= 64 ? 4 : (D <= 128 ? 8 : 16), threads = DR_THREADS;
    const int cols = threads / lpc;
    const dim3 grid((V + cols - 1) / cols, H, requests);
    const size_t smem = ((size_t)2 * DR_TT * ((channel ? 3 : 2) * lpc * ne + cols + 2) + DR_TT) * sizeof(float);
    static bool raised = false;
    if (!raised && smem > 48 * 1024) {
        cudaError_t e = cudaFuncSetAttribute(delta_scan_kernel<16, 16, DR_THREADS, false>, cudaFuncAttributeMaxDynamicSharedMemorySize, 128 * 1024);
        if (e == cudaSuccess) e = cudaFuncSetAttribute(delta_scan_kernel<16, 16, DR_THREADS, true>, cudaFuncAttributeMaxDynamicSharedMemorySize, 128 * 1024);
        if (e == cudaSuccess) e = cudaFuncSetAttribute(delta_scan_kernel<8, 16, DR_THREADS, true>, cudaFuncAttributeMaxDynamicSharedMemorySize, 128 * 1024);
        if (e != cudaSuccess) return 1000 + (int)e;
        raised = true;
    }
#define SCAN2(NE, LPC, TH, C) wllm_launch(delta_scan_kernel<NE, LPC, TH, C>, grid, TH, smem, stream, q, k, v, beta, decay, state, out, \
                                          req_q_start, req_q_len, req_slot, H, G, D, V, below)
#define SCAN(NE, LPC, TH) (channel ? SCAN2(NE, LPC, TH, true) : SCAN2(NE, LPC, TH, false))
    if (D <= 32) return SCAN(4, 8, DR_THREADS);
    if (D <= 64) return SCAN(4, 16, DR_THREADS);
    if (D <= 128) return SCAN(8, 16, DR_THREADS);
    return SCAN(16, 16, DR_THREADS);
#undef SCAN
#undef SCAN2
}

// ---------------------------------------------------------------------------------------------------
// The recurrence in blocks of eight tokens.  The walk above is bound by its chain: every token's state waits for two sums over a
// column's lanes of the state before it, some 600 cycles a token while the arithmetic fills a tenth of them.  Over a block that starts from S
// everything but S and the values can be worked out beforehand.  With G_i the product of the decays of tokens 0 .. i,
// A_ij = k_i . (G_i / G_j) k_j for j < i, P_ij = q_i . (G_i / G_j) k_j for j <= i, and T = (1 + diag(beta) A)^-1 diag(beta):
//
//     r_i = v_i - (G_i k_i)^T S;    o_i = (G_i q_i)^T S + sum_j N_ij r_j,  N = P T;    S <- G_7 S + sum_j M_j r_j^T,  M_j = sum_l T_lj (G_7 / G_l) k_l
//
// so that a block costs one pass over S for sixteen sums, one exchange, and one pass that updates it.  All of it in 32 bits.  The
// triangular solve is that of Joffrain, Low, Quintana-Orti, van de Geijn and Van Zee, "Accumulating Householder transformations, revisited" (2006), which
// Yang, Wang, Zhang, Shen and Kim, "Parallelizing linear transformers with the delta rule over sequence length" (2024), put to this use.  The
// ratios G_i / G_j are running products from token j + 1 on (no quotients, nothing overflows however fast a channel forgets), and
// decays given as g - 1 stay so: G_7 - 1 is carried and S + (G_7 - 1) S taken.
//
//   prepare   a CTA per (block, head, request), a thread a key channel: the 28 + 36 sums over the channels by a transposing tree (a warp's 64
//             values meet in 62 exchanges instead of 320), T by substitution, and the block's matrices in one contiguous piece.
//   walk      a CTA of eight warps has 16 columns of one (request, head), a warp two; a lane holds a thirty-second of the key channels of both,
//             in pairs (two products an instruction).  The 32 sums of a block and warp meet in 31 exchanges.  Shared memory bounds it: a row's
//             16-byte loads take four wavefronts a warp whether its lanes' addresses differ or not, so all 32 lanes lie along the channels.
//             (Four warps of four columns each, sixteen lanes a column: one warp a scheduler waits out its loads and exchanges, 354 us where this
//             form takes 267.)
//             Blocks arrive through a ring of cp.async stages.  The grid seldom exceeds the device's SMs, and a kernel that is
//             launched early finds some SMs still full: it asks for more than half an SM's shared memory then, so that its CTAs do
//             not pile up in pairs (the walk above took 1,490 us for 682 that way in a 2,048-token prompt of 16 heads of 128 x 128).
// Measured, 16 heads of 128 x 128, launches back to back: 2,048 tokens with a decay per channel 1,005 us by the walk above, 276 us here, a decay per head
// 800 and 273 us; 64 tokens 38 and 16, 30 and 16 us.  (The step of a 2,048-token prompt that it first replaced the walk in: 2,879 -> 1,704 us.)
// Which portions come here the caller says (`from`); 32-bit models stay on the walk, whose results do not depend on how a prompt is cut.
// ---------------------------------------------------------------------------------------------------
constexpr int DB = 8;                 // tokens of a block
constexpr int DB_COLS = 16, DB_THREADS = 256;
constexpr int DB_GROUP = 2, DB_STAGES = 3;       // blocks of a stage (the warps meet once a stage and drift apart inside it); stages
__host__ __device__ constexpr int db_channels(int D) { return D <= 64 ? 64 : (D <= 128 ? 128 : 256); }
// a block's piece: [8][DP] G k, [8][DP] G q, [8][DP] M, [DP] G_7 - 1 (or G_7), [8][8] N
__host__ __device__ constexpr int db_floats(int DP) { return (3 * DB + 1) * DP + DB * DB; }
__host__ __device__ constexpr int db_stage_floats(int DP) { return db_floats(DP) + DB * DB_COLS; }      // with the values of the CTA's columns
// A turn takes `turn` blocks of every request from its block b0 on.  The nth request (from 0) of `from` tokens or more that has any: its index (-1 past
// the last) and, in `before`, the turn's blocks of such requests in front of it: where its pieces begin.  The grids count these requests alone: beside decoded tokens a CTA of a request that has none would still take its turn for
// the walk's shared memory.  A warp together.
__device__ __forceinline__ int db_request(const int* __restrict__ req_q_len, int requests, int from, int b0, int turn, int nth, size_t& before) {
    const int lane = threadIdx.x & 31;
    before = 0;
    if (requests == 1) return req_q_len[0] >= from ? 0 : -1;
    for (int r0 = 0; r0 < requests; r0 += 32) {
        const int len = r0 + lane < requests ? req_q_len[r0 + lane] : 0, blocks = len >= from ? min((len + DB - 1) / DB - b0, turn) : 0;
        const unsigned found = __ballot_sync(0xffffffffu, blocks > 0);
        const unsigned here = __ballot_sync(0xffffffffu, blocks > 0 && __popc(found & ((1u << lane) - 1)) == nth);
        const int at = here ? __ffs(here) - 1 : 32;
        before += __reduce_add_sync(0xffffffffu, lane < at ? max(blocks, 0) : 0);
        if (here) return r0 + at;
        nth -= __popc(found);
    }
    return -1;
}

// (the bounds of both kernels keep the compiler from fitting one more CTA an SM with fewer registers: the walk of 2,041 tokens, a decay per channel,
// takes 289 us instead of 276 then)
template <int DP, bool CHANNEL>
__global__ void __launch_bounds__(DP, 896 / DP)
delta_block_prepare_kernel(const float* __restrict__ q, const float* __restrict__ k, const float* __restrict__ beta, const float* __restrict__ decay,
                           float* __restrict__ blocks, const int* __restrict__ req_q_start, const int* __restrict__ req_q_len,
                           const int* __restrict__ req_slot, int requests, int H, int G, int D, int from, int b0, int turn) {
    constexpr int WARPS = DP / 32, PAIRS = DB * (DB - 1) / 2;         // sums: 28 of A, then 36 of P
    __shared__ float sums[WARPS][64], A[DB][DB], P[DB][DB], T[DB][DB], bt[DB];
    pdl_begin();
    size_t before;
    const int r = db_request(req_q_len, requests, from, b0, turn, blockIdx.z, before), h = blockIdx.y;
    if (r < 0 || req_slot[r] < 0) return;
    const int at0 = (b0 + (int)blockIdx.x) * DB, len = req_q_len[r];
    if (at0 >= len) return;
    const int first = req_q_start[r] + at0, count = min(DB, len - at0), g = h / (H / G);
    const int d = threadIdx.x, warp = d >> 5, lane = d & 31;
    float kk[DB], qq[DB], e[DB];
#pragma unroll
    for (int i = 0; i < DB; ++i) {             // tokens past the portion's end: no key, no query, no step, no decay
        const bool in = i < count && d < D;
        const size_t at = ((size_t)(first + i) * G + g) * D + d;
        kk[i] = in ? k[at] : 0.f;
        qq[i] = in ? q[at] : 0.f;
        if (CHANNEL) e[i] = in ? decay[((size_t)(first + i) * H + h) * D + d] : 0.f;
        else e[i] = i < count ? decay[(size_t)(first + i) * H + h] : 1.f;
    }
    if (d < DB) bt[d] = d < count ? beta[(size_t)(first + d) * H + h] : 0.f;
    auto decayed = [&](float x, int i) { return CHANNEL ? fmaf(e[i], x, x) : e[i] * x; };
    float* piece = blocks + ((before + blockIdx.x) * H + h) * db_floats(DP);
    float x[64], last[DB];                      // last[j] = (G_7 / G_j) k_j
#pragma unroll
    for (int j = 0; j < DB; ++j) {
        float w = kk[j];
        x[PAIRS + j * (j + 1) / 2 + j] = qq[j] * w;
#pragma unroll
        for (int i = j + 1; i < DB; ++i) {
            w = decayed(w, i);
            x[i * (i - 1) / 2 + j] = kk[i] * w;
            x[PAIRS + i * (i + 1) / 2 + j] = qq[i] * w;
        }
        last[j] = w;
    }
    float E = CHANNEL ? 0.f : 1.f;               // G_i - 1, or G_i
#pragma unroll
    for (int i = 0; i < DB; ++i) {
        E = CHANNEL ? fmaf(e[i], E, E) + e[i] : e[i] * E;
        piece[i * DP + d] = CHANNEL ? fmaf(E, kk[i], kk[i]) : E * kk[i];
        piece[(DB + i) * DP + d] = CHANNEL ? fmaf(E, qq[i], qq[i]) : E * qq[i];
    }
    piece[3 * DB * DP + d] = E;
    // 64 values over 32 lanes: each exchange halves the values a lane keeps; lane l ends with values 2 l' and 2 l' + 1, l' = l
#pragma unroll
    for (int half = 32, off = 16; off > 0; half >>= 1, off >>= 1) {
        const bool upper = lane & off;
#pragma unroll
        for (int i = 0; i < 32; ++i)
            if (i < half) {
                const float keep = upper ? x[i + half] : x[i], send = upper ? x[i] : x[i + half];
                x[i] = keep + __shfl_xor_sync(0xffffffffu, send, off);
            }
    }
    sums[warp][2 * lane] = x[0];
    sums[warp][2 * lane + 1] = x[1];
    __syncthreads();
    if (d < 64) {
        float v = sums[0][d];
#pragma unroll
        for (int w = 1; w < WARPS; ++w) v += sums[w][d];
        int at = d < PAIRS ? d : d - PAIRS, i = d < PAIRS ? 1 : 0;
        const int width = d < PAIRS ? 0 : 1;       // row i of A holds i sums, of P i + 1
        while (at >= i + width) { at -= i + width; ++i; }
        (d < PAIRS ? A : P)[i][at] = v;
    }
    __syncthreads();
    if (d < DB) {                                // column d of T
        float t[DB];
#pragma unroll
        for (int i = 0; i < DB; ++i) {
            float v = i == d ? 1.f : 0.f;
#pragma unroll
            for (int j = 0; j < DB; ++j)
                if (j < i && j >= d) v = fmaf(-A[i][j], t[j], v);
            t[i] = i >= d ? bt[i] * v : 0.f;
            T[i][d] = t[i];
        }
    }
    __syncthreads();
#pragma unroll
    for (int l = 0; l < DB; ++l) {
        float m = 0.f;
#pragma unroll
        for (int j = l; j < DB; ++j) m = fmaf(T[j][l], last[j], m);
        piece[(2 * DB + l) * DP + d] = m;
    }
    if (d < 64) {
        const int i = d >> 3, l = d & 7;
        float v = 0.f;
        for (int j = l; j <= i; ++j) v = fmaf(P[i][j], T[j][l], v);
        piece[(3 * DB + 1) * DP + d] = v;
    }
}

__device__ __forceinline__ float2 dr_mul2(float2 a, float2 b) { return make_float2(a.x * b.x, a.y * b.y); }

// channels of a lane: 4 lane + 128 j + 0 .. 3 (two: 2 lane, 2 lane + 1), as pairs
template <int NP>
__device__ __forceinline__ void db_row(const float* row, int lane, float2 (&w)[NP]) {
    if constexpr (NP == 1) w[0] = *reinterpret_cast<const float2*>(row + 2 * lane);
    else {
#pragma unroll
        for (int j = 0; j < NP / 2; ++j) {
            const float4 t = *reinterpret_cast<const float4*>(row + 4 * lane + 128 * j);
            w[2 * j] = make_float2(t.x, t.y);
            w[2 * j + 1] = make_float2(t.z, t.w);
        }
    }
}
template <int NP>
__device__ __forceinline__ int db_channel(int lane, int p) { return NP == 1 ? 2 * lane : 4 * lane + 128 * (p >> 1) + 2 * (p & 1); }

template <int DP, bool CHANNEL>
__global__ void __launch_bounds__(DB_THREADS, 2)
delta_block_walk_kernel(const float* __restrict__ blocks, const float* __restrict__ v, float* __restrict__ state, float* __restrict__ out,
                        const int* __restrict__ req_q_start, const int* __restrict__ req_q_len, const int* __restrict__ req_slot, int requests,
                        int H, int D, int V, int from, int b0, int turn) {
    constexpr int FLOATS = db_floats(DP), STAGE = db_stage_floats(DP), NP = DP / 64;        // NP pairs of channels a thread and column
    extern __shared__ __align__(16) float db_smem[];                         // [DB_STAGES][DB_GROUP][STAGE]: a block's piece, [8][16] values
    __shared__ __align__(16) float rs[DB_THREADS / 32][2 * DB];
    pdl_begin();
    size_t before;
    const int r = db_request(req_q_len, requests, from, b0, turn, blockIdx.z, before), h = blockIdx.y;
    if (r < 0) return;
    const int len = min(req_q_len[r] - b0 * DB, turn * DB), slot = req_slot[r];
    if (slot < 0) return;
    const int t0 = req_q_start[r] + b0 * DB, count = (len + DB - 1) / DB;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int col0 = blockIdx.x * DB_COLS, col = col0 + 2 * warp;            // this warp's columns: col, col + 1
    const float* src = blocks + (before * H + h) * FLOATS;
    auto load = [&](int group) {
#pragma unroll
        for (int u = 0; u < DB_GROUP; ++u) {
            const int b = group * DB_GROUP + u;
            if (b >= count) break;
            const float* piece = src + (size_t)b * H * FLOATS;
            float* to = db_smem + ((group % DB_STAGES) * DB_GROUP + u) * STAGE;
            for (int i = threadIdx.x * 4; i < FLOATS; i += DB_THREADS * 4) dr_cp16(to + i, piece + i);
            if (threadIdx.x < DB * DB_COLS) {      // (places outside the portion or the head repeat its last token or column, and reach nothing)
                const int t = min(b * DB + (int)threadIdx.x / DB_COLS, len - 1), c = min(col0 + (int)threadIdx.x % DB_COLS, V - 1);
                dr_cp4(to + FLOATS + threadIdx.x, v + ((size_t)(t0 + t) * H + h) * V + c);
            }
        }
        asm volatile("cp.async.commit_group;" ::: "memory");                 // (an empty group keeps the count of groups)
    };
    for (int a = 0; a < DB_STAGES - 1; ++a) load(a);
    float2 S[2][NP];
    float* Sg = state + (((size_t)slot * H + h) * D) * V;
#pragma unroll
    for (int p = 0; p < NP; ++p) {
        const int c = db_channel<NP>(lane, p);
#pragma unroll
        for (int m = 0; m < 2; ++m) {
            const bool in = col + m < V;
            S[m][p].x = in && c < D ? Sg[(size_t)c * V + col + m] : 0.f;
            S[m][p].y = in && c + 1 < D ? Sg[(size_t)(c + 1) * V + col + m] : 0.f;
        }
    }
    // lane 8 m + i ends with the sum behind r_i of column m, lane 16 + 8 m + i with that behind its output
    const int tok = lane & 7, mine = (lane >> 3) & 1;
    for (int b = 0; b < count; ++b) {
        const int group = b / DB_GROUP;
        if (b % DB_GROUP == 0) {
            asm volatile("cp.async.wait_group %0;" ::"n"(DB_STAGES - 2) : "memory");
            __syncthreads();                    // the stage is here for everyone, and the one before is read to its end
            load(group + DB_STAGES - 1);        // into the stage before
        }
        const float* K = db_smem + ((group % DB_STAGES) * DB_GROUP + b % DB_GROUP) * STAGE;
        const float* M = K + 2 * DB * DP;
        const float* E = M + DB * DP;
        const float* N = E + DP;
        const float vt = K[FLOATS + tok * DB_COLS + 2 * warp + mine];
        float x[32];
#pragma unroll
        for (int i = 0; i < 2 * DB; ++i) {      // rows of G k, then of G q
            float2 w[NP], acc[2] = {make_float2(0.f, 0.f), make_float2(0.f, 0.f)};
            db_row<NP>(K + i * DP, lane, w);
#pragma unroll
            for (int p = 0; p < NP; ++p) {
                acc[0] = fma2(w[p], S[0][p], acc[0]);
                acc[1] = fma2(w[p], S[1][p], acc[1]);
            }
            x[(i & 8) * 2 + (i & 7)] = acc[0].x + acc[0].y;
            x[(i & 8) * 2 + 8 + (i & 7)] = acc[1].x + acc[1].y;
        }
        // 32 sums over 32 lanes in 31 exchanges: lane l ends with sum l
#pragma unroll
        for (int off = 16; off > 0; off >>= 1) {
            const bool upper = lane & off;
#pragma unroll
            for (int i = 0; i < 16; ++i)
                if (i < off) {
                    const float keep = upper ? x[i + off] : x[i], send = upper ? x[i] : x[i + off];
                    x[i] = keep + __shfl_xor_sync(0xffffffffu, send, off);
                }
        }
        if (lane < 16) rs[warp][lane] = b * DB + tok < len ? vt - x[0] : 0.f;        // (past the end a value that is no number must not reach the state)
        __syncwarp();
        float rj[2][DB];
#pragma unroll
        for (int u = 0; u < 4; ++u) *reinterpret_cast<float4*>(&rj[u >> 1][4 * (u & 1)]) = *reinterpret_cast<const float4*>(&rs[warp][4 * u]);
        if (lane >= 16 && b * DB + tok < len && col + mine < V) {
            float nr[DB], o = x[0];
            *reinterpret_cast<float4*>(nr) = *reinterpret_cast<const float4*>(N + tok * DB);
            *reinterpret_cast<float4*>(nr + 4) = *reinterpret_cast<const float4*>(N + tok * DB + 4);
#pragma unroll
            for (int j = 0; j < DB; ++j)        // a select, not N's zeros: a later token's r may be no number
                if (j <= tok) o = fmaf(nr[j], mine ? rj[1][j] : rj[0][j], o);
            out[((size_t)(t0 + b * DB + tok) * H + h) * V + col + mine] = o;
        }
        __syncwarp();                           // r is read to its end before the next block's takes its place
        float2 e[NP];
        db_row<NP>(E, lane, e);
#pragma unroll
        for (int p = 0; p < NP; ++p)
#pragma unroll
            for (int m = 0; m < 2; ++m) S[m][p] = CHANNEL ? fma2(e[p], S[m][p], S[m][p]) : dr_mul2(e[p], S[m][p]);
#pragma unroll
        for (int l = 0; l < DB; ++l) {
            float2 w[NP];
            db_row<NP>(M + l * DP, lane, w);
#pragma unroll
            for (int p = 0; p < NP; ++p)
#pragma unroll
                for (int m = 0; m < 2; ++m) S[m][p] = fma2(w[p], make_float2(rj[m][l], rj[m][l]), S[m][p]);
        }
    }
    asm volatile("cp.async.wait_group 0;" ::: "memory");
#pragma unroll
    for (int p = 0; p < NP; ++p) {
        const int c = db_channel<NP>(lane, p);
#pragma unroll
        for (int m = 0; m < 2; ++m) {
            if (col + m >= V) continue;
            if (c < D) Sg[(size_t)c * V + col + m] = S[m][p].x;
            if (c + 1 < D) Sg[(size_t)(c + 1) * V + col + m] = S[m][p].y;
        }
    }
}

// Floats of scratch that wllm_delta_blocks wants for n tokens of `requests` requests: every block's piece, or DB_SCRATCH floats (128 MB; 5,100 tokens of 16 heads
// of 128), whichever is less, but eight blocks a request.  Longer portions are walked in turns, the state handed on through its slot: the same bits.
constexpr long long DB_SCRATCH = 32ll << 20;
WLLM_API long long wllm_delta_block_floats(int n, int requests, int H, int D) {
    const long long block = (long long)H * db_floats(db_channels(D)), all = (long long)n / DB + requests;
    long long most = DB_SCRATCH / block;
    if (most < 8ll * requests) most = 8ll * requests;
    return (all < most ? all : most) * block;
}

template <int DP, bool CHANNEL>
static int launch_blocks(const float* q, const float* k, const float* v, const float* beta, const float* decay, float* state, float* out,
                         float* blocks, const int* req_q_start, const int* req_q_len, const int* req_slot, int requests, int walked, int most,
                         int H, int G, int D, int V, int from, int turn, int sms, cudaStream_t stream) {
    const dim3 grid((V + DB_COLS - 1) / DB_COLS, H, walked);
    constexpr size_t stage = (size_t)db_stage_floats(DP) * sizeof(float);      // 7,168, 13,568 or 26,368 bytes
    static bool raised = false;
    if (!raised) {
        const cudaError_t e = cudaFuncSetAttribute(delta_block_walk_kernel<DP, CHANNEL>, cudaFuncAttributeMaxDynamicSharedMemorySize, 176 * 1024);
        if (e != cudaSuccess) return 1000 + (int)e;
        raised = true;
    }
    size_t smem = DB_STAGES * DB_GROUP * stage;          // 42, 80 or 155 KB
    const size_t least = ((long long)grid.x * grid.y * grid.z <= sms ? 120 : 80) * 1024;       // at most one CTA an SM, or two
    if (smem < least) smem = least;
    for (int b0 = 0; b0 < most; b0 += turn) {
        const int mine = most - b0 < turn ? most - b0 : turn;
        int code = wllm_launch(delta_block_prepare_kernel<DP, CHANNEL>, dim3(mine, H, walked), DP, 0, stream, q, k, beta, decay, blocks, req_q_start,
                               req_q_len, req_slot, requests, H, G, D, from, b0, mine);
        if (code == WLLM_OK)
            code = wllm_launch(delta_block_walk_kernel<DP, CHANNEL>, grid, DB_THREADS, smem, stream, (const float*)blocks, v, state, out, req_q_start,
                               req_q_len, req_slot, requests, H, D, V, from, b0, mine);
        if (code != WLLM_OK) return code;
    }
    return WLLM_OK;
}

// wllm_delta_scan with the requests of `from` tokens or more among the step's n in blocks (the longest has max_len; `walked`: how many there are, 0: not
// known), the others, if there are any, token by token behind them.  One call, since a step of short portions is bound by the host; launched: how many
// kernels it was.  blocks: scratch, 16-byte aligned, of the floats that wllm_delta_block_floats names or of any less that hold a block of each (more turns, the
// same bits); sms: the device's multiprocessors.
WLLM_API int wllm_delta_blocks(const float* q, const float* k, const float* v, const float* beta, const float* decay, int channel, float* state,
                               float* out, float* blocks, long long blocks_floats, const int* req_q_start, const int* req_q_len, const int* req_slot,
                               int n, int requests, int walked, int max_len, int H, int G, int D, int V, int from, int sms, int* launched,
                               cudaStream_t stream) {
    *launched = 0;
    if (requests <= 0) return WLLM_OK;
    if (max_len < from) {
        *launched = 1;
        return wllm_delta_scan(q, k, v, beta, decay, channel, state, out, req_q_start, req_q_len, req_slot, requests, H, G, D, V, from, 0, stream);
    }
    const bool rest = walked != requests;
    if (walked <= 0) walked = requests;
    if (walked > requests) return WLLM_BAD_SIZE;
    if (H <= 0 || H > 65535 || G <= 0 || H % G != 0 || requests > 65535 || D <= 0 || D > 256 || V <= 0 || from < 1) return WLLM_BAD_SIZE;
    if ((uintptr_t)blocks & 15) return WLLM_BAD_ALIGN;
    const int DP = db_channels(D), most = (max_len + DB - 1) / DB;
    const long long room = blocks_floats / ((long long)H * db_floats(DP));             // blocks of all heads
    const long long each = room >= (long long)n / DB + walked ? most : room / walked;  // (all of them, wherever they lie)
    if (each < 1) return WLLM_BAD_SIZE;
    const int turn = each < most ? (int)each : most;
    *launched = 2 * ((most + turn - 1) / turn) + (rest ? 1 : 0);
#define BLOCKS2(DP, C) launch_blocks<DP, C>(q, k, v, beta, decay, state, out, blocks, req_q_start, req_q_len, req_slot, requests, walked, most, H, \
                                            G, D, V, from, turn, sms, stream)
#define BLOCKS(DP) (channel ? BLOCKS2(DP, true) : BLOCKS2(DP, false))
    const int code = DP == 64 ? BLOCKS(64) : (DP == 128 ? BLOCKS(128) : BLOCKS(256));
#undef BLOCKS
#undef BLOCKS2
    if (code != WLLM_OK || !rest) return code;
    return wllm_delta_scan(q, k, v, beta, decay, channel, state, out, req_q_start, req_q_len, req_slot, requests, H, G, D, V, from, 0, stream);
}
