// Attention over the paged cache, one warp per (token, query head), every size.
//
// A token at position p of request r attends to the keys first..p of r, where
// first = 0, or p - window + 1 when the layer has a window, or the start of p's block of -window positions when `window`
// is negative (a mask of blocks: see first_visible_key); the keys are found
// through the request's row of the block table.  The keys and values of this
// step's own tokens are already in the pages when the kernel runs, so a portion
// of a prompt, a whole prompt and a single decoded token are the same case.
//
// Scores, softmax statistics and the output accumulate in 32-bit (expf, no fast
// math), in an order that is a function of the keys' absolute positions alone:
//   chunk    64 keys that start at an absolute multiple of 64.  Its partial result
//            (max m, sum l, output o) starts from nothing and takes the chunk's keys
//            in tiles of 32 (absolute multiples of 32) with the running-maximum rule.
//   row      the chunks' partial results merged one after the other in ascending
//            order:  m' = max(m, mc), l = l e^(m-m') + lc e^(mc-m'), o likewise.
// So a token's output depends on its own query and keys only: not on what else is
// in the batch, nor on how the sequence was cut into steps, nor on which pages hold
// it, nor on which of the two kernels below computed it, bit for bit:
//   walk     one warp per (token, head) takes the row's chunks in turn.  Steps of
//            many rows (prompts and their portions).
//   split    one warp per (token, head, chunk) leaves its partial result in scratch
//            memory and a second kernel merges a row's chunks in order.  Steps of few
//            rows over long contexts (decoding), where a walk would leave most SMs idle.
//   tiled    a CTA takes 32 rows of one (request, key/value head) and brings every tile
//            of 32 keys and values into shared memory once for all of them; each warp
//            runs its four rows against the tile with the walk's arithmetic.  Portions
//            of prompts, where neighbouring rows read the same keys.
//
// Value heads may have a size of their own (`vd`; the output row of a head has that size), and a head may have a
// sink: a learned number s_h that joins the softmax's denominator as one more term e^(s_h) with no key and no
// value, neither scaled nor counted twice.  It enters when a row is finished, after the last chunk was merged:
//   m' = max(m, s_h);  l' = l e^(m-m') + e^(s_h-m');  out = o e^(m-m') / l'
//
// Two more options of the score rule and the mask.  `cap` > 0: a score becomes cap * tanh(score / cap) after the
// scale.  `keep` > 0 (with a window): the first `keep` keys of a sequence stay visible behind the window, at their
// true positions: key j is seen from position p when j <= p and (p - j < window or j < keep).  A row then touches
// the chunks of its kept keys (from chunk 0 on) and the chunks of its window, each once, in ascending order; tiles
// of 32 keys without a visible key are passed by (their pages may have been given back).
//
// `slopes` (one 32-bit number per query head, or null): a score loses slope_h * (p - j) for the key at position j seen from
// position p, after the scale and the cap: a bias by distance, in 32-bit from the two positions themselves.
//
// `v_ld`: elements between two value rows of the pool; with v_ld = hd and v_pages = k_pages the values are the first vd
// elements of the keys' rows (a cache that holds one row per token for both).
//
// Used for the 32-bit path at every size, and for bfloat16 at the sizes that the
// tensor-core kernels refuse.
#include "common.cuh"

constexpr int WARPS = 4;
constexpr int CHUNK = 64;

template <typename T> struct Vec;
template <> struct Vec<float> {
    static constexpr int N = 4;
    __device__ static void load(const float* p, float* out) {
        const float4 v = *reinterpret_cast<const float4*>(p);
        out[0] = v.x; out[1] = v.y; out[2] = v.z; out[3] = v.w;
    }
};
template <> struct Vec<bf16> {
    static constexpr int N = 8;
    __device__ static void load(const bf16* p, float* out) {
        const uint4 v = *reinterpret_cast<const uint4*>(p);
        const __nv_bfloat162* h = reinterpret_cast<const __nv_bfloat162*>(&v);
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            const float2 f = __bfloat1622float2(h[i]);
            out[2 * i] = f.x; out[2 * i + 1] = f.y;
        }
    }
};


// What a row at position `pos` sees: the keys [0, kept) and [first, pos] (kept = 0: no keys behind the window, or the
// two runs touch and first = 0).  Its chunks: 0 .. head_chunks-1, then first_chunk .. last_chunk.
struct RowKeys { int first, kept, first_chunk, last_chunk, head_chunks; };
__device__ __forceinline__ RowKeys row_keys(int pos, int window, int keep) {
    RowKeys r;
    r.first = first_visible_key(pos, window);
    r.kept = 0;
    if (keep > 0) {
        if (r.first <= keep) r.first = 0; else r.kept = keep;
    }
    r.first_chunk = r.first / CHUNK;
    r.last_chunk = pos / CHUNK;
    r.head_chunks = r.kept > 0 ? min((r.kept - 1) / CHUNK + 1, r.first_chunk) : 0;
    return r;
}
__device__ __forceinline__ int row_chunk(const RowKeys& r, int slot) { return slot < r.head_chunks ? slot : r.first_chunk + slot - r.head_chunks; }
__device__ __forceinline__ int row_chunk_count(const RowKeys& r) { return r.head_chunks + r.last_chunk - r.first_chunk + 1; }

// The partial result of one chunk of one row (every lane holds m and l; lane x holds o of the dimensions e*32+x).
template <typename T, int NE>
__device__ __forceinline__ void chunk_partial(const float* __restrict__ qs, const T* __restrict__ k_pages,
                                              const T* __restrict__ v_pages, const int* __restrict__ table, int nkv,
                                              int kvh, int hd, int vd, int v_ld, int page_size, int first, int kept, int pos, int chunk, float scale,
                                              float cap, float slope, int lane, float& m, float& l, float (&o)[NE]) {
    m = -INFINITY;
    l = 0.f;
#pragma unroll
    for (int e = 0; e < NE; ++e) o[e] = 0.f;
    const int lo = chunk * CHUNK < kept ? chunk * CHUNK : max(chunk * CHUNK, (first >> 5) << 5), hi = min(chunk * CHUNK + CHUNK - 1, pos);
    for (int tile = lo; tile <= hi; tile += 32) {
        const int key = tile + lane;
        const bool valid = (key >= first || key < kept) && key <= pos;
        const unsigned seen = __ballot_sync(0xffffffffu, valid);
        if (seen == 0u) continue;             // a tile between the kept keys and the window
        float s = -INFINITY;
        int row = -1;  // index of the key's row of head_dim elements inside the pool
        if (valid) {
            const int page = table[key / page_size];
            row = (page * nkv + kvh) * page_size + key % page_size;
            const T* kr = k_pages + (size_t)row * hd;
            float acc[4] = {0.f, 0.f, 0.f, 0.f};
            float kv[Vec<T>::N];
#pragma unroll 16
            for (int d = 0; d < hd; d += Vec<T>::N) {
                Vec<T>::load(kr + d, kv);
#pragma unroll
                for (int i = 0; i < Vec<T>::N; ++i) acc[i & 3] = fmaf(qs[d + i], kv[i], acc[i & 3]);
            }
            s = ((acc[0] + acc[1]) + (acc[2] + acc[3])) * scale;
            if (cap > 0.f) s = cap * tanhf(s / cap);
            if (slope != 0.f) s = __fsub_rn(s, __fmul_rn(slope, (float)(pos - key)));
        }
        const float m_new = fmaxf(m, warp_max(s));
        const float p = valid ? expf(s - m_new) : 0.f;
        const float corr = expf(m - m_new);
        l = fmaf(l, corr, warp_sum(p));
#pragma unroll
        for (int e = 0; e < NE; ++e) o[e] *= corr;
        // values of eight keys are requested before the first of them is used; a key outside the row's range
        // (only at its two ends) adds fma(0, v, o) = o with the values of a key inside it
        const int count = min(32, pos - tile + 1);
        const int safe = __shfl_sync(0xffffffffu, row, 31 - __clz(seen));     // the row's last visible key of this tile
        constexpr int VA = NE <= 8 ? 8 : 4;      // value rows asked for together
        for (int j0 = 0; j0 < count; j0 += VA) {
            float pj[VA], vj[VA][NE];
#pragma unroll
            for (int u = 0; u < VA; ++u) {
                const int j = min(j0 + u, 31);
                pj[u] = j0 + u < count ? __shfl_sync(0xffffffffu, p, j) : 0.f;
                const int rj = __shfl_sync(0xffffffffu, row, j);
                const T* vr = v_pages + (size_t)(rj < 0 || j0 + u >= count ? safe : rj) * v_ld;
#pragma unroll
                for (int e = 0; e < NE; ++e) {
                    const int d = e * 32 + lane;
                    vj[u][e] = d < vd ? to_f32(vr[d]) : 0.f;
                }
            }
#pragma unroll
            for (int u = 0; u < VA; ++u)
#pragma unroll
                for (int e = 0; e < NE; ++e) o[e] = fmaf(pj[u], vj[u][e], o[e]);
        }
        m = m_new;
    }
}

// (m, l, o) <- (m, l, o) merged with the next chunk's (mc, lc, oc).  From the empty state (m = -inf, l = 0,
// o = 0) the result is the chunk's own, exactly: e^(-inf) = 0 and e^0 = 1.
template <int NE>
__device__ __forceinline__ void merge_chunk(float& m, float& l, float (&o)[NE], float mc, float lc, const float (&oc)[NE]) {
    const float m_new = fmaxf(m, mc);
    const float a = expf(m - m_new), b = expf(mc - m_new);
    l = fmaf(lc, b, l * a);
#pragma unroll
    for (int e = 0; e < NE; ++e) o[e] = fmaf(oc[e], b, o[e] * a);
    m = m_new;
}

template <typename T, int NE>
__device__ __forceinline__ void store_row(T* __restrict__ orow, int hd, int lane, float l, const float (&o)[NE]) {
    const float inv_l = 1.0f / l;
#pragma unroll
    for (int e = 0; e < NE; ++e) {
        const int d = e * 32 + lane;
        if (d < hd) orow[d] = from_f32<T>(o[e] * inv_l);
    }
}
// the same with a sink (null: none) in the denominator
template <typename T, int NE>
__device__ __forceinline__ void store_row_sink(T* __restrict__ orow, int vd, int lane, float m, float l, const float (&o)[NE],
                                               const float* __restrict__ sinks, int head) {
    if (sinks == nullptr) { store_row<T, NE>(orow, vd, lane, l, o); return; }
    const float sink = sinks[head];
    const float m2 = fmaxf(m, sink);
    const float a = expf(m - m2);
    const float inv_l = 1.0f / fmaf(l, a, expf(sink - m2));
#pragma unroll
    for (int e = 0; e < NE; ++e) {
        const int d = e * 32 + lane;
        if (d < vd) orow[d] = from_f32<T>((o[e] * a) * inv_l);
    }
}

// SPLIT false: grid (items / WARPS), the warp walks its row's chunks and writes the row.
// SPLIT true:  grid (items / WARPS, max_chunks), the warp of (item, slot) computes chunk first_chunk + slot of its
//              row and writes m, l, o[hd] to scratch[(item * max_chunks + slot) * (hd + 2)]; the warp of the last
//              slot also takes whatever chunks lie beyond it (merged in order), so that no key is dropped when a
//              row has more chunks than the caller's bound promised.
template <typename T, int NE, bool SPLIT>  // head_dim <= 32 * NE
__global__ void __launch_bounds__(WARPS * 32)
paged_attention_simt_kernel(const T* __restrict__ q, int q_stride, T* __restrict__ out, int out_stride,
                            const T* __restrict__ k_pages, const T* __restrict__ v_pages,
                            const int* __restrict__ token_req, const int* __restrict__ positions,
                            const int* __restrict__ block_table, int max_pages, int n_tokens, int nq, int nkv, int hd,
                            int page_size, int window, float scale, float* __restrict__ scratch, int max_chunks,
                            int vd, const float* __restrict__ sinks, float cap, int keep, int v_ld,
                            const float* __restrict__ slopes) {
    extern __shared__ float q_smem[];
    pdl_begin();
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int item = blockIdx.x * WARPS + warp;
    if (item >= n_tokens * nq) return;
    const int token = item / nq, head = item % nq;
    const int kvh = head / (nq / nkv);
    const int pos = positions[token];
    const RowKeys rk = row_keys(pos, window, keep);
    int c0 = 0, c1 = row_chunk_count(rk) - 1;           // slots of the row's list of chunks
    if (SPLIT) {
        c0 = (int)blockIdx.y;
        if (c0 > c1) return;
        if ((int)blockIdx.y < max_chunks - 1) c1 = c0;
    }
    const int* table = block_table + (size_t)token_req[token] * max_pages;
    float* qs = q_smem + warp * hd;
    const T* qrow = q + (size_t)token * q_stride + (size_t)head * hd;
    for (int d = lane; d < hd; d += 32) qs[d] = to_f32(qrow[d]);
    __syncwarp();

    const float slope = slopes ? slopes[head] : 0.f;
    float m = -INFINITY, l = 0.f, o[NE];
#pragma unroll
    for (int e = 0; e < NE; ++e) o[e] = 0.f;
    for (int slot = c0; slot <= c1; ++slot) {
        float mc, lc, oc[NE];
        chunk_partial<T, NE>(qs, k_pages, v_pages, table, nkv, kvh, hd, vd, v_ld, page_size, rk.first, rk.kept, pos, row_chunk(rk, slot),
                             scale, cap, slope, lane, mc, lc, oc);
        merge_chunk<NE>(m, l, o, mc, lc, oc);
    }
    if (SPLIT) {
        float* dst = scratch + ((size_t)item * max_chunks + blockIdx.y) * (vd + 2);
        if (lane == 0) { dst[0] = m; dst[1] = l; }
#pragma unroll
        for (int e = 0; e < NE; ++e) {
            const int d = e * 32 + lane;
            if (d < vd) dst[2 + d] = o[e];
        }
    } else {
        store_row_sink<T, NE>(out + (size_t)token * out_stride + (size_t)head * vd, vd, lane, m, l, o, sinks, head);
    }
}

template <typename T, int NE>
__global__ void __launch_bounds__(WARPS * 32)
paged_attention_simt_merge_kernel(T* __restrict__ out, int out_stride, const int* __restrict__ positions, int n_tokens,
                                  int nq, int hd, int window, const float* __restrict__ scratch, int max_chunks,
                                  const float* __restrict__ sinks, int keep) {
    pdl_begin();
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int item = blockIdx.x * WARPS + warp;
    if (item >= n_tokens * nq) return;
    const int token = item / nq, head = item % nq;
    const int pos = positions[token];
    const int slots = min(max_chunks, row_chunk_count(row_keys(pos, window, keep)));
    float m = -INFINITY, l = 0.f, o[NE];
#pragma unroll
    for (int e = 0; e < NE; ++e) o[e] = 0.f;
    // The merges of a row are one chain, in chunk order; the loads are not: a group of chunks is asked for at once and
    // then merged one after the other (one load's latency a chunk made this kernel the longest of a 32-bit decode
    // step: 149 us for 85 chunks of a row).
    constexpr int AHEAD = NE <= 8 ? 8 : 4;
    for (int s0 = 0; s0 < slots; s0 += AHEAD) {
        float mc[AHEAD], lc[AHEAD], oc[AHEAD][NE];
#pragma unroll
        for (int u = 0; u < AHEAD; ++u) {
            const float* src = scratch + ((size_t)item * max_chunks + min(s0 + u, slots - 1)) * (hd + 2);
            mc[u] = src[0];
            lc[u] = src[1];
#pragma unroll
            for (int e = 0; e < NE; ++e) {
                const int d = e * 32 + lane;
                oc[u][e] = d < hd ? src[2 + d] : 0.f;
            }
        }
#pragma unroll
        for (int u = 0; u < AHEAD; ++u)
            if (s0 + u < slots) merge_chunk<NE>(m, l, o, mc[u], lc[u], oc[u]);
    }
    store_row_sink<T, NE>(out + (size_t)token * out_stride + (size_t)head * hd, hd, lane, m, l, o, sinks, head);
}

template <typename T>
static int launch(const void* q, int q_stride, void* out, int out_stride, const void* k_pages, const void* v_pages,
                  const int* token_req, const int* positions, const int* block_table, int max_pages, int n_tokens,
                  int nq, int nkv, int hd, int page_size, int window, float scale, float* scratch, int max_chunks,
                  int vd, const float* sinks, float cap, int keep, int v_ld, const float* slopes, cudaStream_t stream) {
    const int blocks = (n_tokens * nq + WARPS - 1) / WARPS;
    const size_t smem = (size_t)WARPS * hd * sizeof(float);
    const bool split = scratch != nullptr && max_chunks > 1;
#define GO(NE) do { \
        if (!split) \
            return wllm_launch(paged_attention_simt_kernel<T, NE, false>, blocks, WARPS * 32, smem, stream, \
                (const T*)q, q_stride, (T*)out, out_stride, (const T*)k_pages, (const T*)v_pages, token_req, positions, \
                block_table, max_pages, n_tokens, nq, nkv, hd, page_size, window, scale, scratch, max_chunks, vd, sinks, cap, keep, v_ld, slopes); \
        const int st = wllm_launch(paged_attention_simt_kernel<T, NE, true>, dim3(blocks, max_chunks), WARPS * 32, smem, \
                stream, (const T*)q, q_stride, (T*)out, out_stride, (const T*)k_pages, (const T*)v_pages, token_req, \
                positions, block_table, max_pages, n_tokens, nq, nkv, hd, page_size, window, scale, scratch, max_chunks, vd, sinks, cap, keep, v_ld, slopes); \
        if (st != WLLM_OK) return st; \
        return wllm_launch(paged_attention_simt_merge_kernel<T, NE>, blocks, WARPS * 32, 0, stream, (T*)out, out_stride, \
                positions, n_tokens, nq, vd, window, (const float*)scratch, max_chunks, sinks, keep); \
    } while (0)
    if (vd <= 64) GO(2);
    if (vd <= 128) GO(4);
    if (vd <= 256) GO(8);
    GO(16);
#undef GO
}

// scratch (may be null) and max_chunks: with scratch of n_tokens * nq * max_chunks * (hd + 2) floats and
// max_chunks > 1 the split kernels run; max_chunks must be at least the number of chunks of 64 keys that any
// row of the step touches, or the results, still right, are no longer bit-equal to the walk's.
// vd: size of a value head (and of a head's output row); sinks: one 32-bit number per query head, or null.
// v_ld: elements between two value rows (0: vd).
WLLM_API int wllm_paged_attention_simt_strided(const void* q, int q_stride, void* out, int out_stride, const void* k_pages,
                                               const void* v_pages, int dtype, const int* token_req, const int* positions,
                                               const int* block_table, int max_pages, int n_tokens, int nq, int nkv, int hd,
                                               int page_size, int window, float scale, float* scratch, int max_chunks,
                                               int vd, const float* sinks, float cap, int keep, int v_ld, const float* slopes,
                                               cudaStream_t stream) {
    if (n_tokens <= 0) return WLLM_OK;
    if (v_ld == 0) v_ld = vd;
    if (v_ld < vd) return WLLM_BAD_SIZE;
    if (keep < 0 || cap < 0.f || (keep > 0 && window <= 0)) return WLLM_BAD_SIZE;
    // key rows are read with 16-byte loads: key heads come in steps of 8 up to 1024, value heads up to 512
    if (hd <= 0 || hd > 1024 || hd % 8 != 0 || vd <= 0 || vd > 512 || nq <= 0 || nkv <= 0 || nq % nkv != 0 || page_size <= 0 ||
        max_pages <= 0)
        return WLLM_BAD_SIZE;
    if (scratch != nullptr && (max_chunks < 1 || max_chunks > 65535)) return WLLM_BAD_SIZE;
    if (dtype == WLLM_BF16) {
        if (q_stride % 8 != 0) return WLLM_BAD_ALIGN;
        return launch<bf16>(q, q_stride, out, out_stride, k_pages, v_pages, token_req, positions, block_table, max_pages,
                            n_tokens, nq, nkv, hd, page_size, window, scale, scratch, max_chunks, vd, sinks, cap, keep, v_ld, slopes, stream);
    }
    if (dtype == WLLM_F32)
        return launch<float>(q, q_stride, out, out_stride, k_pages, v_pages, token_req, positions, block_table, max_pages,
                             n_tokens, nq, nkv, hd, page_size, window, scale, scratch, max_chunks, vd, sinks, cap, keep, v_ld, slopes, stream);
    return WLLM_BAD_DTYPE;
}

WLLM_API int wllm_paged_attention_simt_general(const void* q, int q_stride, void* out, int out_stride, const void* k_pages,
                                               const void* v_pages, int dtype, const int* token_req, const int* positions,
                                               const int* block_table, int max_pages, int n_tokens, int nq, int nkv, int hd,
                                               int page_size, int window, float scale, float* scratch, int max_chunks,
                                               int vd, const float* sinks, float cap, int keep, cudaStream_t stream) {
    return wllm_paged_attention_simt_strided(q, q_stride, out, out_stride, k_pages, v_pages, dtype, token_req, positions,
                                             block_table, max_pages, n_tokens, nq, nkv, hd, page_size, window, scale, scratch,
                                             max_chunks, vd, sinks, cap, keep, 0, nullptr, stream);
}

WLLM_API int wllm_paged_attention_simt(const void* q, int q_stride, void* out, int out_stride, const void* k_pages,
                                       const void* v_pages, int dtype, const int* token_req, const int* positions,
                                       const int* block_table, int max_pages, int n_tokens, int nq, int nkv, int hd,
                                       int page_size, int window, float scale, float* scratch, int max_chunks,
                                       cudaStream_t stream) {
    if (hd % 16 != 0) return WLLM_BAD_SIZE;
    return wllm_paged_attention_simt_general(q, q_stride, out, out_stride, k_pages, v_pages, dtype, token_req, positions,
                                             block_table, max_pages, n_tokens, nq, nkv, hd, page_size, window, scale, scratch,
                                             max_chunks, hd, nullptr, 0.f, 0, stream);
}

// --------------------------------------------------------------------------------------
// tiled: grid (tiles of 32 rows, kv heads, requests); rows of a request are (token, head of the group)
// --------------------------------------------------------------------------------------
constexpr int TL_WARPS = 8, TL_RPW = 4, TL_ROWS = TL_WARPS * TL_RPW;

__device__ __forceinline__ void cp_async_16(void* smem_dst, const void* src, bool valid) {
    const unsigned dst = (unsigned)__cvta_generic_to_shared(smem_dst);
    const int bytes = valid ? 16 : 0;          // 0: the 16 bytes are filled with zeros, nothing is read
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(dst), "l"(src), "r"(bytes) : "memory");
}

template <typename T, int NE>
__global__ void __launch_bounds__(TL_WARPS * 32)
paged_attention_simt_tiled_kernel(const T* __restrict__ q, int q_stride, T* __restrict__ out, int out_stride,
                                  const T* __restrict__ k_pages, const T* __restrict__ v_pages,
                                  const int* __restrict__ req_q_start, const int* __restrict__ req_q_len,
                                  const int* __restrict__ req_ctx_len, const int* __restrict__ block_table, int max_pages,
                                  int nq, int nkv, int hd, int page_size, int window, float scale, int vd,
                                  const float* __restrict__ sinks, float cap, int keep, int v_ld, const float* __restrict__ slopes) {
    constexpr int VN = Vec<T>::N;                  // elements of a 16-byte piece
    extern __shared__ __align__(16) unsigned char tl_smem[];
    pdl_begin();
    const int g = blockIdx.y, r = blockIdx.z;
    const int q_len = req_q_len[r], rep = nq / nkv, rows = q_len * rep;
    const int m0 = blockIdx.x * TL_ROWS;
    if (m0 >= rows) return;
    const int ctx = req_ctx_len[r], q_start = req_q_start[r], pos0 = ctx - q_len;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int kld = hd + VN;                       // a key's row in shared memory: the head and one piece of padding (banks)
    float* qs = reinterpret_cast<float*>(tl_smem);                          // [32 rows][hd] float
    T* ks = reinterpret_cast<T*>(qs + TL_ROWS * hd);                        // [2][32 keys][kld]
    T* vs = ks + 2 * 32 * kld;                                              // [2][32 keys][vd]
    const int* table = block_table + (size_t)r * max_pages;

    // this warp's rows: position, first key, where they are stored
    int pos_r[TL_RPW], first_r[TL_RPW], kept_r[TL_RPW];
    float slope_r[TL_RPW];
#pragma unroll
    for (int i = 0; i < TL_RPW; ++i) {
        const int m = m0 + warp * TL_RPW + i;
        slope_r[i] = slopes ? slopes[g * rep + m % rep] : 0.f;
        pos_r[i] = m < rows ? pos0 + m / rep : -1;                          // a row past the end takes no key
        const RowKeys rk = row_keys(max(pos_r[i], 0), window, keep);
        first_r[i] = rk.first;
        kept_r[i] = rk.kept;
    }
    for (int idx = threadIdx.x; idx < TL_ROWS * hd; idx += blockDim.x) {
        const int m = m0 + idx / hd, d = idx % hd;
        qs[idx] = m < rows ? to_f32(q[(size_t)(q_start + m / rep) * q_stride + (size_t)(g * rep + m % rep) * hd + d]) : 0.f;
    }
    // the keys that the CTA's rows see, in tiles of 32 at absolute multiples of 32
    const int last_m = min(rows, m0 + TL_ROWS) - 1;
    const int key_hi = pos0 + last_m / rep + 1;                              // one past the last row's position
    const RowKeys top = row_keys(pos0 + m0 / rep, window, keep);             // the CTA's first row reaches furthest back
    const int key_lo = top.first, kept = top.kept;
    const int t_lo = key_lo >> 5, t_hi = (key_hi + 31) >> 5;
    // the tiles of the kept keys that lie before the window's first tile come first; then the window's tiles
    const int head_tiles = kept > 0 ? min((kept + 31) >> 5, t_lo) : 0;
    const int n_tiles = head_tiles + max(t_hi - t_lo, 0);
    auto tile_at = [&](int idx) { return idx < head_tiles ? idx : t_lo + idx - head_tiles; };

    auto load_tile = [&](int t, int stage) {
        const int kp = hd / VN, pieces = kp + vd / VN;      // 16-byte pieces of a key's row and of its value's
        for (int c = threadIdx.x; c < 32 * pieces; c += blockDim.x) {
            const int kl = c / pieces, piece = c % pieces, key = t * 32 + kl;
            const bool valid = (key >= key_lo || key < kept) && key < key_hi;           // others are zero: their weight is zero, their values must be numbers
            size_t row = 0;
            if (valid) row = ((size_t)table[key / page_size] * nkv + g) * page_size + key % page_size;
            if (piece < kp) cp_async_16(ks + ((size_t)stage * 32 + kl) * kld + piece * VN, k_pages + row * hd + piece * VN, valid);
            else cp_async_16(vs + ((size_t)stage * 32 + kl) * vd + (piece - kp) * VN, v_pages + row * v_ld + (piece - kp) * VN, valid);
        }
        asm volatile("cp.async.commit_group;" ::: "memory");
    };

    float m_t[TL_RPW], l_t[TL_RPW], o_t[TL_RPW][NE];      // the rows' results so far (finished chunks)
    float m_c[TL_RPW], l_c[TL_RPW], o_c[TL_RPW][NE];      // the chunk in progress
    bool open_c[TL_RPW];
#pragma unroll
    for (int i = 0; i < TL_RPW; ++i) {
        m_t[i] = m_c[i] = -INFINITY; l_t[i] = l_c[i] = 0.f; open_c[i] = false;
#pragma unroll
        for (int e = 0; e < NE; ++e) o_t[i][e] = o_c[i][e] = 0.f;
    }
    if (n_tiles > 0) load_tile(tile_at(0), 0);
    for (int idx = 0; idx < n_tiles; ++idx) {
        const int t = tile_at(idx), stage = idx & 1;
        if (idx + 1 < n_tiles) load_tile(tile_at(idx + 1), stage ^ 1); else asm volatile("cp.async.commit_group;" ::: "memory");
        asm volatile("cp.async.wait_group 1;" ::: "memory");
        __syncthreads();                          // tile t is here for everyone (and the queries, the first time)
        const T* kt = ks + (size_t)stage * 32 * kld;
        const T* vt = vs + (size_t)stage * 32 * vd;
        const int tile = t * 32, key = tile + lane;
        // a row takes part in the tiles from its first key's to its own position's, as in the walk
        bool act[TL_RPW], any = false;
#pragma unroll
        for (int i = 0; i < TL_RPW; ++i) {
            act[i] = tile <= pos_r[i] && (tile + 31 >= first_r[i] || tile < kept_r[i]);
            any = any || act[i];
        }
        if (any) {
            // scores of the warp's four rows against this lane's key: the key's row is read once for the four
            // (a row that sits this tile out is computed along and dropped; every number it meets is finite)
            const T* kr = kt + (size_t)lane * kld;
            const float* qw = qs + (size_t)(warp * TL_RPW) * hd;
            float acc[TL_RPW][4];
#pragma unroll
            for (int i = 0; i < TL_RPW; ++i) acc[i][0] = acc[i][1] = acc[i][2] = acc[i][3] = 0.f;
#pragma unroll 4
            for (int d = 0; d < hd; d += VN) {
                float kv[VN];
                Vec<T>::load(kr + d, kv);
#pragma unroll
                for (int i = 0; i < TL_RPW; ++i) {
                    float qv[VN];
#pragma unroll
                    for (int u = 0; u < VN; u += 4) {
                        const float4 t4 = *reinterpret_cast<const float4*>(qw + (size_t)i * hd + d + u);
                        qv[u] = t4.x; qv[u + 1] = t4.y; qv[u + 2] = t4.z; qv[u + 3] = t4.w;
                    }
#pragma unroll
                    for (int u = 0; u < VN; ++u) acc[i][u & 3] = fmaf(qv[u], kv[u], acc[i][u & 3]);
                }
            }
            float p[TL_RPW];
#pragma unroll
            for (int i = 0; i < TL_RPW; ++i) {
                p[i] = 0.f;
                if (!act[i]) continue;
                const bool valid = (key >= first_r[i] || key < kept_r[i]) && key <= pos_r[i];
                float s = valid ? ((acc[i][0] + acc[i][1]) + (acc[i][2] + acc[i][3])) * scale : -INFINITY;
                if (valid && cap > 0.f) s = cap * tanhf(s / cap);
                if (valid && slope_r[i] != 0.f) s = __fsub_rn(s, __fmul_rn(slope_r[i], (float)(pos_r[i] - key)));
                const float m_new = fmaxf(m_c[i], warp_max(s));
                p[i] = valid ? expf(s - m_new) : 0.f;
                const float corr = expf(m_c[i] - m_new);
                l_c[i] = fmaf(l_c[i], corr, warp_sum(p[i]));
#pragma unroll
                for (int e = 0; e < NE; ++e) o_c[i][e] *= corr;
                m_c[i] = m_new;
                open_c[i] = true;
            }
            // values: a key's row is read once for the four rows; a weight of 0 (a key outside a row's range, a row
            // that sits the tile out) adds fma(0, v, o) = o
#pragma unroll 2
            for (int j = 0; j < 32; ++j) {
                float v[NE];
#pragma unroll
                for (int e = 0; e < NE; ++e) {
                    const int d = e * 32 + lane;
                    v[e] = d < vd ? to_f32(vt[(size_t)j * vd + d]) : 0.f;
                }
#pragma unroll
                for (int i = 0; i < TL_RPW; ++i) {
                    const float pj = __shfl_sync(0xffffffffu, p[i], j);
#pragma unroll
                    for (int e = 0; e < NE; ++e) o_c[i][e] = fmaf(pj, v[e], o_c[i][e]);
                }
            }
        }
        // the end of a chunk of 64 keys (or of the row): its result joins the row's
        const bool chunk_ends = ((t + 1) & (CHUNK / 32 - 1)) == 0 || idx + 1 == n_tiles || tile_at(idx + 1) != t + 1;
#pragma unroll
        for (int i = 0; i < TL_RPW; ++i) {
            if (open_c[i] && (chunk_ends || tile + 32 > pos_r[i])) {
                merge_chunk<NE>(m_t[i], l_t[i], o_t[i], m_c[i], l_c[i], o_c[i]);
                m_c[i] = -INFINITY; l_c[i] = 0.f; open_c[i] = false;
#pragma unroll
                for (int e = 0; e < NE; ++e) o_c[i][e] = 0.f;
            }
        }
        __syncthreads();                          // everyone is done with this stage before the tile after next lands in it
    }
#pragma unroll
    for (int i = 0; i < TL_RPW; ++i) {
        const int m = m0 + warp * TL_RPW + i;
        if (m < rows)
            store_row_sink<T, NE>(out + (size_t)(q_start + m / rep) * out_stride + (size_t)(g * rep + m % rep) * vd, vd, lane,
                                  m_t[i], l_t[i], o_t[i], sinks, g * rep + m % rep);
    }
}

// --------------------------------------------------------------------------------------
// tiled, chunk by chunk: grid (pairs of a tile of 32 rows and a chunk of 64 keys, over all requests, kv heads), for steps whose tiles are too few to fill the device
// one behind the other.  A request has the pairs of its own rows and keys alone (us by the tiled kernel, with the longest request's pairs for each, and so, 8 heads of
// 256 on one: 250 tokens beside 120 single ones at 60 keys 374, 565 and 50; 509 beside 24 at 1,100 467, 238 and 145; 200 beside 48 at 4,096 1,502, 726 and 317; 509
// alone 228, 93 and 93).  A CTA works out its rows' result over one chunk as the tiled kernel does and leaves m, l, o[vd] in scratch[(row * max_chunks + chunk) * (vd + 2)],
// where the walk's merge kernel takes them up in order: the same bits.  Without a running total and with one tile of keys and values in shared memory (a tile's
// values land while its scores are worked out, the next tile's keys during the weighted sum) two CTAs fit on an SM.  Every key is seen from its position on (no window).
// --------------------------------------------------------------------------------------
// The nth of all pairs: its request (-1 past the last), tile and chunk.  A warp together.
__device__ __forceinline__ int chunk_pair(const int* __restrict__ req_q_len, const int* __restrict__ req_ctx_len, int requests, int rep, int max_chunks, int nth,
                                          int& tile, int& chunk) {
    const int lane = threadIdx.x & 31;
    for (int r0 = 0; r0 < requests; r0 += 32) {
        const int r = r0 + lane;
        const int tiles = r < requests ? (req_q_len[r] * rep + TL_ROWS - 1) / TL_ROWS : 0;
        const int chunks = tiles > 0 ? min((req_ctx_len[r] + CHUNK - 1) / CHUNK, max_chunks) : 0;
        int sum = tiles * chunks;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const int other = __shfl_up_sync(0xffffffffu, sum, o);
            if (lane >= o) sum += other;
        }
        const unsigned behind = __ballot_sync(0xffffffffu, sum > nth);
        if (behind) {
            const int at = __ffs(behind) - 1, each = __shfl_sync(0xffffffffu, chunks, at);
            nth -= __shfl_sync(0xffffffffu, sum - tiles * chunks, at);
            tile = nth / each;
            chunk = nth - tile * each;
            return r0 + at;
        }
        nth -= __shfl_sync(0xffffffffu, sum, 31);
    }
    return -1;
}

template <typename T, int NE>
__global__ void __launch_bounds__(TL_WARPS * 32, 2)
paged_attention_simt_chunk_kernel(const T* __restrict__ q, int q_stride, const T* __restrict__ k_pages, const T* __restrict__ v_pages,
                                  const int* __restrict__ req_q_start, const int* __restrict__ req_q_len, const int* __restrict__ req_ctx_len,
                                  const int* __restrict__ block_table, int max_pages, int requests, int nq, int nkv, int hd, int page_size, float scale, int vd,
                                  float cap, const float* __restrict__ slopes, float* __restrict__ scratch, int max_chunks) {
    constexpr int VN = Vec<T>::N;
    extern __shared__ __align__(16) unsigned char tl_smem[];
    __shared__ size_t row_of[CHUNK];               // the chunk's keys in the pools
    pdl_begin();
    int tile_at, c;
    const int g = blockIdx.y, rep = nq / nkv, r = chunk_pair(req_q_len, req_ctx_len, requests, rep, max_chunks, blockIdx.x, tile_at, c);
    if (r < 0) return;
    const int q_len = req_q_len[r], rows = q_len * rep, m0 = tile_at * TL_ROWS;
    const int ctx = req_ctx_len[r], q_start = req_q_start[r], pos0 = ctx - q_len;
    const int key_hi = pos0 + (min(rows, m0 + TL_ROWS) - 1) / rep + 1;         // one past the last row's position
    if (c * CHUNK >= key_hi) return;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int kld = hd + VN;
    float* qs = reinterpret_cast<float*>(tl_smem);                          // [32 rows][hd] float
    T* ks = reinterpret_cast<T*>(qs + TL_ROWS * hd);                        // [32 keys][kld]
    T* vs = ks + 32 * kld;                                                  // [32 keys][vd]
    if (threadIdx.x < CHUNK) {
        const int key = min(c * CHUNK + (int)threadIdx.x, key_hi - 1);
        row_of[threadIdx.x] = ((size_t)block_table[(size_t)r * max_pages + key / page_size] * nkv + g) * page_size + key % page_size;
    }
    int pos_r[TL_RPW];
    float slope_r[TL_RPW];
#pragma unroll
    for (int i = 0; i < TL_RPW; ++i) {
        const int m = m0 + warp * TL_RPW + i;
        slope_r[i] = slopes ? slopes[g * rep + m % rep] : 0.f;
        pos_r[i] = m < rows ? pos0 + m / rep : -1;                          // a row past the end takes no key
    }
    __syncthreads();
    // 32 rows of `pieces` 16-byte pieces; keys past the last row's are zeros
    auto load = [&](int t, T* to, const T* from, int ld, int width, int to_ld) {
        const int pieces = width / VN, rows_on = (int)blockDim.x / pieces, pieces_on = (int)blockDim.x % pieces;
        int kl = threadIdx.x / pieces, piece = threadIdx.x % pieces;
        while (kl < 32) {
            cp_async_16(to + kl * to_ld + piece * VN, from + row_of[(t & 1) * 32 + kl] * ld + piece * VN, t * 32 + kl < key_hi);
            kl += rows_on;
            piece += pieces_on;
            if (piece >= pieces) { piece -= pieces; ++kl; }
        }
        asm volatile("cp.async.commit_group;" ::: "memory");
    };
    const int t0 = 2 * c, t1 = min(t0 + 2, (key_hi + 31) >> 5);
    load(t0, ks, k_pages, hd, hd, kld);
    load(t0, vs, v_pages, vd, vd, vd);
    for (int idx = threadIdx.x; idx < TL_ROWS * hd; idx += blockDim.x) {
        const int m = m0 + idx / hd, d = idx % hd;
        qs[idx] = m < rows ? to_f32(q[(size_t)(q_start + m / rep) * q_stride + (size_t)(g * rep + m % rep) * hd + d]) : 0.f;
    }
    float m_c[TL_RPW], l_c[TL_RPW], o_c[TL_RPW][NE];
#pragma unroll
    for (int i = 0; i < TL_RPW; ++i) {
        m_c[i] = -INFINITY; l_c[i] = 0.f;
#pragma unroll
        for (int e = 0; e < NE; ++e) o_c[i][e] = 0.f;
    }
    for (int t = t0; t < t1; ++t) {
        const int tile = t * 32, key = tile + lane;
        bool act[TL_RPW], any = false;
#pragma unroll
        for (int i = 0; i < TL_RPW; ++i) { act[i] = tile <= pos_r[i]; any = any || act[i]; }
        asm volatile("cp.async.wait_group 1;" ::: "memory");
        __syncthreads();                          // the tile's keys are here for everyone (and the queries, the first time)
        float p[TL_RPW] = {0.f, 0.f, 0.f, 0.f};
        if (any) {
            const T* kr = ks + (size_t)lane * kld;
            const float* qw = qs + (size_t)(warp * TL_RPW) * hd;
            float acc[TL_RPW][4];
#pragma unroll
            for (int i = 0; i < TL_RPW; ++i) acc[i][0] = acc[i][1] = acc[i][2] = acc[i][3] = 0.f;
#pragma unroll 2
            for (int d = 0; d < hd; d += VN) {
                float kv[VN];
                Vec<T>::load(kr + d, kv);
#pragma unroll
                for (int i = 0; i < TL_RPW; ++i) {
                    float qv[VN];
#pragma unroll
                    for (int u = 0; u < VN; u += 4) {
                        const float4 t4 = *reinterpret_cast<const float4*>(qw + (size_t)i * hd + d + u);
                        qv[u] = t4.x; qv[u + 1] = t4.y; qv[u + 2] = t4.z; qv[u + 3] = t4.w;
                    }
#pragma unroll
                    for (int u = 0; u < VN; ++u) acc[i][u & 3] = fmaf(qv[u], kv[u], acc[i][u & 3]);
                }
            }
#pragma unroll
            for (int i = 0; i < TL_RPW; ++i) {
                if (!act[i]) continue;
                const bool valid = key <= pos_r[i];
                float s = valid ? ((acc[i][0] + acc[i][1]) + (acc[i][2] + acc[i][3])) * scale : -INFINITY;
                if (valid && cap > 0.f) s = cap * tanhf(s / cap);
                if (valid && slope_r[i] != 0.f) s = __fsub_rn(s, __fmul_rn(slope_r[i], (float)(pos_r[i] - key)));
                const float m_new = fmaxf(m_c[i], warp_max(s));
                p[i] = valid ? expf(s - m_new) : 0.f;
                const float corr = expf(m_c[i] - m_new);
                l_c[i] = fmaf(l_c[i], corr, warp_sum(p[i]));
#pragma unroll
                for (int e = 0; e < NE; ++e) o_c[i][e] *= corr;
                m_c[i] = m_new;
            }
        }
        __syncthreads();                          // everyone is done with the keys
        if (t + 1 < t1) load(t + 1, ks, k_pages, hd, hd, kld);
        else asm volatile("cp.async.commit_group;" ::: "memory");
        asm volatile("cp.async.wait_group 1;" ::: "memory");
        __syncthreads();                          // the tile's values are here
        if (any) {
#pragma unroll 2
            for (int j = 0; j < 32; ++j) {
                float v[NE];
#pragma unroll
                for (int e = 0; e < NE; ++e) {
                    const int d = e * 32 + lane;
                    v[e] = d < vd ? to_f32(vs[(size_t)j * vd + d]) : 0.f;
                }
#pragma unroll
                for (int i = 0; i < TL_RPW; ++i) {
                    const float pj = __shfl_sync(0xffffffffu, p[i], j);
#pragma unroll
                    for (int e = 0; e < NE; ++e) o_c[i][e] = fmaf(pj, v[e], o_c[i][e]);
                }
            }
        }
        if (t + 1 < t1) {
            __syncthreads();                      // everyone is done with the values
            load(t + 1, vs, v_pages, vd, vd, vd);
        }
    }
    asm volatile("cp.async.wait_group 0;" ::: "memory");
#pragma unroll
    for (int i = 0; i < TL_RPW; ++i) {
        const int m = m0 + warp * TL_RPW + i;
        if (pos_r[i] < c * CHUNK) continue;
        float* dst = scratch + (((size_t)(q_start + m / rep) * nq + g * rep + m % rep) * max_chunks + c) * (vd + 2);
        if (lane == 0) { dst[0] = m_c[i]; dst[1] = l_c[i]; }
#pragma unroll
        for (int e = 0; e < NE; ++e) {
            const int d = e * 32 + lane;
            if (d < vd) dst[2 + d] = o_c[i][e];
        }
    }
}

template <typename T>
static int launch_tiled(const void* q, int q_stride, void* out, int out_stride, const void* k_pages, const void* v_pages,
                        const int* req_q_start, const int* req_q_len, const int* req_ctx_len, const int* block_table,
                        int max_pages, int requests, int max_q_len, int nq, int nkv, int hd, int page_size, int window,
                        float scale, int vd, const float* sinks, float cap, int keep, int v_ld, const float* slopes,
                        cudaStream_t stream) {
    const int rep = nq / nkv;
    const dim3 grid((max_q_len * rep + TL_ROWS - 1) / TL_ROWS, nkv, requests);
    const size_t smem = (size_t)TL_ROWS * hd * sizeof(float) + 2 * 32 * ((size_t)(hd + Vec<T>::N) + vd) * sizeof(T);
#define GO(NE) do { \
        static bool raised = false; \
        if (!raised) { \
            const cudaError_t e = cudaFuncSetAttribute(paged_attention_simt_tiled_kernel<T, NE>, \
                                                       cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem_max); \
            if (e != cudaSuccess) return 1000 + (int)e; \
            raised = true; \
        } \
        return wllm_launch(paged_attention_simt_tiled_kernel<T, NE>, grid, TL_WARPS * 32, smem, stream, (const T*)q, q_stride, \
                           (T*)out, out_stride, (const T*)k_pages, (const T*)v_pages, req_q_start, req_q_len, req_ctx_len, \
                           block_table, max_pages, nq, nkv, hd, page_size, window, scale, vd, sinks, cap, keep, v_ld, slopes); \
    } while (0)
    const int smem_max = TL_ROWS * 256 * (int)sizeof(float) + 2 * 32 * ((256 + Vec<T>::N) + 256) * (int)sizeof(T);
    if (vd <= 64) GO(2);
    if (vd <= 128) GO(4);
    GO(8);
#undef GO
}

// The tiled kernel for the requests of a step (all of them: a request with one token is a tile with few rows).
// Head sizes up to 256; the result is the walk's bit for bit.
WLLM_API int wllm_paged_attention_simt_tiled_strided(const void* q, int q_stride, void* out, int out_stride, const void* k_pages,
                                                     const void* v_pages, int dtype, const int* req_q_start, const int* req_q_len,
                                                     const int* req_ctx_len, const int* block_table, int max_pages, int requests,
                                                     int max_q_len, int nq, int nkv, int hd, int page_size, int window, float scale,
                                                     int vd, const float* sinks, float cap, int keep, int v_ld, const float* slopes,
                                                     cudaStream_t stream) {
    if (requests <= 0 || max_q_len <= 0) return WLLM_OK;
    if (v_ld == 0) v_ld = vd;
    if (v_ld < vd || v_ld % 8 != 0) return WLLM_BAD_SIZE;
    if (keep < 0 || cap < 0.f || (keep > 0 && window <= 0)) return WLLM_BAD_SIZE;
    if (hd <= 0 || hd > 256 || hd % 8 != 0 || vd <= 0 || vd > 256 || vd % 8 != 0 || nq <= 0 || nkv <= 0 || nq % nkv != 0 || page_size <= 0 || max_pages <= 0 ||
        nkv > 65535 || requests > 65535)
        return WLLM_BAD_SIZE;
    if (dtype == WLLM_BF16) {
        if (q_stride % 8 != 0) return WLLM_BAD_ALIGN;
        return launch_tiled<bf16>(q, q_stride, out, out_stride, k_pages, v_pages, req_q_start, req_q_len, req_ctx_len,
                                  block_table, max_pages, requests, max_q_len, nq, nkv, hd, page_size, window, scale, vd, sinks,
                                  cap, keep, v_ld, slopes, stream);
    }
    if (dtype == WLLM_F32)
        return launch_tiled<float>(q, q_stride, out, out_stride, k_pages, v_pages, req_q_start, req_q_len, req_ctx_len,
                                   block_table, max_pages, requests, max_q_len, nq, nkv, hd, page_size, window, scale, vd, sinks,
                                   cap, keep, v_ld, slopes, stream);
    return WLLM_BAD_DTYPE;
}

WLLM_API int wllm_paged_attention_simt_tiled_general(const void* q, int q_stride, void* out, int out_stride, const void* k_pages,
                                                     const void* v_pages, int dtype, const int* req_q_start, const int* req_q_len,
                                                     const int* req_ctx_len, const int* block_table, int max_pages, int requests,
                                                     int max_q_len, int nq, int nkv, int hd, int page_size, int window, float scale,
                                                     int vd, const float* sinks, float cap, int keep, cudaStream_t stream) {
    return wllm_paged_attention_simt_tiled_strided(q, q_stride, out, out_stride, k_pages, v_pages, dtype, req_q_start, req_q_len,
                                                   req_ctx_len, block_table, max_pages, requests, max_q_len, nq, nkv, hd, page_size,
                                                   window, scale, vd, sinks, cap, keep, 0, nullptr, stream);
}

WLLM_API int wllm_paged_attention_simt_tiled(const void* q, int q_stride, void* out, int out_stride, const void* k_pages,
                                             const void* v_pages, int dtype, const int* req_q_start, const int* req_q_len,
                                             const int* req_ctx_len, const int* block_table, int max_pages, int requests,
                                             int max_q_len, int nq, int nkv, int hd, int page_size, int window, float scale,
                                             cudaStream_t stream) {
    if (hd % 16 != 0) return WLLM_BAD_SIZE;
    return wllm_paged_attention_simt_tiled_general(q, q_stride, out, out_stride, k_pages, v_pages, dtype, req_q_start, req_q_len,
                                                   req_ctx_len, block_table, max_pages, requests, max_q_len, nq, nkv, hd,
                                                   page_size, window, scale, hd, nullptr, 0.f, 0, stream);
}

// The tiled kernel's result over steps without a window, chunk by chunk, bit for bit.  scratch: n_tokens * nq * max_chunks * (vd + 2) floats; max_chunks: chunks of
// 64 keys of the longest context; positions [n_tokens]; pairs: the requests' tiles of 32 rows times their chunks, added up (0: not known, those of the longest for
// each).  32-bit rows of up to 256 elements (the bfloat16 form is not built).
WLLM_API int wllm_paged_attention_simt_chunks(const void* q, int q_stride, void* out, int out_stride, const void* k_pages, const void* v_pages,
                                              const int* positions, const int* req_q_start, const int* req_q_len, const int* req_ctx_len,
                                              const int* block_table, int max_pages, int n_tokens, int requests, int max_q_len, int nq, int nkv, int hd,
                                              int page_size, float scale, int vd, const float* sinks, float cap, const float* slopes, float* scratch,
                                              int max_chunks, long long pairs, cudaStream_t stream) {
    if (n_tokens <= 0 || requests <= 0 || max_q_len <= 0) return WLLM_OK;
    if (hd <= 0 || hd > 256 || hd % 8 != 0 || vd <= 0 || vd > 256 || vd % 8 != 0 || nq <= 0 || nkv <= 0 || nq % nkv != 0 || page_size <= 0 || max_pages <= 0 ||
        max_chunks < 1 || scratch == nullptr || cap < 0.f || requests > 65535 || nkv > 65535)
        return WLLM_BAD_SIZE;
    if (((uintptr_t)k_pages | (uintptr_t)v_pages) & 15) return WLLM_BAD_ALIGN;
    if (pairs <= 0) pairs = ((long long)max_q_len * (nq / nkv) + TL_ROWS - 1) / TL_ROWS * max_chunks * requests;
    if (pairs > 0x7fffffff) return WLLM_BAD_SIZE;
    const dim3 grid((unsigned)pairs, nkv);
    constexpr int VN = Vec<float>::N, most = (TL_ROWS * 256 + 32 * (256 + VN) + 32 * 256) * (int)sizeof(float);
    const size_t smem = ((size_t)TL_ROWS * hd + 32 * (hd + VN) + 32 * vd) * sizeof(float);
    const int blocks = (n_tokens * nq + WARPS - 1) / WARPS;
#define GO(NE) do { \
        static bool raised = false; \
        if (!raised) { \
            const cudaError_t e = cudaFuncSetAttribute(paged_attention_simt_chunk_kernel<float, NE>, cudaFuncAttributeMaxDynamicSharedMemorySize, most); \
            if (e != cudaSuccess) return 1000 + (int)e; \
            raised = true; \
        } \
        const int st = wllm_launch(paged_attention_simt_chunk_kernel<float, NE>, grid, TL_WARPS * 32, smem, stream, (const float*)q, q_stride, \
                                   (const float*)k_pages, (const float*)v_pages, req_q_start, req_q_len, req_ctx_len, block_table, max_pages, requests, \
                                   nq, nkv, hd, page_size, scale, vd, cap, slopes, scratch, max_chunks); \
        if (st != WLLM_OK) return st; \
        return wllm_launch(paged_attention_simt_merge_kernel<float, NE>, blocks, WARPS * 32, 0, stream, (float*)out, out_stride, positions, n_tokens, nq, vd, 0, \
                           (const float*)scratch, max_chunks, sinks, 0); \
    } while (0)
    if (vd <= 64) GO(2);
    if (vd <= 128) GO(4);
    GO(8);
#undef GO
}
