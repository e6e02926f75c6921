// The decayed-state recurrence of linear_attention.cu in chunks of 64 tokens on the tensor cores, for long portions of bfloat16 models:
//
//     S_t = diag(a_t) S_(t-1) + k_t v_t^T,    o_t = S_t^T q_t
//
// With S the state in front of a chunk, G_t the product of the chunk's decays up to t and G_(s..t) that of the tokens behind s up to t,
//
//     o_t = (G_t q_t)^T S + sum_(s <= t) A_ts v_s,   A_ts = q_t . (G_(s..t) k_s)
//     S  <- diag(G_end) S + sum_s (G_(s..end) k_s) v_s^T
//
// (Yang, Wang, Shen, Panda and Kim, "Gated linear attention transformers with hardware-efficient training", 2024).  Kernels:
//
//   prepare   a CTA per (chunk, head): q and k from the fused projection row, turned and scaled in 32 bits as linattn_prepare_kernel does it, then
//             G_t q_t, G_(s..end) k_s, G_end and A.  Every product of decays is a running product of factors that are at most one: blocks of eight tokens
//             carry theirs from their first and to their last token, pairs of blocks the totals of the blocks between, and the pairs inside a block
//             theirs token by token.  No quotients: nothing overflows, however fast a channel forgets.  Entries of A of
//             later tokens are not worked out.  What leaves goes out as operands of the two kernels behind, in the order of a lane's registers.
//   walk      a CTA per (32 key channels by 64 value columns, head, request), S in 32-bit registers: leaves the state in front of every chunk and
//             steps over it.  A chunk's products are summed from zero and join the state in one rounding (the tensor cores cut what they add off, and a
//             state that they added to would drift towards zero).
//   out       a CTA per (chunk, head, 64 value columns): both shares of the outputs.
//   short     requests of fewer than LC_FROM tokens, token by token.
//
// 32-bit factors enter the tensor cores as three bfloat16 pieces each (24 bits together: nothing is lost), of whose nine products the six of
// some weight are taken; values come as the bfloat16 that the projection left.  Large and small products are summed apart and meet at the end.
//
// A value that is no number, or infinite, must not reach earlier tokens through a zero of A: the out kernel looks for such values and then
// adds up their tile token by token.  (Infinite states come out as no number; behind them the head's norm would make them that.)
#include "chunk_common.cuh"

constexpr int LC_COLS = 64, LC_WALK_ROWS = 32, LC_THREADS = 256;

// What the kernels hand on for a (chunk, head), D key channels, V value columns, in 16-byte pieces:
//   Q  [4 row tiles][D / 16][3][32 lanes]     G_t q_t, rows of tokens          K  [D / 16][4][3][32]   (G_(s..end) k_s)^T, rows of channels
//   A  [4][4][3][32]                          rows of tokens (tiles above the diagonal stay empty)
//   G  [D] floats                             S  [3][D][V] bfloat16            the state in front
struct ChunkLayout {
    long long q, k, a, g, s, size;     // offsets and the whole in bytes
    __host__ __device__ ChunkLayout(int D, int V) {
        q = 0;
        k = q + (long long)4 * (D / 16) * 3 * 512;
        a = k + (long long)(D / 16) * 4 * 3 * 512;
        g = a + 4 * 4 * 3 * 512;
        s = g + (long long)D * 4;
        size = s + (long long)3 * D * V * 2;
    }
};

template <int D>
struct PrepareSmem {
    static constexpr int DP = D + 4, AP = LC + 4, PAIRS = LB * (LB + 1) / 2;
    float Q[LC][DP], K[LC][DP];        // q and k; then with their blocks' decays
    float G[LBLOCKS][D];               // the blocks' decays
    float before[LBLOCKS][D], behind[LBLOCKS][D];      // those of the blocks in front of, and behind, a block
    float between[12][D];              // I (I - 1) + J: those between block J and sixteen tokens I, J < 2 I
    float A[LC][AP];
    float sums[LBLOCKS][D / 64][PAIRS];
};

// grid (chunks of the turn, H), 256 threads, two CTAs an SM.  Bound by latency: a round of CTAs that issues in 46 % of its cycles and waits for the fused rows,
// shared memory and the instruction in front by turns (profiles/recurrence_chunks_2048.txt).  (A between blocks by FMA, a thread a channel inside them: 40 us for
// 2,048 tokens of 8 heads of 128 x 256 where this form takes 21.)
template <int D, bool PER_CHANNEL>
__global__ void __launch_bounds__(LC_THREADS, 2)
linattn_chunk_prepare_kernel(const bf16* __restrict__ fused, int row_stride, int q_off, int k_off, const int* __restrict__ positions,
                             const float* __restrict__ inv_freq, int rot_dim, float q_scale, float k_scale, const float* __restrict__ decay,
                             const float* __restrict__ head_decay, const int* __restrict__ req_q_start, const int* __restrict__ req_q_len,
                             const int* __restrict__ req_slot, int requests, int H, int V, int b0, int turn, unsigned char* __restrict__ scratch) {
    typedef PrepareSmem<D> Smem;
    constexpr int GROUPS = 2 * LC_THREADS / D, EACH = LBLOCKS / GROUPS;      // groups of threads that share the blocks, a thread two channels
    extern __shared__ __align__(16) unsigned char lc_raw[];
    Smem& sm = *reinterpret_cast<Smem*>(lc_raw);
    pdl_begin();
    int chunk;
    const int r = lc_find(req_q_len, requests, b0, turn, blockIdx.x, chunk), h = blockIdx.y;
    if (r < 0 || req_slot[r] < 0) return;
    const int first = req_q_start[r] + chunk * LC, count = min(LC, req_q_len[r] - chunk * LC);
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int c2 = 2 * (threadIdx.x % (D / 2)), group = threadIdx.x / (D / 2);
    float2 e[EACH][LB];                // the decays of this thread's blocks and channels; tokens past the end have none
    {
        const float fixed = PER_CHANNEL ? 1.f : head_decay[h];
#pragma unroll
        for (int u = 0; u < EACH; ++u)
#pragma unroll
            for (int i = 0; i < LB; ++i) {
                const int t = (group * EACH + u) * LB + i;
                e[u][i] = make_float2(1.f, 1.f);
                if (t < count) {
                    if (PER_CHANNEL) e[u][i] = *reinterpret_cast<const float2*>(decay + ((size_t)(first + t) * H + h) * D + c2);
                    else e[u][i] = make_float2(fixed, fixed);
                }
            }
    }
    // ---- q and k: pieces of eight channels, a rotated piece with its partner half a turn away; tokens past the end as zeros
    auto widen = [](const uint4& raw, float (&x)[8]) {
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            const float2 f = __bfloat1622float2(reinterpret_cast<const __nv_bfloat162*>(&raw)[i]);
            x[2 * i] = f.x;
            x[2 * i + 1] = f.y;
        }
    };
    auto put = [](float* to, const float (&x)[8], float scale) {
        *reinterpret_cast<float4*>(to) = make_float4(x[0] * scale, x[1] * scale, x[2] * scale, x[3] * scale);
        *reinterpret_cast<float4*>(to + 4) = make_float4(x[4] * scale, x[5] * scale, x[6] * scale, x[7] * scale);
    };
    const uint4 zero = make_uint4(0u, 0u, 0u, 0u);
    if (rot_dim == 0) {
        constexpr int P = D / 8, N = LC * P / LC_THREADS;
        uint4 raw[2][N];
#pragma unroll
        for (int i = 0; i < N; ++i) {
            const int idx = threadIdx.x + i * LC_THREADS, t = idx / P, c = (idx % P) * 8;
            const bf16* src = fused + (size_t)(first + t) * row_stride + h * D + c;
            raw[0][i] = t < count ? *reinterpret_cast<const uint4*>(src + q_off) : zero;
            raw[1][i] = t < count ? *reinterpret_cast<const uint4*>(src + k_off) : zero;
        }
#pragma unroll
        for (int i = 0; i < N; ++i) {
            const int idx = threadIdx.x + i * LC_THREADS, t = idx / P, c = (idx % P) * 8;
            float x[8];
            widen(raw[0][i], x);
            put(&sm.Q[t][c], x, q_scale);
            widen(raw[1][i], x);
            put(&sm.K[t][c], x, k_scale);
        }
    } else {
        const int half = rot_dim >> 1, pieces = D / 8 - half / 8;        // (rot_dim in steps of 16)
        for (int idx = threadIdx.x; idx < LC * pieces; idx += LC_THREADS) {
            const int t = idx / pieces, p = idx - t * pieces, c = p * 8 < half ? p * 8 : p * 8 + half;
            const bool turned = c < half, in = t < count;
            const bf16* src = fused + (size_t)(first + t) * row_stride + h * D + c;
            uint4 raw[2][2] = {{zero, zero}, {zero, zero}};
#pragma unroll
            for (int which = 0; which < 2; ++which)
                if (in) {
                    raw[which][0] = *reinterpret_cast<const uint4*>(src + (which ? k_off : q_off));
                    if (turned) raw[which][1] = *reinterpret_cast<const uint4*>(src + (which ? k_off : q_off) + half);
                }
            float sn[8], cs[8];
            if (turned && in) {
                const float at = (float)positions[first + t];
#pragma unroll
                for (int i = 0; i < 8; ++i) sincosf(at * inv_freq[c + i], &sn[i], &cs[i]);
            }
#pragma unroll
            for (int which = 0; which < 2; ++which) {
                float* to = which ? &sm.K[t][c] : &sm.Q[t][c];
                const float scale = which ? k_scale : q_scale;
                float x[8], y[8];
                widen(raw[which][0], x);
                widen(raw[which][1], y);
                if (turned && in) {
#pragma unroll
                    for (int i = 0; i < 8; ++i) {
                        float u, w;
                        rotate_pair(x[i], y[i], sn[i], cs[i], u, w);
                        x[i] = u;
                        y[i] = w;
                    }
                }
                put(to, x, scale);
                if (turned) put(to + half, y, scale);
            }
        }
    }
    __syncthreads();
    // ---- blocks of eight tokens: a thread two channels
#pragma unroll
    for (int u = 0; u < EACH; ++u) {
        const int B = group * EACH + u;
        float2 kk[LB], qq[LB];
#pragma unroll
        for (int i = 0; i < LB; ++i) {
            qq[i] = *reinterpret_cast<const float2*>(&sm.Q[B * LB + i][c2]);
            kk[i] = *reinterpret_cast<const float2*>(&sm.K[B * LB + i][c2]);
        }
        float x[32], more[4];      // sums of pairs i >= j: i (i + 1) / 2 + j
#pragma unroll
        for (int j = 0; j < LB; ++j) {
            float2 w = kk[j];
#pragma unroll
            for (int i = j; i < LB; ++i) {
                if (i > j) w = lc_mul2(w, e[u][i]);
                const float y = fmaf(qq[i].x, w.x, qq[i].y * w.y);
                const int at = i * (i + 1) / 2 + j;
                if (at < 32) x[at & 31] = y;
                else more[at & 3] = y;
            }
            *reinterpret_cast<float2*>(&sm.K[B * LB + j][c2]) = w;
        }
        float2 E = make_float2(1.f, 1.f);
#pragma unroll
        for (int i = 0; i < LB; ++i) {
            E = lc_mul2(E, e[u][i]);
            *reinterpret_cast<float2*>(&sm.Q[B * LB + i][c2]) = lc_mul2(qq[i], E);
        }
        *reinterpret_cast<float2*>(&sm.G[B][c2]) = E;
        const float s = lc_sums(x, lane), m = lc_sums(more, lane);
        sm.sums[B][c2 / 64][lane] = s;
        if ((lane & 7) == 0) sm.sums[B][c2 / 64][32 + (lane >> 3)] = m;
    }
    __syncthreads();
    // ---- products of the blocks' decays; A inside the blocks
    if (threadIdx.x < D) {
        const int c = threadIdx.x;
        float run = 1.f;
#pragma unroll
        for (int B = 0; B < LBLOCKS; ++B) { sm.before[B][c] = run; run *= sm.G[B][c]; }
#pragma unroll
        for (int I = 1; I < 4; ++I) {
            run = 1.f;
#pragma unroll
            for (int J = 2 * I - 1; J >= 0; --J) { sm.between[I * (I - 1) + J][c] = run; run *= sm.G[J][c]; }
        }
    } else if (threadIdx.x < 2 * D) {
        const int c = threadIdx.x - D;
        float run = 1.f;
#pragma unroll
        for (int B = LBLOCKS - 1; B >= 0; --B) { sm.behind[B][c] = run; run *= sm.G[B][c]; }
    }
    for (int idx = threadIdx.x; idx < LBLOCKS * LB * LB; idx += LC_THREADS) {
        const int B = idx >> 6, i = (idx >> 3) & 7, j = idx & 7;
        float v = 0.f;
        if (j <= i) {
            const int at = i * (i + 1) / 2 + j;
            v = sm.sums[B][0][at];
#pragma unroll
            for (int w = 1; w < D / 64; ++w) v += sm.sums[B][w][at];
        }
        sm.A[B * LB + i][B * LB + j] = v;
        // (the upper half of a tile of 16: a zero that the operand's tile holds)
        if ((B & 1) == 0) sm.A[B * LB + i][(B + 1) * LB + j] = 0.f;
    }
    __syncthreads();
    // ---- A between blocks, tiles of sixteen tokens by a block, two a warp: warps 0 to 5 the tokens I = 1, 2, 2, 3, 3, 3 with blocks J < 2 I in front of
    // them, decays from and to the tokens' first one; warps 6 and 7 the upper half of I with its lower
    {
        const int r0 = lane >> 2, c0 = 2 * (lane & 3);
        const bool inside = warp >= 6;
        const int I = warp == 0 ? 1 : (warp < 3 ? 2 : 3), J0 = warp == 0 ? 0 : (warp < 3 ? 2 * (warp - 1) : 2 * (warp - 3));
        float big[2][4], small[2][4];
#pragma unroll
        for (int u = 0; u < 2; ++u)
#pragma unroll
            for (int i = 0; i < 4; ++i) big[u][i] = small[u][i] = 0.f;
        auto at2 = [](const float* p) { return *reinterpret_cast<const float2*>(p); };
        auto sums = [&](int u, const uint4 (&a)[3], float2 k0, float2 k1) {
            uint32_t b[3][2];
            lc_split(k0.x, k0.y, b[0][0], b[1][0], b[2][0]);
            lc_split(k1.x, k1.y, b[0][1], b[1][1], b[2][1]);
            lc_mma(small[u], a[0], b[2][0], b[2][1]);
            lc_mma(small[u], a[2], b[0][0], b[0][1]);
            lc_mma(small[u], a[1], b[1][0], b[1][1]);
            lc_mma(small[u], a[0], b[1][0], b[1][1]);
            lc_mma(small[u], a[1], b[0][0], b[0][1]);
            lc_mma(big[u], a[0], b[0][0], b[0][1]);
        };
#pragma unroll 2
        for (int c = c0; c < D; c += 16) {
            uint4 a[3];
            if (!inside) {
                const float* q = sm.Q[16 * I + r0];
                const float2 x0 = at2(q + c), x1 = at2(q + c + 8);
                const float2 y0 = lc_mul2(at2(q + 8 * Smem::DP + c), at2(&sm.G[2 * I][c])), y1 = lc_mul2(at2(q + 8 * Smem::DP + c + 8), at2(&sm.G[2 * I][c + 8]));
                lc_split(x0.x, x0.y, a[0].x, a[1].x, a[2].x);
                lc_split(y0.x, y0.y, a[0].y, a[1].y, a[2].y);
                lc_split(x1.x, x1.y, a[0].z, a[1].z, a[2].z);
                lc_split(y1.x, y1.y, a[0].w, a[1].w, a[2].w);
            }
#pragma unroll
            for (int u = 0; u < 2; ++u) {
                const int J = inside ? 4 * (warp - 6) + 2 * u : J0 + u;
                if (inside) {
                    const float* q = sm.Q[8 * J + 8 + r0];
                    const float2 y0 = at2(q + c), y1 = at2(q + c + 8);
#pragma unroll
                    for (int p = 0; p < 3; ++p) a[p].x = a[p].z = 0u;
                    lc_split(y0.x, y0.y, a[0].y, a[1].y, a[2].y);
                    lc_split(y1.x, y1.y, a[0].w, a[1].w, a[2].w);
                }
                float2 k0 = at2(&sm.K[8 * J + r0][c]), k1 = at2(&sm.K[8 * J + r0][c + 8]);
                if (!inside) {
                    const float* f = sm.between[I * (I - 1) + J];
                    k0 = lc_mul2(k0, at2(f + c));
                    k1 = lc_mul2(k1, at2(f + c + 8));
                }
                sums(u, a, k0, k1);
            }
        }
#pragma unroll
        for (int u = 0; u < 2; ++u) {
            const int J = inside ? 4 * (warp - 6) + 2 * u : J0 + u, row = (inside ? 8 * J : 16 * I) + r0, s = 8 * J + c0;
            if (!inside) *reinterpret_cast<float2*>(&sm.A[row][s]) = make_float2(big[u][0] + small[u][0], big[u][1] + small[u][1]);
            *reinterpret_cast<float2*>(&sm.A[row + 8][s]) = make_float2(big[u][2] + small[u][2], big[u][3] + small[u][3]);
        }
    }
    __syncthreads();
    // ---- the operands, in the order of a lane's registers
    const ChunkLayout at(D, V);
    unsigned char* mine = scratch + ((size_t)blockIdx.x * H + h) * at.size;
    const int r0 = lane >> 2, c0 = 2 * (lane & 3);
    auto leave = [&](uint4* to, float2 v0, float2 v1, float2 v2, float2 v3) {
        uint4 p[3];
        lc_split(v0.x, v0.y, p[0].x, p[1].x, p[2].x);
        lc_split(v1.x, v1.y, p[0].y, p[1].y, p[2].y);
        lc_split(v2.x, v2.y, p[0].z, p[1].z, p[2].z);
        lc_split(v3.x, v3.y, p[0].w, p[1].w, p[2].w);
#pragma unroll
        for (int i = 0; i < 3; ++i) to[i * 32 + lane] = p[i];
    };
    for (int tile = warp; tile < 4 * (D / 16); tile += LC_THREADS / 32) {
        const int wm = tile / (D / 16), ks = tile % (D / 16);
        float2 v[4];
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            const int t = wm * 16 + r0 + (i & 1) * 8, c = ks * 16 + c0 + (i >> 1) * 8;
            const float2 x = *reinterpret_cast<const float2*>(&sm.Q[t][c]), f = *reinterpret_cast<const float2*>(&sm.before[t / LB][c]);
            v[i] = make_float2(x.x * f.x, x.y * f.y);
        }
        leave(reinterpret_cast<uint4*>(mine + at.q) + (size_t)tile * 96, v[0], v[1], v[2], v[3]);
    }
    for (int tile = warp; tile < (D / 16) * 4; tile += LC_THREADS / 32) {
        const int dt = tile >> 2, ks = tile & 3;
        float2 v[4];
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            const int d = dt * 16 + r0 + (i & 1) * 8, t = ks * 16 + c0 + (i >> 1) * 8;     // (t and t + 1 lie in one block)
            const float f = sm.behind[t / LB][d];
            v[i] = make_float2(sm.K[t][d] * f, sm.K[t + 1][d] * f);
        }
        leave(reinterpret_cast<uint4*>(mine + at.k) + (size_t)tile * 96, v[0], v[1], v[2], v[3]);
    }
    for (int tile = warp; tile < 16; tile += LC_THREADS / 32) {
        const int wm = tile >> 2, ks = tile & 3;
        if (ks > wm) continue;
        float2 v[4];
#pragma unroll
        for (int i = 0; i < 4; ++i) v[i] = *reinterpret_cast<const float2*>(&sm.A[wm * 16 + r0 + (i & 1) * 8][ks * 16 + c0 + (i >> 1) * 8]);
        leave(reinterpret_cast<uint4*>(mine + at.a) + (size_t)tile * 96, v[0], v[1], v[2], v[3]);
    }
    if (threadIdx.x < D) reinterpret_cast<float*>(mine + at.g)[threadIdx.x] = sm.before[LBLOCKS - 1][threadIdx.x] * sm.G[LBLOCKS - 1][threadIdx.x];
}

struct WalkChunk {
    uint4 K[LC_WALK_ROWS / 16 * 4 * 96];
    bf16 V[LC][LC_COLS + 8];
    float g[LC_WALK_ROWS];
};
constexpr int WALK_GROUP = 2, WALK_STAGES = 3;         // chunks of a stage (worked out side by side), stages

// grid (D / 32 * V / 64, H, requests), 256 threads: warp w channels 16 (w >> 2) .., columns 16 (w & 3) .. of the CTA's 32 by 64.  Bound by the chain of chunks;
// four are on their way while two are worked on.  (128 channels by 16 columns, operands in registers one chunk ahead: 42 us for 2,048 tokens of 8 heads of
// 128 x 256, each CTA reading 50 KB a chunk from the L2 where this one reads 21.)
template <int D>
__global__ void __launch_bounds__(LC_THREADS)
linattn_chunk_walk_kernel(const bf16* __restrict__ v, int row_stride, float* __restrict__ state, const int* __restrict__ req_q_start,
                          const int* __restrict__ req_q_len, const int* __restrict__ req_slot, int H, int V, int b0, int turn,
                          unsigned char* __restrict__ scratch) {
    extern __shared__ __align__(16) unsigned char lc_raw[];
    WalkChunk* ring = reinterpret_cast<WalkChunk*>(lc_raw);
    pdl_begin();
    constexpr int ROWS = D / LC_WALK_ROWS;
    const int r = blockIdx.z, h = blockIdx.y, v0 = blockIdx.x / ROWS * LC_COLS, rows = blockIdx.x % ROWS;
    const int len = req_q_len[r], slot = req_slot[r];
    if (slot < 0) return;
    const int chunks = min(lc_chunks(len) - b0, turn);
    if (chunks <= 0) return;
    const ChunkLayout at(D, V);
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, frow = lane >> 2, fcol = 2 * (lane & 3), wr = warp >> 2, wc = warp & 3;
    unsigned char* mine = scratch + ((size_t)lc_before(req_q_len, r, b0, turn) * H + h) * at.size;
    const size_t next = (size_t)H * at.size;
    const int t0 = req_q_start[r] + b0 * LC, left = len - b0 * LC;
    auto load = [&](int group) {
#pragma unroll
        for (int u = 0; u < WALK_GROUP; ++u) {
            const int c = group * WALK_GROUP + u;
            if (c >= chunks) break;
            WalkChunk& to = ring[(group % WALK_STAGES) * WALK_GROUP + u];
            const unsigned char* p = mine + c * next;
            const uint4* src = reinterpret_cast<const uint4*>(p + at.k) + (size_t)rows * (LC_WALK_ROWS / 16 * 4 * 96);
#pragma unroll
            for (int i = 0; i < 3; ++i) lc_cp16(&to.K[threadIdx.x + i * LC_THREADS], src + threadIdx.x + i * LC_THREADS, true);
#pragma unroll
            for (int i = 0; i < 2; ++i) {
                const int t = (threadIdx.x >> 3) + 32 * i, col = (threadIdx.x & 7) * 8;
                const bool in = c * LC + t < left;
                lc_cp16(&to.V[t][col], in ? v + (size_t)(t0 + c * LC + t) * row_stride + h * V + v0 + col : v, in);
            }
            if (threadIdx.x < LC_WALK_ROWS / 4) lc_cp16(&to.g[4 * threadIdx.x], reinterpret_cast<const float*>(p + at.g) + rows * LC_WALK_ROWS + 4 * threadIdx.x, true);
        }
        asm volatile("cp.async.commit_group;" ::: "memory");                 // (an empty group keeps the count of groups)
    };
#pragma unroll
    for (int g = 0; g < WALK_STAGES - 1; ++g) load(g);
    const int row = rows * LC_WALK_ROWS + wr * 16 + frow, col = v0 + wc * 16 + fcol;
    float* Sg = state + ((size_t)slot * H + h) * D * V;
    float S[2][4];
#pragma unroll
    for (int j = 0; j < 2; ++j)
#pragma unroll
        for (int half = 0; half < 2; ++half) {
            const float2 x = *reinterpret_cast<const float2*>(Sg + (size_t)(row + half * 8) * V + col + j * 8);
            S[j][half * 2] = x.x;
            S[j][half * 2 + 1] = x.y;
        }
    for (int group = 0; group * WALK_GROUP < chunks; ++group) {
        asm volatile("cp.async.wait_group %0;" ::"n"(WALK_STAGES - 2) : "memory");
        __syncthreads();                       // the stage's operands are here; the stage before is read to its end
        load(group + WALK_STAGES - 1);
        float big[WALK_GROUP][2][4], small[WALK_GROUP][2][4];
#pragma unroll
        for (int u = 0; u < WALK_GROUP; ++u) { // (behind the last chunk what a stage held before, or nothing: not used)
            const WalkChunk& from = ring[(group % WALK_STAGES) * WALK_GROUP + u];
            const uint4* k = from.K + wr * 4 * 96 + lane;
#pragma unroll
            for (int j = 0; j < 2; ++j)
#pragma unroll
                for (int e = 0; e < 4; ++e) big[u][j][e] = small[u][j][e] = 0.f;
#pragma unroll
            for (int ks = 0; ks < 4; ++ks) {
                uint32_t b[4];
                lc_ldsm4_t(&from.V[ks * 16 + (lane & 7) + ((lane >> 3) & 1) * 8][wc * 16 + (lane >> 4) * 8], b);
                const uint4 k0 = k[(ks * 3) * 32], k1 = k[(ks * 3 + 1) * 32], k2 = k[(ks * 3 + 2) * 32];
#pragma unroll
                for (int j = 0; j < 2; ++j) {
                    lc_mma(small[u][j], k2, b[2 * j], b[2 * j + 1]);
                    lc_mma(small[u][j], k1, b[2 * j], b[2 * j + 1]);
                    lc_mma(big[u][j], k0, b[2 * j], b[2 * j + 1]);
                }
            }
        }
#pragma unroll
        for (int u = 0; u < WALK_GROUP; ++u) {
            const int c = group * WALK_GROUP + u;
            if (c >= chunks) break;
            bf16* St = reinterpret_cast<bf16*>(mine + c * next + at.s);
#pragma unroll
            for (int half = 0; half < 2; ++half) {
                uint32_t p[2][3];
#pragma unroll
                for (int j = 0; j < 2; ++j) lc_split(S[j][half * 2], S[j][half * 2 + 1], p[j][0], p[j][1], p[j][2]);
                // an even lane and the odd one behind it swap halves: four neighbouring columns each, whole sectors an instruction
                const bool upper = lane & 1;
                bf16* to = St + (size_t)(row + half * 8) * V + v0 + wc * 16 + (upper ? 8 : 0) + 4 * ((lane & 3) >> 1);
#pragma unroll
                for (int i = 0; i < 3; ++i) {
                    const uint32_t got = __shfl_xor_sync(0xffffffffu, upper ? p[0][i] : p[1][i], 1);
                    *reinterpret_cast<uint2*>(to + (size_t)i * D * V) = upper ? make_uint2(got, p[1][i]) : make_uint2(p[0][i], got);
                }
            }
            const WalkChunk& from = ring[(group % WALK_STAGES) * WALK_GROUP + u];
            const float g0 = from.g[wr * 16 + frow], g1 = from.g[wr * 16 + frow + 8];
#pragma unroll
            for (int j = 0; j < 2; ++j)
#pragma unroll
                for (int e = 0; e < 4; ++e) S[j][e] = fmaf(e < 2 ? g0 : g1, S[j][e], big[u][j][e] + small[u][j][e]);
        }
    }
    asm volatile("cp.async.wait_group 0;" ::: "memory");
#pragma unroll
    for (int j = 0; j < 2; ++j)
#pragma unroll
        for (int half = 0; half < 2; ++half)
            *reinterpret_cast<float2*>(Sg + (size_t)(row + half * 8) * V + col + j * 8) = make_float2(S[j][half * 2], S[j][half * 2 + 1]);
}

template <int D>
struct OutSmem {
    bf16 S[3][D][LC_COLS], V[LC][LC_COLS];      // rows of 128 bytes, 16-byte piece p of row r at p ^ (r & 7)
    uint4 Q[4][D / 16 * 96];
};

// grid (V / 64, H, chunks of the turn), 256 threads, two CTAs an SM: warp w rows 16 (w & 3) .., columns 32 (w >> 2) ..  Bound by its operands' latency, so they
// are asked for at once and worked on as they come.
template <int D>
__global__ void __launch_bounds__(LC_THREADS, 2)
linattn_chunk_out_kernel(const bf16* __restrict__ v, int row_stride, float* __restrict__ out, const int* __restrict__ req_q_start,
                         const int* __restrict__ req_q_len, const int* __restrict__ req_slot, int requests, int H, int V, int b0, int turn,
                         const unsigned char* __restrict__ scratch) {
    typedef OutSmem<D> Smem;
    extern __shared__ __align__(16) unsigned char lc_raw[];
    Smem& sm = *reinterpret_cast<Smem*>(lc_raw);
    pdl_begin();
    int chunk;
    const int r = lc_find(req_q_len, requests, b0, turn, blockIdx.z, chunk), h = blockIdx.y, v0 = blockIdx.x * LC_COLS;
    if (r < 0 || req_slot[r] < 0) return;
    const int first = req_q_start[r] + chunk * LC, count = min(LC, req_q_len[r] - chunk * LC);
    const ChunkLayout at(D, V);
    const unsigned char* mine = scratch + ((size_t)blockIdx.z * H + h) * at.size;
    const bf16* St = reinterpret_cast<const bf16*>(mine + at.s);
    for (int idx = threadIdx.x; idx < LC * 8; idx += LC_THREADS) {
        const int t = idx >> 3, p = (idx & 7) * 8;
        lc_cp16(&sm.V[t][p ^ ((t & 7) * 8)], t < count ? v + (size_t)(first + t) * row_stride + h * V + v0 + p : v, t < count);
    }
    constexpr int PARTS = 4, ROWS = D / PARTS;             // the state comes in four runs of channels, the queries' beside it, the first with the values
#pragma unroll
    for (int part = 0; part < PARTS; ++part) {
        for (int idx = threadIdx.x; idx < 3 * ROWS * 8; idx += LC_THREADS) {
            const int piece = idx / (ROWS * 8), row = part * ROWS + (idx / 8) % ROWS, p = (idx & 7) * 8;
            lc_cp16(&sm.S[piece][row][p ^ ((row & 7) * 8)], St + (size_t)(piece * D + row) * V + v0 + p, true);
        }
        constexpr int EACH = D / 16 / PARTS * 96;          // 16-byte pieces of a row tile's operand
        for (int idx = threadIdx.x; idx < 4 * EACH; idx += LC_THREADS) {
            const int tile = idx / EACH, i = part * EACH + idx % EACH;
            lc_cp16(&sm.Q[tile][i], reinterpret_cast<const uint4*>(mine + at.q) + (size_t)tile * (D / 16) * 96 + i, true);
        }
        asm volatile("cp.async.commit_group;" ::: "memory");
    }
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, wm = warp & 3, wn = warp >> 2, frow = lane >> 2, fcol = 2 * (lane & 3);
    const uint4* af = reinterpret_cast<const uint4*>(mine + at.a) + (size_t)wm * 4 * 96 + lane;
    // 16 rows of channels or tokens, 16 columns from 16 jj of this warp's: the lane's place for ldmatrix
    const int krow = (lane & 7) + ((lane >> 3) & 1) * 8, kcol = wn * 32 + (lane >> 4) * 8;
    auto place = [&](int jj) { return (kcol + jj * 16) ^ ((krow & 7) * 8); };
    uint4 a[2][3];                                         // two tiles of A ahead
    float big[4][4], small[4][4], own[4][4];
#pragma unroll
    for (int j = 0; j < 4; ++j)
#pragma unroll
        for (int e = 0; e < 4; ++e) big[j][e] = small[j][e] = own[j][e] = 0.f;
    // ---- the share of the state in front of the chunk
    bool odd = false;                                      // values that are no finite numbers: exponents all ones
#pragma unroll
    for (int part = 0; part < PARTS; ++part) {
        if (part == 0) asm volatile("cp.async.wait_group 3;" ::: "memory");
        if (part == 1) asm volatile("cp.async.wait_group 2;" ::: "memory");
        if (part == 2) asm volatile("cp.async.wait_group 1;" ::: "memory");
        if (part == 3) asm volatile("cp.async.wait_group 0;" ::: "memory");
        if (part == 0) {
#pragma unroll
            for (int i = 0; i < LC * 8 / LC_THREADS; ++i) {              // (what this thread asked for itself)
                const int idx = threadIdx.x + i * LC_THREADS, t = idx >> 3;
                const uint4 x = *reinterpret_cast<const uint4*>(&sm.V[t][((idx & 7) * 8) ^ ((t & 7) * 8)]);
                const uint32_t w[4] = {x.x, x.y, x.z, x.w};
#pragma unroll
                for (int e = 0; e < 4; ++e) odd |= (w[e] & 0x7f80u) == 0x7f80u || (w[e] & 0x7f800000u) == 0x7f800000u;
            }
            odd = __syncthreads_or(odd);
        } else __syncthreads();
        if (part == 2) {
#pragma unroll
            for (int u = 0; u < 2; ++u)
                if (u <= wm) {
#pragma unroll
                    for (int p = 0; p < 3; ++p) a[u][p] = af[(u * 3 + p) * 32];
                }
        }
#pragma unroll
        for (int k = 0; k < D / 16 / PARTS; ++k) {
            const int ks = part * (D / 16 / PARTS) + k;
            uint4 now[3];
#pragma unroll
            for (int p = 0; p < 3; ++p) now[p] = sm.Q[wm][(ks * 3 + p) * 32 + lane];
#pragma unroll
            for (int p = 2; p >= 0; --p) {
                uint32_t b[2][4];
#pragma unroll
                for (int jj = 0; jj < 2; ++jj) lc_ldsm4_t(&sm.S[p][ks * 16 + krow][place(jj)], b[jj]);
#pragma unroll
                for (int q = 2 - p; q >= 0; --q)
#pragma unroll
                    for (int j = 0; j < 4; ++j) lc_mma(p + q == 0 ? big[j] : small[j], now[q], b[j >> 1][2 * (j & 1)], b[j >> 1][2 * (j & 1) + 1]);
            }
        }
    }
    // ---- the share of the chunk's own tokens
    if (!odd) {
#pragma unroll
        for (int ks = 0; ks < 4; ++ks) {
            if (ks > wm) break;
            uint4 now[3];
#pragma unroll
            for (int p = 0; p < 3; ++p) {
                now[p] = a[ks & 1][p];
                if (ks + 2 <= wm) a[ks & 1][p] = af[((ks + 2) * 3 + p) * 32];
            }
            uint32_t b[2][4];
#pragma unroll
            for (int jj = 0; jj < 2; ++jj) lc_ldsm4_t(&sm.V[ks * 16 + krow][place(jj)], b[jj]);
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                const uint32_t b0 = b[j >> 1][2 * (j & 1)], b1 = b[j >> 1][2 * (j & 1) + 1];
                lc_mma(small[j], now[2], b0, b1);
                lc_mma(small[j], now[1], b0, b1);
                lc_mma(own[j], now[0], b0, b1);
            }
        }
    } else {
        for (int half = 0; half < 2; ++half) {
            const int t = wm * 16 + frow + half * 8;
            for (int s = 0; s <= t; ++s) {
                // A_ts from its pieces: row t of tile (wm, s / 16), the register and lane that hold column s
                const int c = s & 15, reg = half + (c >> 3) * 2, from = frow * 4 + ((c & 7) >> 1);
                float weight = 0.f;
#pragma unroll
                for (int p = 2; p >= 0; --p) {
                    const uint32_t pair = reinterpret_cast<const uint32_t*>(af - lane + ((s >> 4) * 3 + p) * 32 + from)[reg];
                    weight += __uint_as_float((c & 1) ? (pair & 0xffff0000u) : (pair << 16));
                }
#pragma unroll
                for (int j = 0; j < 4; ++j)
#pragma unroll
                    for (int e = 0; e < 2; ++e)
                        own[j][half * 2 + e] = fmaf(weight, __bfloat162float(sm.V[s][((wn * 32 + j * 8) ^ ((s & 7) * 8)) + fcol + e]), own[j][half * 2 + e]);
            }
        }
    }
#pragma unroll
    for (int half = 0; half < 2; ++half) {
        const int t = wm * 16 + frow + half * 8;
        if (t >= count) continue;
        float* to = out + ((size_t)(first + t) * H + h) * V + v0 + wn * 32 + fcol;
#pragma unroll
        for (int j = 0; j < 4; ++j)
            *reinterpret_cast<float2*>(to + j * 8) = make_float2(own[j][half * 2] + (big[j][half * 2] + small[j][half * 2]),
                                                                 own[j][half * 2 + 1] + (big[j][half * 2 + 1] + small[j][half * 2 + 1]));
    }
}

// Requests of fewer than LC_FROM tokens, token by token: grid (V / 64, H, requests), 256 threads: a thread a column of a fourth of the channels.  Bound by the
// state's way through the HBM.
template <int D, bool PER_CHANNEL>
__global__ void __launch_bounds__(LC_THREADS)
linattn_short_kernel(const bf16* __restrict__ fused, int row_stride, int q_off, int k_off, int v_off, const int* __restrict__ positions,
                     const float* __restrict__ inv_freq, int rot_dim, float q_scale, float k_scale, const float* __restrict__ decay,
                     const float* __restrict__ head_decay, float* __restrict__ state, float* __restrict__ out, const int* __restrict__ req_q_start,
                     const int* __restrict__ req_q_len, const int* __restrict__ req_slot, int H, int V) {
    constexpr int N = D / 4;
    __shared__ __align__(16) float Q[LC_FROM][D], K[LC_FROM][D], A[PER_CHANNEL ? LC_FROM : 1][D], part[LC_FROM][4][LC_COLS];
    pdl_begin();
    const int r = blockIdx.z, h = blockIdx.y, len = req_q_len[r], slot = req_slot[r];
    if (len <= 0 || len >= LC_FROM || slot < 0) return;
    const int first = req_q_start[r], col = threadIdx.x & 63, c0 = (threadIdx.x >> 6) * N, vc = blockIdx.x * LC_COLS + col;
    float* Sg = state + (((size_t)slot * H + h) * D + c0) * V + vc;
    float S[N];
#pragma unroll
    for (int i = 0; i < N; ++i) S[i] = Sg[(size_t)i * V];
    const int half = rot_dim >> 1, each = D - half;
    for (int idx = threadIdx.x; idx < 2 * len * each; idx += LC_THREADS) {
        const int which = idx >= len * each, t = idx / each - which * len, p = idx % each, c = p < half ? p : p + half;
        const bf16* src = fused + (size_t)(first + t) * row_stride + (which ? k_off : q_off) + h * D;
        float* to = which ? K[t] : Q[t];
        const float scale = which ? k_scale : q_scale, x = __bfloat162float(src[c]);
        if (p < half) {
            float sn, cs, y1, y2;
            sincosf((float)positions[first + t] * inv_freq[p], &sn, &cs);
            rotate_pair(x, __bfloat162float(src[c + half]), sn, cs, y1, y2);
            to[c] = y1 * scale;
            to[c + half] = y2 * scale;
        } else to[c] = x * scale;
    }
    if (PER_CHANNEL)
        for (int idx = threadIdx.x; idx < len * D; idx += LC_THREADS) A[idx / D][idx % D] = decay[((size_t)(first + idx / D) * H + h) * D + idx % D];
    const float fixed = PER_CHANNEL ? 1.f : head_decay[h];
    __syncthreads();
    for (int t = 0; t < len; ++t) {
        const float v = __bfloat162float(fused[(size_t)(first + t) * row_stride + v_off + h * V + vc]);
        float p = 0.f;
#pragma unroll
        for (int i = 0; i < N; ++i) {
            S[i] = fmaf(PER_CHANNEL ? A[t][c0 + i] : fixed, S[i], K[t][c0 + i] * v);
            p = fmaf(S[i], Q[t][c0 + i], p);
        }
        part[t][threadIdx.x >> 6][col] = p;
    }
#pragma unroll
    for (int i = 0; i < N; ++i) Sg[(size_t)i * V] = S[i];
    __syncthreads();
    for (int idx = threadIdx.x; idx < len * LC_COLS; idx += LC_THREADS) {
        const int t = idx >> 6, c = idx & 63;
        out[((size_t)(first + t) * H + h) * V + blockIdx.x * LC_COLS + c] = (part[t][0][c] + part[t][1][c]) + (part[t][2][c] + part[t][3][c]);
    }
}

// Sizes that the chunked form is built for.
static bool lc_sizes(int H, int D, int V) { return H > 0 && H <= 65535 && (D == 64 || D == 128) && V > 0 && V % 64 == 0; }

// Bytes of scratch that wllm_linattn_chunks asks for: 2.56 MB a chunk of 8 heads of 128 x 256, at most 192 MB (4,992 tokens; longer steps go in turns, the state
// handed on through its slot: the same bits) but a chunk of every request that goes in chunks.  lens: the requests' tokens, on the host.  turns: how many with that.
WLLM_API long long wllm_linattn_chunks_bytes(const int* lens, int requests, int H, int D, int V, int* turns) {
    *turns = 0;
    if (!lc_sizes(H, D, V) || requests <= 0) return 0;
    return lc_bytes(lens, requests, H * ChunkLayout(D, V).size, *turns);
}

// Bytes of scratch where chunks are the faster way for a step of these requests, else 0.  rank: of the decay's low-rank map, 0 without one; segments: the walk
// would cut its long requests into segments; most: bytes that a step's chunks may take.
//
// Both ways' us, fitted to B200 measurements from 130 to 8,192 tokens (in brackets the walk's and the chunks' for 8 heads of 128 x 256 with a decay per channel).
// A chunk costs by the bytes that its kernels hand on (2.56 MB of those heads), full or not, a request its state's way; a turn some 45 (2,048 tokens [253, 86],
// 512 [86, 41], 16 x 130 [183, 145], 130 beside 20 of 20 [74, 99], beside 40 [86, 179], beside 90 [176, 447], 512 beside 20 of 20 [206, 108], beside 90
// [286, 678: eight turns], 2,048 beside 90 [837, 1,787: thirty-two]).  The walk is bound by its longest request's chain or by all tokens.  Where segments of the
// long requests fill the device few requests are there, and chunks were the faster way at every size measured (2 to 32 heads).
WLLM_API long long wllm_linattn_chunks_pay(const int* lens, int requests, int H, int D, int V, int rank, int segments, long long most) {
    int turns;
    const long long room = wllm_linattn_chunks_bytes(lens, requests, H, D, V, &turns);
    if (room <= 0 || room > most) return 0;
    if (segments) return room;
    int longest = 0, deepest = 0;
    double tokens = 0, chunks = 0, several = 0;
    for (int r = 0; r < requests; ++r) {
        const int mine = lc_chunks(lens[r]);
        longest = lens[r] > longest ? lens[r] : longest;
        deepest = mine > deepest ? mine : deepest;
        tokens += lens[r];
        chunks += mine;
        several += mine > 0;
    }
    const double size = (double)H * D * V / (1 << 18), unit = H * (double)ChunkLayout(D, V).size / 2.56e6;
    const double chain = 1.05 * deepest, work = 2.0 * unit * chunks + 1.6 * size * several;
    const double in_chunks = 22 + (chain > work ? chain : work) + 45.0 * (turns - 1);
    const double alone = 8 + (0.25 + 0.05 * size) * longest + 0.025 * size * (tokens - longest), all = 0.07 * size * tokens;
    double walked = alone > all ? alone : all;
    if (rank > 0) walked += 5 + (0.006 + 0.014 * H * D * rank / 65536) * tokens;
    return in_chunks < walked ? room : 0;
}

template <int D>
static int launch_chunks(const bf16* fused, int row_stride, int q_off, int k_off, int v_off, const int* positions, const float* inv_freq, int rot_dim,
                         float q_scale, float k_scale, const float* decay, const float* head_decay, float* state, float* out, const int* req_q_start,
                         const int* req_q_len, const int* req_slot, const int* lens, int requests, int H, int V, unsigned char* scratch, int turn,
                         int* launched, cudaStream_t stream) {
    constexpr size_t walk_smem = (size_t)WALK_STAGES * WALK_GROUP * sizeof(WalkChunk);     // 127 KB: one CTA an SM (CTAs that start early would pile up in pairs)
    static bool raised = false;
    if (!raised) {
        cudaError_t e = cudaFuncSetAttribute(linattn_chunk_prepare_kernel<D, true>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sizeof(PrepareSmem<D>));
        if (e == cudaSuccess) e = cudaFuncSetAttribute(linattn_chunk_prepare_kernel<D, false>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sizeof(PrepareSmem<D>));
        if (e == cudaSuccess) e = cudaFuncSetAttribute(linattn_chunk_out_kernel<D>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sizeof(OutSmem<D>));
        if (e == cudaSuccess) e = cudaFuncSetAttribute(linattn_chunk_walk_kernel<D>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)walk_smem);
        if (e != cudaSuccess) return 1000 + (int)e;
        raised = true;
    }
    int longest = 0;
    bool few = false;
    for (int r = 0; r < requests; ++r) {
        longest = lens[r] > longest ? lens[r] : longest;
        few |= lens[r] > 0 && lens[r] < LC_FROM;
    }
    if (few) {
#define SHORT(C) wllm_launch(linattn_short_kernel<D, C>, dim3(V / LC_COLS, H, requests), LC_THREADS, 0, stream, fused, row_stride, q_off, k_off, v_off, positions, \
        inv_freq, rot_dim, q_scale, k_scale, decay, head_decay, state, out, req_q_start, req_q_len, req_slot, H, V)
        const int st = decay ? SHORT(true) : SHORT(false);
#undef SHORT
        if (st != WLLM_OK) return st;
        *launched += 1;
    }
    for (int b0 = 0; b0 < lc_chunks(longest); b0 += turn) {
        const int count = lc_count(lens, requests, b0, turn);
#define PREPARE(C) wllm_launch(linattn_chunk_prepare_kernel<D, C>, dim3(count, H), LC_THREADS, sizeof(PrepareSmem<D>), stream, fused, row_stride, q_off, k_off, \
        positions, inv_freq, rot_dim, q_scale, k_scale, decay, head_decay, req_q_start, req_q_len, req_slot, requests, H, V, b0, turn, scratch)
        int st = decay ? PREPARE(true) : PREPARE(false);
#undef PREPARE
        if (st == WLLM_OK)
            st = wllm_launch(linattn_chunk_walk_kernel<D>, dim3(D / LC_WALK_ROWS * (V / LC_COLS), H, requests), LC_THREADS, walk_smem, stream, fused + v_off,
                             row_stride, state, req_q_start, req_q_len, req_slot, H, V, b0, turn, scratch);
        if (st == WLLM_OK)
            st = wllm_launch(linattn_chunk_out_kernel<D>, dim3(V / LC_COLS, H, count), LC_THREADS, sizeof(OutSmem<D>), stream, fused + v_off, row_stride, out,
                             req_q_start, req_q_len, req_slot, requests, H, V, b0, turn, (const unsigned char*)scratch);
        if (st != WLLM_OK) return st;
        *launched += 3;
    }
    return WLLM_OK;
}

// The recurrence of every request of a step, from and to its state slot.  fused: bfloat16 rows `row_stride` elements apart that hold q [H, D], k [H, D] and
// v [H, V] at the offsets, all in steps of 8 elements; q and k are turned by their position over the first rot_dim channels (a multiple of 16; pairs half a
// turn apart) and scaled.  decay [n, H, D] per key channel, or null with head_decay [H].  D 64 or 128, V in steps of 64.  lens: req_q_len on the host.  Requests
// of LC_FROM tokens go in chunks, shorter ones token by token.
// scratch (16-byte aligned): wllm_linattn_chunks_bytes, or less (more turns, the same bits) but a chunk of every request that goes in chunks.  launched: kernels.
// 8 heads of 128 x 256, captured in a graph, us; behind, linattn_prepare and the walk in segments.  A decay per head: 2,048 tokens 74 and 205 (21 + 32 + 32 kernel by
// kernel under the profiler), 512 34 and 70, 130 27 and 36, 1,531 beside 24 single tokens 85 and 204, 16 requests of 130 139 and 143.  A decay per channel and its map
// (linattn_decay): 2,048 86 and 253, 512 41 and 86, 130 34 and 46, 1,531 beside 24 95 and 244, 16 of 130 145 and 183.  (Products of up to 128 rows leave partial sums,
// which are not read here.)  Distance from 64 bits, decays near one: outputs 2.3e-7 to 2.6e-7 where the walk has 2.4e-7 to 3.0e-7, states 1.8e-7 to 2.4e-7 and 2.3e-7 to 3.0e-7.
WLLM_API int wllm_linattn_chunks(const void* fused, int row_stride, int q_off, int k_off, int v_off, const int* positions, const float* inv_freq,
                                 int rot_dim, float q_scale, float k_scale, const float* decay, const float* head_decay, float* state, float* out,
                                 const int* req_q_start, const int* req_q_len, const int* req_slot, const int* lens, int requests, int H, int D, int V,
                                 void* scratch, long long scratch_bytes, int* launched, cudaStream_t stream) {
    *launched = 0;
    if (requests <= 0) return WLLM_OK;
    if (!lc_sizes(H, D, V) || requests > 65535 || rot_dim < 0 || rot_dim > D || rot_dim % 16 != 0 || (!decay && !head_decay)) return WLLM_BAD_SIZE;
    if (((row_stride | q_off | k_off | v_off) & 7) || (((uintptr_t)fused | (uintptr_t)scratch) & 15) || (((uintptr_t)state | (uintptr_t)out) & 7)) return WLLM_BAD_ALIGN;
    long long chunks;
    const int turn = lc_turn(lens, requests, H * ChunkLayout(D, V).size, scratch_bytes, chunks);
    if (chunks > 65535 || chunks * H * ChunkLayout(D, V).size > scratch_bytes) return WLLM_BAD_SIZE;
#define CHUNKS(DD) launch_chunks<DD>((const bf16*)fused, row_stride, q_off, k_off, v_off, positions, inv_freq, rot_dim, q_scale, k_scale, decay, head_decay, \
        state, out, req_q_start, req_q_len, req_slot, lens, requests, H, V, (unsigned char*)scratch, turn, launched, stream)
    return D == 64 ? CHUNKS(64) : CHUNKS(128);
#undef CHUNKS
}
