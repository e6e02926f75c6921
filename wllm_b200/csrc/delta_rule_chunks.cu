// The gated delta rule of delta_rule.cu in chunks of 64 tokens on the tensor cores, for long portions of bfloat16 models:
//
//     S <- diag(g_t) S;   u_t = beta_t (v_t - S^T k_t);   S <- S + k_t u_t^T;   o_t = S^T q_t
//
// With S the state in front of a chunk, G_t the product of the chunk's decays up to t, G_(s..t) that of the tokens behind s up to t, A_ts = k_t . (G_(s..t) k_s)
// and P_ts = q_t . (G_(s..t) k_s),
//
//     (1 + diag(beta) A, s < t) [W | U] = diag(beta) [G_t k_t | v_t]        worked out beforehand
//     R = U - W S;   o_t = (G_t q_t)^T S + sum_(s <= t) P_ts R_s;   S <- diag(G_end) S + sum_s (G_(s..end) k_s) R_s^T
//
// (Yang, Wang, Zhang, Shen and Kim, "Parallelizing linear transformers with the delta rule over sequence length", 2024).  Kernels:
//
//   prepare   a CTA per (chunk, head): what the other two read, in the order of a lane's registers.  Products of decays are running products of factors that are
//             at most one, as in linear_attention_chunks.cu: no quotients.  [W | U] by forward substitution in 32 bits, a thread a column, sixteen rows at a time.
//   walk      a CTA per (VT value columns, head, request), S in 32-bit registers and as pieces in shared memory: R and the state chunk by chunk.
//   out       a CTA per (chunk, head): both shares of the outputs.
//
// 32-bit numbers are three bfloat16 pieces each (24 bits), and of nine products the six of some weight are taken, large and small ones summed apart.  A chunk's
// products are summed from zero and join the state in one rounding.
//
// Measured, 16 heads, captured in a graph, us; behind, the walk in blocks of eight tokens: 2,048 tokens 194 (prepare 87, walk 90, out 38 kernel by kernel under the
// profiler: profiles/recurrence_chunks_2048.txt) and 274, 8,192 772 and 1,078, 512 59 and 73, 256 47 and 42, 3 x 1,021 310 and 365, 1,531 beside 24 single tokens 187 and 243; a
// decay per key channel within 2 %.  A chunk costs the same full or not, so that steps of many short requests stay with the blocks: 16 x 130 338 and 248.
// Distance from 64 bits where models' decays lie (A softplus(a + bias), A of 1 to 16, steps of 1e-3 to 1e-1), a decay per head and per channel: outputs 1.3e-7 and 1.5e-7
// where the blocks have 1.5e-7 and 1.8e-7, states 0.8e-7 to 1.4e-7 and 1.1e-7 to 1.7e-7; where nearly all is forgotten within two tokens 0.9e-7 for 0.86e-7.
#include "chunk_common.cuh"

constexpr int DC = 128, DCV = 128;     // key channels and value columns of a head
constexpr int DP_THREADS = 256, DW_THREADS = 512, DO_THREADS = 256;       // of prepare, walk and out

// What the kernels hand on for a (chunk, head), in bytes:
//   Q [4 row tiles][8][3][32 lanes] G_t q_t    K [8][4][3][32] (G_(s..end) k_s)^T    P [4][4][3][32] (tiles above the diagonal stay empty)    W [4][8][3][32]
//   G [128] floats (decays given as g - 1: G_end - 1)    U [64][128] floats    S [3][128][128], R [3][64][128] bfloat16
constexpr long long DC_OP = 4ll * 8 * 3 * 512, DC_Q = 0, DC_K = DC_OP, DC_W = 2 * DC_OP, DC_P = 3 * DC_OP, DC_G = DC_P + 4 * 4 * 3 * 512, DC_U = DC_G + DC * 4,
                    DC_S = DC_U + (long long)LC * DCV * 4, DC_R = DC_S + 3ll * DC * DCV * 2, DC_SIZE = DC_R + 3ll * LC * DCV * 2;

struct DeltaPrepareSmem {
    // (pitches: X is read as pairs along its rows, eight rows a warp; K down its columns too)
    static constexpr int XP = DC + 8, DP = DC + 4, AP = LC + 4, PAIRS = LB * (LB + 1) / 2;
    float X[LC][XP], K[LC][DP];                // q (or k) and k; then G_t q_t (G_t k_t) from their block's start on and k_s to its end; then W and U
    float G[LBLOCKS][DC], G1[LBLOCKS][DC];     // the blocks' decays, and those less one
    float before[LBLOCKS][DC], behind[LBLOCKS][DC], between[12][DC];      // those of the blocks in front, behind, and between (linear_attention_chunks.cu)
    float A[LC][AP];                           // P; or diag(beta) A turned: [s][t]
    float sums[LBLOCKS][2][PAIRS];
    float beta[LC];
};

// KEYS: W and U; else Q, K, P and G.
template <bool CHANNEL, bool KEYS>
__device__ __forceinline__ void delta_chunk_prepare(const float* __restrict__ q, const float* __restrict__ k, const float* __restrict__ v,
                                                    const float* __restrict__ beta, const float* __restrict__ decay, int first, int count, int h, int H, int G,
                                                    unsigned char* __restrict__ mine, DeltaPrepareSmem& sm) {
    typedef DeltaPrepareSmem Smem;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    {
        const size_t row = (size_t)G * DC, base = (size_t)(h / (H / G)) * DC;
#pragma unroll
        for (int i = 0; i < LC * (DC / 4) / DP_THREADS; ++i) {
            const int idx = threadIdx.x + i * DP_THREADS, t = idx / (DC / 4), c = (idx % (DC / 4)) * 4;
            const bool in = t < count;
            const size_t at = (size_t)(first + (in ? t : 0)) * row + base + c;
            if (!KEYS) lc_cp16(&sm.X[t][c], q + at, in);
            lc_cp16(&sm.K[t][c], k + at, in);
        }
        asm volatile("cp.async.commit_group;" ::: "memory");
    }
    if (KEYS && threadIdx.x < LC) sm.beta[threadIdx.x] = threadIdx.x < count ? beta[(size_t)(first + threadIdx.x) * H + h] : 0.f;
    // ---- blocks of eight tokens: a thread two blocks, two channels
    const int c2 = 2 * (threadIdx.x & 63), side = warp & 1;
    float2 e[2][LB];                   // decays, or those less one
#pragma unroll
    for (int u = 0; u < 2; ++u)
#pragma unroll
        for (int i = 0; i < LB; ++i) {
            const int t = (2 * (threadIdx.x >> 6) + u) * LB + i;
            e[u][i] = CHANNEL ? make_float2(0.f, 0.f) : make_float2(1.f, 1.f);
            if (t < count) {
                if (CHANNEL) e[u][i] = *reinterpret_cast<const float2*>(decay + ((size_t)(first + t) * H + h) * DC + c2);
                else e[u][i].x = e[u][i].y = decay[(size_t)(first + t) * H + h];
            }
        }
    auto fade = [](float2 x, float2 d) { return CHANNEL ? fma2(x, d, x) : lc_mul2(x, d); };
    asm volatile("cp.async.wait_group 0;" ::: "memory");
    __syncthreads();
#pragma unroll
    for (int u = 0; u < 2; ++u) {
        const int B = 2 * (threadIdx.x >> 6) + u;
        float2 kk[LB], xx[LB];
#pragma unroll
        for (int i = 0; i < LB; ++i) {
            kk[i] = *reinterpret_cast<const float2*>(&sm.K[B * LB + i][c2]);
            xx[i] = KEYS ? kk[i] : *reinterpret_cast<const float2*>(&sm.X[B * LB + i][c2]);
        }
        float x[32], more[4];          // sums of pairs i >= j: i (i + 1) / 2 + j; of keys i > j: i (i - 1) / 2 + j
        if (KEYS)
#pragma unroll
            for (int i = 28; i < 32; ++i) x[i] = 0.f;
#pragma unroll
        for (int j = 0; j < LB; ++j) {
            float2 w = kk[j];
#pragma unroll
            for (int i = j; i < LB; ++i) {
                if (i > j) w = fade(w, e[u][i]);
                else if (KEYS) continue;
                const float y = fmaf(xx[i].x, w.x, xx[i].y * w.y);
                const int at = KEYS ? i * (i - 1) / 2 + j : i * (i + 1) / 2 + j;
                if (at < 32) x[at & 31] = y;
                else more[at & 3] = y;
            }
            *reinterpret_cast<float2*>(&sm.K[B * LB + j][c2]) = w;
        }
        sm.sums[B][side][lane] = lc_sums(x, lane);
        if (!KEYS) {
            const float m = lc_sums(more, lane);
            if ((lane & 7) == 0) sm.sums[B][side][32 + (lane >> 3)] = m;
        }
        float2 E = make_float2(1.f, 1.f), E1 = make_float2(0.f, 0.f);
#pragma unroll
        for (int i = 0; i < LB; ++i) {
            if (CHANNEL && !KEYS) E1 = make_float2(fmaf(E1.x, e[u][i].x, E1.x + e[u][i].x), fmaf(E1.y, e[u][i].y, E1.y + e[u][i].y));
            E = fade(E, e[u][i]);
            *reinterpret_cast<float2*>(&sm.X[B * LB + i][c2]) = lc_mul2(xx[i], E);
        }
        *reinterpret_cast<float2*>(&sm.G[B][c2]) = E;
        if (CHANNEL && !KEYS) *reinterpret_cast<float2*>(&sm.G1[B][c2]) = E1;
    }
    __syncthreads();
    // ---- products of the blocks' decays; sums inside the blocks
    if (threadIdx.x < DC) {
        const int c = threadIdx.x;
        float run = 1.f;
#pragma unroll
        for (int b = 0; b < LBLOCKS; ++b) { sm.before[b][c] = run; run *= sm.G[b][c]; }
        if (!KEYS) {
            if (CHANNEL) {
                run = 0.f;
#pragma unroll
                for (int b = 0; b < LBLOCKS; ++b) run = fmaf(run, sm.G1[b][c], run + sm.G1[b][c]);
            }
            reinterpret_cast<float*>(mine + DC_G)[c] = run;
            run = 1.f;
#pragma unroll
            for (int b = LBLOCKS - 1; b >= 0; --b) { sm.behind[b][c] = run; run *= sm.G[b][c]; }
        }
    } else {
        const int c = threadIdx.x - DC;
#pragma unroll
        for (int I = 1; I < 4; ++I) {
            float run = 1.f;
#pragma unroll
            for (int J = 2 * I - 1; J >= 0; --J) { sm.between[I * (I - 1) + J][c] = run; run *= sm.G[J][c]; }
        }
    }
#pragma unroll
    for (int u = 0; u < 2; ++u) {
        const int idx = threadIdx.x + u * DP_THREADS, b = idx >> 6, i = (idx >> 3) & 7, j = idx & 7;
        float x = 0.f;
        if (KEYS ? j < i : j <= i) {
            const int at = KEYS ? i * (i - 1) / 2 + j : i * (i + 1) / 2 + j;
            x = sm.sums[b][0][at] + sm.sums[b][1][at];
        }
        if (KEYS) sm.A[b * LB + j][b * LB + i] = sm.beta[b * LB + i] * x;
        else {
            sm.A[b * LB + i][b * LB + j] = x;
            if ((b & 1) == 0) sm.A[b * LB + i][(b + 1) * LB + j] = 0.f;      // (the upper half of a tile of 16: a zero that the operand's tile holds)
        }
    }
    // the first values of a column
    float ahead[16];
    const int column = threadIdx.x & (DC - 1);
    const float* vc = v + (size_t)h * DCV + column;
    auto look = [&](int I) {
#pragma unroll
        for (int i = 0; i < 16; ++i) ahead[i] = 16 * I + i < count ? vc[(size_t)(first + 16 * I + i) * H * DCV] : 0.f;
    };
    if (KEYS && threadIdx.x >= DC) look(0);
    __syncthreads();
    // ---- sums between blocks, tiles of sixteen tokens by a block, two a warp: warps 0 to 5 the tokens I = 1, 2, 2, 3, 3, 3 with blocks J < 2 I in front of
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
#pragma unroll 2
        for (int c = c0; c < DC; c += 16) {
            uint4 a[3];
            if (!inside) {
                const float* x = sm.X[16 * I + r0];
                const float2 x0 = at2(x + c), x1 = at2(x + c + 8);
                const float2 y0 = lc_mul2(at2(x + 8 * Smem::XP + c), at2(&sm.G[2 * I][c])), y1 = lc_mul2(at2(x + 8 * Smem::XP + c + 8), at2(&sm.G[2 * I][c + 8]));
                lc_split(x0.x, x0.y, a[0].x, a[1].x, a[2].x);
                lc_split(y0.x, y0.y, a[0].y, a[1].y, a[2].y);
                lc_split(x1.x, x1.y, a[0].z, a[1].z, a[2].z);
                lc_split(y1.x, y1.y, a[0].w, a[1].w, a[2].w);
            }
#pragma unroll
            for (int u = 0; u < 2; ++u) {
                const int J = inside ? 4 * (warp - 6) + 2 * u : J0 + u;
                if (inside) {
                    const float* x = sm.X[8 * J + 8 + r0];
                    const float2 y0 = at2(x + c), y1 = at2(x + c + 8);
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
                uint32_t b[3][2];
                lc_split(k0.x, k0.y, b[0][0], b[1][0], b[2][0]);
                lc_split(k1.x, k1.y, b[0][1], b[1][1], b[2][1]);
                lc_mma(small[u], a[0], b[2][0], b[2][1]);
                lc_mma(small[u], a[2], b[0][0], b[0][1]);
                lc_mma(small[u], a[1], b[1][0], b[1][1]);
                lc_mma(small[u], a[0], b[1][0], b[1][1]);
                lc_mma(small[u], a[1], b[0][0], b[0][1]);
                lc_mma_add(big[u], a[0], b[0][0], b[0][1]);
            }
        }
#pragma unroll
        for (int u = 0; u < 2; ++u) {
            const int J = inside ? 4 * (warp - 6) + 2 * u : J0 + u, row = (inside ? 8 * J : 16 * I) + r0, s = 8 * J + c0;
            float x[4];
#pragma unroll
            for (int i = 0; i < 4; ++i) x[i] = big[u][i] + small[u][i];
            if (KEYS) {
                const float b0 = sm.beta[row], b8 = sm.beta[row + 8];
                if (!inside) {
                    sm.A[s][row] = b0 * x[0];
                    sm.A[s + 1][row] = b0 * x[1];
                }
                sm.A[s][row + 8] = b8 * x[2];
                sm.A[s + 1][row + 8] = b8 * x[3];
            } else {
                if (!inside) *reinterpret_cast<float2*>(&sm.A[row][s]) = make_float2(x[0], x[1]);
                *reinterpret_cast<float2*>(&sm.A[row + 8][s]) = make_float2(x[2], x[3]);
            }
        }
    }
    __syncthreads();
    const int r0 = lane >> 2, c0 = 2 * (lane & 3);
    // a tile of an operand, in the order of a lane's registers
    auto leave = [&](uint4* to, float2 v0, float2 v1, float2 v2, float2 v3) {
        uint4 p[3];
        lc_split(v0.x, v0.y, p[0].x, p[1].x, p[2].x);
        lc_split(v1.x, v1.y, p[0].y, p[1].y, p[2].y);
        lc_split(v2.x, v2.y, p[0].z, p[1].z, p[2].z);
        lc_split(v3.x, v3.y, p[0].w, p[1].w, p[2].w);
#pragma unroll
        for (int i = 0; i < 3; ++i) to[i * 32 + lane] = p[i];
    };
    if (KEYS) {
        // ---- W and U by forward substitution, sixteen rows at a time: a thread a column
        const bool values = threadIdx.x >= DC;
        float* X = values ? &sm.K[0][column] : &sm.X[0][column];
        const int pitch = values ? Smem::DP : Smem::XP;
        float* to = reinterpret_cast<float*>(mine + DC_U) + column;
        for (int I = 0; I < 4; ++I) {
            // (what the tokens in front take away is summed for itself, small beside what it is taken from, and taken away in one rounding)
            float x[16], own[16];
#pragma unroll
            for (int i = 0; i < 16; ++i) {
                x[i] = 0.f;
                own[i] = values ? ahead[i] : X[(16 * I + i) * pitch] * sm.before[2 * I + (i >> 3)][column];
            }
            if (values && I < 3) look(I + 1);
#pragma unroll 4
            for (int s = 0; s < 16 * I; ++s) {
                const float y = X[s * pitch];
                const float4* l = reinterpret_cast<const float4*>(&sm.A[s][16 * I]);
#pragma unroll
                for (int i = 0; i < 4; ++i) {
                    const float4 w = l[i];
                    x[4 * i] = fmaf(w.x, y, x[4 * i]);
                    x[4 * i + 1] = fmaf(w.y, y, x[4 * i + 1]);
                    x[4 * i + 2] = fmaf(w.z, y, x[4 * i + 2]);
                    x[4 * i + 3] = fmaf(w.w, y, x[4 * i + 3]);
                }
            }
#pragma unroll
            for (int j = 0; j < 16; ++j) {
                const float y = x[j] = fmaf(sm.beta[16 * I + j], own[j], -x[j]);
                if (j == 15) break;
                const float4* l = reinterpret_cast<const float4*>(&sm.A[16 * I + j][16 * I]);
#pragma unroll
                for (int i = (j + 1) / 4; i < 4; ++i) {
                    const float4 w = l[i];
                    if (4 * i > j) x[4 * i] = fmaf(w.x, y, x[4 * i]);
                    if (4 * i + 1 > j) x[4 * i + 1] = fmaf(w.y, y, x[4 * i + 1]);
                    if (4 * i + 2 > j) x[4 * i + 2] = fmaf(w.z, y, x[4 * i + 2]);
                    if (4 * i + 3 > j) x[4 * i + 3] = fmaf(w.w, y, x[4 * i + 3]);
                }
            }
#pragma unroll
            for (int i = 0; i < 16; ++i) {
                X[(16 * I + i) * pitch] = x[i];
                if (values) to[(16 * I + i) * DCV] = x[i];
            }
        }
        __syncthreads();
    }
    for (int tile = warp; tile < 32; tile += DP_THREADS / 32) {
        const int wm = tile >> 3, ks = tile & 7;
        float2 x[4];
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            const int t = wm * 16 + r0 + (i & 1) * 8, c = ks * 16 + c0 + (i >> 1) * 8;
            x[i] = *reinterpret_cast<const float2*>(&sm.X[t][c]);
            if (!KEYS) x[i] = lc_mul2(x[i], *reinterpret_cast<const float2*>(&sm.before[t / LB][c]));
        }
        leave(reinterpret_cast<uint4*>(mine + (KEYS ? DC_W : DC_Q)) + (size_t)tile * 96, x[0], x[1], x[2], x[3]);
    }
    if (!KEYS) {
        for (int tile = warp; tile < 32; tile += DP_THREADS / 32) {
            const int dt = tile >> 2, ks = tile & 3;
            float2 x[4];
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                const int d = dt * 16 + r0 + (i & 1) * 8, t = ks * 16 + c0 + (i >> 1) * 8;     // (t and t + 1 lie in one block)
                const float f = sm.behind[t / LB][d];
                x[i] = make_float2(sm.K[t][d] * f, sm.K[t + 1][d] * f);
            }
            leave(reinterpret_cast<uint4*>(mine + DC_K) + (size_t)tile * 96, x[0], x[1], x[2], x[3]);
        }
        for (int tile = warp; tile < 16; tile += DP_THREADS / 32) {
            const int wm = tile >> 2, ks = tile & 3;
            if (ks > wm) continue;
            float2 x[4];
#pragma unroll
            for (int i = 0; i < 4; ++i) x[i] = *reinterpret_cast<const float2*>(&sm.A[wm * 16 + r0 + (i & 1) * 8][ks * 16 + c0 + (i >> 1) * 8]);
            leave(reinterpret_cast<uint4*>(mine + DC_P) + (size_t)tile * 96, x[0], x[1], x[2], x[3]);
        }
    }
}

// grid (2, chunks of the turn, H), 256 threads, two CTAs an SM: one of a (chunk, head)'s queries, one of its keys.  Bound by latency and
// shared memory (64 % of its throughput): few of a phase's instructions are independent.  87 us for 2,048 tokens of 16 heads under the profiler (both in one CTA of 512
// threads, one an SM: 92).
template <bool CHANNEL>
__global__ void __launch_bounds__(DP_THREADS, 2)
delta_chunk_prepare_kernel(const float* __restrict__ q, const float* __restrict__ k, const float* __restrict__ v, const float* __restrict__ beta,
                           const float* __restrict__ decay, const int* __restrict__ req_q_start, const int* __restrict__ req_q_len,
                           const int* __restrict__ req_slot, int requests, int H, int G, int b0, int turn, unsigned char* __restrict__ scratch) {
    extern __shared__ __align__(16) unsigned char dc_raw[];
    DeltaPrepareSmem& sm = *reinterpret_cast<DeltaPrepareSmem*>(dc_raw);
    pdl_begin();
    int chunk;
    const int r = lc_find(req_q_len, requests, b0, turn, blockIdx.y, chunk), h = blockIdx.z;
    if (r < 0 || req_slot[r] < 0) return;
    const int first = req_q_start[r] + chunk * LC, count = min(LC, req_q_len[r] - chunk * LC);
    unsigned char* mine = scratch + ((size_t)blockIdx.y * H + h) * DC_SIZE;
    if (blockIdx.x) delta_chunk_prepare<CHANNEL, false>(q, k, v, beta, decay, first, count, h, H, G, mine, sm);
    else delta_chunk_prepare<CHANNEL, true>(q, k, v, beta, decay, first, count, h, H, G, mine, sm);
}

constexpr int VT = 16, DW_PITCH = VT + 8;      // value columns of a CTA of the walk

struct DeltaWalkSmem {
    uint4 ring[3][4 * 8 * 96];         // W and K in turn
    float U[2][LC][DW_PITCH], g[2][DC];
    bf16 S[3][DC][DW_PITCH], R[3][LC][DW_PITCH];
    float2 part[DW_THREADS / 32][4][32];       // what warps hand one another
};

// grid (128 / VT, H, requests), 512 threads.  R: warps w, w + 4, w + 8, w + 12 rows 16 w .., a fourth of the channels each; the state: warps w and w + 8 channels
// 16 w .., half of the tokens each.  Warps of the same rows hand one another their sums and finish a part of the columns.  Bound by shared memory (72 % of its
// throughput) and the latency of two products a chunk.  90 us for 2,048 tokens of 16 heads under the profiler.  (In turn: this form 88, eight warps a CTA 89, 32 columns a CTA 130; operands
// straight to the registers of the one warp that reads them, without the ring, 96.)
template <bool CHANNEL>
__global__ void __launch_bounds__(DW_THREADS, 1)
delta_chunk_walk_kernel(float* __restrict__ state, const int* __restrict__ req_q_len, const int* __restrict__ req_slot, int H, int b0, int turn,
                        unsigned char* __restrict__ scratch) {
    extern __shared__ __align__(16) unsigned char dc_raw[];
    DeltaWalkSmem& sm = *reinterpret_cast<DeltaWalkSmem*>(dc_raw);
    pdl_begin();
    const int r = blockIdx.z, h = blockIdx.y, v0 = blockIdx.x * VT, len = req_q_len[r], slot = req_slot[r];
    if (slot < 0) return;
    const int chunks = min(lc_chunks(len) - b0, turn);
    if (chunks <= 0) return;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, frow = lane >> 2, fcol = 2 * (lane & 3);
    unsigned char* mine = scratch + ((size_t)lc_before(req_q_len, r, b0, turn) * H + h) * DC_SIZE;
    const size_t next = (size_t)H * DC_SIZE;
    auto load = [&](int m) {           // W (even) and K (odd) of the chunks, one behind the other
        const int c = m >> 1;
        if (c < chunks) {
            const unsigned char* p = mine + c * next;
            const uint4* src = reinterpret_cast<const uint4*>(p + ((m & 1) ? DC_K : DC_W));
            uint4* to = sm.ring[m % 3];
#pragma unroll
            for (int i = 0; i < 4 * 8 * 96 / DW_THREADS; ++i) lc_cp16(&to[threadIdx.x + i * DW_THREADS], src + threadIdx.x + i * DW_THREADS, true);
            if (m & 1) {
                if (threadIdx.x < DC / 4) lc_cp16(&sm.g[c & 1][4 * threadIdx.x], reinterpret_cast<const float*>(p + DC_G) + 4 * threadIdx.x, true);
            } else if (threadIdx.x < LC * (VT / 4)) {
                const int t = threadIdx.x / (VT / 4), col = (threadIdx.x % (VT / 4)) * 4;
                lc_cp16(&sm.U[c & 1][t][col], reinterpret_cast<const float*>(p + DC_U) + (size_t)t * DCV + v0 + col, true);
            }
        }
        asm volatile("cp.async.commit_group;" ::: "memory");                 // (an empty group keeps the count of groups)
    };
    load(0);
    load(1);
    // pieces of shared memory to their place in the chunk
    auto copy = [&](const bf16* from, long long offset, int rows, int c) {
        bf16* far = reinterpret_cast<bf16*>(mine + c * next + offset) + v0;
        for (int idx = threadIdx.x; idx < 3 * rows * (VT / 8); idx += DW_THREADS) {
            const int row = idx / (VT / 8), p = (idx % (VT / 8)) * 8;
            *reinterpret_cast<uint4*>(far + (size_t)row * DCV + p) = *reinterpret_cast<const uint4*>(from + row * DW_PITCH + p);
        }
    };
    const int wm = warp & 3, quarter = warp >> 2;                            // of R
    const int ct = warp & 7, half_k = warp >> 3;                             // of the state
    // this warp's 16 channels by 8 columns of the state
    float* Sg = state + ((size_t)slot * H + h) * DC * DCV + (size_t)(ct * 16 + frow) * DCV + v0 + half_k * 8 + fcol;
    float S[4];
#pragma unroll
    for (int half = 0; half < 2; ++half) {
        const float2 x = *reinterpret_cast<const float2*>(Sg + (size_t)half * 8 * DCV);
        S[half * 2] = x.x;
        S[half * 2 + 1] = x.y;
    }
    auto put_state = [&]() {
#pragma unroll
        for (int half = 0; half < 2; ++half) {
            uint32_t p[3];
            lc_split(S[half * 2], S[half * 2 + 1], p[0], p[1], p[2]);
#pragma unroll
            for (int i = 0; i < 3; ++i) *reinterpret_cast<uint32_t*>(&sm.S[i][ct * 16 + frow + half * 8][half_k * 8 + fcol]) = p[i];
        }
    };
    put_state();
    const int krow = (lane & 7) + ((lane >> 3) & 1) * 8, kcol = (lane >> 4) * 8;
    // 16 rows of A times the 16 columns of the pieces B, two steps of 16
    auto product = [&](const uint4* A, const bf16* B, int plane, float (&sum)[2][4]) {
        float big[2][4], small[2][2][4];
#pragma unroll
        for (int j = 0; j < 2; ++j)
#pragma unroll
            for (int i = 0; i < 4; ++i) big[j][i] = small[0][j][i] = small[1][j][i] = 0.f;
#pragma unroll
        for (int ks = 0; ks < 2; ++ks) {
            uint4 a[3];
#pragma unroll
            for (int p = 0; p < 3; ++p) a[p] = A[(ks * 3 + p) * 32];
#pragma unroll
            for (int p = 2; p >= 0; --p) {
                uint32_t b[4];
                lc_ldsm4_t(B + p * plane + (ks * 16 + krow) * DW_PITCH + kcol, b);
#pragma unroll
                for (int i = 2 - p; i >= 0; --i)
#pragma unroll
                    for (int j = 0; j < 2; ++j) {
                        if (p + i == 0) lc_mma_add(big[j], a[i], b[2 * j], b[2 * j + 1]);
                        else lc_mma(small[ks][j], a[i], b[2 * j], b[2 * j + 1]);
                    }
            }
        }
#pragma unroll
        for (int j = 0; j < 2; ++j)
#pragma unroll
            for (int i = 0; i < 4; ++i) sum[j][i] = big[j][i] + (small[0][j][i] + small[1][j][i]);
    };
    for (int c = 0; c < chunks; ++c) {
        float x[2][4];
        // ---- R = U - W S
        asm volatile("cp.async.wait_group 1;" ::: "memory");
        __syncthreads();               // W, U and the state's pieces are here; K of the chunk before is read to its end
        load(2 * c + 2);
        product(sm.ring[(2 * c) % 3] + (wm * 8 + quarter * 2) * 96 + lane, &sm.S[0][quarter * 32][0], DC * DW_PITCH, x);
        // (warp `quarter` finishes tile quarter >> 1, rows quarter & 1 of the eights)
#pragma unroll
        for (int i = 0; i < 4; ++i) sm.part[warp][i][lane] = make_float2(x[i >> 1][2 * (i & 1)], x[i >> 1][2 * (i & 1) + 1]);
        asm volatile("bar.sync %0, 128;" ::"r"(1 + wm) : "memory");          // the four warps of these rows
        {
            const int row = wm * 16 + frow + (quarter & 1) * 8, col = (quarter >> 1) * 8 + fcol;
            const float2 u = *reinterpret_cast<const float2*>(&sm.U[c & 1][row][col]);
            const float2 s0 = sm.part[wm][quarter][lane], s1 = sm.part[wm + 4][quarter][lane], s2 = sm.part[wm + 8][quarter][lane],
                         s3 = sm.part[wm + 12][quarter][lane];
            uint32_t p[3];
            lc_split(u.x - ((s0.x + s1.x) + (s2.x + s3.x)), u.y - ((s0.y + s1.y) + (s2.y + s3.y)), p[0], p[1], p[2]);
#pragma unroll
            for (int i = 0; i < 3; ++i) *reinterpret_cast<uint32_t*>(&sm.R[i][row][col]) = p[i];
        }
        copy(&sm.S[0][0][0], DC_S, DC, c);
        // ---- the state behind the chunk
        asm volatile("cp.async.wait_group 1;" ::: "memory");
        __syncthreads();               // K, its decays and R's pieces are here; W is read to its end
        load(2 * c + 3);
        product(sm.ring[(2 * c + 1) % 3] + (ct * 4 + half_k * 2) * 96 + lane, &sm.R[0][half_k * 32][0], LC * DW_PITCH, x);
#pragma unroll
        for (int i = 0; i < 2; ++i) sm.part[warp][i][lane] = half_k ? make_float2(x[0][2 * i], x[0][2 * i + 1]) : make_float2(x[1][2 * i], x[1][2 * i + 1]);
        asm volatile("bar.sync %0, 64;" ::"r"(5 + ct) : "memory");           // the two warps of these channels
#pragma unroll
        for (int half = 0; half < 2; ++half) {
            const float2 other = sm.part[warp ^ 8][half][lane];
            const float g = sm.g[c & 1][ct * 16 + frow + half * 8];
            const float add[2] = {(half_k ? x[1][2 * half] : x[0][2 * half]) + other.x, (half_k ? x[1][2 * half + 1] : x[0][2 * half + 1]) + other.y};
#pragma unroll
            for (int e = 0; e < 2; ++e) {
                float& s = S[2 * half + e];
                s = CHANNEL ? s + fmaf(g, s, add[e]) : fmaf(g, s, add[e]);
            }
        }
        copy(&sm.R[0][0][0], DC_R, LC, c);
        if (c + 1 < chunks) put_state();       // (the pieces of the state in front are copied and read to their end)
    }
    asm volatile("cp.async.wait_group 0;" ::: "memory");
#pragma unroll
    for (int half = 0; half < 2; ++half) *reinterpret_cast<float2*>(Sg + (size_t)half * 8 * DCV) = make_float2(S[half * 2], S[half * 2 + 1]);
}

constexpr int DO_COLS = 64;

struct DeltaOutSmem {
    bf16 S[3][DC][DO_COLS];            // rows of 128 bytes, 16-byte piece p of row r at p ^ (r & 7); then R in the first 64 rows
    uint4 Q[4][DC / 16 * 96];
};

// grid (128 / 64, H, chunks of the turn), 256 threads, two CTAs an SM: warp w rows 16 (w & 3) .., columns 32 (w >> 2) ..  Bound by its operands' way from memory:
// 38 us for 2,048 tokens of 16 heads under the profiler.  (In turn: this form 36, 128 columns and 512 threads, one CTA an SM, 41.)
__global__ void __launch_bounds__(DO_THREADS, 2)
delta_chunk_out_kernel(float* __restrict__ out, const int* __restrict__ req_q_start, const int* __restrict__ req_q_len, const int* __restrict__ req_slot,
                       int requests, int H, int b0, int turn, const unsigned char* __restrict__ scratch) {
    extern __shared__ __align__(16) unsigned char dc_raw[];
    DeltaOutSmem& sm = *reinterpret_cast<DeltaOutSmem*>(dc_raw);
    pdl_begin();
    int chunk;
    const int r = lc_find(req_q_len, requests, b0, turn, blockIdx.z, chunk), h = blockIdx.y, v0 = blockIdx.x * DO_COLS;
    if (r < 0 || req_slot[r] < 0) return;
    const int first = req_q_start[r] + chunk * LC, count = min(LC, req_q_len[r] - chunk * LC);
    const unsigned char* mine = scratch + ((size_t)blockIdx.z * H + h) * DC_SIZE;
    const bf16 *St = reinterpret_cast<const bf16*>(mine + DC_S) + v0, *Rt = reinterpret_cast<const bf16*>(mine + DC_R) + v0;
    constexpr int PARTS = 4, ROWS = DC / PARTS, PIECES = DO_COLS / 8;        // the state comes in four runs of channels, the queries' beside it
#pragma unroll
    for (int part = 0; part < PARTS; ++part) {
        for (int idx = threadIdx.x; idx < 3 * ROWS * PIECES; idx += DO_THREADS) {
            const int piece = idx / (ROWS * PIECES), row = part * ROWS + (idx / PIECES) % ROWS, p = idx % PIECES;
            lc_cp16(&sm.S[piece][row][(p ^ (row & 7)) * 8], St + (size_t)(piece * DC + row) * DCV + p * 8, true);
        }
        constexpr int EACH = DC / 16 / PARTS * 96;
        for (int idx = threadIdx.x; idx < 4 * EACH; idx += DO_THREADS) {
            const int tile = idx / EACH, i = part * EACH + idx % EACH;
            lc_cp16(&sm.Q[tile][i], reinterpret_cast<const uint4*>(mine + DC_Q) + (size_t)tile * (DC / 16) * 96 + i, true);
        }
        asm volatile("cp.async.commit_group;" ::: "memory");
    }
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, wm = warp & 3, wn = warp >> 2, frow = lane >> 2, fcol = 2 * (lane & 3);
    const uint4* af = reinterpret_cast<const uint4*>(mine + DC_P) + (size_t)wm * 4 * 96 + lane;
    const int krow = (lane & 7) + ((lane >> 3) & 1) * 8, kcol = wn * 32 + (lane >> 4) * 8;
    auto place = [&](int jj) { return (kcol + jj * 16) ^ ((krow & 7) * 8); };
    uint4 a[2][3];                                         // two tiles of P ahead
    float big[4][4], small[4][4], own[4][4];
#pragma unroll
    for (int j = 0; j < 4; ++j)
#pragma unroll
        for (int e = 0; e < 4; ++e) big[j][e] = small[j][e] = own[j][e] = 0.f;
    // ---- the share of the state in front of the chunk
#pragma unroll
    for (int part = 0; part < PARTS; ++part) {
        if (part == 0) asm volatile("cp.async.wait_group 3;" ::: "memory");
        if (part == 1) asm volatile("cp.async.wait_group 2;" ::: "memory");
        if (part == 2) asm volatile("cp.async.wait_group 1;" ::: "memory");
        if (part == 3) asm volatile("cp.async.wait_group 1;" ::: "memory");
        __syncthreads();
        if (part == 2) {
            // the first half of the state is read to its end: R takes its place
            for (int idx = threadIdx.x; idx < 3 * LC * PIECES; idx += DO_THREADS) {
                const int piece = idx / (LC * PIECES), t = (idx / PIECES) % LC, p = idx % PIECES;
                lc_cp16(&sm.S[piece][t][(p ^ (t & 7)) * 8], Rt + (size_t)(piece * LC + t) * DCV + p * 8, true);
            }
            asm volatile("cp.async.commit_group;" ::: "memory");
#pragma unroll
            for (int u = 0; u < 2; ++u)
                if (u <= wm) {
#pragma unroll
                    for (int p = 0; p < 3; ++p) a[u][p] = af[(u * 3 + p) * 32];
                }
        }
#pragma unroll
        for (int k = 0; k < DC / 16 / PARTS; ++k) {
            const int ks = part * (DC / 16 / PARTS) + k;
            uint4 now[3];
#pragma unroll
            for (int p = 0; p < 3; ++p) now[p] = sm.Q[wm][(ks * 3 + p) * 32 + lane];
#pragma unroll
            for (int p = 2; p >= 0; --p) {
                uint32_t b[2][4];
#pragma unroll
                for (int jj = 0; jj < 2; ++jj) lc_ldsm4_t(&sm.S[p][ks * 16 + krow][place(jj)], b[jj]);
#pragma unroll
                for (int i = 2 - p; i >= 0; --i)
#pragma unroll
                    for (int j = 0; j < 4; ++j) {
                        if (p + i == 0) lc_mma_add(big[j], now[i], b[j >> 1][2 * (j & 1)], b[j >> 1][2 * (j & 1) + 1]);
                        else lc_mma(small[j], now[i], b[j >> 1][2 * (j & 1)], b[j >> 1][2 * (j & 1) + 1]);
                    }
            }
        }
    }
    // ---- the share of the chunk's own tokens
    asm volatile("cp.async.wait_group 0;" ::: "memory");
    bool odd = false;                                      // values that are no finite numbers (exponents all ones) must not reach earlier tokens through a zero of P
#pragma unroll
    for (int i = 0; i < LC * PIECES / DO_THREADS; ++i) {   // (what this thread asked for itself: the first piece's rows)
        const int idx = threadIdx.x + i * DO_THREADS, t = idx / PIECES, p = idx % PIECES;
        const uint4 x = *reinterpret_cast<const uint4*>(&sm.S[0][t][(p ^ (t & 7)) * 8]);
        const uint32_t w[4] = {x.x, x.y, x.z, x.w};
#pragma unroll
        for (int e = 0; e < 4; ++e) odd |= (w[e] & 0x7f80u) == 0x7f80u || (w[e] & 0x7f800000u) == 0x7f800000u;
    }
    odd = __syncthreads_or(odd);
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
#pragma unroll
            for (int p = 2; p >= 0; --p) {
                uint32_t b[2][4];
#pragma unroll
                for (int jj = 0; jj < 2; ++jj) lc_ldsm4_t(&sm.S[p][ks * 16 + krow][place(jj)], b[jj]);
#pragma unroll
                for (int i = 2 - p; i >= 0; --i)
#pragma unroll
                    for (int j = 0; j < 4; ++j) {
                        if (p + i == 0) lc_mma_add(own[j], now[i], b[j >> 1][2 * (j & 1)], b[j >> 1][2 * (j & 1) + 1]);
                        else lc_mma(small[j], now[i], b[j >> 1][2 * (j & 1)], b[j >> 1][2 * (j & 1) + 1]);
                    }
            }
        }
    } else {
        for (int half = 0; half < 2; ++half) {
            const int t = wm * 16 + frow + half * 8;
            for (int s = 0; s <= t; ++s) {
                // P_ts from its pieces: row t of tile (wm, s / 16), the register and lane that hold column s
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
                    for (int e = 0; e < 2; ++e) {
                        const int col = ((wn * 32 + j * 8) ^ ((s & 7) * 8)) + fcol + e;
                        const float x = __bfloat162float(sm.S[0][s][col]) + (__bfloat162float(sm.S[1][s][col]) + __bfloat162float(sm.S[2][s][col]));
                        own[j][half * 2 + e] = fmaf(weight, x, own[j][half * 2 + e]);
                    }
            }
        }
    }
#pragma unroll
    for (int half = 0; half < 2; ++half) {
        const int t = wm * 16 + frow + half * 8;
        if (t >= count) continue;
        float* to = out + ((size_t)(first + t) * H + h) * DCV + v0 + wn * 32 + fcol;
#pragma unroll
        for (int j = 0; j < 4; ++j)
            *reinterpret_cast<float2*>(to + j * 8) = make_float2(own[j][half * 2] + (big[j][half * 2] + small[j][half * 2]),
                                                                 own[j][half * 2 + 1] + (big[j][half * 2 + 1] + small[j][half * 2 + 1]));
    }
}

// Bytes of scratch that wllm_delta_chunks asks for: 5.6 MB a chunk of 16 heads, at most 192 MB (longer steps go in turns, the state handed on through its slot:
// the same bits) but a chunk of every request that goes in chunks.  lens: the requests' tokens, on the host.  turns: how many with that.
WLLM_API long long wllm_delta_chunks_bytes(const int* lens, int requests, int H, int* turns) {
    *turns = 0;
    if (H <= 0 || H > 65535 || requests <= 0) return 0;
    return lc_bytes(lens, requests, H * DC_SIZE, *turns);
}

// Bytes of scratch where chunks are the faster way for a step of these requests, else 0 (the walk in blocks of eight tokens).  sms: of the device; most: bytes
// that a step's chunks may take.
//
// Both ways' us, fitted to B200 measurements with 2 to 64 heads (in brackets blocks and chunks).  Blocks have eight CTAs a request and head, two an SM, each a chain:
// 0.133 a token where one has an SM to itself, 0.225 where two share it, and so many SMs for all tokens.  Chunks have a chain of their own, 2.85 a chunk, and cost
// by heads and chunks, full or not; a turn brings every request's states once more, and shorter requests are walked in front of them, not beside.
// 16 heads: 2,048 tokens [274, 194], 512 [73, 59], 384 [57, 54], 256 [42, 47], 1,021 + 680 + 340 [240, 203], 1,531 beside 24 single ones [243, 187], 16 x 512
// [864, 846], 4 x 300 [147, 134], 16 x 130 [248, 338], 512 beside 100 of 20 [433, 1,122].  4 heads: 256 [39, 39], 4 x 300 [48, 52], 16 x 130 [74, 92].  32 heads:
// 2,048 [458, 388], 512 [121, 108], 1,021 + 680 + 340 [434, 456], 4 x 300 [259, 269], 16 x 512 [1,856, 1,919].  64 heads: 2,048 [922, 792], 1,021 + 680 + 340
// [895, 943], 4 x 300 [507, 549].
WLLM_API long long wllm_delta_chunks_pay(const int* lens, int requests, int H, int sms, long long most) {
    int turns;
    const long long room = wllm_delta_chunks_bytes(lens, requests, H, &turns);
    if (room <= 0 || room > most) return 0;
    int longest = 0;
    double tokens = 0, chunks = 0, several = 0, few = 0;
    for (int r = 0; r < requests; ++r) {
        const int mine = lc_chunks(lens[r]);
        few += lens[r] > 0 && mine == 0;
        if (mine == 0) continue;
        longest = lens[r] > longest ? lens[r] : longest;
        tokens += lens[r];
        chunks += mine;
        several += 1;
    }
    const double each = 8.0 * H * several > sms ? 0.225 * ((8 * H + 2 * sms - 1) / (2 * sms)) : 0.133;
    const double alone = each * longest, all = 0.0069 * H * tokens, in_blocks = 8 + (alone > all ? alone : all);
    const double chain = 23 + (1.4 * H < 11 ? 1.4 * H : 11) + 2.85 * lc_chunks(longest), work = 20 + 0.36 * H * chunks + 0.07 * H * several * turns;
    const double in_chunks = (chain > work ? chain : work) + 12.0 * (turns - 1) + 0.015 * H * few;
    return in_chunks < in_blocks ? room : 0;
}

// The requests of LC_FROM tokens or more, from and to their state slots; shorter ones are left to wllm_delta_scan.  q, k [n, G, 128], v, out [n, H, 128],
// beta [n, H], decay [n, H] or (channel) decays less one [n, H, 128], state [slots, H, 128, 128]; lens: req_q_len on the host.
// scratch (16-byte aligned): wllm_delta_chunks_bytes, or less (more turns, the same bits) but a chunk of every request that goes in chunks.  launched: kernels.
WLLM_API int wllm_delta_chunks(const float* q, const float* k, const float* v, const float* beta, const float* decay, int channel, float* state, float* out,
                               const int* req_q_start, const int* req_q_len, const int* req_slot, const int* lens, int requests, int H, int G,
                               void* scratch, long long scratch_bytes, int* launched, cudaStream_t stream) {
    *launched = 0;
    if (requests <= 0) return WLLM_OK;
    if (H <= 0 || H > 65535 || G <= 0 || H % G != 0 || requests > 65535) return WLLM_BAD_SIZE;
    if ((((uintptr_t)q | (uintptr_t)k | (uintptr_t)v | (uintptr_t)scratch) & 15) || (((uintptr_t)decay | (uintptr_t)state | (uintptr_t)out) & 7)) return WLLM_BAD_ALIGN;
    long long all;
    const int turn = lc_turn(lens, requests, H * DC_SIZE, scratch_bytes, all);
    if (all > 65535 || all * H * DC_SIZE > scratch_bytes) return WLLM_BAD_SIZE;
    static bool raised = false;
    if (!raised) {
        cudaError_t e = cudaSuccess;
#define RAISE(K, S) if (e == cudaSuccess) e = cudaFuncSetAttribute(K, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sizeof(S))
        RAISE(delta_chunk_prepare_kernel<true>, DeltaPrepareSmem);
        RAISE(delta_chunk_prepare_kernel<false>, DeltaPrepareSmem);
        RAISE((delta_chunk_walk_kernel<true>), DeltaWalkSmem);
        RAISE((delta_chunk_walk_kernel<false>), DeltaWalkSmem);
        RAISE(delta_chunk_out_kernel, DeltaOutSmem);
#undef RAISE
        if (e != cudaSuccess) return 1000 + (int)e;
        raised = true;
    }
    int longest = 0;
    for (int r = 0; r < requests; ++r) longest = lens[r] > longest ? lens[r] : longest;
    unsigned char* room = (unsigned char*)scratch;
    for (int b0 = 0; b0 < lc_chunks(longest); b0 += turn) {
        const int count = lc_count(lens, requests, b0, turn);
#define PREPARE(C) wllm_launch(delta_chunk_prepare_kernel<C>, dim3(2, count, H), DP_THREADS, sizeof(DeltaPrepareSmem), stream, q, k, v, beta, decay, req_q_start, \
        req_q_len, req_slot, requests, H, G, b0, turn, room)
#define WALK(C) wllm_launch(delta_chunk_walk_kernel<C>, dim3(DCV / VT, H, requests), DW_THREADS, sizeof(DeltaWalkSmem), stream, state, req_q_len, req_slot, \
        H, b0, turn, room)
        int st = channel ? PREPARE(true) : PREPARE(false);
        if (st == WLLM_OK) st = channel ? WALK(true) : WALK(false);
#undef PREPARE
#undef WALK
        if (st == WLLM_OK)
            st = wllm_launch(delta_chunk_out_kernel, dim3(DCV / DO_COLS, H, count), DO_THREADS, sizeof(DeltaOutSmem), stream, out, req_q_start, req_q_len, req_slot, requests, H,
                             b0, turn, (const unsigned char*)room);
        if (st != WLLM_OK) return st;
        *launched += 3;
    }
    return WLLM_OK;
}
