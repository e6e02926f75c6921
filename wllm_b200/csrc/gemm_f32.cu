// True 32-bit matrix product  C[M, N] = A[M, K] * W[N, K]^T  on the FMA pipes.
//
// No tensor cores and no reduced-precision mode.  Every element of C is computed in one order, whatever
// kernel and tile it falls in:
//   segment   1,024 consecutive k that start at a multiple of 1,024: one chain of fused multiply-adds over
//             the segment's k in ascending order, starting from zero;
//   element   the segments' sums added one after the other in ascending order.
// A row of C therefore depends on its own row of A only, bit for bit, which makes the 32-bit path of the
// engine independent of batching.  (Zero padding past K adds fma(0, 0, acc) = acc.)
//
// Three kernels with that same arithmetic:
//   tile kernel    steps of more than 32 rows, bound by the FMA pipes: BM x 128 x 16 tiles (BM = 64 or 128), 256
//                  threads with 4 x 8 or 8 x 8 outputs each, operands transposed in shared memory and read
//                  as float4, the next tile fetched into registers while the current one is multiplied; the
//                  sums of finished segments wait in shared memory.
//   wide kernel    steps of more than 64 rows (K and the pitches in steps of 4 floats, 16-byte aligned operands) where it is faster: tiles cut by
//                  segments, a CTA each, and very many tiles; see gemm_f32_wide_kernel and wide_segments.
//   skinny kernel  steps of at most 32 rows, bound by streaming W once: a warp owns 32 rows of W and one
//                  segment (so a matrix of few rows and long K still gives every SM many warps), streams it
//                  through its own ring of cp.async stages and keeps one chain per row of A in each lane;
//                  a second kernel adds the segments' sums in order.
#include "common.cuh"

// ------------------------------------------------------------------------------------------------
// tile kernel
// ------------------------------------------------------------------------------------------------
constexpr int SEG = 1024;              // k per segment
constexpr int TBN = 128, TBK = 16;

template <int ROWS, bool VEC>
__device__ __forceinline__ void tile_fetch(const float* __restrict__ src, int ld, int rows, int K, int r0, int k0,
                                           int tid, float4 (&reg)[ROWS * 4 / 256]) {
    // ROWS rows x 16 k = ROWS * 4 groups of 4 along k
#pragma unroll
    for (int i = 0; i < ROWS * 4 / 256; ++i) {
        const int f = tid + i * 256;
        const int row = f >> 2, kq = (f & 3) * 4;
        const int gr = r0 + row, gk = k0 + kq;
        float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
        if (gr < rows) {
            const float* p = src + (size_t)gr * ld + gk;
            if (VEC) {
                if (gk < K) v = *reinterpret_cast<const float4*>(p);
            } else {
                if (gk < K) v.x = p[0];
                if (gk + 1 < K) v.y = p[1];
                if (gk + 2 < K) v.z = p[2];
                if (gk + 3 < K) v.w = p[3];
            }
        }
        reg[i] = v;
    }
}

template <int ROWS>
__device__ __forceinline__ void tile_stash(float (*dst)[ROWS + 4], int tid, const float4 (&reg)[ROWS * 4 / 256]) {
#pragma unroll
    for (int i = 0; i < ROWS * 4 / 256; ++i) {
        const int f = tid + i * 256;
        const int row = f >> 2, kq = (f & 3) * 4;
        dst[kq + 0][row] = reg[i].x;
        dst[kq + 1][row] = reg[i].y;
        dst[kq + 2][row] = reg[i].z;
        dst[kq + 3][row] = reg[i].w;
    }
}

template <int BM, bool VEC>
__global__ void __launch_bounds__(256, 2)
gemm_f32_tile_kernel(const float* __restrict__ A, int lda, const float* __restrict__ W, int ldw, float* __restrict__ C,
                     int ldc, int M, int N, int K) {
    constexpr int TM = BM / 16;            // 4 or 8 rows a thread: ty*4 + 0..3, and BM/2 + ty*4 + 0..3 when TM = 8
    __shared__ __align__(16) float As[2][TBK][BM + 4];
    __shared__ __align__(16) float Ws[2][TBK][TBN + 4];
    pdl_begin();
    const int tid = threadIdx.x;
    const int m0 = blockIdx.x * BM, n0 = blockIdx.y * TBN;   // neighbours in the grid share a tile of W
    const int ty = tid >> 4, tx = tid & 15;
    extern __shared__ float totals[];      // [TM * 8][256]: the sum of the finished segments, when K has several
    float acc[TM][8];
#pragma unroll
    for (int i = 0; i < TM; ++i)
#pragma unroll
        for (int j = 0; j < 8; ++j) acc[i][j] = 0.f;

    float4 ra[BM * 4 / 256], rw[TBN * 4 / 256];
    const int tiles = (K + TBK - 1) / TBK;
    tile_fetch<BM, VEC>(A, lda, M, K, m0, 0, tid, ra);
    tile_fetch<TBN, VEC>(W, ldw, N, K, n0, 0, tid, rw);
    tile_stash<BM>(As[0], tid, ra);
    tile_stash<TBN>(Ws[0], tid, rw);
    __syncthreads();
    for (int t = 0; t < tiles; ++t) {
        const int cur = t & 1;
        if (t + 1 < tiles) {
            tile_fetch<BM, VEC>(A, lda, M, K, m0, (t + 1) * TBK, tid, ra);
            tile_fetch<TBN, VEC>(W, ldw, N, K, n0, (t + 1) * TBK, tid, rw);
        }
#pragma unroll
        for (int k = 0; k < TBK; ++k) {
            const float4 a0 = *reinterpret_cast<const float4*>(&As[cur][k][ty * 4]);
            const float4 a1 = TM == 8 ? *reinterpret_cast<const float4*>(&As[cur][k][BM / 2 + ty * 4]) : a0;
            const float4 b0 = *reinterpret_cast<const float4*>(&Ws[cur][k][tx * 4]);
            const float4 b1 = *reinterpret_cast<const float4*>(&Ws[cur][k][TBN / 2 + tx * 4]);
            const float a[8] = {a0.x, a0.y, a0.z, a0.w, a1.x, a1.y, a1.z, a1.w};
            const float b[8] = {b0.x, b0.y, b0.z, b0.w, b1.x, b1.y, b1.z, b1.w};
#pragma unroll
            for (int i = 0; i < TM; ++i)
#pragma unroll
                for (int j = 0; j < 8; ++j) acc[i][j] = fmaf(a[i], b[j], acc[i][j]);
        }
        if (t + 1 < tiles) {
            tile_stash<BM>(As[cur ^ 1], tid, ra);
            tile_stash<TBN>(Ws[cur ^ 1], tid, rw);
            if (((t + 1) & (SEG / TBK - 1)) == 0) {     // a segment ends here and another follows
                const bool first = (t + 1) == SEG / TBK;
#pragma unroll
                for (int i = 0; i < TM; ++i)
#pragma unroll
                    for (int j = 0; j < 8; ++j) {
                        float* tot = &totals[(i * 8 + j) * 256 + tid];
                        *tot = first ? acc[i][j] : *tot + acc[i][j];
                        acc[i][j] = 0.f;
                    }
            }
        }
        __syncthreads();
    }
    if (tiles > SEG / TBK) {
#pragma unroll
        for (int i = 0; i < TM; ++i)
#pragma unroll
            for (int j = 0; j < 8; ++j) acc[i][j] = totals[(i * 8 + j) * 256 + tid] + acc[i][j];
    }
    const bool vec_out = (ldc % 4 == 0) && ((uintptr_t)C % 16 == 0);
#pragma unroll
    for (int i = 0; i < TM; ++i) {
        const int gm = m0 + (i < 4 ? ty * 4 + i : BM / 2 + ty * 4 + (i - 4));
        if (gm >= M) continue;
#pragma unroll
        for (int h = 0; h < 2; ++h) {
            const int gn = n0 + h * (TBN / 2) + tx * 4;
            float* dst = C + (size_t)gm * ldc + gn;
            if (vec_out && gn + 3 < N) {
                *reinterpret_cast<float4*>(dst) = make_float4(acc[i][h * 4], acc[i][h * 4 + 1], acc[i][h * 4 + 2], acc[i][h * 4 + 3]);
            } else {
#pragma unroll
                for (int j = 0; j < 4; ++j)
                    if (gn + j < N) dst[j] = acc[i][h * 4 + j];
            }
        }
    }
}

// ------------------------------------------------------------------------------------------------
// skinny kernel (K and the pitches in steps of 4 floats, 16-byte aligned operands)
// ------------------------------------------------------------------------------------------------
constexpr int SBN = 32, SBK = 32, SLD = SBK + 4;    // a warp's stage: 32 rows of 32 floats (128 contiguous bytes of W) + 4 of padding
constexpr int SWARPS = 4;
// Stages of a warp's ring.  Four (12 KB of W a warp ahead of its arithmetic, two CTAs an SM) is what a launch with
// tasks for every warp slot runs fastest with.  A launch of few tasks (the o projection of a 32-bit Gemma-7B step
// is 384 tasks for 148 SMs) lives on what each warp has in flight: it takes the deep ring, as deep as four warps'
// shared memory allows (28 KB a warp with up to 8 rows of A, 20 KB with 16; with 32 rows there is no room).
constexpr int SSTAGES_FULL = 4;
template <int BM> __host__ __device__ constexpr int skinny_deep_stages() { return BM <= 8 ? 8 : (BM <= 16 ? 6 : 4); }

__device__ __forceinline__ void cp_async_16(float* smem_dst, const float* src, bool valid) {
    const unsigned dst = (unsigned)__cvta_generic_to_shared(smem_dst);
    const int bytes = valid ? 16 : 0;          // 0: the 16 bytes are filled with zeros, nothing is read
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(dst), "l"(src), "r"(bytes) : "memory");
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N> __device__ __forceinline__ void cp_async_wait() { asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory"); }

// A warp's task: rows n0..n0+31 of W, segment `seg`.  Lane x keeps BM chains, out[m][n0 + x], m < BM.
// `dst` is C when K has one segment, else the partial sums [segment][M][N].
template <int BM, int SSTAGES>
__global__ void __launch_bounds__(SWARPS * 32)
gemm_f32_skinny_kernel(const float* __restrict__ A, int lda, const float* __restrict__ W, int ldw,
                       float* __restrict__ dst, int ld_dst, long long seg_stride, int M, int N, int K, int segs,
                       int tasks) {
    extern __shared__ __align__(16) float smem[];
    pdl_launch_dependents();
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int task = blockIdx.x * SWARPS + warp;
    if (task >= tasks) return;
    float (*Ws)[SBN][SLD] = reinterpret_cast<float (*)[SBN][SLD]>(smem + (size_t)warp * SSTAGES * (SBN + BM) * SLD);
    float (*As)[BM][SLD] = reinterpret_cast<float (*)[BM][SLD]>(&Ws[SSTAGES][0][0]);
    const int n0 = (task / segs) * SBN, seg = task % segs;
    const int k_begin = seg * SEG, k_end = min(K, k_begin + SEG);
    const int tiles = (k_end - k_begin + SBK - 1) / SBK;

    auto issue_w = [&](int t, int stage) {        // 32 rows x 8 chunks of 16 bytes: an instruction takes 4 rows of 128 bytes
#pragma unroll
        for (int c = lane; c < SBN * (SBK / 4); c += 32) {
            const int row = c >> 3, gk = k_begin + t * SBK + (c & 7) * 4;
            const bool valid = n0 + row < N && gk < k_end;
            cp_async_16(&Ws[stage][row][(c & 7) * 4], valid ? W + (size_t)(n0 + row) * ldw + gk : W, valid);
        }
    };
    auto issue_a = [&](int t, int stage) {
#pragma unroll
        for (int c = lane; c < BM * (SBK / 4); c += 32) {
            const int row = c >> 3, gk = k_begin + t * SBK + (c & 7) * 4;
            const bool valid = row < M && gk < k_end;
            cp_async_16(&As[stage][row][(c & 7) * 4], valid ? A + (size_t)row * lda + gk : A, valid);
        }
    };
    // the weights are no kernel's output: their first stages are on the way before this kernel waits for the
    // kernel that writes A
#pragma unroll
    for (int s = 0; s < SSTAGES - 1; ++s)
        if (s < tiles) issue_w(s, s);
    pdl_wait();
#pragma unroll
    for (int s = 0; s < SSTAGES - 1; ++s) {
        if (s < tiles) issue_a(s, s);
        cp_async_commit();
    }
    float acc[BM];
#pragma unroll
    for (int i = 0; i < BM; ++i) acc[i] = 0.f;
    for (int t = 0; t < tiles; ++t) {
        cp_async_wait<SSTAGES - 2>();
        __syncwarp();                        // tile t has landed for every lane, and every lane is done with tile t-1
        const int ahead = t + SSTAGES - 1;
        if (ahead < tiles) {
            issue_w(ahead, ahead % SSTAGES);
            issue_a(ahead, ahead % SSTAGES);
        }
        cp_async_commit();
        const int st = t % SSTAGES;
#pragma unroll
        for (int kk = 0; kk < SBK; kk += 4) {
            const float4 w4 = *reinterpret_cast<const float4*>(&Ws[st][lane][kk]);
#pragma unroll
            for (int i = 0; i < BM; ++i) {
                const float4 a4 = *reinterpret_cast<const float4*>(&As[st][i][kk]);
                acc[i] = fmaf(a4.x, w4.x, acc[i]);
                acc[i] = fmaf(a4.y, w4.y, acc[i]);
                acc[i] = fmaf(a4.z, w4.z, acc[i]);
                acc[i] = fmaf(a4.w, w4.w, acc[i]);
            }
        }
    }
    cp_async_wait<0>();
    const int gn = n0 + lane;
    if (gn < N) {
        float* out = dst + (size_t)seg * seg_stride;
#pragma unroll
        for (int i = 0; i < BM; ++i)
            if (i < M) out[(size_t)i * ld_dst + gn] = acc[i];
    }
}

// ------------------------------------------------------------------------------------------------
// wide kernel: 128 x 128 tiles, 128 threads with 8 x 16 outputs each, two CTAs an SM.
//
// The tile kernel's scheme with two changes.  Neighbouring columns are multiplied two an instruction (fma.rn.f32x2: each half is the fused
// multiply-add of its own chain, so the bits are the same): the pipes' peak is no higher for it (73.4 against 71.9 TFLOP/s in a loop), but half the
// instructions compete for the schedulers and the register ports.  And a thread has twice the columns, 24 floats read from shared memory
// for 128 products instead of 16 for 64.  A launch's last round
// finds its SMs half empty and runs faster, so the tiles need not divide evenly.  Tiles cut by segments leave their
// sums in slabs that the fold kernel adds in the same ascending order, in turns of as many segments as WIDE_SLABS floats hold; a tile that walks several
// segments keeps their running total in C.  (Rows left as they lie in memory, brought by cp.async and read four k at a time, cannot be paired: 39 TFLOP/s;
// A that way and W transposed: 51.)  Which products come here: wide_segments.  Measured in turn with the tile kernel, us: 509 x 2,048 x 16,384 cut 1,766 ->
// 766, 509 x 2,048 x 2,048 cut 261 -> 212, 4,096 x 32,768 x 2,048 whole 11,347 -> 11,084 (49.6 TFLOP/s).
// ------------------------------------------------------------------------------------------------
constexpr int WT = 128, WTHREADS = 128;

// grid (row tiles, column tiles, segments with CTAs of their own, or 1); dst: C, or slabs [segment][M][N]
__global__ void __launch_bounds__(WTHREADS, 2)
gemm_f32_wide_kernel(const float* __restrict__ A, int lda, const float* __restrict__ W, int ldw, float* __restrict__ dst, int ld_dst,
                     long long seg_stride, int M, int N, int K) {
    __shared__ __align__(16) float As[2][TBK][WT + 4];
    __shared__ __align__(16) float Ws[2][TBK][WT + 4];
    constexpr int CHUNKS = WT * TBK / 4 / WTHREADS;         // groups of four k a thread and operand: rows crow + 32 i, k ck .. ck + 3
    pdl_launch_dependents();
    const int tid = threadIdx.x, m0 = blockIdx.x * WT, n0 = blockIdx.y * WT;       // neighbours in the grid share a tile of W
    const int k_begin = gridDim.z > 1 ? blockIdx.z * SEG : 0, k_end = gridDim.z > 1 ? min(K, k_begin + SEG) : K;
    const int tiles = (k_end - k_begin + TBK - 1) / TBK;
    float* out = dst + (gridDim.z > 1 ? (size_t)blockIdx.z * seg_stride : 0);
    const int crow = tid >> 2, ck = (tid & 3) * 4;
    auto fetch = [&](const float* __restrict__ src, int ld, int rows, int r0, int t, float4 (&reg)[CHUNKS]) {
        const int gk = k_begin + t * TBK + ck;
#pragma unroll
        for (int i = 0; i < CHUNKS; ++i) {
            const int row = r0 + crow + 32 * i;
            reg[i] = row < rows && gk < k_end ? *reinterpret_cast<const float4*>(src + (size_t)row * ld + gk) : make_float4(0.f, 0.f, 0.f, 0.f);
        }
    };
    auto stash = [&](float (*to)[WT + 4], const float4 (&reg)[CHUNKS]) {
#pragma unroll
        for (int i = 0; i < CHUNKS; ++i) {
            const int row = crow + 32 * i;
            to[ck][row] = reg[i].x; to[ck + 1][row] = reg[i].y; to[ck + 2][row] = reg[i].z; to[ck + 3][row] = reg[i].w;
        }
    };
    const int tx = tid & 7, ty = tid >> 3;      // outputs: rows 4 ty .. and 64 + 4 ty .., columns 4 tx .. + 32 h (h < 4), four each
    float2 acc[8][8];
#pragma unroll
    for (int i = 0; i < 8; ++i)
#pragma unroll
        for (int j = 0; j < 8; ++j) acc[i][j] = make_float2(0.f, 0.f);
    // what the accumulators hold joins the running total (add) or becomes it
    const bool vec_out = (ld_dst & 3) == 0 && (seg_stride & 3) == 0 && ((uintptr_t)dst & 15) == 0;
    auto leave = [&](bool add) {
#pragma unroll
        for (int i = 0; i < 8; ++i) {
            const int gm = m0 + (i < 4 ? 4 * ty + i : WT / 2 + 4 * ty + i - 4);
            if (gm >= M) continue;
#pragma unroll
            for (int h = 0; h < 4; ++h) {
                const int gn = n0 + 32 * h + 4 * tx;
                float* to = out + (size_t)gm * ld_dst + gn;
                float4 v = make_float4(acc[i][2 * h].x, acc[i][2 * h].y, acc[i][2 * h + 1].x, acc[i][2 * h + 1].y);
                if (vec_out && gn + 3 < N) {
                    if (add) {
                        const float4 b = *reinterpret_cast<const float4*>(to);
                        v = make_float4(b.x + v.x, b.y + v.y, b.z + v.z, b.w + v.w);
                    }
                    *reinterpret_cast<float4*>(to) = v;
                } else {
                    if (gn < N) to[0] = add ? to[0] + v.x : v.x;
                    if (gn + 1 < N) to[1] = add ? to[1] + v.y : v.y;
                    if (gn + 2 < N) to[2] = add ? to[2] + v.z : v.z;
                    if (gn + 3 < N) to[3] = add ? to[3] + v.w : v.w;
                }
            }
        }
    };
    float4 ra[CHUNKS], rw[CHUNKS];
    fetch(W, ldw, N, n0, 0, rw);                // the weights are no kernel's output
    pdl_wait();
    fetch(A, lda, M, m0, 0, ra);
    stash(As[0], ra);
    stash(Ws[0], rw);
    __syncthreads();
    for (int t = 0; t < tiles; ++t) {
        const int cur = t & 1;
        if (t + 1 < tiles) {
            fetch(A, lda, M, m0, t + 1, ra);
            fetch(W, ldw, N, n0, t + 1, rw);
        }
#pragma unroll
        for (int k = 0; k < TBK; ++k) {
            float a[8];
            float2 b[8];
            *reinterpret_cast<float4*>(a) = *reinterpret_cast<const float4*>(&As[cur][k][4 * ty]);
            *reinterpret_cast<float4*>(a + 4) = *reinterpret_cast<const float4*>(&As[cur][k][WT / 2 + 4 * ty]);
#pragma unroll
            for (int h = 0; h < 4; ++h) *reinterpret_cast<float4*>(&b[2 * h]) = *reinterpret_cast<const float4*>(&Ws[cur][k][32 * h + 4 * tx]);
#pragma unroll
            for (int i = 0; i < 8; ++i)
#pragma unroll
                for (int j = 0; j < 8; ++j) acc[i][j] = fma2(make_float2(a[i], a[i]), b[j], acc[i][j]);
        }
        if (t + 1 < tiles) {
            stash(As[cur ^ 1], ra);
            stash(Ws[cur ^ 1], rw);
            if (((t + 1) & (SEG / TBK - 1)) == 0) {        // a segment ends here and another follows
                leave(t + 1 > SEG / TBK);
#pragma unroll
                for (int i = 0; i < 8; ++i)
#pragma unroll
                    for (int j = 0; j < 8; ++j) acc[i][j] = make_float2(0.f, 0.f);
            }
        }
        __syncthreads();
    }
    leave(tiles > SEG / TBK);
}

// C[m][n] = the segments' sums added in ascending order, behind (add) those that it holds.
__global__ void __launch_bounds__(256)
gemm_f32_fold_kernel(const float* __restrict__ parts, float* __restrict__ C, int ldc, int M, int N, int segs, bool add) {
    pdl_begin();
    const size_t idx = (size_t)blockIdx.x * 256 + threadIdx.x;
    if (idx >= (size_t)M * N) return;
    float* to = C + (idx / N) * ldc + idx % N;
    float total = add ? *to + parts[idx] : parts[idx];
    for (int s = 1; s < segs; ++s) total = total + parts[(size_t)s * M * N + idx];
    *to = total;
}

template <int BM, int STAGES>
static int launch_skinny_as(const float* A, int lda, const float* W, int ldw, float* C, int ldc, int M, int N, int K,
                            float* scratch, cudaStream_t stream) {
    const int segs = (K + SEG - 1) / SEG;
    const size_t smem = (size_t)SWARPS * STAGES * (SBN + BM) * SLD * sizeof(float);
    static bool raised = false;          // per instantiation; the attribute is a property of the function
    if (!raised) {
        const cudaError_t e = cudaFuncSetAttribute(gemm_f32_skinny_kernel<BM, STAGES>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                                   (int)smem);
        if (e != cudaSuccess) return 1000 + (int)e;
        raised = true;
    }
    const int tasks = ((N + SBN - 1) / SBN) * segs;
    float* dst = segs > 1 ? scratch : C;
    const int st = wllm_launch(gemm_f32_skinny_kernel<BM, STAGES>, dim3((tasks + SWARPS - 1) / SWARPS), SWARPS * 32, smem, stream,
                               A, lda, W, ldw, dst, segs > 1 ? N : ldc, (long long)M * N, M, N, K, segs, tasks);
    if (st != WLLM_OK || segs == 1) return st;
    return wllm_launch(gemm_f32_fold_kernel, dim3((unsigned)(((size_t)M * N + 255) / 256)), 256, 0, stream,
                       (const float*)scratch, C, ldc, M, N, segs, false);
}

template <int BM>
static int launch_skinny(const float* A, int lda, const float* W, int ldw, float* C, int ldc, int M, int N, int K,
                         float* scratch, long long scratch_floats, cudaStream_t stream) {
    const int segs = (K + SEG - 1) / SEG;
    if (segs > 1 && (scratch == nullptr || scratch_floats < (long long)segs * M * N)) return WLLM_BAD_SIZE;
    static int sms = 0;
    if (!sms) {
        int dev = 0;
        if (cudaGetDevice(&dev) != cudaSuccess || cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess)
            sms = 148;
    }
    const int tasks = ((N + SBN - 1) / SBN) * segs;
    constexpr int DEEP = skinny_deep_stages<BM>();
    if (DEEP != SSTAGES_FULL && tasks <= sms * SWARPS)      // at most one CTA's worth of warps an SM: few tasks
        return launch_skinny_as<BM, DEEP>(A, lda, W, ldw, C, ldc, M, N, K, scratch, stream);
    return launch_skinny_as<BM, SSTAGES_FULL>(A, lda, W, ldw, C, ldc, M, N, K, scratch, stream);
}

template <int BM, bool VEC>
static int launch_tile(const float* A, int lda, const float* W, int ldw, float* C, int ldc, int M, int N, int K,
                       cudaStream_t stream) {
    const size_t totals = K > SEG ? (size_t)(BM / 16) * 8 * 256 * sizeof(float) : 0;
    static bool raised = false;
    if (totals > 0 && !raised) {
        const cudaError_t e = cudaFuncSetAttribute(gemm_f32_tile_kernel<BM, VEC>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                                   (int)((size_t)(BM / 16) * 8 * 256 * sizeof(float)));
        if (e != cudaSuccess) return 1000 + (int)e;
        raised = true;
    }
    const dim3 grid((M + BM - 1) / BM, (N + TBN - 1) / TBN);
    return wllm_launch(gemm_f32_tile_kernel<BM, VEC>, grid, 256, totals, stream, A, lda, W, ldw, C, ldc, M, N, K);
}

// The most slabs' floats that a product asks for (256 MB).  A product that is cut has at most 592 tiles, so that a turn has some 4,000 CTAs and more,
// fourteen rounds of two an SM; slabs without a bound were 600 MB for 4,608 x 2,048 x 16,384.  (4,096 x 2,048 x 16,384: 5,672 us at once, 6,071 in turns of four.)
constexpr long long WIDE_SLABS = 64ll << 20;

// Segments of a turn for `floats` of scratch.
static int turn_of(int M, int N, int segs, long long floats) {
    const long long room = floats / ((long long)M * N);
    return (int)(room < segs ? (room < 65535 ? room : 65535) : (segs < 65535 ? segs : 65535));
}

// Half rounds of two CTAs an SM: a last round that leaves every SM one CTA or none takes half a round's time.
static long long half_rounds(long long ctas, int sms) {
    const long long rest = ctas % (2 * sms);
    return 2 * (ctas / (2 * sms)) + (rest == 0 ? 0 : (rest <= sms ? 1 : 2));
}

// How a product of more than 64 rows runs: its segments (more than one), each with CTAs of its own; 1: the wide kernel's tiles walk them; 0: the tile
// kernel's do.  Cut, where the tiles leave SMs idle, or where that takes fewer half rounds of a segment each by more than the slabs' five per cent.
// Whole, the tile kernel is the faster one until some fourteen tiles an SM.  us by the tile kernel, cut, whole, K 2,048: 64 tiles 261, 212, 257;
// 192 416, 335, 432; 256 414, 442, 432; 320 636, 552, 646; 384 635, 658, 666; 512 826, 767, 843; 576 828, 875, 851; 1,024 1,445 and 1,482
// whole, 1,536 2,246 and 2,227 to 2,270, 2,048 2,851 and 2,859, 3,072 4,268 and 4,222, 8,192 11,347 and 11,084.  K 508: 32 tiles 58 and 67.
static int wide_segments(int M, int N, int K) {
    static int sms = 0;
    if (!sms) {
        int dev = 0;
        if (cudaGetDevice(&dev) != cudaSuccess || cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess) sms = 148;
    }
    const int segs = (K + SEG - 1) / SEG;
    const long long tiles = (long long)((M + WT - 1) / WT) * ((N + WT - 1) / WT);
    if (segs > 1 && tiles < 4ll * sms) {
        const int turn = turn_of(M, N, segs, WIDE_SLABS);
        if (tiles <= sms && turn > 1) return segs;
        if (turn > 1 && 21 * (segs / turn * half_rounds(tiles * turn, sms) + half_rounds(tiles * (segs % turn), sms)) < 20 * segs * half_rounds(tiles, sms))
            return segs;
    }
    return tiles >= 14ll * sms ? 1 : 0;
}

// turn: segments with CTAs of their own at a time; 1: a tile's CTA walks them all
static int launch_wide(const float* A, int lda, const float* W, int ldw, float* C, int ldc, int M, int N, int K, float* scratch, int turn,
                       cudaStream_t stream) {
    const int segs = (K + SEG - 1) / SEG;
    dim3 grid((M + WT - 1) / WT, (N + WT - 1) / WT);
    if (turn < 2) return wllm_launch(gemm_f32_wide_kernel, grid, WTHREADS, 0, stream, A, lda, W, ldw, C, ldc, (long long)M * N, M, N, K);
    for (int s0 = 0; s0 < segs; s0 += turn) {
        grid.z = segs - s0 < turn ? segs - s0 : turn;
        int st = wllm_launch(gemm_f32_wide_kernel, grid, WTHREADS, 0, stream, A + (size_t)s0 * SEG, lda, W + (size_t)s0 * SEG, ldw, scratch, N,
                             (long long)M * N, M, N, K - s0 * SEG);
        if (st == WLLM_OK)
            st = wllm_launch(gemm_f32_fold_kernel, dim3((unsigned)(((size_t)M * N + 255) / 256)), 256, 0, stream, (const float*)scratch, C, ldc, M, N,
                             (int)grid.z, s0 > 0);
        if (st != WLLM_OK) return st;
    }
    return WLLM_OK;
}

static bool vec_operands(const void* A, int lda, const void* W, int ldw, int K) {
    return K % 4 == 0 && lda % 4 == 0 && ldw % 4 == 0 && (uintptr_t)A % 16 == 0 && (uintptr_t)W % 16 == 0;
}

// Floats of scratch that a product of these operands and sizes wants (0: none): partial sums of the skinny kernel, which needs them, or of the wide one,
// which does with any less.
WLLM_API long long wllm_gemm_f32_scratch_floats(const float* A, int lda, const float* W, int ldw, int M, int N, int K) {
    if (M <= 0 || N <= 0 || K <= 0 || !vec_operands(A, lda, W, ldw, K)) return 0;
    if (M <= 32) return K > SEG ? (long long)((K + SEG - 1) / SEG) * M * N : 0;
    const int segs = M > 64 ? wide_segments(M, N, K) : 0, turn = segs > 1 ? turn_of(M, N, segs, WIDE_SLABS) : 0;
    return turn > 1 ? (long long)turn * M * N : 0;
}

WLLM_API int wllm_gemm_f32(const float* A, int lda, const float* W, int ldw, float* C, int ldc, int M, int N, int K,
                           float* scratch, long long scratch_floats, cudaStream_t stream) {
    if (M <= 0 || N <= 0) return WLLM_OK;
    if (K <= 0 || lda < K || ldw < K || ldc < N || (M > 32 && (N + TBN - 1) / TBN > 65535)) return WLLM_BAD_SIZE;
    const bool vec = vec_operands(A, lda, W, ldw, K);
    if (vec && M <= 8) return launch_skinny<8>(A, lda, W, ldw, C, ldc, M, N, K, scratch, scratch_floats, stream);
    if (vec && M <= 16) return launch_skinny<16>(A, lda, W, ldw, C, ldc, M, N, K, scratch, scratch_floats, stream);
    if (vec && M <= 32) return launch_skinny<32>(A, lda, W, ldw, C, ldc, M, N, K, scratch, scratch_floats, stream);
    if (M <= 64) {
        if (vec) return launch_tile<64, true>(A, lda, W, ldw, C, ldc, M, N, K, stream);
        return launch_tile<64, false>(A, lda, W, ldw, C, ldc, M, N, K, stream);
    }
    const int segs = vec ? wide_segments(M, N, K) : 0;
    // without room for two slabs the tile kernel's tiles walk their segments: the same bits
    const int turn = segs > 1 ? turn_of(M, N, segs, scratch == nullptr ? 0 : scratch_floats) : segs;
    if (turn > 1 || segs == 1) return launch_wide(A, lda, W, ldw, C, ldc, M, N, K, scratch, turn, stream);
    if (vec) return launch_tile<128, true>(A, lda, W, ldw, C, ldc, M, N, K, stream);
    return launch_tile<128, false>(A, lda, W, ldw, C, ldc, M, N, K, stream);
}

// ------------------------------------------------------------------------------------------------
// What the FMA pipes give when nothing else is asked of them: the denominator of the products above.
// Every thread runs 8 independent chains of `iters` fused multiply-adds; out[blocks * 256] takes the sums.
// ------------------------------------------------------------------------------------------------
__global__ void __launch_bounds__(256) fma_loop_kernel(float* __restrict__ out, int iters, float a, float b) {
    float x[8];
#pragma unroll
    for (int j = 0; j < 8; ++j) x[j] = (float)(threadIdx.x + j) * 1e-3f;
    for (int i = 0; i < iters; ++i) {
#pragma unroll
        for (int j = 0; j < 8; ++j) x[j] = fmaf(x[j], a, b);
    }
    float total = 0.f;
#pragma unroll
    for (int j = 0; j < 8; ++j) total += x[j];
    out[(size_t)blockIdx.x * 256 + threadIdx.x] = total;
}

WLLM_API int wllm_fma_loop(float* out, int blocks, int iters, cudaStream_t stream) {
    if (blocks <= 0 || iters <= 0) return WLLM_BAD_SIZE;
    fma_loop_kernel<<<blocks, 256, 0, stream>>>(out, iters, 0.999f, 1e-4f);
    return wllm_launch_status();
}
