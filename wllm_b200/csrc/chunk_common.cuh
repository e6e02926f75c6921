// What the recurrences that go in chunks of 64 tokens share (linear_attention_chunks.cu, delta_rule_chunks.cu): sizes, pieces, products and sums, and the places of
// the requests' chunks.
#pragma once
#include "common.cuh"

constexpr int LC = 64;                 // tokens of a chunk
constexpr int LB = 8, LBLOCKS = LC / LB;
constexpr int LC_FROM = 16;            // tokens of a request from which on it goes in chunks

__host__ __device__ inline int lc_chunks(int len) { return len < LC_FROM ? 0 : (len + LC - 1) / LC; }

__device__ __forceinline__ void lc_mma(float (&c)[4], const uint4& a, uint32_t b0, uint32_t b1) {
    asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, {%0, %1, %2, %3};"
                 : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3]) : "r"(a.x), "r"(a.y), "r"(a.z), "r"(a.w), "r"(b0), "r"(b1));
}
// A product of its own, added with a rounding: the tensor cores cut off what they add to a sum that is there, and cuts all go one way.
__device__ __forceinline__ void lc_mma_add(float (&sum)[4], const uint4& a, uint32_t b0, uint32_t b1) {
    float c[4] = {0.f, 0.f, 0.f, 0.f};
    lc_mma(c, a, b0, b1);
#pragma unroll
    for (int i = 0; i < 4; ++i) sum[i] += c[i];
}
__device__ __forceinline__ float2 lc_mul2(float2 a, float2 b) {         // two products an instruction
    unsigned long long d;
    asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(*reinterpret_cast<unsigned long long*>(&a)), "l"(*reinterpret_cast<unsigned long long*>(&b)));
    return *reinterpret_cast<float2*>(&d);
}
__device__ __forceinline__ void lc_ldsm4_t(const bf16* p, uint32_t (&r)[4]) {
    asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0, %1, %2, %3}, [%4];"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"((uint32_t)__cvta_generic_to_shared(p)));
}
__device__ __forceinline__ void lc_cp16(void* dst, const void* src, bool valid) {       // 16 bytes, or zeros
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"((uint32_t)__cvta_generic_to_shared(dst)), "l"(src), "r"(valid ? 16 : 0) : "memory");
}
// two neighbouring values as three bfloat16 pieces each
__device__ __forceinline__ void lc_split(float x, float y, uint32_t& hi, uint32_t& mid, uint32_t& lo) {
    const __nv_bfloat162 h = __floats2bfloat162_rn(x, y);
    const float2 fh = __bfloat1622float2(h);
    x -= fh.x;
    y -= fh.y;
    const __nv_bfloat162 m = __floats2bfloat162_rn(x, y);
    const float2 fm = __bfloat1622float2(m);
    const __nv_bfloat162 l = __floats2bfloat162_rn(x - fm.x, y - fm.y);
    hi = *reinterpret_cast<const uint32_t*>(&h);
    mid = *reinterpret_cast<const uint32_t*>(&m);
    lo = *reinterpret_cast<const uint32_t*>(&l);
}

// A turn takes `turn` chunks of every request from its chunk b0 on.  The nth of all of them: its request (-1 past the last) and, in `chunk`, its place in the
// request.  A warp together.
__device__ __forceinline__ int lc_find(const int* __restrict__ req_q_len, int requests, int b0, int turn, int nth, int& chunk) {
    const int lane = threadIdx.x & 31;
    for (int r0 = 0; r0 < requests; r0 += 32) {
        const int len = r0 + lane < requests ? req_q_len[r0 + lane] : 0;
        const int mine = max(0, min(lc_chunks(len) - b0, turn));
        int sum = mine;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const int other = __shfl_up_sync(0xffffffffu, sum, o);
            if (lane >= o) sum += other;
        }
        const unsigned behind = __ballot_sync(0xffffffffu, sum > nth);
        if (behind) {
            const int at = __ffs(behind) - 1;
            chunk = b0 + nth - __shfl_sync(0xffffffffu, sum - mine, at);
            return r0 + at;
        }
        nth -= __shfl_sync(0xffffffffu, sum, 31);
    }
    return -1;
}
// The turn's chunks of the requests in front of request r.  A warp together.
__device__ __forceinline__ int lc_before(const int* __restrict__ req_q_len, int r, int b0, int turn) {
    int sum = 0;
    for (int i = threadIdx.x & 31; i < r; i += 32) sum += max(0, min(lc_chunks(req_q_len[i]) - b0, turn));
    return __reduce_add_sync(0xffffffffu, sum);
}

// N values a lane over a warp's lanes, N a power of two: value i's sum ends in lane i * (32 / N) and those behind it.
template <int N>
__device__ __forceinline__ float lc_sums(float (&x)[N], int lane) {
    int half = N / 2;
#pragma unroll
    for (int off = 16; off > 0; off >>= 1) {
        const bool upper = lane & off;
        if (half >= 1) {
#pragma unroll
            for (int i = 0; i < N / 2; ++i)
                if (i < half) {
                    const float keep = upper ? x[i + half] : x[i], send = upper ? x[i] : x[i + half];
                    x[i] = keep + __shfl_xor_sync(0xffffffffu, send, off);
                }
            half >>= 1;
        } else x[0] += __shfl_xor_sync(0xffffffffu, x[0], off);
    }
    return x[0];
}

// The chunks that one turn takes of every request, `most` bytes of scratch at hand and `each` a chunk of all heads; in `chunks` how many that are of all requests.
// lens: the requests' tokens, on the host.
inline int lc_turn(const int* lens, int requests, long long each, long long most, long long& chunks) {
    int longest = 0;
    for (int r = 0; r < requests; ++r) longest = lens[r] > longest ? lens[r] : longest;
    int turn = lc_chunks(longest);
    for (;; turn = (turn + 1) / 2) {
        chunks = 0;
        for (int r = 0; r < requests; ++r) {
            const int mine = lc_chunks(lens[r]);
            chunks += mine < turn ? mine : turn;
        }
        if (turn <= 1 || (chunks * each <= most && chunks <= 65535)) return turn;
    }
}
// Bytes that a step's chunks ask for, at most LC_SCRATCH but a chunk of every request that goes in chunks, and the turns with them.
constexpr long long LC_SCRATCH = 192ll << 20;
inline long long lc_bytes(const int* lens, int requests, long long each, int& turns) {
    long long chunks;
    const int turn = lc_turn(lens, requests, each, LC_SCRATCH, chunks);
    turns = 0;
    for (int r = 0; r < requests; ++r) {
        const int mine = turn > 0 ? (lc_chunks(lens[r]) + turn - 1) / turn : 0;
        turns = mine > turns ? mine : turns;
    }
    return chunks * each;
}
// Chunks of a turn from chunk b0 on.
inline int lc_count(const int* lens, int requests, int b0, int turn) {
    int count = 0;
    for (int r = 0; r < requests; ++r) {
        const int mine = lc_chunks(lens[r]) - b0;
        count += mine < 0 ? 0 : (mine < turn ? mine : turn);
    }
    return count;
}
