// Float matrix product  Y[M,N] = X[M,K] * W[N,K]^T  for large weights, on tcgen05: every float is taken as the sum of two
// half-precision numbers, and a product of floats as the sum of three products of those.
//
// 64 k of a row have a power of two s in common that brings the largest of them to 2^14 .. 2^15.  Then
//     s x = x0 + x1 + rest:   x0 = half(s x), x1 = half(s x - x0),   |rest| <= 2^-24 |s x|, or 2^-25 where s x is small
//     x w = (x0 w0 + (x0 w1 + x1 w0)) / (s s') + ...                 what is left out: at most 2^-24 |x w| more
// so a product is as good as one of numbers rounded to float.  Products of two half-precision numbers are exact in float.
// The tensor core adds 16 of them at a time to a float accumulator and cuts off what lies below its last place, so its sums
// are kept short: the 64 k of the three products, the small ones first, make a partial sum; the partial sums of a slice of K
// are scaled back and added by float fmas in ascending order, and the slices likewise.  How K is cut hangs on N and K alone, so
// a row's bits depend neither on M nor on its place among the rows, nor on how X lies in memory.
//
// A block owns 128 rows of W (the M side of the instruction), up to NT tokens (the N side) and one slice of K.  The sums of
// the slices are added through the shared memory of a cluster of blocks, or by the kernel behind this one.  Roles:
//   TMA     one thread fetches W, 32 floats of every row at a time, ahead of the kernel before it;
//   SPLIT   a lane takes 64 k of a row of W apart and puts the two rows of halves into tensor memory (the A operand);
//   X       these do the same for the tokens, into shared memory (the B operand).  Many tokens are taken apart once, by a
//           kernel ahead of this one, instead of by every block; then FETCH_X, one thread, brings the halves in by TMA;
//   MMA     one thread issues 12 tcgen05.mma for 64 k (M 128, N tokens, K 16) into one of two accumulators;
//   ADD     these add an accumulator to the sums in their registers, and at the end store them.
// The thread that issues is what all wait for, so its stage of 64 k has one barrier to wait on, which all that its products
// need arrive at (A, the tokens, the emptied accumulator), and one commit, which frees all of it.
// For W = [gate; up] a block has 64 rows of each, and stores act(gate) * up.
//
// Bound: up to 32 tokens by the memory and by the start and end of short slices, beyond by the warps that split and add (a
// stage of 64 k with 150 tokens takes 1.5 us, of which the products are 0.5).  us, the kernels of linear_f32.cu / here:
//     tokens                     3              16              150             300             1,000
//     4,096 x 2,304         11.2 / 14.1     25.2 / 14.4     91.7 / 28.2     150 / 48.6      445 / 159
//     2,304 x 2,048          9.8 / 10.6     18.5 / 11.2     54.5 / 20.9    87.4 / 36.1      220 / 153
//     18,432 x 2,304        38.4 / 34.6     53.0 / 34.7      357 / 58.8     591 / 110     1,845 / 350
//     2,304 x 9,216         23.0 / 29.2     44.6 / 29.0      182 / 39.6     298 / 73.4      976 / 303
// (few tokens would be as fast there; they are here because a row's bits are to be the same however many there are).  The
// error against 64 bits, as a share of the result's norm: 2.8 to 3.0e-7 there, 1.5 to 1.7e-7 here.  The same with three
// bfloat16 parts a float and six products: 1.4e-7, but 170 us for 300 tokens of 18,432 x 2,304 and 69 us for 3.
// An infinity or a NaN among the operands ends as a NaN here (infinity minus infinity, infinity times zero), and numbers
// near the smallest lose their low parts: a slice's sum that is not finite, or so small that this may show, is made again
// from the floats themselves by the thread that has it.
#include "tcgen05.cuh"

#include <cuda_fp16.h>

namespace {

using namespace tc;

constexpr int BR = 128, KW = 32, KX = 64;          // rows of W; k of a slot of W, and of a stage
constexpr int W_SLOT = BR * KW * 4;
constexpr int A_PLANE = KX / 2, A_COLS = 2 * A_PLANE;        // tensor memory: two k a column, two planes a stage
constexpr int SCALES = 4;                          // stages whose scales are kept: one that is written is not read any more

enum class Role { TMA, MMA, SPLIT, ADD, X, FETCH_X, NONE };

// Up to 32 tokens two blocks share an SM, or one has a ring of twice the slots where there are no more blocks than SMs and
// their clusters are small enough to find room (18,432 x 2,304 with 3 tokens, 144 blocks: 40.6 us with four slots, 34.4 with
// ten; the memory's latency asks for more than two stages on their way).  For more tokens one block takes the SM, with 28 warps
// that share its registers by need.
template <int NT, int BLOCKS>
struct Shape {
    static constexpr bool FEW = NT <= 32;
    static constexpr int PER_SM = BLOCKS;
    static_assert(FEW || BLOCKS == 1, "many tokens take the SM");
    static constexpr int WARPS = FEW ? 16 : 28, THREADS = 32 * WARPS;
    static constexpr int GROUPS = FEW ? 1 : 2, COLS = NT / GROUPS;          // warps of a quarter that add, each its share of the tokens
    static constexpr int X_WARPS = FEW ? 2 : 8;
    static constexpr int READY = 4 + X_WARPS + 4 * GROUPS;                  // arrivals that a stage waits for
    static constexpr int X_RAW = NT * KX * 4;                               // bytes of a stage of X as it is
    static constexpr int W_SLOTS = !FEW ? 8 : PER_SM == 1 ? 10 : NT == 16 ? 5 : 4;
    static constexpr int AHEAD = !FEW ? 0 : PER_SM == 1 ? 4 : 3;           // stages of X that are on their way (FEW)
    static constexpr int X_PLANE = NT * KX * 2, X_SLOT = 2 * X_PLANE;
    static constexpr int TMEM = FEW ? 256 : 512;
    static constexpr int RING = W_SLOTS * W_SLOT + 2 * X_SLOT + AHEAD * X_RAW;
    static constexpr int BARS = 2 * W_SLOTS + 7;
    static constexpr int SMEM = RING + SCALES * (BR + NT) * 4 + BARS * 8 + 24;
    static_assert(2 * NT + 2 * A_COLS <= TMEM && TMEM * PER_SM <= 512, "accumulators and A");
    static_assert((SMEM + 1024) * PER_SM <= 228 * 1024, "the blocks of an SM");
    static_assert(NT * BR * 4 <= RING, "the sums of a slice lie where the rings were");

    static __device__ __forceinline__ Role role(int warp, int& index) {     // index: within the role
        if (warp < 2) return warp == 0 ? Role::TMA : Role::MMA;
        if (warp < 4) return index = warp - 2, FEW ? Role::X : warp == 3 ? Role::FETCH_X : Role::NONE;
        if (warp < 12) return index = warp - 4, Role::SPLIT;
        if (warp < 12 + 4 * GROUPS) return index = warp - 12, Role::ADD;
        return index = warp - 20, Role::X;
    }
};
// Registers of a thread: 896 threads are launched with 72 each; what 640 of them give back lets 256 hold 80 sums.
template <int N> __device__ __forceinline__ void fewer_registers() { asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(N)); }
template <int N> __device__ __forceinline__ void more_registers() { asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;" ::"n"(N)); }

__device__ int g_linear_f32_tc_error;

struct Args {
    const float* x;
    const float* w;
    float* y;
    const float* x_scale;    // X taken apart ahead: [M][stages of K] scales, and the halves under a map of their own; null: here
    float* parts;            // the slices' sums, [slice][M][N], are added by the kernel behind; null: by the cluster
    int ldx, ldw, ldy;
    int M, N, K;
    int tokens;              // of a token tile: a multiple of 16
    int slice;               // k of a slice: a multiple of 64
    int x_vec;               // X's rows lie on 16-byte boundaries
    int x_stages;            // columns of x_scale
    int gated;               // W is [gate; up] of 2 N rows, a block has 64 of each, and y = act(gate) * up
    int act;
    float limit;
};

// The power of two that brings `most` to 2^14 .. 2^15, and its inverse; both are normal numbers for every `most`.
__device__ __forceinline__ void scales_of(float most, float& up, float& down) {
    const uint32_t e = max((__float_as_uint(most) >> 23) & 255u, 16u);
    up = __uint_as_float((268u - e) << 23);
    down = __uint_as_float((e - 14u) << 23);
}
// Two neighbours along k, taken apart.
__device__ __forceinline__ void take_apart(float a, float b, float scale, uint32_t& p0, uint32_t& p1) {
    a *= scale;
    b *= scale;
    const __half2 h = __floats2half2_rn(a, b);
    const float2 f = __half22float2(h);
    const __half2 l = __floats2half2_rn(a - f.x, b - f.y);
    p0 = *reinterpret_cast<const uint32_t*>(&h);
    p1 = *reinterpret_cast<const uint32_t*>(&l);
}
__device__ __forceinline__ float largest(float most, const float4& v) {
    return fmaxf(fmaxf(fmaxf(most, fabsf(v.x)), fmaxf(fabsf(v.y), fabsf(v.z))), fabsf(v.w));
}
__device__ __forceinline__ float4 lds_float4(uint32_t at) {
    float4 v;
    asm volatile("ld.shared.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "r"(at) : "memory");
    return v;
}
__device__ __forceinline__ void tmem_st8(uint32_t taddr, const uint32_t (&v)[8]) {
    asm volatile("tcgen05.st.sync.aligned.32x32b.x8.b32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8};" ::"r"(taddr), "r"(v[0]), "r"(v[1]),
                 "r"(v[2]), "r"(v[3]), "r"(v[4]), "r"(v[5]), "r"(v[6]), "r"(v[7]) : "memory");
}
// Instruction descriptor of kind::f16: half x half -> f32, both K-major.
__device__ __forceinline__ uint32_t idesc_half(int m, int n) {
    return (1u << 4) | ((uint32_t)(n >> 3) << 17) | ((uint32_t)(m >> 4) << 24);
}

__device__ __noinline__ float plain_dot(const float* x, const float* w, int k, int end) {
    float y = 0.0f;
    for (; k < end; k += 512) {
        float even = 0.0f, odd = 0.0f;
        const int stop = min(end, k + 512);
        for (int i = k; i < stop; i += 2) {                   // the ends are multiples of 4
            even = __fmaf_rn(x[i], w[i], even);
            odd = __fmaf_rn(x[i + 1], w[i + 1], odd);
        }
        y += even + odd;
    }
    return y;
}
__device__ __forceinline__ bool doubtful(float y) {
    const float size = fabsf(y);
    return !(size <= 3.402823466e38f) || (size < 1e-25f && y != 0.0f);
}

template <int NT, int BLOCKS>
__global__ void __launch_bounds__(Shape<NT, BLOCKS>::THREADS, BLOCKS) linear_f32_tc_kernel(const __grid_constant__ CUtensorMap map_w,
                                                                                                     const __grid_constant__ CUtensorMap map_x, Args g) {
    using S = Shape<NT, BLOCKS>;
    extern __shared__ __align__(1024) uint8_t smem_raw[];
    const uint32_t w_ring = smem_u32(smem_raw), x_ring = w_ring + S::W_SLOTS * W_SLOT;
    float* row_scale = reinterpret_cast<float*>(smem_raw + S::RING);        // [SCALES][BR]: what a partial sum is multiplied by
    float* token_scale = row_scale + SCALES * BR;                           // [SCALES][NT]
    uint64_t* bars = reinterpret_cast<uint64_t*>(token_scale + SCALES * NT);
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + S::BARS);
    volatile int* give_up = reinterpret_cast<volatile int*>(tmem_slot + 1);
    const uint32_t w_full = smem_u32(bars), w_empty = w_full + 8 * S::W_SLOTS, ready = w_empty + 8 * S::W_SLOTS, made = ready + 16,
                   all_made = made + 16, x_full = all_made + 8;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;

    const int n_slices = gridDim.x, part = blockIdx.x;
    const int out_rows = g.gated ? BR / 2 : BR;                // columns of Y that the block makes
    const int m0 = blockIdx.y * g.tokens, n0 = blockIdx.z * out_rows;
    const int second = g.gated ? g.N + n0 : n0 + BR / 2;       // the row of W of lane 64
    const int tokens = min(g.tokens, g.M - m0), wide = (tokens + 15) & ~15;
    const int k_lo = part * g.slice, stages = (min(g.K, k_lo + g.slice) - k_lo + KX - 1) / KX;      // (zeros are read behind K)

    if (threadIdx.x == 0) {
        for (int s = 0; s < S::W_SLOTS; ++s) mbar_init(w_full + 8 * s, 1), mbar_init(w_empty + 8 * s, 4);
        for (int s = 0; s < 2; ++s) mbar_init(ready + 8 * s, S::READY), mbar_init(made + 8 * s, 1), mbar_init(x_full + 8 * s, 1);
        mbar_init(all_made, 1);
        give_up[0] = 0;
        give_up[1] = 0;
        give_up[2] = tc::g_stall_code;
        mbar_init_fence();
    }
    if (warp == 2) tmem_alloc(smem_u32(tmem_slot), S::TMEM);
    fence_before_sync();
    __syncthreads();
    fence_after_sync();
    const uint32_t tmem = *tmem_slot, tmem_a = tmem + 2 * NT;

    auto wait_on = [&](uint32_t bar, uint32_t parity, int code) { return mbar_wait(bar, parity, give_up, &g_linear_f32_tc_error, code); };
    auto all_wait_on = [&](uint32_t bar, uint32_t parity, int code) { return __all_sync(0xffffffffu, wait_on(bar, parity, code)) != 0; };

    int index = 0;
    const Role role = S::role(warp, index);
    if (role == Role::TMA || role == Role::MMA || role == Role::FETCH_X || role == Role::NONE) {
        if constexpr (!S::FEW) fewer_registers<48>();
        if (role == Role::TMA && lane == 0) {
            int i = 0;
            for (; i < 2 * stages; ++i) {
                const int s = i % S::W_SLOTS;
                if (i >= S::W_SLOTS && !wait_on(w_empty + 8 * s, ((i / S::W_SLOTS) & 1) ^ 1, 1)) break;
                mbar_expect_tx(w_full + 8 * s, W_SLOT);
                tma_load_2d(w_ring + s * W_SLOT, &map_w, k_lo + i * KW, n0, w_full + 8 * s);
                tma_load_2d(w_ring + s * W_SLOT + W_SLOT / 2, &map_w, k_lo + i * KW, second, w_full + 8 * s);
            }
            pdl_trigger();                                     // W is on its way: the next kernel may move in
            if (*give_up)
                for (int j = max(0, i - S::W_SLOTS); j < i; ++j)
                    mbar_wait(w_full + 8 * (j % S::W_SLOTS), (j / S::W_SLOTS) & 1, give_up, &g_linear_f32_tc_error, 7, true);
        }
        if (role == Role::MMA && lane == 0) {
            const uint32_t id = idesc_half(BR, wide);
            for (int j = 0; j < stages; ++j) {
                const int s = j & 1;
                if (!wait_on(ready + 8 * s, (j >> 1) & 1, 2)) break;
                if (g.x_scale && !wait_on(x_full + 8 * s, (j >> 1) & 1, 3)) break;
                fence_after_sync();
                const uint32_t acc = tmem + s * NT, a = tmem_a + s * A_COLS;
                const uint64_t b = desc_kmajor(x_ring + s * S::X_SLOT);
                // (plane of W, plane of X), the small products first
                constexpr int P[3][2] = {{1, 0}, {0, 1}, {0, 0}};
#pragma unroll
                for (int p = 0; p < 3; ++p)
#pragma unroll
                    for (int k = 0; k < 4; ++k)
                        umma_ts(acc, a + P[p][0] * A_PLANE + 8 * k, b + (uint64_t)(P[p][1] * (S::X_PLANE >> 4) + 2 * k), id, p + k > 0);
                umma_commit(made + 8 * s);
            }
            if (*give_up) {                                    // products in flight end before their operands go
                umma_commit(all_made);
                mbar_wait(all_made, 0, give_up, &g_linear_f32_tc_error, 10, true);
            }
        }
        if (role == Role::FETCH_X && lane == 0 && g.x_scale) {
            pdl_wait();
            int j = 0;
            for (; j < stages; ++j) {
                const int s = j & 1;
                if (j >= 2 && !wait_on(made + 8 * s, ((j >> 1) & 1) ^ 1, 9)) break;
                mbar_expect_tx(x_full + 8 * s, 2 * g.tokens * KX * 2);
                for (int q = 0; q < 2; ++q)
                    tma_load_3d(x_ring + s * S::X_SLOT + q * S::X_PLANE, &map_x, k_lo + j * KX, m0, q, x_full + 8 * s);
            }
            if (*give_up)
                for (int i = max(0, j - 2); i < j; ++i)
                    mbar_wait(x_full + 8 * (i & 1), (i >> 1) & 1, give_up, &g_linear_f32_tc_error, 11, true);
        }
    } else if (role == Role::SPLIT) {
        if constexpr (!S::FEW) fewer_registers<48>();
        const int row = (warp & 3) * 32 + lane;
        for (int j = index >> 2; j < stages; j += 2) {         // two sets of four warps take turns
            const int s0 = 2 * j % S::W_SLOTS, s1 = (2 * j + 1) % S::W_SLOTS;
            // A wait on a slot's phase asks that the phase before it is known to be over.  That was a stage at least four back
            // where there are eight slots, which this set has seen; where there are fewer, the stage two back has to be over first.
            constexpr bool AT_ONCE = S::W_SLOTS >= 8;
            static_assert(S::W_SLOTS >= 4, "two stages");
            if (!AT_ONCE && j >= 2 && !all_wait_on(made + 8 * (j & 1), ((j >> 1) & 1) ^ 1, 6)) break;
            if (!all_wait_on(w_full + 8 * s0, (2 * j / S::W_SLOTS) & 1, 5)) break;
            if (!all_wait_on(w_full + 8 * s1, ((2 * j + 1) / S::W_SLOTS) & 1, 5)) break;
            const uint32_t src[2] = {w_ring + s0 * W_SLOT + row * 128, w_ring + s1 * W_SLOT + row * 128};
            float most = 0.0f, up, down;
#pragma unroll
            for (int c = 0; c < 16; ++c) most = largest(most, lds_float4(src[c >> 3] + (((c & 7) ^ (row & 7)) << 4)));
            scales_of(most, up, down);
            if (AT_ONCE && j >= 2 && !all_wait_on(made + 8 * (j & 1), ((j >> 1) & 1) ^ 1, 6)) break;
            fence_after_sync();
            row_scale[(j % SCALES) * BR + row] = down;
            const uint32_t a = tmem_a + (j & 1) * A_COLS + ((uint32_t)((warp & 3) * 32) << 16);
#pragma unroll
            for (int h = 0; h < 4; ++h) {
                uint32_t p0[8], p1[8];
#pragma unroll
                for (int c = 0; c < 4; ++c) {
                    const float4 v = lds_float4(src[h >> 1] + ((((h & 1) * 4 + c) ^ (row & 7)) << 4));
                    take_apart(v.x, v.y, up, p0[2 * c], p1[2 * c]);
                    take_apart(v.z, v.w, up, p0[2 * c + 1], p1[2 * c + 1]);
                }
                tmem_st8(a + 8 * h, p0);
                tmem_st8(a + A_PLANE + 8 * h, p1);
            }
            __syncwarp();
            if (lane == 0) mbar_arrive(w_empty + 8 * s0), mbar_arrive(w_empty + 8 * s1);       // (every lane has its floats)
            tmem_wait_st();
            fence_before_sync();
            __syncwarp();
            if (lane == 0) mbar_arrive(ready + 8 * (j & 1));
        }
    } else if (role == Role::ADD) {
        if constexpr (!S::FEW) more_registers<112>();
        const int quarter = warp & 3, first = (index >> 2) * S::COLS, row = quarter * 32 + lane;
        float sum[S::COLS];
#pragma unroll
        for (int c = 0; c < S::COLS; ++c) sum[c] = 0.0f;
        if (lane == 0) mbar_arrive(ready), mbar_arrive(ready + 8);          // both accumulators are free
        int j = 0;
        for (; j < stages; ++j) {
            if (!all_wait_on(made + 8 * (j & 1), (j >> 1) & 1, 8)) break;
            if (!all_wait_on(ready + 8 * (j & 1), (j >> 1) & 1, 8)) break;          // (it has long been: for the scales' sake)
            fence_after_sync();
            const uint32_t acc = tmem + (j & 1) * NT + first + ((uint32_t)(quarter * 32) << 16);
            const float mine = row_scale[(j % SCALES) * BR + row];
            const float4* theirs = reinterpret_cast<const float4*>(token_scale + (j % SCALES) * NT + first);
#pragma unroll
            for (int c = 0; c < S::COLS; c += 16) {
                if (first + c < wide) {
                    uint32_t v[16];
                    tmem_ld16(acc + c, v);
                    tmem_wait_ld();
#pragma unroll
                    for (int e = 0; e < 16; e += 4) {
                        const float4 t = theirs[(c + e) / 4];
                        sum[c + e] = __fmaf_rn(__uint_as_float(v[e]) * mine, t.x, sum[c + e]);
                        sum[c + e + 1] = __fmaf_rn(__uint_as_float(v[e + 1]) * mine, t.y, sum[c + e + 1]);
                        sum[c + e + 2] = __fmaf_rn(__uint_as_float(v[e + 2]) * mine, t.z, sum[c + e + 2]);
                        sum[c + e + 3] = __fmaf_rn(__uint_as_float(v[e + 3]) * mine, t.w, sum[c + e + 3]);
                    }
                }
            }
            fence_before_sync();
            __syncwarp();
            if (lane == 0) mbar_arrive(ready + 8 * (j & 1));
        }
        if (j == stages && g.parts && g.y) {
            // the kernel behind this one looks for doubtful sums itself
            float* dst = g.parts + ((size_t)part * g.M + m0 + first) * g.N + n0 + row;
            if (n0 + row < g.N) {
#pragma unroll
                for (int c = 0; c < S::COLS; ++c)
                    if (first + c < tokens) dst[(size_t)c * g.N] = sum[c];
            }
        } else if (j == stages) {
            // the rings are done with: all products have been made
            float* sums = reinterpret_cast<float*>(smem_raw) + row;
            bool fine = true;
#pragma unroll
            for (int c = 0; c < S::COLS; ++c)
                if (first + c < tokens) {
                    sums[(first + c) * BR] = sum[c];
                    fine &= !doubtful(sum[c]);
                }
            const int w_row = row < BR / 2 ? n0 + row : second + row - BR / 2;
            if (!fine && w_row < (g.gated ? 2 * g.N : g.N))
                for (int c = first; c < min(first + S::COLS, tokens); ++c)
                    if (doubtful(sums[c * BR]))
                        sums[c * BR] = plain_dot(g.x + (size_t)(m0 + c) * g.ldx, g.w + (size_t)w_row * g.ldw, k_lo, min(g.K, k_lo + g.slice));
        }
    } else {
        // X: eight k of a token at a time, the eight lanes of a token side by side
        if constexpr (!S::FEW) fewer_registers<64>();
        constexpr int T = S::X_WARPS * 32, PER = (NT * 8 + T - 1) / T;
        const int xt = index * 32 + lane, chunk = xt & 7;
        pdl_wait();                                            // X is the kernel before this one's result
        auto load = [&](int j, float (&v)[PER][8]) {
            const int k = k_lo + j * KX + chunk * 8;
#pragma unroll
            for (int u = 0; u < PER; ++u) {
                const int token = u * (T / 8) + (xt >> 3);
#pragma unroll
                for (int e = 0; e < 8; ++e) v[u][e] = 0.0f;
                if (token < tokens) {
                    const float* p = g.x + (size_t)(m0 + token) * g.ldx + k;
                    if (g.x_vec) {
#pragma unroll
                        for (int e = 0; e < 8; e += 4)
                            if (k + e < g.K) {
                                const float4 f = *reinterpret_cast<const float4*>(p + e);
                                v[u][e] = f.x, v[u][e + 1] = f.y, v[u][e + 2] = f.z, v[u][e + 3] = f.w;
                            }
                    } else {
#pragma unroll
                        for (int e = 0; e < 8; ++e)
                            if (k + e < g.K) v[u][e] = p[e];
                    }
                }
            }
        };
        auto put = [&](int j, const float (&v)[PER][8]) {      // false: gave up
            if (j >= 2 && !all_wait_on(made + 8 * (j & 1), ((j >> 1) & 1) ^ 1, 9)) return false;
            const uint32_t slot = x_ring + (j & 1) * S::X_SLOT;
#pragma unroll
            for (int u = 0; u < PER; ++u) {
                const int token = u * (T / 8) + (xt >> 3);
                float most = 0.0f, up, down;
#pragma unroll
                for (int e = 0; e < 8; ++e) most = fmaxf(most, fabsf(v[u][e]));
#pragma unroll
                for (int o = 4; o > 0; o >>= 1) most = fmaxf(most, __shfl_xor_sync(0xffffffffu, most, o));
                scales_of(most, up, down);
                if (token < wide) {
                    uint32_t p[2][4];
#pragma unroll
                    for (int e = 0; e < 4; ++e) take_apart(v[u][2 * e], v[u][2 * e + 1], up, p[0][e], p[1][e]);
                    const uint32_t at = slot + token * 128 + ((chunk ^ (token & 7)) << 4);
#pragma unroll
                    for (int q = 0; q < 2; ++q)
                        asm volatile("st.shared.v4.b32 [%0], {%1, %2, %3, %4};" ::"r"(at + q * S::X_PLANE), "r"(p[q][0]), "r"(p[q][1]),
                                     "r"(p[q][2]), "r"(p[q][3]) : "memory");
                    if (chunk == 0) token_scale[(j % SCALES) * NT + token] = down;
                }
            }
            fence_proxy_async();
            __syncwarp();
            if (lane == 0) mbar_arrive(ready + 8 * (j & 1));
            return true;
        };
        if constexpr (S::FEW) {
            // every thread brings in what it will take apart, some stages ahead
            const uint32_t raw = x_ring + 2 * S::X_SLOT + xt * 32;
            auto fetch = [&](int j) {
                const int k = k_lo + j * KX + chunk * 8;
#pragma unroll
                for (int u = 0; u < PER; ++u) {
                    const int token = u * (T / 8) + (xt >> 3);
                    const float* p = g.x + (size_t)(m0 + token) * g.ldx + k;
                    const uint32_t dst = raw + (j % S::AHEAD) * S::X_RAW + u * T * 32;
                    const bool there = token < tokens && j < stages;
                    if (g.x_vec) {
#pragma unroll
                        for (int e = 0; e < 8; e += 4) copy16(dst + e * 4, there && k + e < g.K ? p + e : g.x, there && k + e < g.K);
                    } else {
#pragma unroll
                        for (int e = 0; e < 8; ++e) {
                            const bool ok = there && k + e < g.K;
                            asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;\n" ::"r"(dst + e * 4), "l"(ok ? p + e : g.x), "r"(ok ? 4 : 0) : "memory");
                        }
                    }
                }
                copy_commit();
            };
#pragma unroll
            for (int j = 0; j < S::AHEAD - 1; ++j) fetch(j);
            for (int j = 0; j < stages; ++j) {
                fetch(j + S::AHEAD - 1);
                copy_wait<S::AHEAD - 1>();
                float v[PER][8];
#pragma unroll
                for (int u = 0; u < PER; ++u)
#pragma unroll
                    for (int e = 0; e < 8; e += 4) {
                        const float4 f = lds_float4(raw + (j % S::AHEAD) * S::X_RAW + u * T * 32 + e * 4);
                        v[u][e] = f.x, v[u][e + 1] = f.y, v[u][e + 2] = f.z, v[u][e + 3] = f.w;
                    }
                if (!put(j, v)) break;
            }
            copy_wait<0>();
        } else if (g.x_scale) {
            // the halves come by TMA: the scales alone
            const float* src = g.x_scale + (size_t)(m0 + xt) * g.x_stages + k_lo / KX;
            const bool there = xt < tokens;
            float next = there ? src[0] : 1.0f;
            for (int j = 0; j < stages; ++j) {
                const float now = next;
                if (there && j + 1 < stages) next = src[j + 1];
                if (j >= 2 && !all_wait_on(made + 8 * (j & 1), ((j >> 1) & 1) ^ 1, 9)) break;
                if (xt < NT) token_scale[(j % SCALES) * NT + xt] = now;
                __syncwarp();
                if (lane == 0) mbar_arrive(ready + 8 * (j & 1));
            }
        } else {
            float v[PER][8];
            for (int j = 0; j < stages; ++j) {
                load(j, v);
                if (!put(j, v)) break;
            }
        }
    }
    __syncwarp();
    const bool cluster = n_slices > 1 && !g.parts;
    auto all_here = [&] {
        if (cluster) asm volatile("barrier.cluster.arrive.release;\nbarrier.cluster.wait.acquire;" ::: "memory");
        else __syncthreads();
    };
    all_here();
    if (!(g.parts && g.y) && !give_up[0]) {
        // the blocks of the cluster deal the tokens among them; a thread makes four neighbours of a row of Y, or of this slice's sums
        const int quads = out_rows / 4, ranks = g.parts ? 1 : n_slices, rank = g.parts ? 0 : part;
        float* dst_rows = g.parts ? g.parts + (size_t)part * g.M * g.N : g.y;
        const int ld = g.parts ? g.N : g.ldy;
        const bool wide_store = ld % 4 == 0 && ((uintptr_t)dst_rows & 15) == 0;
        auto total = [&](int t, int row, float (&y)[4]) {
            const uint32_t at = w_ring + (t * BR + row) * 4;
            for (int r = 0; r < ranks; ++r) {
                float4 v;
                if (ranks > 1) {
                    uint32_t far;
                    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(far) : "r"(at), "r"(r));
                    asm volatile("ld.shared::cluster.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "r"(far) : "memory");
                } else {
                    v = lds_float4(at);
                }
                y[0] = r ? y[0] + v.x : v.x;
                y[1] = r ? y[1] + v.y : v.y;
                y[2] = r ? y[2] + v.z : v.z;
                y[3] = r ? y[3] + v.w : v.w;
            }
        };
        const int mine = (tokens - rank + ranks - 1) / ranks;  // tokens rank, rank + ranks, ...
        for (int idx = threadIdx.x; idx < mine * quads; idx += S::THREADS) {
            const int t = rank + ranks * (idx / quads), c = idx % quads * 4, left = g.N - n0 - c;
            if (left <= 0) continue;
            float y[4], u[4];
            total(t, c, y);
            if (g.gated) {
                total(t, c + BR / 2, u);
#pragma unroll
                for (int e = 0; e < 4; ++e) y[e] = gate_pair(y[e], u[e], g.act, g.limit);
            }
            float* dst = dst_rows + (size_t)(m0 + t) * ld + n0 + c;
            if (wide_store && left >= 4) {
                *reinterpret_cast<float4*>(dst) = make_float4(y[0], y[1], y[2], y[3]);
            } else {
                for (int e = 0; e < 4; ++e)
                    if (e < left) dst[e] = y[e];
            }
        }
    }
    if (cluster) all_here();                                   // no block's shared memory goes while another reads it
    pdl_trigger();
    fence_before_sync();
    __syncthreads();
    if (warp == 2) tmem_dealloc(tmem, S::TMEM);
}

// X taken apart ahead: eight lanes take 64 k of a token.  halves [2][M][Kp], Kp = 64 stages; scale [M][stages]
__global__ void __launch_bounds__(256) split_rows_kernel(Args g, __half* __restrict__ halves, float* __restrict__ scale, int stages) {
    pdl_trigger();
    const size_t kp = (size_t)stages * KX;
    const long long unit = ((long long)blockIdx.x * 256 + threadIdx.x) >> 3;
    const int chunk = threadIdx.x & 7, token = (int)(unit / stages), st = (int)(unit % stages), k = st * KX + chunk * 8;
    pdl_wait();
    const bool there = token < g.M;
    const float* p = g.x + (size_t)(there ? token : 0) * g.ldx + k;
    float v[8], most = 0.0f, up, down;
#pragma unroll
    for (int e = 0; e < 8; e += 4) {                          // (X's rows lie on 16-byte boundaries)
        const float4 f = there && k + e < g.K ? *reinterpret_cast<const float4*>(p + e) : make_float4(0.0f, 0.0f, 0.0f, 0.0f);
        v[e] = f.x, v[e + 1] = f.y, v[e + 2] = f.z, v[e + 3] = f.w;
    }
#pragma unroll
    for (int e = 0; e < 8; ++e) most = fmaxf(most, fabsf(v[e]));
#pragma unroll
    for (int o = 4; o > 0; o >>= 1) most = fmaxf(most, __shfl_xor_sync(0xffffffffu, most, o));
    scales_of(most, up, down);
    if (!there) return;
    uint4 q[2];
    uint32_t* q0 = &q[0].x;
    uint32_t* q1 = &q[1].x;
#pragma unroll
    for (int e = 0; e < 4; ++e) take_apart(v[2 * e], v[2 * e + 1], up, q0[e], q1[e]);
    __half* dst = halves + (size_t)token * kp + k;
    *reinterpret_cast<uint4*>(dst) = q[0];
    *reinterpret_cast<uint4*>(dst + (size_t)g.M * kp) = q[1];
    if (chunk == 0) scale[(size_t)token * stages + st] = down;
}

// y = parts[0] + parts[1] + ... in order
__global__ void __launch_bounds__(256) add_slices_kernel(Args g, int slices) {
    pdl_trigger();
    pdl_wait();
    const size_t total = (size_t)g.M * g.N;
    for (size_t idx = (size_t)blockIdx.x * 256 + threadIdx.x; idx < total; idx += (size_t)gridDim.x * 256) {
        const size_t token = idx / g.N, n = idx % g.N;
        float v[8];                                            // at most eight slices, all on their way at once
        bool fine = true;
#pragma unroll
        for (int s = 0; s < 8; ++s) v[s] = s < slices ? g.parts[s * total + idx] : 0.0f;
#pragma unroll
        for (int s = 0; s < 8; ++s) fine &= !doubtful(v[s]);
        if (!fine)
#pragma unroll
            for (int s = 0; s < 8; ++s)
                if (doubtful(v[s])) v[s] = plain_dot(g.x + token * g.ldx, g.w + n * g.ldw, s * g.slice, min(g.K, (s + 1) * g.slice));
        float y = v[0];
#pragma unroll
        for (int s = 1; s < 8; ++s)
            if (s < slices) y += v[s];
        g.y[token * g.ldy + n] = y;
    }
}

template <int NT, int BLOCKS>
int launch(const CUtensorMap& mw, const CUtensorMap& mx, const Args& g, dim3 grid, cudaStream_t stream) {
    using S = Shape<NT, BLOCKS>;
    static OncePerDevice allowed;
    if (const int e = allow_shared_memory(linear_f32_tc_kernel<NT, BLOCKS>, S::SMEM, allowed)) return e;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = grid;
    cfg.blockDim = dim3(S::THREADS);
    cfg.dynamicSmemBytes = S::SMEM;
    cfg.stream = stream;
    cudaLaunchAttribute attr[2];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = pdl_enabled() ? 1 : 0;
    attr[1].id = cudaLaunchAttributeClusterDimension;
    attr[1].val.clusterDim.x = grid.x;
    attr[1].val.clusterDim.y = attr[1].val.clusterDim.z = 1;
    cfg.attrs = attr;
    cfg.numAttrs = grid.x > 1 && !g.parts ? 2 : 1;
    const int st = (int)cudaLaunchKernelEx(&cfg, linear_f32_tc_kernel<NT, BLOCKS>, mw, mx, g);
    if (st || !g.parts || !g.y) return st;
    const size_t blocks = ((size_t)g.M * g.N + 255) / 256;
    return launch_pdl(add_slices_kernel, dim3((unsigned)(blocks < 2368 ? blocks : 2368)), dim3(256), 0, stream, g, (int)grid.x);
}

}  // namespace

// Y = X W^T over `slices` slices of K of `slice` k each (a multiple of 64, none empty; at most 8 slices); gated: Y =
// act(X Wg^T) * (X Wu^T) for W = [Wg; Wu] of 2 N rows.  W's rows lie on 16-byte boundaries, K is a multiple of 4; X's rows
// may lie anywhere.  parts: room for slices * M * N floats, with which a second kernel adds the slices (y null: the caller's does); null: clusters do.
// halves: room for X taken apart ahead (more than 32 rows on 16-byte boundaries), 16-byte aligned, M * ceil(K / 64) * 260 bytes;
// null: every block does it.
BROLM_API int brolm_linear_f32_tc(const void* x, int ldx, const void* w, int ldw, void* y, int ldy, int M, int N, int K,
                                  int slices, int slice, int gated, int act, float limit, void* parts, void* halves, cudaStream_t stream) {
    if (M <= 0 || N <= 0) return BROLM_OK;
    if (K <= 0 || K % 4 || ldw % 4 || ((uintptr_t)w & 15)) return BROLM_ERR_ALIGNMENT;
    if (slices < 1 || slices > 8 || slice < 64 || slice % 64 || (long long)(slices - 1) * slice >= K || (long long)slices * slice < K) return BROLM_ERR_BAD_SIZE;
    if (gated && (act < 0 || act > 2)) return BROLM_ERR_BAD_SIZE;
    if (parts && (gated || slices < 2)) return BROLM_ERR_BAD_SIZE;
    const int most = M <= 16 ? 16 : M <= 32 ? 32 : 160;
    const int tiles = (M + most - 1) / most;
    const int out_rows = gated ? BR / 2 : BR;
    const long long row_tiles = (N + out_rows - 1) / out_rows;
    if (tiles > 65535 || row_tiles > 65535) return BROLM_ERR_TOO_LARGE;
    CUtensorMap mw;
    EncodeTiled enc = encoder();
    if (!enc) return BROLM_ERR_BAD_SIZE;
    const cuuint64_t dims[2] = {(cuuint64_t)K, (cuuint64_t)N * (gated ? 2 : 1)}, strides[1] = {(cuuint64_t)ldw * 4};
    const cuuint32_t box[2] = {KW, BR / 2}, elem[2] = {1, 1};
    if (enc(&mw, CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 2, const_cast<void*>(w), dims, strides, box, elem, CU_TENSOR_MAP_INTERLEAVE_NONE,
            CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) != CUDA_SUCCESS)
        return BROLM_ERR_ALIGNMENT;
    Args g;
    g.x = (const float*)x; g.w = (const float*)w; g.y = (float*)y; g.parts = (float*)parts;
    g.ldx = ldx; g.ldw = ldw; g.ldy = ldy;
    g.M = M; g.N = N; g.K = K;
    g.tokens = ((M + tiles - 1) / tiles + 15) / 16 * 16;
    g.slice = slice;
    g.gated = gated; g.act = act; g.limit = limit;
    g.x_vec = ldx % 4 == 0 && ((uintptr_t)x & 15) == 0;
    g.x_scale = nullptr;
    g.x_stages = (K + KX - 1) / KX;
    CUtensorMap mx = mw;
    if (halves) {
        if (most <= 32 || !g.x_vec || ((uintptr_t)halves & 15)) return BROLM_ERR_ALIGNMENT;
        const cuuint64_t kp = (cuuint64_t)g.x_stages * KX;
        const cuuint64_t xdims[3] = {kp, (cuuint64_t)M, 2}, xstrides[2] = {kp * 2, kp * M * 2};
        const cuuint32_t xbox[3] = {KX, (cuuint32_t)g.tokens, 1}, xelem[3] = {1, 1, 1};
        if (enc(&mx, CU_TENSOR_MAP_DATA_TYPE_FLOAT16, 3, halves, xdims, xstrides, xbox, xelem, CU_TENSOR_MAP_INTERLEAVE_NONE,
                CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) != CUDA_SUCCESS)
            return BROLM_ERR_ALIGNMENT;
        float* scale = reinterpret_cast<float*>((uint8_t*)halves + (size_t)M * kp * 4);
        g.x_scale = scale;
        const long long units = (long long)M * g.x_stages;
        const int st = launch_pdl(split_rows_kernel, dim3((unsigned)((units * 8 + 255) / 256)), dim3(256), 0, stream, g, (__half*)halves, scale, g.x_stages);
        if (st) return st;
    }
    const dim3 grid(slices, (M + g.tokens - 1) / g.tokens, (unsigned)row_tiles);
    const bool alone = (grid.x <= 4 || parts) && (long long)grid.x * grid.y * grid.z <= device_sm_count();
    if (most == 16) return alone ? launch<16, 1>(mw, mx, g, grid, stream) : launch<16, 2>(mw, mx, g, grid, stream);
    if (most == 32) return alone ? launch<32, 1>(mw, mx, g, grid, stream) : launch<32, 2>(mw, mx, g, grid, stream);
    return launch<160, 1>(mw, mx, g, grid, stream);
}

BROLM_API int brolm_linear_f32_tc_status(int reset) {
    int v = 0;
    if (cudaMemcpyFromSymbol(&v, g_linear_f32_tc_error, sizeof(int)) != cudaSuccess) return -1;
    if (reset && v) {
        const int zero = 0;
        cudaMemcpyToSymbol(g_linear_f32_tc_error, &zero, sizeof(int));
    }
    return v;
}

BROLM_WAIT_CONTROL(linear_f32_tc)
