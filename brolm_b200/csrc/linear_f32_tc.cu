// Float matrix product  Y[M,N] = X[M,K] * W[N,K]^T  for large weights, on tcgen05: every float is taken as the sum of three
// bfloat16 numbers, and a product of floats as the sum of six products of those (Henry, Tang and Heinecke, "Leveraging the
// bfloat16 Artificial Intelligence Datatype For Higher-Precision Computations", 2019).
//
//     x = x0 + x1 + x2:   x0 = bfloat16(x), x1 = bfloat16(x - x0), x2 = x - x0 - x1,   exact: 8 + 8 + 8 bits, and their signs
//     x w = x2 w0 + x0 w2 + x1 w1 + x1 w0 + x0 w1 + x0 w0 + ...      what is left out: less than 2^-25 |x w|
// A bfloat16 has the exponents of a float, so this holds for each number by itself, whatever stands beside it in its row (two
// halves under a power of two in common, three products, were a sixth faster for 300 tokens and lost what lay 2^15 below its
// neighbours).
// Products of two bfloat16 numbers are exact in float.
// The tensor core adds 16 of them at a time to a float accumulator and cuts off what lies below its last place, so its sums
// are kept short: the 64 k of the six products, the small ones first, make a partial sum; the partial sums of a slice of K
// are added by float additions in ascending order, and the slices likewise.  How K is cut hangs on N and K alone, so
// a row's bits depend neither on M nor on its place among the rows, nor on how X lies in memory.
//
// A block owns 128 rows of W (the M side of the instruction), up to NT tokens (the N side) and one slice of K.  The sums of
// the slices are added through the shared memory of a cluster of blocks, or by the kernel behind this one.  Roles:
//   TMA     one thread fetches W, 32 floats of every row at a time, ahead of the kernel before it where W stands;
//   SPLIT   a lane takes 64 k of a row of W apart and puts the three rows of parts into tensor memory (the A operand);
//   X       these do the same for the tokens, into shared memory (the B operand).  Many tokens are taken apart once, by a
//           kernel ahead of this one, instead of by every block; then FETCH_X, one thread, brings the parts in by TMA;
//   MMA     one lane issues 24 tcgen05.mma for 64 k (M 128, N tokens, K 16) into one of two or four accumulators;
//   ADD     these add an accumulator to the sums in their registers, and at the end store them.
// The thread that issues is what all wait for, so its stage of 64 k has one barrier to wait on, which all that its products
// need arrive at (A, the tokens, the emptied accumulator), and one commit, which frees all of it.
// For W = [gate; up] a block has 64 rows of each, and stores act(gate) * up.
//
// Bound: up to 32 tokens by the memory and by the start and end of short slices, beyond by the warps that split and add (a
// stage of 64 k with 150 tokens takes 1.6 us, of which the products are 0.9: there is room for two stages of X and of W's parts,
// so each waits for the products two back, and then for its own X and W).  us, the kernels of linear_f32.cu / here:
//     tokens                     3              16              150             300             1,000
//     4,096 x 2,304         11.3 / 12.2     25.3 / 12.3     91.4 / 28.7     150 / 48.1      446 / 155
//     2,304 x 2,048          9.6 / 8.8      18.5 / 9.3      54.0 / 20.2    87.4 / 35.6      220 / 141
//     18,432 x 2,304        37.7 / 30.6     53.3 / 30.9      358 / 67.3     592 / 128     1,847 / 400
//     2,304 x 9,216         23.8 / 20.2     44.6 / 21.1      182 / 43.5     298 / 78.0      978 / 309
// (a decode step leaves the slices of the second and the fourth to the kernel behind them: 3 tokens 7.4 and 17.6).  The error
// against 64 bits, as a share of the result's norm: 2.8 to 3.0e-7 there, 1.0 to 1.4e-7 here for normal numbers; 0.7 to 1.2e-7 and
// 0.9 to 1.2e-7 for sums of one sign, which lose half a last place at each step of the tensor core and none on average to fmas.
//
// What three parts cannot say is said by the floats themselves: the warp that has a doubtful sum of a slice makes it again
// by fmas.  Doubtful are (see doubtful())
//   a sum that is not finite: an infinity among the operands ends as a NaN here, infinity minus infinity (a NaN among them
//   is a NaN in any case, and stays);
//   a sum below 1e-16: the products of low parts end at 2^-126;
//   a sum with a number below 2^-60 (or a zero, which is not told from it) on one side and one of 2^32 or more on the other:
//   numbers below 2^-102 lose their low parts, up to 2^-125 of each; times less than 2^32 and 2^15 such terms that is below the
//   last place of a sum of 1e-16;
//   a zero, where a side has numbers below 2^-60 (or zeros) and neither has zeros alone.
#include "tcgen05.cuh"

namespace {

using namespace tc;

constexpr int BR = 128, KW = 32, KX = 64;          // rows of W; k of a slot of W, and of a stage
constexpr int W_SLOT = BR * KW * 4;
constexpr int PARTS = 3;                           // of a float
constexpr int A_PLANE = KX / 2, A_COLS = PARTS * A_PLANE;    // tensor memory: two k a column, a plane for each part

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
    static constexpr int BUFFERS = FEW && PER_SM == 1 ? 4 : 2;              // of A, the tokens and the accumulator
    static constexpr int W_SLOTS = !FEW ? 6 : PER_SM == 1 ? NT == 16 ? 10 : 8 : NT == 16 ? 5 : 4;
    static constexpr int AHEAD = !FEW ? 0 : PER_SM == 1 ? 4 : 3;           // stages of X that are on their way (FEW)
    static constexpr int X_PLANE = NT * KX * 2, X_SLOT = PARTS * X_PLANE;
    static constexpr int TMEM = PER_SM == 1 ? 512 : 256;
    static constexpr int RING = W_SLOTS * W_SLOT + BUFFERS * X_SLOT + AHEAD * X_RAW;
    static constexpr int BARS = 2 * W_SLOTS + 3 * BUFFERS + 1;
    static constexpr int SMEM = RING + 2 * BR + NT + BARS * 8 + 24;
    static_assert(BUFFERS * (NT + A_COLS) <= TMEM && TMEM * PER_SM <= 512, "accumulators and A");
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
    const uint8_t* x_flags;  // X taken apart ahead: flags [M][stages of K], and the parts under a map of their own; null: here
    float* parts;            // the slices' sums, [slice][M][N], are added by the kernel behind; null: by the cluster
    int ldx, ldw, ldy;
    int M, N, K;
    int tokens;              // of a token tile: a multiple of 16
    int slice;               // k of a slice: a multiple of 64
    int x_vec;               // X's rows lie on 16-byte boundaries
    int x_stages;            // columns of x_flags
    int w_behind;            // W may be the result of the kernel before this one
    int gated;               // W is [gate; up] of 2 N rows, a block has 64 of each, and y = act(gate) * up
    int act;
    float limit;
};

// What a row's or a token's numbers of a slice are like, for doubtful().
enum : uint32_t { SMALL = 1, BIG = 2, SOME = 4, BROKEN = 8 };
struct Extent {
    float low = INFINITY, high = 0.0f;                         // (a NaN among them makes `high` one)
    __device__ __forceinline__ void add(float v) {
        low = fminf(low, fabsf(v));
        asm("max.NaN.f32 %0, %0, %1;" : "+f"(high) : "f"(fabsf(v)));
    }
    __device__ __forceinline__ void add(const float4& v) { add(v.x), add(v.y), add(v.z), add(v.w); }
    __device__ __forceinline__ uint32_t flags() const {
        return (low < 8.67361738e-19f ? SMALL : 0) | (high >= 4.294967296e9f ? BIG : 0) | (high > 0.0f ? SOME : 0) |
               (high != high ? BROKEN : 0);
    }
    // of the eight lanes that share a row's 64 k
    __device__ __forceinline__ uint32_t flags_of_eight(int lane) const {
        const uint32_t mine = flags(), eight = 0xffu << (lane & 24);
        uint32_t all = 0;
#pragma unroll
        for (uint32_t bit = SMALL; bit <= BROKEN; bit <<= 1) all |= __ballot_sync(0xffffffffu, mine & bit) & eight ? bit : 0;
        return all;
    }
};
// The same of first parts, two at a time: one instruction a number where that of the floats takes two (few tokens, whose pace
// the warps that split set beside the memory: 3 of 18,432 x 2,304 30.5 us for 32.0).
struct PairExtent {
    uint32_t low = 0x7f807f80u, high = 0;
    __device__ __forceinline__ void add(uint32_t p) {
        asm("min.xorsign.abs.bf16x2 %0, %0, %1;" : "+r"(low) : "r"(p));
        asm("max.NaN.xorsign.abs.bf16x2 %0, %0, %1;" : "+r"(high) : "r"(p));
    }
    __device__ __forceinline__ uint32_t flags() const {
        Extent e;
        e.add(__uint_as_float(high << 16)), e.add(__uint_as_float(high & 0xffff0000u));
        e.low = fminf(fabsf(__uint_as_float(low << 16)), fabsf(__uint_as_float(low & 0xffff0000u)));
        return e.flags();
    }
};
// Two neighbours along k, taken apart.
__device__ __forceinline__ uint32_t take_part(float& a, float& b) {
    uint32_t p;
    asm("cvt.rn.bf16x2.f32 %0, %1, %2;" : "=r"(p) : "f"(b), "f"(a));
    a -= __uint_as_float(p << 16);
    b -= __uint_as_float(p & 0xffff0000u);
    return p;
}
__device__ __forceinline__ void take_apart(float a, float b, uint32_t& p0, uint32_t& p1, uint32_t& p2) {
    p0 = take_part(a, b);
    p1 = take_part(a, b);
    p2 = take_part(a, b);
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
// A sum from the floats themselves, by a whole warp: a lane's chain of fmas over every 32nd four k, then the lanes' sums in pairs.
// A token with an infinity is doubtful in all its sums (18,432 x 2,304, 3 tokens: 160 us with one such token, 256 where a thread
// makes a sum).
__device__ __noinline__ float plain_dot(const float* x, const float* w, int k, int end, int lane) {
    float y = 0.0f;
    for (k += 4 * lane; k < end; k += 128) {                  // (the ends are multiples of 4, W's rows lie on 16-byte boundaries)
        const float4 v = *reinterpret_cast<const float4*>(w + k);
        y = __fmaf_rn(x[k], v.x, y);
        y = __fmaf_rn(x[k + 1], v.y, y);
        y = __fmaf_rn(x[k + 2], v.z, y);
        y = __fmaf_rn(x[k + 3], v.w, y);
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) y += __shfl_xor_sync(0xffffffffu, y, o);
    return y;
}
// The same for every lane of a warp whose sum is doubtful, one after the other.
__device__ __forceinline__ void make_again(bool again, float& y, const float* x, const float* w, int k, int end, int lane) {
    for (uint32_t left = __ballot_sync(0xffffffffu, again); left; left &= left - 1) {
        const int whose = __ffs(left) - 1;
        const float* xs = reinterpret_cast<const float*>(__shfl_sync(0xffffffffu, reinterpret_cast<unsigned long long>(x), whose));
        const float* ws = reinterpret_cast<const float*>(__shfl_sync(0xffffffffu, reinterpret_cast<unsigned long long>(w), whose));
        const float sum = plain_dot(xs, ws, k, end, lane);
        if (lane == whose) y = sum;
    }
}
__device__ __forceinline__ bool far_apart(uint32_t row, uint32_t token) { return (((row & token >> 1) | (row >> 1 & token)) & SMALL) != 0; }
__device__ __forceinline__ bool doubtful(float y, uint32_t row, uint32_t token) {
    const float size = fabsf(y);                               // (no branches: every sum of a block is asked)
    const uint32_t either = row | token;
    const bool zero = y == 0.0f && !((row & token & SOME) && (either & SMALL));       // (a true one)
    const bool odd = !(size <= 3.402823466e38f) | ((size < 1e-16f) & !zero) | far_apart(row, token);
    return odd & !(either & BROKEN);                           // (a NaN among the numbers: the sum is one)
}
constexpr uint32_t AGAIN = 0x7fc0a6a1u;            // a NaN that no sum is: the kernel that adds the slices makes this one again

// One lane of a warp that is there as a whole, always the same one.  The compiler knows of this one that it is alone, and keeps
// what the products are given in uniform registers: 24 products of 16 tokens are issued in 0.7 us where `lane == 0` takes 1.2.
__device__ __forceinline__ bool elect_one() {
    uint32_t one;
    asm volatile("{\n.reg .pred p;\nelect.sync _|p, 0xffffffff;\nselp.u32 %0, 1, 0, p;\n}" : "=r"(one));
    return one != 0;
}

__device__ __noinline__ void mark_doubtful(float* sums, int ld, int c, int end, uint32_t row, const uint8_t* token_flags) {
    for (; c < end; ++c)
        if (doubtful(sums[(size_t)c * ld], row, token_flags[c])) sums[(size_t)c * ld] = __uint_as_float(AGAIN);
}

template <int NT, int BLOCKS>
__global__ void __launch_bounds__(Shape<NT, BLOCKS>::THREADS, BLOCKS) linear_f32_tc_kernel(const __grid_constant__ CUtensorMap map_w,
                                                                                                     const __grid_constant__ CUtensorMap map_x, Args g) {
    using S = Shape<NT, BLOCKS>;
    constexpr int NB = S::BUFFERS;
    extern __shared__ __align__(1024) uint8_t smem_raw[];
    const uint32_t w_ring = smem_u32(smem_raw), x_ring = w_ring + S::W_SLOTS * W_SLOT;
    uint8_t* row_flags = smem_raw + S::RING;               // [2][BR]: of the stages that a set of SPLIT had
    uint8_t* token_flags = row_flags + 2 * BR;             // [NT]
    uint64_t* bars = reinterpret_cast<uint64_t*>(token_flags + NT);
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + S::BARS);
    volatile int* give_up = reinterpret_cast<volatile int*>(tmem_slot + 1);
    const uint32_t w_full = smem_u32(bars), w_empty = w_full + 8 * S::W_SLOTS, ready = w_empty + 8 * S::W_SLOTS,
                   made = ready + 8 * NB, x_full = made + 8 * NB, all_made = x_full + 8 * NB;
    const int warp = __shfl_sync(0xffffffffu, threadIdx.x >> 5, 0), lane = threadIdx.x & 31;

    const int n_slices = gridDim.x, part = blockIdx.x;
    const int out_rows = g.gated ? BR / 2 : BR;                // columns of Y that the block makes
    const int m0 = blockIdx.y * g.tokens, n0 = blockIdx.z * out_rows;
    const int second = g.gated ? g.N + n0 : n0 + BR / 2;       // the row of W of lane 64
    const int tokens = min(g.tokens, g.M - m0), wide = (tokens + 15) & ~15;
    const int k_lo = part * g.slice, stages = (min(g.K, k_lo + g.slice) - k_lo + KX - 1) / KX;      // (zeros are read behind K)

    if (threadIdx.x == 0) {
        for (int s = 0; s < S::W_SLOTS; ++s) mbar_init(w_full + 8 * s, 1), mbar_init(w_empty + 8 * s, 4);
        for (int s = 0; s < NB; ++s) mbar_init(ready + 8 * s, S::READY), mbar_init(made + 8 * s, 1), mbar_init(x_full + 8 * s, 1);
        mbar_init(all_made, 1);
        give_up[0] = 0;
        give_up[1] = 0;
        give_up[2] = tc::g_stall_code;
        mbar_init_fence();
    }
    if (threadIdx.x < 2 * BR + NT) row_flags[threadIdx.x] = 0;              // (the tokens' too)
    if (warp == 2) tmem_alloc(smem_u32(tmem_slot), S::TMEM);
    fence_before_sync();
    __syncthreads();
    fence_after_sync();
    const uint32_t tmem = *tmem_slot, tmem_a = tmem + NB * NT;

    auto wait_on = [&](uint32_t bar, uint32_t parity, int code) { return mbar_wait<2>(bar, parity, give_up, &g_linear_f32_tc_error, code); };
    auto all_wait_on = [&](uint32_t bar, uint32_t parity, int code) { return __all_sync(0xffffffffu, wait_on(bar, parity, code)) != 0; };

    int index = 0;
    const Role role = S::role(warp, index);
    if (role == Role::TMA || role == Role::MMA || role == Role::FETCH_X || role == Role::NONE) {
        if constexpr (!S::FEW) fewer_registers<48>();
        if (role == Role::TMA && lane == 0) {
            if (g.w_behind) pdl_wait();
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
        if (role == Role::MMA) {
            const uint32_t id = idesc_bf16(BR, wide);
            for (int j = 0; j < stages; ++j) {
                const int s = j % NB;
                if (!all_wait_on(ready + 8 * s, (j / NB) & 1, 2)) break;
                if (g.x_flags && !all_wait_on(x_full + 8 * s, (j / NB) & 1, 3)) break;
                fence_after_sync();
                if (elect_one()) {
                    const uint32_t acc = tmem + s * NT, a = tmem_a + s * A_COLS;
                    const uint64_t b = desc_kmajor(x_ring + s * S::X_SLOT);
                    // (plane of W, plane of X), the small products first
                    constexpr int P[6][2] = {{2, 0}, {0, 2}, {1, 1}, {1, 0}, {0, 1}, {0, 0}};
#pragma unroll
                    for (int p = 0; p < 6; ++p)
#pragma unroll
                        for (int k = 0; k < 4; ++k)
                            umma_ts(acc, a + P[p][0] * A_PLANE + 8 * k, b + (uint64_t)(P[p][1] * (S::X_PLANE >> 4) + 2 * k), id, p + k > 0);
                    umma_commit(made + 8 * s);
                }
                __syncwarp();
            }
            if (__any_sync(0xffffffffu, *give_up) && elect_one()) {                     // products in flight end before their operands go
                umma_commit(all_made);
                mbar_wait(all_made, 0, give_up, &g_linear_f32_tc_error, 10, true);
            }
        }
        if (role == Role::FETCH_X && lane == 0 && g.x_flags) {
            pdl_wait();
            int j = 0;
            for (; j < stages; ++j) {
                const int s = j % NB;
                if (j >= NB && !wait_on(made + 8 * s, ((j / NB) & 1) ^ 1, 9)) break;
                mbar_expect_tx(x_full + 8 * s, PARTS * g.tokens * KX * 2);
                for (int q = 0; q < PARTS; ++q)
                    tma_load_3d(x_ring + s * S::X_SLOT + q * S::X_PLANE, &map_x, k_lo + j * KX, m0, q, x_full + 8 * s);
            }
            if (*give_up)
                for (int i = max(0, j - NB); i < j; ++i)
                    mbar_wait(x_full + 8 * (i % NB), (i / NB) & 1, give_up, &g_linear_f32_tc_error, 11, true);
        }
    } else if (role == Role::SPLIT) {
        if constexpr (!S::FEW) fewer_registers<48>();
        const int row = (warp & 3) * 32 + lane;
        PairExtent extent;
        for (int j = index >> 2; j < stages; j += 2) {         // two sets of four warps take turns
            const int s0 = 2 * j % S::W_SLOTS, s1 = (2 * j + 1) % S::W_SLOTS;
            // A wait on a slot's phase asks that the phase before it is known to be over: it was at least NB stages back.
            static_assert(S::W_SLOTS >= 2 * NB, "the slots of NB stages");
            if (j >= NB && !all_wait_on(made + 8 * (j % NB), ((j / NB) & 1) ^ 1, 6)) break;
            if (!all_wait_on(w_full + 8 * s0, (2 * j / S::W_SLOTS) & 1, 5)) break;
            if (!all_wait_on(w_full + 8 * s1, ((2 * j + 1) / S::W_SLOTS) & 1, 5)) break;
            const uint32_t src[2] = {w_ring + s0 * W_SLOT + row * 128, w_ring + s1 * W_SLOT + row * 128};
            fence_after_sync();
            const uint32_t a = tmem_a + (j % NB) * A_COLS + ((uint32_t)((warp & 3) * 32) << 16);
#pragma unroll
            for (int h = 0; h < 4; ++h) {
                uint32_t p0[8], p1[8], p2[8];
#pragma unroll
                for (int c = 0; c < 4; ++c) {
                    const float4 v = lds_float4(src[h >> 1] + ((((h & 1) * 4 + c) ^ (row & 7)) << 4));
                    take_apart(v.x, v.y, p0[2 * c], p1[2 * c], p2[2 * c]);
                    take_apart(v.z, v.w, p0[2 * c + 1], p1[2 * c + 1], p2[2 * c + 1]);
                    extent.add(p0[2 * c]), extent.add(p0[2 * c + 1]);
                }
                tmem_st8(a + 8 * h, p0);
                tmem_st8(a + A_PLANE + 8 * h, p1);
                tmem_st8(a + 2 * A_PLANE + 8 * h, p2);
            }
            if (j + 2 >= stages) row_flags[(index >> 2) * BR + row] = extent.flags();
            __syncwarp();
            if (lane == 0) mbar_arrive(w_empty + 8 * s0), mbar_arrive(w_empty + 8 * s1);       // (every lane has its floats)
            tmem_wait_st();
            fence_before_sync();
            __syncwarp();
            if (lane == 0) mbar_arrive(ready + 8 * (j % NB));
        }
    } else if (role == Role::ADD) {
        if constexpr (!S::FEW) more_registers<112>();
        const int quarter = warp & 3, first = (index >> 2) * S::COLS, row = quarter * 32 + lane;
        float sum[S::COLS];
#pragma unroll
        for (int c = 0; c < S::COLS; ++c) sum[c] = 0.0f;
        if (lane == 0)
            for (int s = 0; s < NB; ++s) mbar_arrive(ready + 8 * s);       // the accumulators are free
        int j = 0;
        for (; j < stages; ++j) {
            if (!all_wait_on(made + 8 * (j % NB), (j / NB) & 1, 8)) break;
            // (it has long been: for the flags' sake)
            if (j + 2 >= stages && !all_wait_on(ready + 8 * (j % NB), (j / NB) & 1, 8)) break;
            fence_after_sync();
            const uint32_t acc = tmem + (j % NB) * NT + first + ((uint32_t)(quarter * 32) << 16);
#pragma unroll
            for (int c = 0; c < S::COLS; c += 16) {
                if (first + c < wide) {
                    uint32_t v[16];
                    tmem_ld16(acc + c, v);
                    tmem_wait_ld();
#pragma unroll
                    for (int e = 0; e < 16; ++e) sum[c + e] += __uint_as_float(v[e]);
                }
            }
            fence_before_sync();
            __syncwarp();
            if (lane == 0) mbar_arrive(ready + 8 * (j % NB));
        }
        // Whether any of the sums can be doubtful: one of ordinary size only by numbers far apart (a zero is not of ordinary size).
        const uint32_t mine = row_flags[row] | row_flags[BR + row];
        const int w_row = row < BR / 2 ? n0 + row : second + row - BR / 2, end = min(first + S::COLS, tokens);
        uint32_t theirs = 0;
        for (int c = first + lane; c < end; c += 32) theirs |= token_flags[c];
        theirs = __reduce_or_sync(0xffffffffu, theirs);
        bool ask = far_apart(mine, theirs);
        const auto odd = [](float y) { return !(fabsf(y) <= 3.402823466e38f) | (fabsf(y) < 1e-16f); };
        const bool real = w_row < (g.gated ? 2 * g.N : g.N);
        if (j == stages && g.parts && g.y) {
            // the kernel behind this one makes the doubtful sums again
            float* dst = g.parts + ((size_t)part * g.M + m0) * g.N + n0 + row;
            if (n0 + row < g.N) {
#pragma unroll
                for (int c = 0; c < S::COLS; ++c)
                    if (first + c < tokens) dst[(size_t)(first + c) * g.N] = sum[c], ask |= odd(sum[c]);
                if (ask) mark_doubtful(dst, g.N, first, end, mine, token_flags);
            }
        } else if (j == stages) {
            // the rings are done with: all products have been made
            float* sums = reinterpret_cast<float*>(smem_raw) + row;
#pragma unroll
            for (int c = 0; c < S::COLS; ++c)
                if (first + c < tokens) sums[(first + c) * BR] = sum[c], ask |= odd(sum[c]);
            ask &= real;
            if (__any_sync(0xffffffffu, ask))
                for (int c = first; c < end; ++c) {
                    float y = sums[c * BR];
                    make_again(ask && doubtful(y, mine, token_flags[c]), y, g.x + (size_t)(m0 + c) * g.ldx, g.w + (size_t)w_row * g.ldw, k_lo,
                               min(g.K, k_lo + g.slice), lane);
                    sums[c * BR] = y;
                }
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
            if (j >= NB && !all_wait_on(made + 8 * (j % NB), ((j / NB) & 1) ^ 1, 9)) return false;
            const uint32_t slot = x_ring + (j % NB) * S::X_SLOT;
#pragma unroll
            for (int u = 0; u < PER; ++u) {
                const int token = u * (T / 8) + (xt >> 3);
                Extent extent;
#pragma unroll
                for (int e = 0; e < 8; ++e) extent.add(v[u][e]);
                const uint32_t flags = extent.flags_of_eight(lane);
                if (token < wide) {
                    uint32_t p[PARTS][4];
#pragma unroll
                    for (int e = 0; e < 4; ++e) take_apart(v[u][2 * e], v[u][2 * e + 1], p[0][e], p[1][e], p[2][e]);
                    const uint32_t at = slot + token * 128 + ((chunk ^ (token & 7)) << 4);
#pragma unroll
                    for (int q = 0; q < PARTS; ++q)
                        asm volatile("st.shared.v4.b32 [%0], {%1, %2, %3, %4};" ::"r"(at + q * S::X_PLANE), "r"(p[q][0]), "r"(p[q][1]),
                                     "r"(p[q][2]), "r"(p[q][3]) : "memory");
                    if (chunk == 0) token_flags[token] |= flags;
                }
            }
            fence_proxy_async();
            __syncwarp();
            if (lane == 0) mbar_arrive(ready + 8 * (j % NB));
            return true;
        };
        if constexpr (S::FEW) {
            // every thread brings in what it will take apart, some stages ahead
            const uint32_t raw = x_ring + NB * S::X_SLOT + xt * 32;
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
        } else if (g.x_flags) {
            // the parts come by TMA: the flags alone
            const uint8_t* src = g.x_flags + (size_t)(m0 + xt) * g.x_stages + k_lo / KX;
            const bool there = xt < tokens;
            uint32_t all = 0, next = there ? src[0] : 0;
            for (int j = 0; j < stages; ++j) {
                all |= next;
                if (there && j + 1 < stages) next = src[j + 1];
                if (j >= NB && !all_wait_on(made + 8 * (j % NB), ((j / NB) & 1) ^ 1, 9)) break;
                if (j + 1 == stages && xt < NT) token_flags[xt] = all;
                __syncwarp();
                if (lane == 0) mbar_arrive(ready + 8 * (j % NB));
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

// X taken apart ahead: eight lanes take 64 k of a token.  parts [3][M][Kp] bfloat16, Kp = 64 stages; flags [M][stages]
__global__ void __launch_bounds__(256) split_rows_kernel(Args g, uint16_t* __restrict__ parts, uint8_t* __restrict__ flags, int stages) {
    pdl_trigger();
    const size_t kp = (size_t)stages * KX;
    const long long unit = ((long long)blockIdx.x * 256 + threadIdx.x) >> 3;
    const int chunk = threadIdx.x & 7, token = (int)(unit / stages), st = (int)(unit % stages), k = st * KX + chunk * 8;
    pdl_wait();
    const bool there = token < g.M;
    const float* p = g.x + (size_t)(there ? token : 0) * g.ldx + k;
    float4 v[2];
    Extent extent;
#pragma unroll
    for (int h = 0; h < 2; ++h) {                             // (X's rows lie on 16-byte boundaries)
        const bool here = there && k + 4 * h < g.K;
        v[h] = here ? *reinterpret_cast<const float4*>(p + 4 * h) : make_float4(0.0f, 0.0f, 0.0f, 0.0f);
        extent.add(v[h]);
    }
    const uint32_t all = extent.flags_of_eight(threadIdx.x & 31);
    if (!there) return;
    uint4 q[PARTS];
    take_apart(v[0].x, v[0].y, q[0].x, q[1].x, q[2].x);
    take_apart(v[0].z, v[0].w, q[0].y, q[1].y, q[2].y);
    take_apart(v[1].x, v[1].y, q[0].z, q[1].z, q[2].z);
    take_apart(v[1].z, v[1].w, q[0].w, q[1].w, q[2].w);
    uint16_t* dst = parts + (size_t)token * kp + k;
#pragma unroll
    for (int i = 0; i < PARTS; ++i) *reinterpret_cast<uint4*>(dst + i * g.M * kp) = q[i];
    if (chunk == 0) flags[(size_t)token * stages + st] = (uint8_t)all;
}

// y = parts[0] + parts[1] + ... in order
__global__ void __launch_bounds__(256) add_slices_kernel(Args g, int slices) {
    pdl_trigger();
    pdl_wait();
    const size_t total = (size_t)g.M * g.N;
    const int lane = threadIdx.x & 31;
    for (size_t first = (size_t)blockIdx.x * 256 + threadIdx.x - lane; first < total; first += (size_t)gridDim.x * 256) {
        const bool there = first + lane < total;              // (a warp stays whole)
        const size_t idx = there ? first + lane : total - 1, token = idx / g.N, n = idx % g.N;
        float v[8];                                            // at most eight slices, all on their way at once
        bool fine = true;
#pragma unroll
        for (int s = 0; s < 8; ++s) v[s] = s < slices ? g.parts[s * total + idx] : 0.0f;
#pragma unroll
        for (int s = 0; s < 8; ++s) fine &= __float_as_uint(v[s]) != AGAIN;
        float y = v[0];
#pragma unroll
        for (int s = 1; s < 8; ++s)
            if (s < slices) y += v[s];
        if (!__all_sync(0xffffffffu, fine))
            for (int s = 0; s < slices; ++s) {
                float t = g.parts[s * total + idx];
                make_again(there && __float_as_uint(t) == AGAIN, t, g.x + token * g.ldx, g.w + n * g.ldw, s * g.slice, min(g.K, (s + 1) * g.slice), lane);
                y = s ? y + t : t;
            }
        if (there) g.y[token * g.ldy + n] = y;
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
// split: room for X taken apart ahead (more than 32 rows on 16-byte boundaries), 16-byte aligned, M * ceil(K / 64) * 385 bytes;
// null: every block does it.  w_behind: W may be the result of a kernel that is still running when this one is let in.
BROLM_API int brolm_linear_f32_tc(const void* x, int ldx, const void* w, int ldw, void* y, int ldy, int M, int N, int K,
                                  int slices, int slice, int gated, int act, float limit, int w_behind, void* parts, void* split, cudaStream_t stream) {
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
    g.w_behind = w_behind;
    g.gated = gated; g.act = act; g.limit = limit;
    g.x_vec = ldx % 4 == 0 && ((uintptr_t)x & 15) == 0;
    g.x_flags = nullptr;
    g.x_stages = (K + KX - 1) / KX;
    CUtensorMap mx = mw;
    if (split) {
        if (most <= 32 || !g.x_vec || ((uintptr_t)split & 15)) return BROLM_ERR_ALIGNMENT;
        const cuuint64_t kp = (cuuint64_t)g.x_stages * KX;
        const cuuint64_t xdims[3] = {kp, (cuuint64_t)M, PARTS}, xstrides[2] = {kp * 2, kp * M * 2};
        const cuuint32_t xbox[3] = {KX, (cuuint32_t)g.tokens, 1}, xelem[3] = {1, 1, 1};
        if (enc(&mx, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 3, split, xdims, xstrides, xbox, xelem, CU_TENSOR_MAP_INTERLEAVE_NONE,
                CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) != CUDA_SUCCESS)
            return BROLM_ERR_ALIGNMENT;
        uint8_t* flags = (uint8_t*)split + (size_t)M * kp * 2 * PARTS;
        g.x_flags = flags;
        const long long units = (long long)M * g.x_stages;
        const int st = launch_pdl(split_rows_kernel, dim3((unsigned)((units * 8 + 255) / 256)), dim3(256), 0, stream, g, (uint16_t*)split, flags, g.x_stages);
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
