// True 32-bit matrix product  Y[M,N] = X[M,K] * W[N,K]^T  on CUDA cores
// (wlejon/brolm include/brolm/detail/compute.h:49-86, the float branch).
//
// For weights of up to a million numbers, those off 16-byte boundaries, and a K below 256 (linear_f32_tc.cu takes the others).
// The largest of them, 1,024 x 1,024, take 6.8 / 8.6 / 12.1 / 17.2 us for 1 / 3 / 8 / 16 rows and 22 / 23 / 36 / 62 for 33 / 150 /
// 300 / 1,000; figures below at more weights than that were measured on these kernels all the same, to see what bounds them.
// No tensor cores and no reduced-precision mode: every product and sum is an IEEE float fma.  One order of sums holds for all kernels of this file,
// whatever M is, wherever the row stands in the batch and however the work is
// cut:
//
//     y = C_0 + C_1 + C_2 + ...                    in ascending order,
//     C_s = (sum over the even k) + (sum over the odd k)   of k in [512 s, 512 s + 512),
//
// each of the two sums being a chain of fmas over ascending k from zero.  So
// a row gives the same bits alone, in a prompt or in a batch, and there are
// independent sums to give to different warps and blocks (one chain over
// K = 9216 leaves a decode step nothing to run in parallel, and a chain that
// long also rounds more).  Even and odd k are the two halves of a packed
// fma.rn.f32x2, whose operands are neighbours in a row of X and of W: both
// are read from shared memory as they lie in memory.
//
// Three kernels:
//   rows_kernel   M <= 16: the product is a stream of W.  Bound by memory.
//   tiles_kernel  M > 16: tiles of 32 or 64 rows by 128 columns.  Bound by the fma pipes.
//   any_kernel    operands whose rows do not lie on 16-byte boundaries, and K of a few elements.
// Which one, and how K is cut: linear_f32_plan in kernels/__init__.py.
#include "common.cuh"

namespace {

constexpr int SEG = 512;        // k of one C_s

__device__ __forceinline__ float halves_sum(uint64_t v) {
    float lo, hi;
    asm("mov.b64 {%0, %1}, %2;\n" : "=f"(lo), "=f"(hi) : "l"(v));
    return lo + hi;
}
__device__ __forceinline__ Pair2 lds4(uint32_t addr) {
    Pair2 v;
    asm volatile("ld.shared.v2.b64 {%0, %1}, [%2];\n" : "=l"(v.x), "=l"(v.y) : "r"(addr));
    return v;
}

// ---------------------------------------------------------------------------
// M <= MP <= 16.  A block owns RG * R rows of W over the whole of K, a lane R rows of one segment at a time: the
// 32 / RG segments a warp works on lie side by side in its lanes, and its warps take them in turns.  Every warp has a
// queue of its own in shared memory (cp.async, no barrier): slices of 32 k of its rows, 128 bytes each from memory,
// rows 144 bytes apart so that eight lanes' 16-byte reads fall into different banks; x's part of the slice comes along
// and is read by all lanes of a segment at once.  The sums of all segments meet in shared memory and are added in
// ascending order.
// A warp's 16-byte read takes shared memory four cycles even where all lanes read one address, so with one row a lane
// the reads of x set the pace from M = 8 on (256,000 x 2,304: 680 us at M = 8 and 987 us at M = 16, against 370 us at
// M = 1, which is 6.4 TB/s): a lane then takes two rows for every x it reads (533 and 836 us).
constexpr int PITCH = 144;                       // bytes of a pair's 32 k, with padding

template <int R> __host__ __device__ constexpr int slots() { return R == 1 ? 5 : 4; }
template <int MP, int RG> __host__ __device__ constexpr int x_bytes() { return (32 / RG) * (MP * 128 + 16); }
template <int MP, int RG, int R> __host__ __device__ constexpr int slot_bytes() { return 32 * R * PITCH + x_bytes<MP, RG>(); }

template <int MP, int RG, int R>
__global__ void __launch_bounds__(256) rows_kernel(const float* __restrict__ X, int ldx, const float* __restrict__ W, int ldw,
                                                   float* __restrict__ Y, int ldy, int M, int N, int K) {
    constexpr int SUBS = 32 / RG, SLOTS = slots<R>(), ROWS = RG * R;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, n_warps = blockDim.x >> 5;
    const int n_seg = (K + SEG - 1) / SEG, units = (n_seg + SUBS - 1) / SUBS;
    const int n0 = blockIdx.x * ROWS;
    extern __shared__ __align__(16) uint8_t raw[];
    const uint32_t queue = (uint32_t)__cvta_generic_to_shared(raw) + warp * (SLOTS * slot_bytes<MP, RG, R>());
    float* sums = reinterpret_cast<float*>(raw + (size_t)n_warps * (SLOTS * slot_bytes<MP, RG, R>()));   // [seg][MP][ROWS]

    constexpr int SLICES = SEG / 32;
    const int my_units = warp < units ? (units - warp + n_warps - 1) / n_warps : 0;
    // the last unit ends with K
    const int tail = min(SLICES, (K - (units - 1) * SUBS * SEG + 31) / 32);
    const int total = my_units * SLICES - (my_units && (units - 1) % n_warps == warp ? SLICES - tail : 0);
    // slice i of this warp: unit warp + n_warps * (i / SLICES), k from 32 * (i % SLICES) of each of its segments
    auto slice_k = [&](int i, int sub) {
        return ((warp + n_warps * (i / SLICES)) * SUBS + sub) * SEG + (i % SLICES) * 32;
    };
    auto fetch_w = [&](int i) {
        if (i >= total) return;
        const uint32_t dst = queue + (i % SLOTS) * slot_bytes<MP, RG, R>();
#pragma unroll
        for (int j = 0; j < 8 * R; ++j) {                           // [row of the lane][segment][row]
            const int p = j * 4 + (lane >> 3), row = n0 + p % RG + (p / 32) * RG, k = slice_k(i, p % 32 / RG) + (lane & 7) * 4;
            const bool ok = row < N && k < K;                       // K is a multiple of 4
            copy16(dst + p * PITCH + (lane & 7) * 16, W + (ok ? (size_t)row * ldw + k : 0), ok);
        }
    };
    auto fetch_x = [&](int i) {
        if (i >= total) return;
        const uint32_t dst = queue + (i % SLOTS) * slot_bytes<MP, RG, R>() + 32 * R * PITCH;
#pragma unroll
        for (int j = 0; j < (SUBS * MP * 8 + 31) / 32; ++j) {
            const int idx = j * 32 + lane, m = (idx >> 3) % MP, sub = idx / (MP * 8);
            if (idx < SUBS * MP * 8) {
                const int k = slice_k(i, sub) + (idx & 7) * 4;
                const bool ok = m < M && k < K;
                copy16(dst + sub * (MP * 128 + 16) + m * 128 + (idx & 7) * 16, X + (ok ? (size_t)m * ldx + k : 0), ok);
            }
        }
    };

    // W depends on nothing that ran before; X is the kernel before this one's result
#pragma unroll
    for (int i = 0; i < SLOTS - 1; ++i) fetch_w(i);
    pdl_wait();
#pragma unroll
    for (int i = 0; i < SLOTS - 1; ++i) {
        fetch_x(i);
        copy_commit();
    }
    uint64_t acc[R][MP];
#pragma unroll
    for (int r = 0; r < R; ++r)
#pragma unroll
        for (int m = 0; m < MP; ++m) acc[r][m] = 0;
    const int sub = lane / RG;
    for (int i = 0; i < total; ++i) {
        copy_wait<SLOTS - 2>();
        __syncwarp();                            // the slice has landed for all lanes, and slice i - 1 has been read by all
        fetch_w(i + SLOTS - 1);
        fetch_x(i + SLOTS - 1);
        copy_commit();
        const uint32_t slot = queue + (i % SLOTS) * slot_bytes<MP, RG, R>();
        const uint32_t wp = slot + lane * PITCH, xp = slot + 32 * R * PITCH + sub * (MP * 128 + 16);
#pragma unroll
        for (int c = 0; c < 8; ++c) {
            Pair2 w[R];
#pragma unroll
            for (int r = 0; r < R; ++r) w[r] = lds4(wp + r * 32 * PITCH + c * 16);
#pragma unroll
            for (int m = 0; m < MP; ++m) {
                const Pair2 x = lds4(xp + m * 128 + c * 16);
#pragma unroll
                for (int r = 0; r < R; ++r) {
                    fma2(acc[r][m], w[r].x, x.x);
                    fma2(acc[r][m], w[r].y, x.y);
                }
            }
        }
        if (i % SLICES == SLICES - 1 || i == total - 1) {
            const int seg = (warp + n_warps * (i / SLICES)) * SUBS + sub;
#pragma unroll
            for (int r = 0; r < R; ++r)
#pragma unroll
                for (int m = 0; m < MP; ++m) {
                    if (seg < n_seg) sums[(seg * MP + m) * ROWS + r * RG + lane % RG] = halves_sum(acc[r][m]);
                    acc[r][m] = 0;
                }
        }
    }
    copy_wait<0>();
    pdl_trigger();
    __syncthreads();
    for (int idx = threadIdx.x; idx < MP * ROWS; idx += blockDim.x) {
        const int m = idx / ROWS, n = n0 + idx % ROWS;
        if (m >= M || n >= N) continue;
        float y = sums[idx];
        for (int s = 1; s < n_seg; ++s) y += sums[s * MP * ROWS + idx];
        Y[(size_t)m * ldy + n] = y;
    }
}

template <int MP, int RG, int R>
int launch_rows(const float* x, int ldx, const float* w, int ldw, float* y, int ldy, int M, int N, int K, cudaStream_t stream) {
    const int n_seg = (K + SEG - 1) / SEG, units = (n_seg + 32 / RG - 1) / (32 / RG);
    constexpr int ROWS = RG * R;
    const size_t sums = (size_t)n_seg * MP * ROWS * sizeof(float);
    constexpr size_t queue = (size_t)slots<R>() * slot_bytes<MP, RG, R>();
    // two blocks an SM where that leaves at least two warps; of the counts that fit, the largest that leaves no warp
    // of the last round of units without one
    int fit = sums < 112 * 1024 ? (int)((112 * 1024 - sums) / queue) : 0;
    if (fit < 2) fit = sums < 224 * 1024 ? (int)((224 * 1024 - sums) / queue) : 0;
    if (fit < 1) return BROLM_ERR_TOO_LARGE;
    fit = fit < 8 ? fit : 8;
    int warps = fit < units ? fit : units;
    warps = (units + (units + warps - 1) / warps - 1) / ((units + warps - 1) / warps);
    const size_t smem = warps * queue + sums;
    static OncePerDevice allowed;
    if (const int e = allow_shared_memory(rows_kernel<MP, RG, R>, 227 * 1024, allowed)) return e;
    return launch_pdl(rows_kernel<MP, RG, R>, dim3((N + ROWS - 1) / ROWS), dim3(warps * 32), smem, stream, x, ldx, w, ldw, y, ldy, M, N, K);
}

// Rows of W per block: as many as leave two blocks for every SM, since the memory wants all SMs at work (a block of
// fewer rows has the segments beside one another in its lanes, and reads x once per segment instead of once).  Two rows
// a lane for more than four tokens, if that leaves lanes for about four warps an SM: 2,304 x 9,216 with 8 tokens 38.8 ->
// 28.6 us, 18,432 x 2,304 with 16 tokens 82 -> 63 us, but 2,304 x 2,048 with 16 tokens 18.8 -> 23.4 us, and with 3
// tokens 256,000 x 2,304 takes 464 us with one and 494 us with two.
template <int MP, int R>
int dispatch_groups(const float* x, int ldx, const float* w, int ldw, float* y, int ldy, int M, int N, int K, cudaStream_t stream) {
    const int want = 2 * device_sm_count() - 40;
    if (N / (32 * R) >= want) return launch_rows<MP, 32, R>(x, ldx, w, ldw, y, ldy, M, N, K, stream);
    if (N / (16 * R) >= want) return launch_rows<MP, 16, R>(x, ldx, w, ldw, y, ldy, M, N, K, stream);
    return launch_rows<MP, 8, R>(x, ldx, w, ldw, y, ldy, M, N, K, stream);
}
template <int MP>
int dispatch_rows(const float* x, int ldx, const float* w, int ldw, float* y, int ldy, int M, int N, int K, cudaStream_t stream) {
    if constexpr (MP > 4)
        if ((long long)N * ((K + SEG - 1) / SEG) >= 2 * 4 * 32 * (long long)device_sm_count())
            return dispatch_groups<MP, 2>(x, ldx, w, ldw, y, ldy, M, N, K, stream);
    return dispatch_groups<MP, 1>(x, ldx, w, ldw, y, ldy, M, N, K, stream);
}

// ---------------------------------------------------------------------------
// Tiles of BM x 128, BM / 8 x 8 outputs a thread (rows 8 apart, columns 16 apart: the eight lanes of a 16-byte read take
// eight neighbouring rows of W, 144 bytes apart).  Shared memory hands out 128 bytes a cycle, so a thread's outputs have
// to be as many as its registers hold: 8 x 8 reads 64 bytes for 64 fmas, which is what the fma pipes take in that time
// (18,432 x 2,304: 43 TFLOP/s at M = 300 and 47 at M = 1024, 0.63 of the 74.5 that the fma pipes do at 1,965 MHz; 38 and 42 with
// 8 x 4 and twice the warps; 24 and 25 before, with 4 x 4 and scalar fmas).  Two stages of 32 k; the sum over
// the finished segments waits in shared memory, [output][thread].  The segments of K may be dealt to blocks along
// z: the first of them adds its own in slice 0 of Y, the others leave every segment's sums in a slice of its own.
constexpr int BN = 128, STAGES = 2;

template <int BM>
__global__ void __launch_bounds__(128, 2) tiles_kernel(const float* __restrict__ X, int ldx, const float* __restrict__ W, int ldw,
                                                       float* __restrict__ Y, int ldy, int M, int N, int K, int seg_per_block,
                                                       long long part_stride) {
    constexpr int TM = BM / 8, TN = BN / 16;
    constexpr int STAGE = (BM + BN) * PITCH;
    extern __shared__ __align__(16) uint8_t raw[];
    const uint32_t base = (uint32_t)__cvta_generic_to_shared(raw);
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int tn = (lane & 7) + 8 * (warp & 1), tm = (lane >> 3) + 4 * (warp >> 1);
    const int m0 = blockIdx.x * BM, n0 = blockIdx.y * BN;
    const int seg0 = blockIdx.z * seg_per_block;
    const int k_end = min(K, (seg0 + seg_per_block) * SEG);
    const int steps = (k_end - seg0 * SEG + 31) / 32;
    // the slice of this block's first segment; -1: the segments are added here (into slice 0, where there are several)
    const int slice = seg0 > 0 ? seg0 - seg_per_block + 1 : -1;

    auto fetch = [&](int i) {
        if (i < steps) {
            const int k = seg0 * SEG + i * 32 + (tid & 7) * 4;
            const uint32_t dst = base + (i % STAGES) * STAGE + (tid >> 3) * PITCH + (tid & 7) * 16;
#pragma unroll
            for (int j = 0; j < (BM + BN) / 16; ++j) {
                const int row = j * 16 + (tid >> 3);
                const float* p = row < BM ? X : W;
                const long long r = row < BM ? m0 + row : n0 + row - BM;
                const bool ok = k < K && r < (row < BM ? M : N);
                copy16(dst + j * 16 * PITCH, p + (ok ? r * (row < BM ? ldx : ldw) + k : 0), ok);
            }
        }
        copy_commit();
    };

    uint64_t acc[TM][TN];
    float* tot = reinterpret_cast<float*>(raw + STAGES * STAGE) + tid;
#pragma unroll
    for (int i = 0; i < TM; ++i)
#pragma unroll
        for (int j = 0; j < TN; ++j) acc[i][j] = 0;
    pdl_wait();
#pragma unroll
    for (int i = 0; i < STAGES - 1; ++i) fetch(i);
    for (int i = 0; i < steps; ++i) {
        copy_wait<STAGES - 2>();
        __syncthreads();                         // stage i has landed for all threads, and stage i - 1 has been read
        fetch(i + STAGES - 1);
        const uint32_t xs = base + (i % STAGES) * STAGE + tm * PITCH, ws = base + (i % STAGES) * STAGE + (BM + tn) * PITCH;
#pragma unroll
        for (int c = 0; c < 8; ++c) {
            Pair2 w[TN];
#pragma unroll
            for (int j = 0; j < TN; ++j) w[j] = lds4(ws + j * 16 * PITCH + c * 16);
#pragma unroll
            for (int t = 0; t < TM; ++t) {
                const Pair2 x = lds4(xs + t * 8 * PITCH + c * 16);
#pragma unroll
                for (int j = 0; j < TN; ++j) fma2(acc[t][j], w[j].x, x.x);
#pragma unroll
                for (int j = 0; j < TN; ++j) fma2(acc[t][j], w[j].y, x.y);
            }
        }
        if (i % (SEG / 32) == SEG / 32 - 1 || i == steps - 1) {
            const int seg = i / (SEG / 32);
            if (slice >= 0) {
                float* dst = Y + (slice + seg) * part_stride;
#pragma unroll
                for (int t = 0; t < TM; ++t)
#pragma unroll
                    for (int j = 0; j < TN; ++j) {
                        const int m = m0 + tm + 8 * t, n = n0 + tn + 16 * j;
                        if (m < M && n < N) dst[(size_t)m * ldy + n] = halves_sum(acc[t][j]);
                        acc[t][j] = 0;
                    }
            } else {
#pragma unroll
                for (int t = 0; t < TM; ++t)
#pragma unroll
                    for (int j = 0; j < TN; ++j) {
                        const float c = halves_sum(acc[t][j]);
                        tot[(t * TN + j) * 128] = seg == 0 ? c : tot[(t * TN + j) * 128] + c;
                        acc[t][j] = 0;
                    }
            }
        }
    }
    pdl_trigger();
    if (slice >= 0) return;
#pragma unroll
    for (int t = 0; t < TM; ++t)
#pragma unroll
        for (int j = 0; j < TN; ++j) {
            const int m = m0 + tm + 8 * t, n = n0 + tn + 16 * j;
            if (m < M && n < N) Y[(size_t)m * ldy + n] = tot[(t * TN + j) * 128];
        }
}

// y = parts[0] + parts[1] + ... in order; parts [n_parts][M][N]
__global__ void __launch_bounds__(256) sum_parts_kernel(const float* __restrict__ parts, int n_parts, float* __restrict__ Y,
                                                        int ldy, int M, int N) {
    pdl_trigger();
    pdl_wait();
    const size_t stride = (size_t)M * N;
    for (size_t idx = (size_t)blockIdx.x * 256 + threadIdx.x; idx < stride; idx += (size_t)gridDim.x * 256) {
        float y = parts[idx];
#pragma unroll 4
        for (int s = 1; s < n_parts; ++s) y += parts[s * stride + idx];
        Y[idx / N * ldy + idx % N] = y;
    }
}

template <int BM>
int launch_tiles(const float* x, int ldx, const float* w, int ldw, float* y, int ldy, int M, int N, int K, float* parts,
                 int seg_per_block, cudaStream_t stream) {
    constexpr int smem = STAGES * (BM + BN) * PITCH + BM * BN * (int)sizeof(float);
    static OncePerDevice allowed;
    if (const int e = allow_shared_memory(tiles_kernel<BM>, smem, allowed)) return e;
    const int n_seg = (K + SEG - 1) / SEG;
    const dim3 grid((M + BM - 1) / BM, (N + BN - 1) / BN, parts ? (n_seg + seg_per_block - 1) / seg_per_block : 1);
    // Blocks that are let in early, beside what is left of the kernel before them, lie two on one SM and none on another,
    // which costs where they do not fill all places (300 x 2,304 x 256, 90 blocks: 22.1 us and 19.7 in order; 17 x 2,304 x 2,304
    // in 90, behind the sums of the product before: 30.9 and 22.5); a handful finds SMs of its own, and starts sooner
    // (17 x 1,000 x 516, 8 blocks: 21.2 and 22.5).
    const long long blocks_all = (long long)grid.x * grid.y * grid.z;
    const bool in_order = blocks_all < 2LL * device_sm_count() && (parts || blocks_all > device_sm_count() / 4);
    auto run = [&](float* dst, int ld, int per, long long stride) {
        return in_order ? launch_in_order(tiles_kernel<BM>, grid, dim3(128), smem, stream, x, ldx, w, ldw, dst, ld, M, N, K, per, stride)
                        : launch_pdl(tiles_kernel<BM>, grid, dim3(128), smem, stream, x, ldx, w, ldw, dst, ld, M, N, K, per, stride);
    };
    if (!parts) return run(y, ldy, n_seg, 0LL);
    const int st = run(parts, N, seg_per_block, (long long)M * N);
    if (st) return st;
    const size_t blocks = ((size_t)M * N + 255) / 256;
    return launch_pdl(sum_parts_kernel, dim3((unsigned)(blocks < 2368 ? blocks : 2368)), dim3(256), 0, stream, parts,
                      1 + (n_seg > seg_per_block ? n_seg - seg_per_block : 0), y, ldy, M, N);
}

// ---------------------------------------------------------------------------
// Any strides and sizes, one element at a time: 64 x 64 tiles, 4 x 4 outputs a thread, pairs of an even and an odd k side
// by side in shared memory; the next 16 k are on their way while a tile is multiplied.
constexpr int AM = 64, AN = 64, AK = 16;
constexpr int APITCH = AM + 4;                         // pairs

__global__ void __launch_bounds__(256) any_kernel(const float* __restrict__ X, int ldx, const float* __restrict__ W, int ldw,
                                                  float* __restrict__ Y, int ldy, int M, int N, int K) {
    __shared__ __align__(16) float2 As[2][AK / 2][APITCH];
    __shared__ __align__(16) float2 Bs[2][AK / 2][APITCH];
    const int tid = threadIdx.x;
    const int tx = tid & 15, ty = tid >> 4;            // rows 4 ty .. 4 ty + 3; columns 2 tx, 2 tx + 1 and the two 32 further on
    const int m0 = blockIdx.y * AM, n0 = blockIdx.x * AN;
    const int lr = tid >> 2, lk = (tid & 3) * 4;       // loader: row lr, k offset lk..lk+3
    const float* xp = X + (size_t)min(m0 + lr, M - 1) * ldx + lk;
    const float* wp = W + (size_t)min(n0 + lr, N - 1) * ldw + lk;
    const bool x_ok = m0 + lr < M, w_ok = n0 + lr < N;

    float a[4], b[4];
    auto load = [&](int k0) {
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            const bool ok = k0 + lk + i < K;
            a[i] = ok && x_ok ? xp[k0 + i] : 0.0f;
            b[i] = ok && w_ok ? wp[k0 + i] : 0.0f;
        }
    };
    uint64_t acc[4][4];
    float tot[4][4];
#pragma unroll
    for (int i = 0; i < 4; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            acc[i][j] = 0;
            tot[i][j] = 0.0f;
        }
    load(0);
    for (int k0 = 0; k0 < K; k0 += AK) {
        const int st = (k0 / AK) & 1;
        As[st][lk / 2][lr] = make_float2(a[0], a[1]);
        As[st][lk / 2 + 1][lr] = make_float2(a[2], a[3]);
        Bs[st][lk / 2][lr] = make_float2(b[0], b[1]);
        Bs[st][lk / 2 + 1][lr] = make_float2(b[2], b[3]);
        __syncthreads();   // this tile is written, and the one before it is consumed by all (its stage is written next)
        if (k0 + AK < K) load(k0 + AK);
#pragma unroll
        for (int kk = 0; kk < AK / 2; ++kk) {
            const ulonglong2 a0 = *reinterpret_cast<const ulonglong2*>(&As[st][kk][ty * 4]);
            const ulonglong2 a1 = *reinterpret_cast<const ulonglong2*>(&As[st][kk][ty * 4 + 2]);
            const ulonglong2 b0 = *reinterpret_cast<const ulonglong2*>(&Bs[st][kk][tx * 2]);
            const ulonglong2 b1 = *reinterpret_cast<const ulonglong2*>(&Bs[st][kk][tx * 2 + 32]);
            const uint64_t ar[4] = {a0.x, a0.y, a1.x, a1.y}, br[4] = {b0.x, b0.y, b1.x, b1.y};
#pragma unroll
            for (int i = 0; i < 4; ++i)
#pragma unroll
                for (int j = 0; j < 4; ++j) fma2(acc[i][j], ar[i], br[j]);
        }
        if ((k0 + AK) % SEG == 0 || k0 + AK >= K) {
#pragma unroll
            for (int i = 0; i < 4; ++i)
#pragma unroll
                for (int j = 0; j < 4; ++j) {
                    const float c = halves_sum(acc[i][j]);
                    tot[i][j] = k0 < SEG ? c : tot[i][j] + c;
                    acc[i][j] = 0;
                }
        }
    }
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        const int m = m0 + ty * 4 + i;
        if (m >= M) continue;
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            const int n = n0 + tx * 2 + (j & 1) + (j >> 1) * 32;
            if (n < N) Y[(size_t)m * ldy + n] = tot[i][j];
        }
    }
}

}  // namespace

// kind: which kernel (rows and tiles want operands whose rows lie on 16-byte boundaries, K % 4 == 0; rows M <= 16).
// parts (tiles only): the blocks take seg_per_block segments of 512 k each, and their sums lie here before they are added,
// 1 + ceil(K / 512) - seg_per_block times M * N floats; null: a block takes all of K.
enum : int { KIND_ANY = 0, KIND_ROWS = 1, KIND_TILES32 = 32, KIND_TILES64 = 64 };

BROLM_API int brolm_linear_f32(const void* x, int ldx, const void* w, int ldw, void* y, int ldy, int M, int N, int K,
                               int kind, void* parts, int seg_per_block, cudaStream_t stream) {
    if (M <= 0 || N <= 0) return BROLM_OK;
    if (K <= 0 || (parts && seg_per_block < 1)) return BROLM_ERR_BAD_SIZE;
    const float *xf = (const float*)x, *wf = (const float*)w;
    float* yf = (float*)y;
    if (kind != KIND_ANY && (K % 4 || ldx % 4 || ldw % 4 || ((uintptr_t)x & 15) || ((uintptr_t)w & 15))) return BROLM_ERR_ALIGNMENT;
    if (kind == KIND_ROWS) {
        if (M > 16) return BROLM_ERR_BAD_SIZE;
        const int st = M <= 1 ? dispatch_rows<1>(xf, ldx, wf, ldw, yf, ldy, M, N, K, stream)
                     : M <= 2 ? dispatch_rows<2>(xf, ldx, wf, ldw, yf, ldy, M, N, K, stream)
                     : M <= 4 ? dispatch_rows<4>(xf, ldx, wf, ldw, yf, ldy, M, N, K, stream)
                     : M <= 8 ? dispatch_rows<8>(xf, ldx, wf, ldw, yf, ldy, M, N, K, stream)
                              : dispatch_rows<16>(xf, ldx, wf, ldw, yf, ldy, M, N, K, stream);
        if (st != BROLM_ERR_TOO_LARGE) return st;
        kind = KIND_TILES32;                             // a K beyond what the sums have room for
    }
    if ((N + BN - 1) / BN <= 65535) {
        if (kind == KIND_TILES32) return launch_tiles<32>(xf, ldx, wf, ldw, yf, ldy, M, N, K, (float*)parts, seg_per_block, stream);
        if (kind == KIND_TILES64) return launch_tiles<64>(xf, ldx, wf, ldw, yf, ldy, M, N, K, (float*)parts, seg_per_block, stream);
    }
    const long long gy = (M + AM - 1) / AM;
    if (gy > 65535) return BROLM_ERR_TOO_LARGE;
    dim3 grid((N + AN - 1) / AN, (unsigned)gy);
    any_kernel<<<grid, 256, 0, stream>>>(xf, ldx, wf, ldw, yf, ldy, M, N, K);
    return launch_status();
}
