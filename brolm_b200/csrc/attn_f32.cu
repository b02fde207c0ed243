// Float attention over a prompt's packed keys or the paged cache, on CUDA cores: the float model's path where rows are
// whole 16-byte pieces of at most 256 elements (attn_simt.cu has the masks and options, and takes everything else).
//
// One order of operations for a query, whatever step, batch or split it runs in, so that a prompt pass and a decode pass
// give the same bits for finite values.  (A tile reads the values of all keys that any of its rows sees, and gives those
// that a row does not see the weight zero: zero times an infinity or a NaN of a later token reaches the rows before it in the
// tile, and a decode pass does not read it.)  Keys come in spans of 128, anchored at multiples of 128 of the absolute position:
//
//   score    s_j = (sum over even c of q_c k_c) + (sum over odd c), each a chain of fmas over ascending c; then the
//            scale, the cap, the slope, the distance bias and the mask
//   span     m = max s_j, p_j = exp(s_j - m), l = the 32-key sums of p (a butterfly over lanes) added in order,
//            a_d = a chain of fmas p_j v_jd over ascending j
//   merge    of the spans in ascending order: M' = max(M, m), L = L e^(M - M') + l e^(m - M'), A alike
//
// and the result is A / L (with a sink: A / (L + e^(sink - M))).
//
// A block owns 32 rows of one (sequence, kv head), a row being a (query token, query head of the group) pair, or 8 where
// a step has no more (decode), and either walks all spans it sees or, where that leaves SMs idle, one of them, with
// merge_kernel behind it (attn_f32_splits and attn_f32_worth_sharing in kernels/__init__.py have the rule and what both take): a decode step of three
// sequences of 420 keys, 4 kv heads of 256, is otherwise twelve blocks (79 us; 27 shared, 11.5 in clusters of four blocks, which
// take such a span where there are few; 337 in attn_simt.cu, which served all sizes before).  Prompts in tiles of 16 rows where
// those of 32 leave SMs idle (300 tokens, 8 heads of 256 on 4: 50 us, 62 in tiles of 32).  Of a span only the 32-key parts that some row sees are worked on: one,
// two or all four (16 tokens, 4 heads of 16: 8.9 us, 13.8 with whole spans; 1,000 tokens, 32 heads of 128 on 8 kv heads, window 64:
// 129 and 183).  K comes through a ring of cp.async stages in slices of 32 c of all 128 keys, V in
// slices of 16 keys; both products run on packed fma.rn.f32x2, the scores paired along c, the values along d.  Bound by
// shared memory: a thread's outputs are what its registers hold (4 x 8 scores, 4 x 16 values).
#include "common.cuh"

namespace {

constexpr int SPAN = 128;
constexpr int THREADS = 128;
constexpr int STAGES = 3;
constexpr int KC = 32;                        // c of a slice of keys
constexpr int PITCH = 144;                    // its bytes, padded: eight neighbouring rows lie in different banks
constexpr int VK = 16;                        // keys of a slice of values
constexpr int P_PITCH = SPAN + 4;             // floats

struct F32Args {
    const float* q;
    float* out;
    int q_stride, out_stride;
    const int32_t* cu_q;
    const int32_t* kv_len;
    const float* k;
    const float* v;
    int k_stride, v_stride;
    const float* k_pages;                     // null: packed keys
    const float* v_pages;
    const int32_t* page_table;
    int pt_stride, ring, page_size;
    int n_kv, group, hd, vd;
    float scale, cap;
    int window, chunk;
    const float* sink;
    const float* slopes;
    const float* dist_bias;
    int dist_len;
    int max_parts;                            // 32-key parts of a span that hold keys: 4, or fewer in steps of so few keys
    int splits;                               // spans a tile can see; 0: a block walks them all
    float* part_acc;                          // [token][head][split][vd]
    float* part_ml;                           // [token][head][split][2]
};

__device__ __forceinline__ uint64_t pack2(float lo, float hi) {
    uint64_t v;
    asm("mov.b64 %0, {%1, %2};\n" : "=l"(v) : "f"(lo), "f"(hi));
    return v;
}
__device__ __forceinline__ float2 unpack2(uint64_t v) {
    float2 f;
    asm("mov.b64 {%0, %1}, %2;\n" : "=f"(f.x), "=f"(f.y) : "l"(v));
    return f;
}
__device__ __forceinline__ Pair2 lds4(const float* p) {
    const ulonglong2 v = *reinterpret_cast<const ulonglong2*>(p);
    return Pair2{v.x, v.y};
}

// a slice of keys, or of values
__host__ __device__ __forceinline__ int stage_bytes(const F32Args& a) {
    const int k = a.max_parts * 32 * PITCH, v = VK * a.vd * 4;
    return k > v ? k : v;
}

// The merge of one more span into (M, L): factors for what is held and for what comes.
__device__ __forceinline__ void merge_factors(float& M, float& L, float m, float l, float& held, float& fresh) {
    const float top = fmaxf(M, m);
    held = M > -INFINITY ? expf(M - top) : 0.0f;
    fresh = m > -INFINITY ? expf(m - top) : 0.0f;
    L = __fmaf_rn(L, held, __fmul_rn(l, fresh));
    M = top;
}
__device__ __forceinline__ float merged(float held_sum, float held, float fresh_sum, float fresh) {
    return __fmaf_rn(held_sum, held, __fmul_rn(fresh_sum, fresh));
}
__device__ __forceinline__ float share(const F32Args& a, float M, float L, int head) {
    if (a.sink && M > -INFINITY) L += expf(a.sink[head] - M);
    return L > 0.0f ? 1.0f / L : 0.0f;
}

// The rows of a tile and the spans they see: [first, last].
struct Tile { int q0, row0, rows, first_pos, key_lo, first, last; };
template <int ROWS>
__device__ __forceinline__ Tile tile_of(const F32Args& a, int b, int tile) {
    Tile t;
    t.q0 = a.cu_q[b];
    const int q_len = a.cu_q[b + 1] - t.q0, kv_len = a.kv_len[b];
    t.row0 = tile * ROWS;
    t.rows = kv_len > 0 ? max(0, min(ROWS, q_len * a.group - t.row0)) : 0;
    t.first_pos = kv_len - q_len;
    if (t.rows <= 0) return t;
    const int lo = t.first_pos + t.row0 / a.group;
    int key = a.window > 0 ? max(0, lo - a.window + 1) : 0;
    if (a.chunk > 0) key = max(key, lo - lo % a.chunk);
    t.key_lo = key;
    t.first = key / SPAN;
    t.last = (t.first_pos + (t.row0 + t.rows - 1) / a.group) / SPAN;
    return t;
}

template <int N> struct Count { static constexpr int value = N; };

template <int ROWS, int VJ>
__global__ void __launch_bounds__(THREADS, ROWS == 8 ? 4 : VJ == 4 && ROWS == 32 ? 2 : 3) attn_f32_kernel(F32Args a) {
    constexpr int LN = ROWS == 8 ? 32 : 16;           // threads side by side over keys, and over value dims
    constexpr int RI = ROWS / (THREADS / LN);          // rows of a thread, THREADS / LN apart
    constexpr int RSTEP = THREADS / LN;
    extern __shared__ __align__(16) uint8_t raw[];
    const int q_pitch = (a.hd + KC - 1) / KC * KC + 4;  // floats; zeros behind hd
    const int stage = stage_bytes(a);
    uint8_t* ring = raw;
    const uint32_t ring_at = (uint32_t)__cvta_generic_to_shared(ring);
    float* Qs = reinterpret_cast<float*>(raw + STAGES * stage);
    float* P = Qs + ROWS * q_pitch;
    float* stats = P + ROWS * P_PITCH;                  // [ROWS]: M, L, and from the second span on the factors of what is held and of what comes
    long long* k_off = reinterpret_cast<long long*>(stats + 4 * ROWS);
    long long* v_off = k_off + SPAN;

    const int b = blockIdx.z, g = blockIdx.y;
    const int tile = a.splits ? blockIdx.x / a.splits : blockIdx.x;
    pdl_wait();
    const Tile t = tile_of<ROWS>(a, b, tile);
    if (t.rows <= 0) return;
    int span = t.first, last = t.last;
    if (a.splits) {
        const int share = blockIdx.x % a.splits;
        span += share;
        if (span > last) return;
        if (share < a.splits - 1) last = span;          // (the last block walks what is left, should the bound not have held)
    }
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int tn = tid % LN, tm = tid / LN;
    const int key_hi = t.first_pos + (t.row0 + t.rows - 1) / a.group;

    auto load_q = [&] {
        for (int idx = tid; idx < ROWS * (q_pitch / 4); idx += THREADS) {
            const int r = idx / (q_pitch / 4), c = (idx - r * (q_pitch / 4)) * 4;
            float4 v = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
            if (r < t.rows && c < a.hd) {
                const int row = t.row0 + r;
                v = *reinterpret_cast<const float4*>(a.q + (size_t)(t.q0 + row / a.group) * a.q_stride +
                                                     (g * a.group + row % a.group) * a.hd + c);
            }
            *reinterpret_cast<float4*>(Qs + r * q_pitch + c) = v;
        }
    };
    if (ROWS == 8) load_q();

    const int k_slices = (a.hd + KC - 1) / KC;
    float tot[RI][VJ][4];
#pragma unroll
    for (int i = 0; i < RI; ++i)
#pragma unroll
        for (int j = 0; j < VJ; ++j) tot[i][j][0] = tot[i][j][1] = tot[i][j][2] = tot[i][j][3] = 0.0f;

    for (bool first = true; span <= last; ++span, first = false) {
        const int key0 = span * SPAN;
        const int keys = min(a.max_parts * 32, key_hi + 1 - key0);      // keys behind the tile's last query are not read
        // the 32-key parts of the span that any row sees: part0 and as many as make one, two or all four.  (Tiles of eight
        // rows, decoding, always work on all four: a step runs each instruction about once, and what a launch of three
        // variants fetches of them is a tenth of its time, 30 us against 26 a layer of 4 kv heads of 256 at 420 keys.)
        int part0 = max(0, t.key_lo - key0) / 32, n_parts = (keys - 1) / 32 - part0 + 1;
        if (ROWS == 8 || n_parts > 2) part0 = 0, n_parts = 4;
        __syncthreads();                                // the span before this one is done with
        {
            const int kp = key0 + tid;
            long long ko = -1, vo = -1;
            if (tid < keys && kp >= t.key_lo) {          // (a ring's places of older positions hold other keys)
                if (a.k_pages) {
                    const int place = kp % a.ring, page = a.page_table[(size_t)b * a.pt_stride + place / a.page_size];
                    const long long at = ((long long)page * a.n_kv + g) * a.page_size + place % a.page_size;
                    ko = at * a.hd;
                    vo = at * a.vd;
                } else {
                    ko = (long long)(t.q0 + kp) * a.k_stride + (long long)g * a.hd;
                    vo = (long long)(t.q0 + kp) * a.v_stride + (long long)g * a.vd;
                }
            }
            k_off[tid] = ko;
            v_off[tid] = vo;
        }
        __syncthreads();
        const float* kb = a.k_pages ? a.k_pages : a.k;
        const float* vb = a.k_pages ? a.v_pages : a.v;
        const int v_from = part0 * 32, slices = k_slices + (keys - v_from + VK - 1) / VK;
        auto fetch_v = [&](int i) {
            if (i < slices) {
                const uint32_t dst = ring_at + (i % STAGES) * stage;
                const int pieces = a.vd / 4;
                for (int idx = tid; idx < VK * pieces; idx += THREADS) {
                    const int j = idx / pieces, c = (idx - j * pieces) * 4;
                    const long long o = v_off[v_from + (i - k_slices) * VK + j];
                    copy16(dst + (j * a.vd + c) * 4, vb + (o >= 0 ? o + c : 0), o >= 0);
                }
            }
            copy_commit();
        };
        auto parts = [&](auto count) {
            constexpr int N = decltype(count)::value, NJ = N * 32 / LN;
            auto fetch = [&](int i) {
                if (i >= k_slices) return fetch_v(i);
                const uint32_t dst = ring_at + (i % STAGES) * stage;
                const int c = i * KC + (tid & 7) * 4;
#pragma unroll
                for (int j = 0; j < N * 2; ++j) {
                    const int key = part0 * 32 + j * 16 + (tid >> 3);
                    const long long o = k_off[key];
                    const bool ok = o >= 0 && c < a.hd;
                    copy16(dst + key * PITCH + (tid & 7) * 16, kb + (ok ? o + c : 0), ok);
                }
                copy_commit();
            };
#pragma unroll
            for (int i = 0; i < STAGES - 1; ++i) fetch(i);
            if (ROWS != 8 && first) load_q();              // (seen by all behind the first slice's barrier)
            uint64_t s[RI][NJ];
#pragma unroll
            for (int i = 0; i < RI; ++i)
#pragma unroll
                for (int j = 0; j < NJ; ++j) s[i][j] = 0;
            for (int i = 0; i < k_slices; ++i) {
                copy_wait<STAGES - 2>();
                __syncthreads();
                fetch(i + STAGES - 1);
                const float* ks = reinterpret_cast<const float*>(ring + (i % STAGES) * stage) + (part0 * 32 + tn) * (PITCH / 4);
                const float* qs = Qs + tm * q_pitch + i * KC;
#pragma unroll
                for (int c = 0; c < KC; c += 4) {
                    Pair2 q[RI];
#pragma unroll
                    for (int r = 0; r < RI; ++r) q[r] = lds4(qs + r * RSTEP * q_pitch + c);
#pragma unroll
                    for (int j = 0; j < NJ; ++j) {
                        const Pair2 k = lds4(ks + j * LN * (PITCH / 4) + c);
#pragma unroll
                        for (int r = 0; r < RI; ++r) {
                            fma2(s[r][j], q[r].x, k.x);
                            fma2(s[r][j], q[r].y, k.y);
                        }
                    }
                }
            }
#pragma unroll
            for (int r = 0; r < RI; ++r)
#pragma unroll
                for (int j = 0; j < NJ; ++j) {
                    const float2 h = unpack2(s[r][j]);
                    P[(tm + r * RSTEP) * P_PITCH + part0 * 32 + tn + j * LN] = h.x + h.y;
                }
            __syncthreads();
            // a warp's rows, two at a time: scores out of the products, then the span's maximum, probabilities and sum
            constexpr int RB = 2;
            for (int r0 = warp * (ROWS / 4); r0 < (warp + 1) * (ROWS / 4); r0 += RB) {
                float sc[RB][N], m[RB], l[RB];
#pragma unroll
                for (int r = 0; r < RB; ++r) {
                    const int row = t.row0 + r0 + r, head = g * a.group + row % a.group;
                    const int pos = r0 + r < t.rows ? t.first_pos + row / a.group : -1;
                    const float slope = a.slopes && pos >= 0 ? a.slopes[head] : 0.0f;
                    const int from = max(a.window > 0 ? pos - a.window + 1 : 0, a.chunk > 0 && pos >= 0 ? pos - pos % a.chunk : 0);
                    m[r] = -INFINITY;
#pragma unroll
                    for (int e = 0; e < N; ++e) {
                        const int kp = key0 + (part0 + e) * 32 + lane;
                        float v = -INFINITY;
                        if (kp <= pos && kp >= from) {
                            v = soft_cap(__fmul_rn(P[(r0 + r) * P_PITCH + (part0 + e) * 32 + lane], a.scale), a.cap);
                            if (a.slopes) v = __fmaf_rn(-slope, (float)(pos - kp), v);
                            if (a.dist_bias) v += a.dist_bias[(size_t)head * a.dist_len + min(pos - kp, a.dist_len - 1)];
                        }
                        sc[r][e] = v;
                        m[r] = fmaxf(m[r], v);
                    }
                }
#pragma unroll
                for (int o = 16; o > 0; o >>= 1)
#pragma unroll
                    for (int r = 0; r < RB; ++r) m[r] = fmaxf(m[r], __shfl_xor_sync(0xffffffffu, m[r], o));
#pragma unroll
                for (int r = 0; r < RB; ++r)
#pragma unroll
                    for (int e = 0; e < N; ++e) {
                        sc[r][e] = sc[r][e] == -INFINITY ? 0.0f : expf(sc[r][e] - m[r]);       // (a NaN stays one)
                        P[(r0 + r) * P_PITCH + (part0 + e) * 32 + lane] = sc[r][e];
                    }
#pragma unroll
                for (int o = 16; o > 0; o >>= 1)
#pragma unroll
                    for (int r = 0; r < RB; ++r)
#pragma unroll
                        for (int e = 0; e < N; ++e) sc[r][e] += __shfl_xor_sync(0xffffffffu, sc[r][e], o);
#pragma unroll
                for (int r = 0; r < RB; ++r) {
                    l[r] = sc[r][0];
#pragma unroll
                    for (int e = 1; e < N; ++e) l[r] += sc[r][e];
                }
                if (lane < RB) {
                    const float mine = lane == 0 ? m[0] : m[1], sum = lane == 0 ? l[0] : l[1];
                    const int r = r0 + lane;
                    if (first) {                             // nothing is held: what comes is taken as it is
                        stats[r] = mine;
                        stats[ROWS + r] = sum;
                    } else {
                        float M = stats[r], L = stats[ROWS + r], held, fresh;
                        merge_factors(M, L, mine, sum, held, fresh);
                        stats[r] = M;
                        stats[ROWS + r] = L;
                        stats[2 * ROWS + r] = held;
                        stats[3 * ROWS + r] = fresh;
                    }
                }
            }
        };
        if constexpr (ROWS == 8) parts(Count<4>());
        else if (n_parts == 1) parts(Count<1>());
        else if (n_parts == 2) parts(Count<2>());
        else parts(Count<4>());
        uint64_t acc[RI][VJ][2];
#pragma unroll
        for (int r = 0; r < RI; ++r)
#pragma unroll
            for (int j = 0; j < VJ; ++j) acc[r][j][0] = acc[r][j][1] = 0;
        for (int i = k_slices; i < slices; ++i) {
            copy_wait<STAGES - 2>();
            __syncthreads();                            // (the first time round: P and the factors are written, too)
            fetch_v(i + STAGES - 1);
            const float* vs = reinterpret_cast<const float*>(ring + (i % STAGES) * stage);
            const float* ps = P + tm * P_PITCH + v_from + (i - k_slices) * VK;
#pragma unroll
            for (int j0 = 0; j0 < VK; j0 += 4) {
                float p[RI][4];
#pragma unroll
                for (int r = 0; r < RI; ++r) {
                    const float4 f = *reinterpret_cast<const float4*>(ps + r * RSTEP * P_PITCH + j0);
                    p[r][0] = f.x; p[r][1] = f.y; p[r][2] = f.z; p[r][3] = f.w;
                }
#pragma unroll
                for (int e = 0; e < 4; ++e) {
                    uint64_t pp[RI];
#pragma unroll
                    for (int r = 0; r < RI; ++r) pp[r] = pack2(p[r][e], p[r][e]);
#pragma unroll
                    for (int j = 0; j < VJ; ++j) {
                        const int d = 4 * (tn + j * LN);
                        if (d < a.vd) {
                            const Pair2 v = lds4(vs + (j0 + e) * a.vd + d);
#pragma unroll
                            for (int r = 0; r < RI; ++r) {
                                fma2(acc[r][j][0], pp[r], v.x);
                                fma2(acc[r][j][1], pp[r], v.y);
                            }
                        }
                    }
                }
            }
        }
        copy_wait<0>();                                 // (only empty groups are left)
#pragma unroll
        for (int r = 0; r < RI; ++r) {
            const int rr = tm + r * RSTEP;
            const float held = first ? 0.0f : stats[2 * ROWS + rr], fresh = first ? 1.0f : stats[3 * ROWS + rr];
#pragma unroll
            for (int j = 0; j < VJ; ++j) {
                const float2 lo = unpack2(acc[r][j][0]), hi = unpack2(acc[r][j][1]);
                tot[r][j][0] = merged(tot[r][j][0], held, lo.x, fresh);
                tot[r][j][1] = merged(tot[r][j][1], held, lo.y, fresh);
                tot[r][j][2] = merged(tot[r][j][2], held, hi.x, fresh);
                tot[r][j][3] = merged(tot[r][j][3], held, hi.y, fresh);
            }
        }
    }
    pdl_trigger();
#pragma unroll
    for (int r = 0; r < RI; ++r) {
        const int rr = tm + r * RSTEP;
        if (rr >= t.rows) continue;
        const int row = t.row0 + rr, token = t.q0 + row / a.group, head = g * a.group + row % a.group;
        float* dst;
        float inv = 1.0f;
        if (a.splits) {
            const size_t at = ((size_t)token * a.n_kv * a.group + head) * a.splits + blockIdx.x % a.splits;
            dst = a.part_acc + at * a.vd;
            if (tn == 0) {
                a.part_ml[2 * at] = stats[rr];
                a.part_ml[2 * at + 1] = stats[ROWS + rr];
            }
        } else {
            dst = a.out + (size_t)token * a.out_stride + (size_t)head * a.vd;
            inv = share(a, stats[rr], stats[ROWS + rr], head);
        }
#pragma unroll
        for (int j = 0; j < VJ; ++j) {
            const int d = 4 * (tn + j * LN);
            if (d < a.vd)
#pragma unroll
                for (int e = 0; e < 4; ++e) dst[d + e] = a.splits ? tot[r][j][e] : __fmul_rn(tot[r][j][e], inv);
        }
    }
}

// Tiles of eight rows whose spans are shared (decode steps): a cluster of four blocks takes a span, each the scores of 32
// keys for all rows, and then, with every score handed round through shared memory, a quarter of the value's entries for
// all 128 keys.  All keys and values of a block are on their way at once, 64 KB with heads of 256, and every chain of fmas
// has a thread of its own: what is left is the chains' length and the memory's latency.  The same order of operations.  For no more spans than SMs: the
// cluster's exchange costs more than it gives once blocks queue (brolm_attn_f32 has the figures).
constexpr int FEW = 8, FEW_THREADS = 32 * FEW, SHARERS = 4;

__host__ __device__ __forceinline__ int few_quarter(int vd) { return (vd + 15) / 16 * 4; }      // value entries of a block
__host__ __device__ __forceinline__ int few_bytes(const F32Args& a) {
    return 32 * (a.hd * 4 + 16) + SPAN * few_quarter(a.vd) * 4 + (FEW * a.hd + FEW * P_PITCH + 4 * FEW) * 4 + (32 + SPAN) * 8;
}

__global__ void __launch_bounds__(FEW_THREADS) __cluster_dims__(SHARERS, 1, 1) attn_f32_few_kernel(F32Args a) {
    extern __shared__ __align__(16) uint8_t raw[];
    const int k_pitch = a.hd * 4 + 16, vq = few_quarter(a.vd);
    const uint32_t ks = (uint32_t)__cvta_generic_to_shared(raw), vs = ks + 32 * k_pitch;
    float* Vs = reinterpret_cast<float*>(raw + 32 * k_pitch);
    float* Qs = Vs + SPAN * vq;
    float* P = Qs + FEW * a.hd;
    float* stats = P + FEW * P_PITCH;                   // [FEW]: M, L, the factors of what is held and of what comes
    long long* k_off = reinterpret_cast<long long*>(stats + 4 * FEW);
    long long* v_off = k_off + 32;
    const int b = blockIdx.z, g = blockIdx.y, part = blockIdx.x % SHARERS, split = blockIdx.x / SHARERS;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    pdl_wait();
    const Tile t = tile_of<FEW>(a, b, 0);
    if (t.rows <= 0) return;
    int span = t.first + split, last = t.last;
    if (span > last) return;
    if (split < a.splits - 1) last = span;              // (the last one walks what is left, should the bound not have held)
    asm volatile("barrier.cluster.arrive.release;" ::: "memory");
    const int key_hi = t.first_pos + (t.row0 + t.rows - 1) / a.group;
    const int v0 = part * vq, v_wide = min(vq, a.vd - v0);              // (nothing is left for the last blocks of small rows)
    const float* kb = a.k_pages ? a.k_pages : a.k;
    const float* vb = a.k_pages ? a.v_pages : a.v;
    for (int idx = tid; idx < t.rows * (a.hd / 4); idx += FEW_THREADS) {
        const int r = idx / (a.hd / 4), c = (idx - r * (a.hd / 4)) * 4, row = t.row0 + r;
        copy16((uint32_t)__cvta_generic_to_shared(Qs + r * a.hd + c),
               a.q + (size_t)(t.q0 + row / a.group) * a.q_stride + (g * a.group + row % a.group) * a.hd + c, true);
    }
    // a thread's chain over the keys: two neighbouring value entries of a row
    const int chains = max(0, v_wide / 2), my_row = chains ? tid / chains : FEW, my_d = chains ? (tid - my_row * chains) * 2 : 0;
    float tot[2] = {0.0f, 0.0f};
    for (bool first = true; span <= last; ++span, first = false) {
        const int key0 = span * SPAN, keys = min(SPAN, key_hi + 1 - key0);
        if (tid < SPAN) {
            const int kp = key0 + tid;
            long long ko = -1, vo = -1;
            if (tid < keys && kp >= t.key_lo) {          // (a ring's places of older positions hold other keys)
                if (a.k_pages) {
                    const int place = kp % a.ring, page = a.page_table[(size_t)b * a.pt_stride + place / a.page_size];
                    const long long at = ((long long)page * a.n_kv + g) * a.page_size + place % a.page_size;
                    ko = at * a.hd;
                    vo = at * a.vd;
                } else {
                    ko = (long long)(t.q0 + kp) * a.k_stride + (long long)g * a.hd;
                    vo = (long long)(t.q0 + kp) * a.v_stride + (long long)g * a.vd;
                }
            }
            if (tid >> 5 == part) k_off[lane] = ko;
            v_off[tid] = vo;
        }
        __syncthreads();
        for (int key = warp; key < 32; key += FEW) {
            const long long o = k_off[key];
            for (int c = lane * 4; c < a.hd; c += 128) copy16(ks + key * k_pitch + c * 4, kb + (o >= 0 ? o + c : 0), o >= 0);
        }
        copy_commit();
        if (v_wide > 0) {
            const int pieces = v_wide / 4;
            for (int idx = tid; idx < SPAN * pieces; idx += FEW_THREADS) {
                const int j = idx / pieces, c = (idx - j * pieces) * 4;
                const long long o = v_off[j];
                copy16(vs + (j * vq + c) * 4, vb + (o >= 0 ? o + v0 + c : 0), o >= 0);
            }
        }
        copy_commit();
        copy_wait<1>();
        __syncthreads();
        float score = 0.0f;
        if (warp < t.rows) {                             // a warp's row, a lane's key
            uint64_t s = 0;
            const float* q = Qs + warp * a.hd;
            const float* k = reinterpret_cast<const float*>(raw + lane * k_pitch);
#pragma unroll 8
            for (int c = 0; c < a.hd; c += 4) {
                const Pair2 qq = lds4(q + c), kk = lds4(k + c);
                fma2(s, qq.x, kk.x);
                fma2(s, qq.y, kk.y);
            }
            const float2 h = unpack2(s);
            score = h.x + h.y;
        }
        if (first) asm volatile("barrier.cluster.wait.acquire;" ::: "memory");          // (the other blocks are there)
        if (warp < t.rows) {
            const uint32_t at = (uint32_t)__cvta_generic_to_shared(P + warp * P_PITCH + part * 32 + lane);
#pragma unroll
            for (int r = 0; r < SHARERS; ++r) {
                uint32_t far;
                asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(far) : "r"(at), "r"(r));
                asm volatile("st.shared::cluster.f32 [%0], %1;" ::"r"(far), "f"(score) : "memory");
            }
        }
        asm volatile("barrier.cluster.arrive.release;\nbarrier.cluster.wait.acquire;" ::: "memory");
        if (warp < t.rows) {                             // as in the kernel above, one row a warp
            const int row = t.row0 + warp, head = g * a.group + row % a.group, pos = t.first_pos + row / a.group;
            const float slope = a.slopes ? a.slopes[head] : 0.0f;
            const int from = max(a.window > 0 ? pos - a.window + 1 : 0, a.chunk > 0 ? pos - pos % a.chunk : 0);
            float sc[4], m = -INFINITY;
#pragma unroll
            for (int e = 0; e < 4; ++e) {
                const int kp = key0 + e * 32 + lane;
                float v = -INFINITY;
                if (kp <= pos && kp >= from) {
                    v = soft_cap(__fmul_rn(P[warp * P_PITCH + e * 32 + lane], a.scale), a.cap);
                    if (a.slopes) v = __fmaf_rn(-slope, (float)(pos - kp), v);
                    if (a.dist_bias) v += a.dist_bias[(size_t)head * a.dist_len + min(pos - kp, a.dist_len - 1)];
                }
                sc[e] = v;
                m = fmaxf(m, v);
            }
            m = warp_max(m);
#pragma unroll
            for (int e = 0; e < 4; ++e) {
                sc[e] = sc[e] == -INFINITY ? 0.0f : expf(sc[e] - m);                    // (a NaN stays one)
                P[warp * P_PITCH + e * 32 + lane] = sc[e];
            }
#pragma unroll
            for (int o = 16; o > 0; o >>= 1)
#pragma unroll
                for (int e = 0; e < 4; ++e) sc[e] += __shfl_xor_sync(0xffffffffu, sc[e], o);
            if (lane == 0) {
                const float sum = ((sc[0] + sc[1]) + sc[2]) + sc[3];
                if (first) {
                    stats[warp] = m;
                    stats[FEW + warp] = sum;
                } else {
                    float M = stats[warp], L = stats[FEW + warp], held, fresh;
                    merge_factors(M, L, m, sum, held, fresh);
                    stats[warp] = M;
                    stats[FEW + warp] = L;
                    stats[2 * FEW + warp] = held;
                    stats[3 * FEW + warp] = fresh;
                }
            }
        }
        copy_wait<0>();
        __syncthreads();
        if (my_row < t.rows) {
            uint64_t acc = 0;
            const float* p = P + my_row * P_PITCH;
            const float* v = Vs + my_d;
#pragma unroll 4
            for (int j = 0; j < SPAN; j += 4) {
                const float4 w = *reinterpret_cast<const float4*>(p + j);
                fma2(acc, pack2(w.x, w.x), *reinterpret_cast<const uint64_t*>(v + j * vq));
                fma2(acc, pack2(w.y, w.y), *reinterpret_cast<const uint64_t*>(v + (j + 1) * vq));
                fma2(acc, pack2(w.z, w.z), *reinterpret_cast<const uint64_t*>(v + (j + 2) * vq));
                fma2(acc, pack2(w.w, w.w), *reinterpret_cast<const uint64_t*>(v + (j + 3) * vq));
            }
            const float held = first ? 0.0f : stats[2 * FEW + my_row], fresh = first ? 1.0f : stats[3 * FEW + my_row];
            const float2 f = unpack2(acc);
            tot[0] = merged(tot[0], held, f.x, fresh);
            tot[1] = merged(tot[1], held, f.y, fresh);
        }
        if (span < last) {                               // the scores of the next span come into P from all blocks
            __syncthreads();
            asm volatile("barrier.cluster.arrive.release;\nbarrier.cluster.wait.acquire;" ::: "memory");
        }
    }
    pdl_trigger();
    const auto place = [&](int r) {
        const int row = t.row0 + r;
        return ((size_t)(t.q0 + row / a.group) * a.n_kv * a.group + g * a.group + row % a.group) * a.splits + split;
    };
    if (part == 0 && tid < t.rows) {
        a.part_ml[2 * place(tid)] = stats[tid];
        a.part_ml[2 * place(tid) + 1] = stats[FEW + tid];
    }
    if (my_row < t.rows) *reinterpret_cast<float2*>(a.part_acc + place(my_row) * a.vd + v0 + my_d) = make_float2(tot[0], tot[1]);
}

// One row (blockIdx.x: a row of the sequence's, blockIdx.y: kv head, blockIdx.z: sequence): its spans in order.
template <int ROWS>
__global__ void __launch_bounds__(64) merge_kernel(F32Args a) {
    const int b = blockIdx.z, row = blockIdx.x;
    pdl_trigger();
    pdl_wait();
    const Tile t = tile_of<ROWS>(a, b, row / ROWS);
    if (row - t.row0 >= t.rows) return;
    const int token = t.q0 + row / a.group, head = blockIdx.y * a.group + row % a.group;
    const size_t at = ((size_t)token * a.n_kv * a.group + head) * a.splits;
    const int n = min(t.last - t.first + 1, a.splits);  // (never more: the caller's bound; and no read behind its room)
    const float* acc = a.part_acc + at * a.vd + threadIdx.x * 4;
    const bool mine = (int)threadIdx.x * 4 < a.vd;
    float M = -INFINITY, L = 0.0f, A[4] = {0.0f, 0.0f, 0.0f, 0.0f};
#pragma unroll 4
    for (int s = 0; s < n; ++s) {
        float held, fresh;
        const float2 ml = reinterpret_cast<const float2*>(a.part_ml)[at + s];
        const float4 f = mine ? *reinterpret_cast<const float4*>(acc + (size_t)s * a.vd) : make_float4(0.0f, 0.0f, 0.0f, 0.0f);
        merge_factors(M, L, ml.x, ml.y, held, fresh);
        A[0] = merged(A[0], held, f.x, fresh);
        A[1] = merged(A[1], held, f.y, fresh);
        A[2] = merged(A[2], held, f.z, fresh);
        A[3] = merged(A[3], held, f.w, fresh);
    }
    const float inv = share(a, M, L, head);
    if (!mine) return;
    float* dst = a.out + (size_t)token * a.out_stride + (size_t)head * a.vd + threadIdx.x * 4;
#pragma unroll
    for (int e = 0; e < 4; ++e) dst[e] = __fmul_rn(A[e], inv);
}

int launch_few(const F32Args& a, int batch, int max_q_len, cudaStream_t stream) {
    static OncePerDevice allowed;
    if (const int e = allow_shared_memory(attn_f32_few_kernel, 112 * 1024, allowed)) return e;
    const int st = launch_pdl(attn_f32_few_kernel, dim3(a.splits * SHARERS, a.n_kv, batch), dim3(FEW_THREADS), few_bytes(a), stream, a);
    if (st) return st;
    return launch_pdl(merge_kernel<FEW>, dim3(max_q_len * a.group, a.n_kv, batch), dim3(64), 0, stream, a);
}

template <int ROWS, int VJ>
int launch(const F32Args& a, int batch, int max_q_len, cudaStream_t stream) {
    const int q_pitch = (a.hd + KC - 1) / KC * KC + 4;
    const int smem = STAGES * stage_bytes(a) + (ROWS * q_pitch + ROWS * P_PITCH + 4 * ROWS) * (int)sizeof(float) + 2 * SPAN * 8;
    static OncePerDevice allowed;
    if (const int e = allow_shared_memory(attn_f32_kernel<ROWS, VJ>, 112 * 1024, allowed)) return e;
    const int rows = max_q_len * a.group, tiles = (rows + ROWS - 1) / ROWS;
    int st = launch_pdl(attn_f32_kernel<ROWS, VJ>, dim3(tiles * (a.splits ? a.splits : 1), a.n_kv, batch), dim3(THREADS), smem,
                        stream, a);
    if (st || !a.splits) return st;
    return launch_pdl(merge_kernel<ROWS>, dim3(rows, a.n_kv, batch), dim3(64), 0, stream, a);
}

}  // namespace

// Sizes: hd and vd multiples of 8, at most 256; all rows and strides whole 16-byte pieces.  splits > 0: at least as many
// spans of 128 keys as any tile of rows sees, with part_acc [tokens][heads][splits][vd] and part_ml [..][splits][2].
BROLM_API int brolm_attn_f32(const void* q, int q_stride, void* out, int out_stride, const void* cu_q, const void* kv_len,
                             const void* k, const void* v, int k_stride, int v_stride, const void* k_pages, const void* v_pages,
                             const void* page_table, int pt_stride, int ring, int page_size, int n_kv, int group, int hd, int vd,
                             float scale, float cap, int window, int chunk, const void* sink, const void* slopes,
                             const void* dist_bias, int dist_len, int batch, int max_q_len, int splits, void* part_acc,
                             void* part_ml, cudaStream_t stream) {
    if (batch <= 0 || max_q_len <= 0) return BROLM_OK;
    if (hd <= 0 || hd > 256 || vd <= 0 || vd > 256 || group <= 0 || n_kv <= 0 || splits < 0) return BROLM_ERR_BAD_SIZE;
    if (hd % 8 || vd % 8 || q_stride % 4 || ((uintptr_t)q & 15)) return BROLM_ERR_ALIGNMENT;
    if (splits && (!part_acc || !part_ml)) return BROLM_ERR_BAD_SIZE;
    if (dist_bias && dist_len <= 0) return BROLM_ERR_BAD_SIZE;
    if (batch > 65535 || n_kv > 65535) return BROLM_ERR_TOO_LARGE;
    if (k_pages) {
        if (ring <= 0 || page_size <= 0 || page_size % 32 != 0 || ring % page_size != 0) return BROLM_ERR_BAD_SIZE;
    } else if (!k || !v || k_stride % 4 || v_stride % 4 || ((uintptr_t)k & 15) || ((uintptr_t)v & 15)) {
        return BROLM_ERR_ALIGNMENT;
    }
    F32Args a;
    a.q = (const float*)q; a.out = (float*)out; a.q_stride = q_stride; a.out_stride = out_stride;
    a.cu_q = (const int32_t*)cu_q; a.kv_len = (const int32_t*)kv_len;
    a.k = (const float*)k; a.v = (const float*)v; a.k_stride = k_stride; a.v_stride = v_stride;
    a.k_pages = (const float*)k_pages; a.v_pages = (const float*)v_pages; a.page_table = (const int32_t*)page_table;
    a.pt_stride = pt_stride; a.ring = ring; a.page_size = page_size;
    a.n_kv = n_kv; a.group = group; a.hd = hd; a.vd = vd; a.scale = scale; a.cap = cap; a.window = window; a.chunk = chunk;
    a.sink = (const float*)sink; a.slopes = (const float*)slopes; a.dist_bias = (const float*)dist_bias; a.dist_len = dist_len;
    a.splits = splits; a.part_acc = (float*)part_acc; a.part_ml = (float*)part_ml;
    // a prompt's keys are its tokens: with few of them a block takes less of an SM (16 prompts of 20 tokens, 32 heads of 128 on
    // 8 kv heads, 384 blocks: 27 us where two share an SM)
    a.max_parts = k_pages || max_q_len > 64 || (long long)max_q_len * group <= 8 ? 4 : max_q_len > 32 ? 2 : 1;
    if ((long long)max_q_len * group <= 8) {
        // us, a block a span / a cluster a span, by spans (of all sequences and kv heads): heads of 256, two a kv head, 64 28.1 /
        // 12.5, 128 31.2 / 20.1, 256 36.2 / 35.1, 512 64.6 / 68.2, 1,024 97.7 / 122; heads of 64, one, 128 15.9 / 11.9, 256 19.5 /
        // 18.6, 512 29.8 / 30.7, 1,024 44.0 / 53.8; heads of 16, two, 128 14.8 / 11.2, 256 16.5 / 17.2, 1,024 37.5 / 49.2
        if (splits && (long long)splits * n_kv * batch <= device_sm_count()) return launch_few(a, batch, max_q_len, stream);
        if (vd <= 128) return launch<8, 1>(a, batch, max_q_len, stream);
        return launch<8, 2>(a, batch, max_q_len, stream);
    }
    // Shared spans that give an SM hardly more than one block of 32 rows go in tiles of 16: two blocks an SM hide each other's
    // waits (us in tiles of 32 / of 16, prompts of 160 to 400 tokens: 8 heads of 256 on 4 kv heads 59 to 62 / 47 to 50, 8 of 128
    // on 4 38 to 40 / 32 to 34, 16 of 128 on 4 39.6 / 33.3, 4 of 64 on 2 25 to 27 / 19 to 23).  Beyond, tiles of 16 lose with heads
    // of 256 (400 tokens, 8 on 4: 63 / 86; 300, 16 on 8: 66 / 94) and gain up to 15 % or lose up to 10 with smaller ones.
    const long long tiles = ((long long)max_q_len * group + 31) / 32;
    if (splits && 2 * tiles * n_kv * batch * (splits + 1) <= 5LL * device_sm_count()) {
        if (vd <= 64) return launch<16, 1>(a, batch, max_q_len, stream);
        if (vd <= 128) return launch<16, 2>(a, batch, max_q_len, stream);
        return launch<16, 4>(a, batch, max_q_len, stream);
    }
    if (vd <= 64) return launch<32, 1>(a, batch, max_q_len, stream);
    if (vd <= 128) return launch<32, 2>(a, batch, max_q_len, stream);
    return launch<32, 4>(a, batch, max_q_len, stream);
}
