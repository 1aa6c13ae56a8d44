// Attention on the CUDA cores over the paged cache for head sizes 64 and 128, in tiles of 64 keys: the true 32-bit path (causal,
// grouped heads, with an optional window or chunked visibility), and the decode steps in bfloat16 whose options no tensor-core kernel
// has (kept first keys, heads whose weights are mixed).  Scores, softmax and sums are float; key tiles, splits and the
// order of every sum are fixed in absolute position, so in float32 a query's bits depend on nothing but its own sequence (and on
// whether that brings one token to the step or more).
// (attention_simt.cu takes every other size and option.)
//
//  * decode: a CTA takes one (sequence, key/value head, split), up to eight heads of the group, and tiles of 64 keys.  Bound by the
//    chain of lookups, one trip
//    to memory, scores, softmax and values: all of a tile's keys and values are asked for at once, and with splits of 64 keys
//    (attention.py) a CTA has one tile.
//  * prompts: a CTA takes up to 64 rows (query, head of the group) and walks the keys in tiles of 64; scores and value sums
//    are register tiles of 8 x 4 and 8 x HD/16 per thread.  Bound by the FMA pipes and what shared memory delivers.
#include <math.h>

#include "attention.cuh"

namespace fd {

namespace {

constexpr int FT = 64;             // keys per tile
constexpr int FTHREADS = 128;
constexpr int GDEC = 8;            // most query heads of a CTA of the decode kernel; larger groups are cut (p.kv_div pieces)

__device__ __forceinline__ void cp16(void* dst, const void* src, bool on) {
    const unsigned d = (unsigned)__cvta_generic_to_shared(dst);
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" :: "r"(d), "l"(src), "r"(on ? 16 : 0) : "memory");
}
__device__ __forceinline__ void commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N> __device__ __forceinline__ void wait() { asm volatile("cp.async.wait_group %0;" :: "n"(N) : "memory"); }

// The rows in the key and value pools of the tile's FT tokens from t0 on (-1: outside the visible keys or not in the cache), by the
// first FT threads.  vhead: the pool head of the values.
__device__ __forceinline__ void tile_rows(const AttnParams& p, int slot, int kvh, int vhead, int t0, int lo, int hi, int kf, int s_lo,
                                          int* row_s, int* vrow_s) {
    const int t = t0 + (int)threadIdx.x;
    if (threadIdx.x >= FT) return;
    int row = -1, vrow = -1;
    if ((t >= lo || (t < kf && t >= s_lo)) && t < hi) {
        const int blk = p.block_table[(size_t)slot * p.max_blocks + t / p.block_size];
        if (blk < 0 || blk >= p.num_blocks) set_status(p.status, STATUS_BAD_BLOCK);
        else {
            row = (blk * p.n_kv_pool + kvh) * p.block_size + t % p.block_size;
            vrow = (blk * p.n_kv_pool + vhead) * p.block_size + t % p.block_size;
        }
    }
    row_s[threadIdx.x] = row;
    if (vrow_s != nullptr) vrow_s[threadIdx.x] = vrow;
}

// A tile of keys (or values) to shared memory, rows LD apart; rows of -1 read as zero.  `ahead`: rows added to each.
template <typename T, int HD, int LD>
__device__ __forceinline__ void load_tile(T* dst, const T* pool, const int* row_s, int ahead = 0) {
    constexpr int E = 16 / sizeof(T), CH = HD / E;
#pragma unroll 8
    for (int c = threadIdx.x; c < FT * CH; c += FTHREADS) {
        const int t = c / CH, e = (c % CH) * E, row = row_s[t];
        cp16(dst + t * LD + e, row >= 0 ? pool + ((size_t)row + ahead) * HD + e : pool, row >= 0);
    }
}

// 16 bytes of a row, and four values of one, as float.
__device__ __forceinline__ void chunk16(const float* p, float v[4]) { *reinterpret_cast<float4*>(v) = *reinterpret_cast<const float4*>(p); }
__device__ __forceinline__ void chunk16(const __nv_bfloat16* p, float v[8]) {
    const uint4 r = *reinterpret_cast<const uint4*>(p);
    const __nv_bfloat162* h = reinterpret_cast<const __nv_bfloat162*>(&r);
#pragma unroll
    for (int e = 0; e < 4; ++e) { const float2 f = __bfloat1622float2(h[e]); v[2 * e] = f.x; v[2 * e + 1] = f.y; }
}
__device__ __forceinline__ float4 four(const float* p) { return *reinterpret_cast<const float4*>(p); }
__device__ __forceinline__ float4 four(const __nv_bfloat16* p) {
    const uint2 r = *reinterpret_cast<const uint2*>(p);
    const float2 a = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&r.x)), b = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&r.y));
    return make_float4(a.x, a.y, b.x, b.y);
}
template <typename T> __device__ __forceinline__ float exp_for(float x) { return sizeof(T) == 4 ? expf(x) : __expf(x); }

// VR value heads (1, or all of the pool's: mixed heads), GM query heads per key head at most.
template <typename T, int HD, int VR>
constexpr int decode_smem() {
    return (FT * (HD + 16 / (int)sizeof(T)) + VR * FT * HD) * (int)sizeof(T) + (GDEC * HD + FT * GDEC + 3 * GDEC) * (int)sizeof(float);
}

template <typename T, int HD, int VR, int GM>
__global__ void __launch_bounds__(FTHREADS)
attn_rows_decode_kernel(const AttnParams p) {
    constexpr int E = 16 / sizeof(T), LD = HD + E, DW = HD / 4;      // DW: threads that hold a row's dims, four each
    extern __shared__ __align__(16) unsigned char sm_raw[];
    T* k_s = reinterpret_cast<T*>(sm_raw);                   // [FT][LD]
    T* v_s = k_s + FT * LD;                                  // [VR][FT][HD]
    float* q_s = reinterpret_cast<float*>(v_s + VR * FT * HD);       // [GDEC][HD]
    float* p_s = q_s + GDEC * HD;                            // [FT][GDEC]: scores, then weights
    float* m_s = p_s + FT * GDEC;                            // [GDEC] running maximum, sum, factor of the tile before
    float* l_s = m_s + GDEC;
    float* a_s = l_s + GDEC;
    __shared__ int row_s[FT], vrow_s[FT];
    // pieces of a group of more than GDEC heads are as equal as whole heads allow: the last one may have fewer
    // (heads whose weights are mixed are not cut)
    const int split = blockIdx.x, kvh = VR > 1 ? blockIdx.y : blockIdx.y / p.kv_div, per = VR > 1 ? p.G : (p.G + p.kv_div - 1) / p.kv_div, b = blockIdx.z;
    const int g0 = VR > 1 ? 0 : (blockIdx.y - kvh * p.kv_div) * per, G = VR > 1 ? p.G : min(per, p.G - g0), head = kvh * p.G + g0;
    const int slot = p.row_slot[b];
    if (slot < 0 || p.row_q_len[b] != 1) return;
    const int tok = p.row_q_start[b], pos = p.row_ctx_len[b];
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    int lo = p.window > 0 ? max(0, pos - p.window + 1) : 0, hi = pos + 1;
    if (p.chunk > 0) lo = max(lo, (pos / p.chunk) * p.chunk);
    int kf = p.window > 0 ? min(p.keep_first, lo) : 0, s_lo = 0;     // kept first keys before the window: [s_lo, kf)
    if (p.n_splits > 1) {
        s_lo = split * p.split_len;
        lo = max(lo, s_lo);
        hi = min(hi, (split + 1) * p.split_len);
        kf = min(kf, hi);
    }
    if (kf <= s_lo) kf = 0;
    const size_t head0 = (size_t)tok * p.n_q + head;         // the CTA's first (token, head), and that of its partial sums
    const size_t part0 = p.row_kind == ROWS_SINGLE ? (size_t)b * p.n_q + head : head0;
    if (lo >= hi && kf == 0) {                               // (a split without keys: only its sums are looked at)
        if (p.n_splits > 1 && tid < G * VR) p.part_l[(part0 * VR + tid) * p.n_splits + split] = 0.f;
        return;
    }
    const T* qg = static_cast<const T*>(p.q) + head0 * HD;
    for (int e = tid; e < G * HD; e += FTHREADS) q_s[e] = to_float(qg[e]) * p.scale;
    if (tid < GDEC) { m_s[tid] = -INFINITY; l_s[tid] = 0.f; }
    float acc[VR][GM][4];
#pragma unroll
    for (int j = 0; j < VR; ++j)
#pragma unroll
        for (int g = 0; g < GM; ++g) acc[j][g][0] = acc[j][g][1] = acc[j][g][2] = acc[j][g][3] = 0.f;
    constexpr int KS = FTHREADS / DW;                        // shares of a tile's keys in the value phase
    const int d4 = (tid % DW) * 4, share = tid / DW;
    const int kf_end = (kf + FT - 1) / FT * FT, lo_tile = lo / FT * FT;

    for (int t0 = kf > 0 ? s_lo / FT * FT : lo_tile; t0 < hi; t0 += FT) {
        if (t0 >= kf_end && t0 < lo_tile) t0 = lo_tile;      // nothing visible between the kept keys and the window
        if (t0 >= hi) break;
        __syncthreads();                                     // the tile before is consumed
        tile_rows(p, slot, kvh, VR > 1 ? 0 : kvh, t0, lo, hi, kf, s_lo, row_s, vrow_s);
        __syncthreads();
        load_tile<T, HD, LD>(k_s, static_cast<const T*>(p.k_pool), row_s);
        commit();
#pragma unroll
        for (int j = 0; j < VR; ++j) load_tile<T, HD, HD>(v_s + j * FT * HD, static_cast<const T*>(p.v_pool), vrow_s, j * p.block_size);
        commit();
        wait<1>();
        __syncthreads();
        // scores: a thread has one key and every second head
        {
            const int key = tid & (FT - 1), h0 = tid / FT, t = t0 + key;
            float s[GM / 2];
#pragma unroll
            for (int i = 0; i < GM / 2; ++i) s[i] = 0.f;
            const T* kr = k_s + key * LD;
#pragma unroll 4
            for (int e = 0; e < HD; e += E) {
                float kc[E];
                chunk16(kr + e, kc);
#pragma unroll
                for (int i = 0; i < GM / 2; ++i) {
                    if (h0 + 2 * i >= G) break;
#pragma unroll
                    for (int c = 0; c < E; c += 4) {
                        const float4 q4 = *reinterpret_cast<const float4*>(q_s + (h0 + 2 * i) * HD + e + c);
                        s[i] = fmaf(q4.x, kc[c], s[i]); s[i] = fmaf(q4.y, kc[c + 1], s[i]);
                        s[i] = fmaf(q4.z, kc[c + 2], s[i]); s[i] = fmaf(q4.w, kc[c + 3], s[i]);
                    }
                }
            }
            const bool valid = (t >= lo || (t < kf && t >= s_lo)) && t < hi;
#pragma unroll
            for (int i = 0; i < GM / 2; ++i) {
                if (p.softcap > 0.f) s[i] = p.softcap * tanhf(s[i] / p.softcap);
                if (h0 + 2 * i < G) p_s[key * GDEC + h0 + 2 * i] = valid ? s[i] : -INFINITY;
            }
        }
        __syncthreads();
        for (int g = warp; g < G; g += FTHREADS / 32) {      // softmax: a warp per head, two keys per lane
            const float s0 = p_s[lane * GDEC + g], s1 = p_s[(lane + 32) * GDEC + g];
            const float m_old = m_s[g], m_new = fmaxf(m_old, warp_max(fmaxf(s0, s1)));
            const float e0 = s0 == -INFINITY ? 0.f : exp_for<T>(s0 - m_new), e1 = s1 == -INFINITY ? 0.f : exp_for<T>(s1 - m_new);
            const float sum = warp_sum(e0 + e1);
            p_s[lane * GDEC + g] = e0;
            p_s[(lane + 32) * GDEC + g] = e1;
            __syncwarp();
            if (lane == 0) {
                const float alpha = m_old == -INFINITY ? 0.f : exp_for<T>(m_old - m_new);
                a_s[g] = alpha;
                l_s[g] = l_s[g] * alpha + sum;
                m_s[g] = m_new;
            }
        }
        wait<0>();
        __syncthreads();
#pragma unroll
        for (int g = 0; g < GM; ++g) {
            if (g >= G) break;
            const float al = a_s[g];
#pragma unroll
            for (int j = 0; j < VR; ++j) { acc[j][g][0] *= al; acc[j][g][1] *= al; acc[j][g][2] *= al; acc[j][g][3] *= al; }
        }
#pragma unroll 4
        for (int t = share * (FT / KS); t < (share + 1) * (FT / KS); ++t) {
            float w[GM];
#pragma unroll
            for (int g = 0; g < GM; g += 4) *reinterpret_cast<float4*>(w + g) = *reinterpret_cast<const float4*>(p_s + t * GDEC + g);
#pragma unroll
            for (int j = 0; j < VR; ++j) {
                const float4 v4 = four(v_s + (j * FT + t) * HD + d4);
#pragma unroll
                for (int g = 0; g < GM; ++g) {
                    if (g >= G) break;
                    acc[j][g][0] = fmaf(w[g], v4.x, acc[j][g][0]); acc[j][g][1] = fmaf(w[g], v4.y, acc[j][g][1]);
                    acc[j][g][2] = fmaf(w[g], v4.z, acc[j][g][2]); acc[j][g][3] = fmaf(w[g], v4.w, acc[j][g][3]);
                }
            }
        }
    }
    // the shares' sums, added in order (through the keys' and values' place), one value head at a time
    float* x_s = reinterpret_cast<float*>(sm_raw);           // [KS][GM][HD]
    static_assert(KS * GM * HD * 4 <= (FT * LD + VR * FT * HD) * (int)sizeof(T), "the sums take the tiles' place");
#pragma unroll
    for (int j = 0; j < VR; ++j) {
        __syncthreads();
#pragma unroll
        for (int g = 0; g < GM; ++g) {
            if (g >= G) break;
            *reinterpret_cast<float4*>(x_s + (share * GM + g) * HD + d4) = make_float4(acc[j][g][0], acc[j][g][1], acc[j][g][2], acc[j][g][3]);
        }
        __syncthreads();
        for (int c = tid; c < G * DW; c += FTHREADS) {
            const int g = c / DW, e = (c % DW) * 4;
            float4 o = *reinterpret_cast<const float4*>(x_s + g * HD + e);
#pragma unroll
            for (int s = 1; s < KS; ++s) {
                const float4 x = *reinterpret_cast<const float4*>(x_s + (s * GM + g) * HD + e);
                o.x += x.x; o.y += x.y; o.z += x.z; o.w += x.w;
            }
            if (p.n_splits > 1) {
                const size_t pi = ((part0 + g) * VR + j) * p.n_splits + split;
                if (e == 0) { p.part_m[pi] = m_s[g]; p.part_l[pi] = l_s[g]; }
                *reinterpret_cast<float4*>(p.part_acc + pi * HD + e) = o;
                continue;
            }
            float l = l_s[g], f = 1.f;
            if (p.sink != nullptr) {                         // one more term in the denominator: exp(sink), no key, no value
                const float sk = p.sink[head + g], m2 = fmaxf(m_s[g], sk);
                f = expf(m_s[g] - m2);
                l = l * f + expf(sk - m2);
            }
            const float inv = l > 0.f ? f * p.out_scale / l : 0.f;
            const size_t at = (size_t)tok * p.out_ld + ((head + g) * VR + j) * HD + e;
            if (sizeof(T) == 4 || p.out_f32)
                *reinterpret_cast<float4*>(static_cast<float*>(p.out) + at) = make_float4(o.x * inv, o.y * inv, o.z * inv, o.w * inv);
            else {
                const __nv_bfloat162 a = __floats2bfloat162_rn(o.x * inv, o.y * inv), c2 = __floats2bfloat162_rn(o.z * inv, o.w * inv);
                *reinterpret_cast<uint2*>(static_cast<__nv_bfloat16*>(p.out) + at) =
                    make_uint2(*reinterpret_cast<const uint32_t*>(&a), *reinterpret_cast<const uint32_t*>(&c2));
            }
        }
    }
}

// Rows (query, head) per CTA of the prompt kernel: 64, eight per thread, or 8 in steps whose rows of a group are no more (a few
// queries of heads without groups: 2 queries of 8 heads of 128 12.0 us in the general kernel, 13.9 in tiles of 64 rows, 7.0 in tiles of 8).
// A row's sums are the same in either.
constexpr int PR_MAX = 64;

template <int HD, int TM>
constexpr int prompt_smem_floats() { return 8 * TM * (HD + 4) + FT * (HD + 4) + FT * HD; }

template <int HD, int TM>
__global__ void __launch_bounds__(FTHREADS, 2)
attn_f32_prompt_kernel(const AttnParams p) {
    constexpr int PR = 8 * TM;
    constexpr int LD = HD + 4, PLD = FT + 4, TN = 4, TV = HD / 16;             // a thread: TM rows, 4 keys, TV dims
    static_assert(PR * PLD <= FT * LD, "the weights take the keys' place");
    extern __shared__ __align__(16) float sm[];
    float* q_s = sm;                                         // [PR][LD]
    float* k_s = q_s + PR * LD;                              // [FT][LD]; then the weights, [PR][PLD]
    float* p_s = k_s;
    float* v_s = k_s + FT * LD;                              // [FT][HD]
    __shared__ int row_s[FT];
    const int b = blockIdx.z, kvh = blockIdx.y, tile = gridDim.x - 1 - blockIdx.x;      // the longest chains first
    const int slot = p.row_slot[b];
    if (slot < 0) return;
    const int q_len = p.row_q_len[b], G = p.G, QT = p.QT;
    if (tile * QT >= q_len || (p.row_kind == ROWS_LONGER && q_len == 1)) return;
    const int nq = min(QT, q_len - tile * QT), R = nq * G;
    const int tok0 = p.row_q_start[b] + tile * QT, p_first = p.row_ctx_len[b] + tile * QT;
    int lo = p.window > 0 ? max(0, p_first - p.window + 1) : 0;
    if (p.chunk > 0) lo = max(lo, (p_first / p.chunk) * p.chunk);
    const int hi = p_first + nq;
    const int tid = threadIdx.x, tx = tid & 15, ty = tid >> 4;
    // queries of this CTA, scaled (rows beyond R are zero)
    for (int c = tid; c < PR * (HD / 4); c += FTHREADS) {
        const int r = c / (HD / 4), e = (c % (HD / 4)) * 4;
        float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
        if (r < R) {
            const int qi = r / G, g = r - qi * G;
            v = *reinterpret_cast<const float4*>(static_cast<const float*>(p.q) + ((size_t)(tok0 + qi) * p.n_q + kvh * G + g) * HD + e);
        }
        *reinterpret_cast<float4*>(q_s + r * LD + e) = make_float4(v.x * p.scale, v.y * p.scale, v.z * p.scale, v.w * p.scale);
    }
    float m_run[TM], l_run[TM], acc[TM][TV];
    int qpos[TM], first[TM];                                 // position of a row's query, first key it sees
#pragma unroll
    for (int i = 0; i < TM; ++i) {
        m_run[i] = -INFINITY; l_run[i] = 0.f;
        const int r = i * (PR / TM) + ty;
        qpos[i] = r < R ? p_first + r / G : -1;
        first[i] = p.window > 0 ? max(0, qpos[i] - p.window + 1) : 0;
        if (p.chunk > 0) first[i] = max(first[i], (qpos[i] / p.chunk) * p.chunk);
#pragma unroll
        for (int j = 0; j < TV; ++j) acc[i][j] = 0.f;
    }
    for (int t0 = lo / FT * FT; t0 < hi; t0 += FT) {
        __syncthreads();                                     // the tile before is consumed (first time: nothing yet)
        tile_rows(p, slot, kvh, kvh, t0, lo, hi, 0, 0, row_s, nullptr);
        __syncthreads();
        load_tile<float, HD, LD>(k_s, static_cast<const float*>(p.k_pool), row_s);
        commit();
        load_tile<float, HD, HD>(v_s, static_cast<const float*>(p.v_pool), row_s);
        commit();
        wait<1>();
        __syncthreads();
        float s[TM][TN];
#pragma unroll
        for (int i = 0; i < TM; ++i)
#pragma unroll
            for (int j = 0; j < TN; ++j) s[i][j] = 0.f;
#pragma unroll 2
        for (int e = 0; e < HD; e += 4) {
            float4 k4[TN];
#pragma unroll
            for (int j = 0; j < TN; ++j) k4[j] = *reinterpret_cast<const float4*>(k_s + (j * (FT / TN) + tx) * LD + e);
#pragma unroll
            for (int i = 0; i < TM; ++i) {
                const float4 q4 = *reinterpret_cast<const float4*>(q_s + (i * (PR / TM) + ty) * LD + e);
#pragma unroll
                for (int j = 0; j < TN; ++j) {
                    s[i][j] = fmaf(q4.x, k4[j].x, s[i][j]); s[i][j] = fmaf(q4.y, k4[j].y, s[i][j]);
                    s[i][j] = fmaf(q4.z, k4[j].z, s[i][j]); s[i][j] = fmaf(q4.w, k4[j].w, s[i][j]);
                }
            }
        }
        __syncthreads();                                     // the keys are read: their place takes the weights
#pragma unroll
        for (int i = 0; i < TM; ++i) {
            float mx = -INFINITY;
#pragma unroll
            for (int j = 0; j < TN; ++j) {
                const int t = t0 + j * (FT / TN) + tx;
                if (t < first[i] || t > qpos[i]) s[i][j] = -INFINITY;
                mx = fmaxf(mx, s[i][j]);
            }
#pragma unroll
            for (int o = 8; o > 0; o >>= 1) mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, o));
            const float m_new = fmaxf(m_run[i], mx);
            float alpha = 1.f, sum = 0.f;
            if (m_new != -INFINITY) {
                alpha = expf(m_run[i] - m_new);
#pragma unroll
                for (int j = 0; j < TN; ++j) { s[i][j] = expf(s[i][j] - m_new); sum += s[i][j]; }
            } else {
#pragma unroll
                for (int j = 0; j < TN; ++j) s[i][j] = 0.f;
            }
#pragma unroll
            for (int o = 8; o > 0; o >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, o);
            l_run[i] = l_run[i] * alpha + sum;
            m_run[i] = m_new;
#pragma unroll
            for (int j = 0; j < TN; ++j) p_s[(i * (PR / TM) + ty) * PLD + j * (FT / TN) + tx] = s[i][j];
#pragma unroll
            for (int j = 0; j < TV; ++j) acc[i][j] *= alpha;
        }
        wait<0>();
        __syncthreads();
        for (int t = 0; t < FT; t += 4) {
            float4 w4[TM];
#pragma unroll
            for (int i = 0; i < TM; ++i) w4[i] = *reinterpret_cast<const float4*>(p_s + (i * (PR / TM) + ty) * PLD + t);
#pragma unroll
            for (int u = 0; u < 4; ++u) {
                float v[TV];
#pragma unroll
                for (int j = 0; j < TV; j += 4)
                    *reinterpret_cast<float4*>(v + j) = *reinterpret_cast<const float4*>(v_s + (t + u) * HD + (j / 4) * 64 + tx * 4);
#pragma unroll
                for (int i = 0; i < TM; ++i) {
                    const float w = u == 0 ? w4[i].x : (u == 1 ? w4[i].y : (u == 2 ? w4[i].z : w4[i].w));
#pragma unroll
                    for (int j = 0; j < TV; ++j) acc[i][j] = fmaf(w, v[j], acc[i][j]);
                }
            }
        }
    }
#pragma unroll
    for (int i = 0; i < TM; ++i) {
        const int r = i * (PR / TM) + ty;
        if (r >= R) continue;
        const int qi = r / G, g = r - qi * G;
        const float inv = l_run[i] > 0.f ? p.out_scale / l_run[i] : 0.f;
        float* o = static_cast<float*>(p.out) + (size_t)(tok0 + qi) * p.out_ld + (kvh * G + g) * HD;
#pragma unroll
        for (int j = 0; j < TV; j += 4)
            *reinterpret_cast<float4*>(o + (j / 4) * 64 + tx * 4) =
                make_float4(acc[i][j] * inv, acc[i][j + 1] * inv, acc[i][j + 2] * inv, acc[i][j + 3] * inv);
    }
}

template <typename KernelT>
int configure(KernelT k, int smem, bool& done) {
    if (done) return 0;
    const cudaError_t e = cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
    if (e != cudaSuccess) return fail(-3, "attention: cannot get %d bytes of shared memory: %s", smem, cudaGetErrorString(e));
    done = true;
    return 0;
}

template <typename T, int HD, int VR, int GM>
int launch_decode(const AttnParams& p, int n_rows, cudaStream_t stream) {
    constexpr int smem = decode_smem<T, HD, VR>();
    static bool done = false;
    const int rc = configure(attn_rows_decode_kernel<T, HD, VR, GM>, smem, done);
    if (rc != 0) return rc;
    attn_rows_decode_kernel<T, HD, VR, GM><<<dim3(p.n_splits, p.n_kv * p.kv_div, n_rows), FTHREADS, smem, stream>>>(p);
    return check_launch("attention_rows_decode");
}

template <int HD, int TM>
int launch_prompt(AttnParams p, int n_rows, int max_q_len, cudaStream_t stream) {
    constexpr int smem = prompt_smem_floats<HD, TM>() * (int)sizeof(float);
    static bool done = false;
    const int rc = configure(attn_f32_prompt_kernel<HD, TM>, smem, done);
    if (rc != 0) return rc;
    p.QT = 8 * TM / p.G < max_q_len ? 8 * TM / p.G : max_q_len;
    attn_f32_prompt_kernel<HD, TM><<<dim3((max_q_len + p.QT - 1) / p.QT, p.n_kv, n_rows), FTHREADS, smem, stream>>>(p);
    return check_launch("attention_f32_prompt");
}

template <int HD>
int launch_f32(const AttnParams& p0, int n_rows, int max_q_len, cudaStream_t stream) {
    AttnParams p = p0;
    // Which kernel takes a row depends on its group and on how many tokens it brings, never on the splits: those follow from the
    // batch's longest sequence, and a row's bits must not.
    if (p.G > PR_MAX) return 1;
    if (max_q_len == 1) {
        p.kv_div = (p.G + GDEC - 1) / GDEC;
        return p.n_kv * p.kv_div <= 65535 ? launch_decode<float, HD, 1, GDEC>(p, n_rows, stream) : 1;
    }
    if (p.n_splits > 1) return 1;
    return (long long)max_q_len * p.G <= 8 ? launch_prompt<HD, 1>(p, n_rows, max_q_len, stream) : launch_prompt<HD, 8>(p, n_rows, max_q_len, stream);
}

}  // namespace

// Heads of 64 or 128 for keys and values alike, no cap, kept first keys, keyless term, repeated heads or 16-bit output; output rows
// 16-byte aligned.  Returns 1 if it does not take the sizes.
int launch_attn_f32(const AttnParams& p, int n_rows, int max_q_len, cudaStream_t stream) {
    if (p.d != p.dv || p.v_ld != p.dv || p.kv_div != 1 || p.softcap > 0.f || (p.keep_first > 0 && p.window > 0) ||
        p.sink != nullptr || p.v_rep != 1 || (uintptr_t)p.out % 16 != 0 || p.out_ld % 4 != 0)
        return 1;
    if (p.d == 128) return launch_f32<128>(p, n_rows, max_q_len, stream);
    if (p.d == 64) return launch_f32<64>(p, n_rows, max_q_len, stream);
    return 1;
}

// bfloat16 decode steps with the options that the tensor-core kernel has not: kept first keys, and weights applied to every value
// head for the caller to mix.  The number of value heads and the most query heads of a group are the kernel's register tile (value heads x
// query heads x 4 sums a thread, 64 at most), so it is built for 2 and 4 value heads under groups of up to 4, which
// the sizes at hand have (33 us in the general kernel, 13 here), and returns 1 for others: three or eight value heads, larger groups.
int launch_attn_rows_ext(const AttnParams& p, int n_rows, cudaStream_t stream) {
    if (p.d != p.dv || p.v_ld != p.dv || p.kv_div != 1 || (uintptr_t)p.out % 16 != 0 || p.out_ld % 4 != 0) return 1;
    if (p.v_rep > 1 && p.v_rep != p.n_kv_pool) return 1;
    typedef __nv_bfloat16 bf16;
    if (p.d == 128) {
        if (p.v_rep == 1 && p.G <= 8) return launch_decode<bf16, 128, 1, 8>(p, n_rows, stream);
        if (p.v_rep == 2 && p.G <= 4) return launch_decode<bf16, 128, 2, 4>(p, n_rows, stream);
        if (p.v_rep == 4 && p.G <= 4) return launch_decode<bf16, 128, 4, 4>(p, n_rows, stream);
    } else if (p.d == 64) {
        if (p.v_rep == 1 && p.G <= 8) return launch_decode<bf16, 64, 1, 8>(p, n_rows, stream);
        if (p.v_rep == 2 && p.G <= 4) return launch_decode<bf16, 64, 2, 4>(p, n_rows, stream);
        if (p.v_rep == 4 && p.G <= 4) return launch_decode<bf16, 64, 4, 4>(p, n_rows, stream);
    }
    return 1;
}

}  // namespace fd
