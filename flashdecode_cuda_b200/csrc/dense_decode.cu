// A decode step of a dense model (one new token of up to 24 sequences, bfloat16) in ONE kernel: every layer's norms, q/k/v projection
// with rotation and cache append, attention over the paged cache, output projection and gated feed-forward.
//
// What bounds it.  The step reads every weight once, so HBM does: 14.3 us per layer at the 1.5B sizes.  As seven kernels per layer it took
// 42 us (one sequence): each kernel starts its loads only when the one before has drained, and its own last reductions and first
// trips to memory leave HBM idle.  Here one persistent CTA per SM copies ITS share of all weights, layer after layer, through one ring
// of shared-memory stages: weights depend on nothing, so the ring runs ahead through every exchange of activations.  With
// everything but the ring left out a layer takes 14.0 us; what remains on top is the chain of exchanges below.  Measured, us of a replayed
// step by its layers (head and sampler included), parts / one kernel: 1.5B sizes, 1 sequence of 1,300 tokens 41.3 / 30.8, 2 of 1,500 43.9 /
// 35.5, 8 of 2,200 47.2 / 42.2, 16 of 600 52.4 / 45.2, 24 of 1,200 67.0 / 58.8; 7B 1 of 1,800 103.4 / 89.2, 8 of 1,800 108.2 / 106.0, of 1,100
// to 2,600 113.0 / 109.1; 14B 1 of 1,000 127.5 / 99.4, 8 of 1,000 134.9 / 125.0.  Counters: HBM reads 1.008 of the matrices, keys and values.
//
// What is exchanged, and how.  A layer is a chain of exchanges through L2: normed stream -> q, k, v -> partial attention -> attention
// -> normed stream -> gated activations -> partial sums -> stream.  Each 32-bit word (two bfloat16, or a float) travels in an 8-byte
// packet with the number of its layer, written and read whole; the reader reads until the number is the awaited one.  There is no
// fence, no barrier over the grid and no second trip for the data: one exchange is one write to L2 and one read (about 1 us).  A buffer is
// written again a layer later, when (through the chain) every reader has handed on what it made of the words, so one buffer of
// each kind is enough.  Numbers go on from launch to launch (`ctrl`), so nothing has to be cleared.
//
// The norm has no phase of its own: the owner of 16 elements of the stream keeps them (float) in its shared memory for the whole
// step and hands out bfloat16(r w) and the sum of r^2; the product's epilogue multiplies by 1 / rms.  One rounding to bfloat16, as
// with the norm before the product.
//
// Split.  Weight rows in tiles of 16 (the M side of mma.sync.m16n8k16: at most 24 rows of x cannot feed a 128-row tcgen05 tile
// from a matrix that is read once), in stages of 16 rows x 768 or 1,024 k, one copy each (3-D tensor map, 128-byte swizzle); the eight
// consumer warps take 32 k of a stage in turn, the warps' sums meet in shared memory, where one of three finishing warps takes them:
// what becomes of a tile's sums passes beside the next tiles.  The down projection has few rows and a long k: its k is cut into S
// slices and `tp` row tiles share a CTA so that tiles x slices fill the grid (dd_plan), the partial sums go to the tile's owner in
// packets.  Keys and values go from global memory straight to registers as MMA fragments, the first tile before the queries arrive;
// a row's keys in as many splits of at least 128 as are its share of the grid.
//
// No local memory.  Beside 227 KB of shared memory an SM has some 20 KB of L1, and every word of a stack that 384 threads share goes
// to L2: with 100 to 600 bytes of stack a thread (arguments by reference to functions that were not inlined, arrays that were filled
// conditionally) a layer took 35 to 52 us instead of 29.  So everything is inlined, loops over phases keep one copy of the
// code, and batches of loads have a fixed number (beyond the end: an earlier one once more).
//
// Waits: on mbarriers and on packets, all bounded (fd_tc_test_hook's limit does for both): a wait that runs out sets the abort flag
// of its CTA and STATUS_WAIT_TIMEOUT, and everything after it goes on without waiting.  Where a warp votes on what its lanes saw, the lanes
// give up together.  The launch is cooperative, so that all CTAs are on the GPU together or the launch is refused.
#include <string.h>

#include <type_traits>

#include "dense_step.cuh"
#include "mma_utils.cuh"
#include "tcgen05.cuh"

// A decode step: the stream [M, hidden], the index arrays, the exchange memory (zeroed once, fd_dense_decode_plan says how much), the
// cache's pools by group and the rotation tables by position.
struct FdDenseDecode {
    float* resid;
    const int *tok_pos, *row_slot, *row_ctx_len;
    int* status;
    cudaStream_t stream;
    void* exchange;
    long long M, num_blocks, block_size;
    char *k_base[8], *v_base[8];
    const int* table[8];
    long long k_stride[8], v_stride[8], max_blocks[8];
    const float *cos_t[4], *sin_t[4];
    long long table_len[4];
    const void* next;                    // what the step streams after this, or null, and how much of it to ask L2 for
    long long next_bytes;
};

namespace fd {

constexpr int DD_WARPS = 8, DD_CONS = DD_WARPS * 32, DD_FIN = 3;                     // consumer warps, finishing warps; and one producer
constexpr int DD_THREADS = DD_CONS + 32 + DD_FIN * 32;
constexpr int DD_LAYERS = 48;                                                       // per launch: the kernel's parameters are at most 32 KB
constexpr int DD_SPLITS = 32, DD_ROWS = 24, DD_OWN = 16, DD_CTAS = 160, DD_MAX_STAGES = 13;
constexpr int DD_FLYING = 4;                                                        // copies of a CTA under way at a time
constexpr int DD_BLOCK = 2048;                                                      // 16 rows x 64 k; a stage is kbs of them, one copy
constexpr unsigned long long DD_WAIT_NS = 2000ull * 1000 * 1000;

struct alignas(64) DdLayer {
    CUtensorMap map[4];                  // q/k/v, o, gate/up, down
    const void *norm1, *norm2, *bias;
    __nv_bfloat16 *kp, *vp;
    const int* table;
    const float *cos_t, *sin_t;
    float eps1, eps2, scale;
    int window, chunk, max_blocks, table_len, f32;      // f32: bit 0 norm1, 1 norm2, 2 bias
};

struct DdParams {
    DdLayer layer[DD_LAYERS];
    float* resid;
    const int *tok_pos, *row_slot, *row_ctx;
    int* status;
    unsigned* ctrl;                      // [0] the number that the next launch counts from, [1] CTAs that are through
    unsigned long long bs_inv;           // 2^32 / block size, rounded up: key / block size for keys x block size below 2^32
    unsigned long long *x[2], *ss[2], *q, *kv, *part, *attn, *act, *dpart;
    const unsigned char* pf_ptr;         // what the step streams next: the last CTAs ask L2 for its beginning
    unsigned long long pf_bytes, wait_ns;
    int n_layers, M, H, I, n_q, n_kv, num_blocks, block_size;
    int S, tp, n_groups, n_stages;
    int skip;                            // tests: what one CTA keeps to itself in the last layer: 1 normed stream, 2 queries, 3 attention, 4 partial sums
    int flying;                          // copies of a CTA under way at a time
    int kbs;                             // blocks of 64 k in a stage
    int splits;                          // of a row's keys, at the most
    int x_bytes;                         // shared memory for the rows of x
    short gu[DD_CTAS + 1];               // gate/up tiles of CTA c: gu[c] .. gu[c + 1]
};
static_assert(sizeof(DdParams) <= 32764, "kernel parameters");

typedef unsigned long long u64;

__device__ __forceinline__ void put(u64* p, uint32_t word, uint32_t num) {
    asm volatile("st.relaxed.gpu.global.b64 [%0], %1;" ::"l"(p), "l"((u64)num << 32 | word) : "memory");
}
__device__ __forceinline__ void put2(u64* p, uint32_t a, uint32_t b, uint32_t num) {
    asm volatile("st.relaxed.gpu.global.v2.b64 [%0], {%1, %2};" ::"l"(p), "l"((u64)num << 32 | a), "l"((u64)num << 32 | b) : "memory");
}
// a load that is issued where it stands: the compiler moves plain ones behind the waits
__device__ __forceinline__ uint4 load16(const uint4* p) {
    uint4 v;
    asm volatile("ld.global.cg.v4.u32 {%0, %1, %2, %3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "l"(p) : "memory");
    return v;
}
struct Pair { u64 a, b; };
__device__ __forceinline__ Pair get2(const u64* p) {
    Pair v;
    asm volatile("ld.relaxed.gpu.global.v2.b64 {%0, %1}, [%2];" : "=l"(v.a), "=l"(v.b) : "l"(p) : "memory");
    return v;
}
__device__ __forceinline__ bool fresh(const Pair& v, uint32_t num) { return (uint32_t)(v.a >> 32) == num && (uint32_t)(v.b >> 32) == num; }

// What a wait looks at now and then: whether another thread of the CTA has given up, and the clock.
struct DdShared;
struct Waiter {
    volatile int* abort;                          // in shared memory
    int* status;
    u64 limit;
    // Having said no it goes on saying so: where a warp looks at its words together, a lane that has given up drops out of the vote on
    // who still waits, and the lanes leave together when nobody does.
    __device__ __forceinline__ bool more(uint32_t& spins, u64& since) const {
        if ((++spins & 63) != 0) return true;
        if (!*abort) {
            const u64 now = global_ns();
            if (since == 0) since = now;
            if (now - since <= limit) return true;
            *abort = 1;
            set_status(status, STATUS_WAIT_TIMEOUT);
        }
        --spins;
        return false;
    }
    __device__ __forceinline__ bool bar(uint32_t bar, uint32_t parity) const {
        uint32_t spins = 0;
        u64 since = 0;
        for (;;) {
            uint32_t ok;
            asm volatile(
                "{\n\t.reg .pred p;\n\t"
                "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
                "selp.u32 %0, 1, 0, p;\n\t}"
                : "=r"(ok) : "r"(bar), "r"(parity) : "memory");
            if (ok) return true;
            if (!more(spins, since)) return false;
        }
    }
    // Before a warp looks at all of its words: one lane looks at one of them until it is there.  Words that are awaited are asked for by
    // every SM; with all threads at it the L2 slices that hold them had no time for anything else.
    __device__ __forceinline__ void first(const u64* p, uint32_t num, int lane) const {
        if (lane == 0) wait2(p, num);
        __syncwarp();
    }
    __device__ __forceinline__ Pair wait2(const u64* p, uint32_t num) const {
        Pair v = get2(p);
        uint32_t spins = 0;
        u64 t0 = 0;
        while (!fresh(v, num) && more(spins, t0)) v = get2(p);
        return v;
    }
};

__device__ __forceinline__ void cons_sync() { asm volatile("bar.sync 1, %0;" ::"n"(DD_CONS) : "memory"); }

struct DdShared {
    uint64_t full[DD_MAX_STAGES], empty[DD_MAX_STAGES], sums[DD_FIN], taken[DD_FIN];
    int abort;
    uint32_t base;
    int slot[DD_ROWS], pos[DD_ROWS], ctx[DD_ROWS];
    // attention: keys that row b sees from lo[b] on, cut into ns[b] splits of cut[b] keys; items of one KV head before row b
    int lo[DD_ROWS], ns[DD_ROWS], cut[DD_ROWS], before[DD_ROWS + 1];
    float inv[2][DD_ROWS];
    float m[DD_WARPS][8], l[DD_WARPS][8];
    float merge[DD_WARPS][132];
};

// the warps' sums of a tile, for each finishing warp
__host__ __device__ constexpr int dd_red_bytes(int NT) { return DD_FIN * DD_WARPS * 128 * NT * 4; }
__host__ __device__ constexpr int dd_own_bytes(int NT, int own) { return own * 128 * NT * 4; }

__device__ __forceinline__ float vec_at(const void* v, int i, bool f32) {
    return f32 ? static_cast<const float*>(v)[i] : __bfloat162float(static_cast<const __nv_bfloat16*>(v)[i]);
}

// Rows [M][units of 4 elements] of packets (row_ld packets apart) to shared memory as bfloat16 rows of `stride` bytes; B units of a thread
// on their way together (beyond the end: its first one once more).
template <int B>
__device__ __forceinline__ void load_batch(const u64* src, int row_ld, int units, int all, uint32_t inv, unsigned char* dst, int stride,
                                           uint32_t num, const Waiter& w, int i0, int lane) {
    Pair v[B];
    uint32_t from[B], to[B];
#pragma unroll
    for (int k = 0; k < B; ++k) {
        int i = i0 + k * DD_CONS;
        i = i < all ? i : min(i0, all - 1);
        const int row = __umulhi(i, inv), u = i - row * units;
        from[k] = row * row_ld + u * 2;
        to[k] = row * stride + u * 8;
    }
    uint32_t spins = 0;
    u64 since = 0;
#pragma unroll 1
    for (;;) {
#pragma unroll
        for (int k = 0; k < B; ++k) v[k] = get2(src + from[k]);
        uint32_t at = 0xffffffffu;                // the last one that is not there
#pragma unroll
        for (int k = 0; k < B; ++k) at = fresh(v[k], num) ? at : from[k];
        const uint32_t who = __ballot_sync(0xffffffffu, at != 0xffffffffu && w.more(spins, since));
        if (who == 0) break;
        // many words: one lane waits for that one; few (by a per cent or two): all look again
        if (B > 6) w.first(src + at, num, lane - (__ffs(who) - 1));
    }
#pragma unroll
    for (int k = 0; k < B; ++k) *reinterpret_cast<uint2*>(dst + to[k]) = make_uint2((uint32_t)v[k].a, (uint32_t)v[k].b);
}
__device__ __forceinline__ void load_rows(const u64* src, int row_ld, int units, int M, unsigned char* dst, int stride, uint32_t num,
                                          const Waiter& w, int tid) {
    const int all = units * M;
    const uint32_t inv = (uint32_t)((0x100000000ull + units - 1) / units);        // i / units = the high word of i * inv (i and units below 2^16)
    int i0 = tid, left = (all + DD_CONS - 1) / DD_CONS;
#pragma unroll 1
    for (; left > 6; left -= 12, i0 += 12 * DD_CONS) load_batch<12>(src, row_ld, units, all, inv, dst, stride, num, w, i0, tid & 31);
    if (left > 2) load_batch<6>(src, row_ld, units, all, inv, dst, stride, num, w, i0, tid & 31);
    else if (left > 0) load_batch<2>(src, row_ld, units, all, inv, dst, stride, num, w, i0, tid & 31);
}

// A place in the ring.
struct Place {
    uint32_t slot = 0, phase = 0;
    __device__ __forceinline__ void next(int n) {
        if (++slot == (uint32_t)n) { slot = 0; phase ^= 1; }
    }
};

// A tile of 16 weight rows over the next `nst` stages of the ring: each warp's share of the sums (32 k in turn), left in red.
// kb_n: blocks of 64 k there are from the first stage on (beyond them the stage holds zeros and x nothing).
template <int NT>
__device__ __forceinline__ void tile_sums(const DdParams& p, const Waiter& w, DdShared* sh, unsigned char* ring, Place& at, int f, uint32_t& turns,
                                          int nst, int kb_n, uint32_t x_s, int x_stride, float* red_all, int warp, int lane) {
    float acc[2][NT][4];
#pragma unroll
    for (int h = 0; h < 2; ++h)
#pragma unroll
        for (int nt = 0; nt < NT; ++nt) acc[h][nt][0] = acc[h][nt][1] = acc[h][nt][2] = acc[h][nt][3] = 0.f;
    const int arow = lane & 15;
    uint32_t b_row[NT];
#pragma unroll
    for (int nt = 0; nt < NT; ++nt) b_row[nt] = x_s + min(nt * 8 + (lane & 7), p.M - 1) * x_stride + (lane >> 3) * 16;
    const uint32_t a_row = smem_u32(ring) + arow * 128;
    const uint32_t a_sw = (lane >> 4) ^ (arow & 7);           // chunk 2 k + (lane >> 4) of the row, swizzled: (2 k) ^ a_sw
    const int units = 2 * p.kbs, left = 2 * kb_n;             // units of 32 k, dealt to the warps in turn: at most four each
#pragma unroll 1
    for (int st = 0; st < nst; ++st) {
        w.bar(s_addr(&sh->full[at.slot]), at.phase);
        __syncwarp();
        const uint32_t a_s = a_row + at.slot * p.kbs * DD_BLOCK;
        const int u1 = min(units, left - st * units);
        auto load = [&](int u, uint32_t (&a)[2][4], uint32_t (&b)[NT][4]) {
            const uint32_t a_u = a_s + (u >> 1) * DD_BLOCK;
            const int c0 = (u & 1) * 4;
            ldmatrix_x4(a_u + ((c0 ^ a_sw) << 4), a[0][0], a[0][1], a[0][2], a[0][3]);
            ldmatrix_x4(a_u + (((c0 + 2) ^ a_sw) << 4), a[1][0], a[1][1], a[1][2], a[1][3]);
#pragma unroll
            for (int nt = 0; nt < NT; ++nt) ldmatrix_x4(b_row[nt] + (st * units + u) * 64, b[nt][0], b[nt][1], b[nt][2], b[nt][3]);
        };
        auto multiply = [&](const uint32_t (&a)[2][4], const uint32_t (&b)[NT][4]) {
#pragma unroll
            for (int nt = 0; nt < NT; ++nt) {
                mma_bf16(acc[0][nt], a[0][0], a[0][1], a[0][2], a[0][3], b[nt][0], b[nt][1]);
                mma_bf16(acc[1][nt], a[1][0], a[1][1], a[1][2], a[1][3], b[nt][2], b[nt][3]);
            }
        };
        // whole stages: all fragments first, then the MMAs (a loop of load and use waits for shared memory once per unit)
        auto whole = [&](auto count) {
            constexpr int U = decltype(count)::value;
            uint32_t a[U][2][4], b[U][NT][4];
#pragma unroll
            for (int k = 0; k < U; ++k) load(warp + k * DD_WARPS, a[k], b[k]);
#pragma unroll
            for (int k = 0; k < U; ++k) multiply(a[k], b[k]);
        };
        if (u1 == 4 * DD_WARPS) whole(std::integral_constant<int, 4>());
        else if (u1 == 3 * DD_WARPS) whole(std::integral_constant<int, 3>());
        else {
#pragma unroll 1
            for (int u = warp; u < u1; u += DD_WARPS) {
                uint32_t a[2][4], b[NT][4];
                load(u, a, b);
                multiply(a, b);
            }
        }
        __syncwarp();
        if (lane == 0) mbar_arrive(s_addr(&sh->empty[at.slot]));
        at.next(p.n_stages);
    }
    // to finishing warp f (bit f of `turns`: the parity of its turn), when it has taken its tile before
    w.bar(s_addr(&sh->taken[f]), (turns >> f & 1) ^ 1);
    __syncwarp();
    turns ^= 1u << f;
    float* red = red_all + f * (DD_WARPS * NT * 128);
#pragma unroll
    for (int nt = 0; nt < NT; ++nt) {
        float* r = red + (warp * NT + nt) * 128 + (lane >> 2) * 8 + (lane & 3) * 2;
        *reinterpret_cast<float2*>(r) = make_float2(acc[0][nt][0] + acc[1][nt][0], acc[0][nt][1] + acc[1][nt][1]);
        *reinterpret_cast<float2*>(r + 64) = make_float2(acc[0][nt][2] + acc[1][nt][2], acc[0][nt][3] + acc[1][nt][3]);
    }
    __syncwarp();
    if (lane == 0) mbar_arrive(s_addr(&sh->sums[f]));
}

// A finishing thread's values of a tile: rows r = lane / 4 and r + 8, columns 8 nt + 2 (lane % 4) and the next.  [nt][column] = (row r, row r + 8)
template <int NT>
__device__ __forceinline__ void take_sums(const Waiter& w, DdShared* sh, const float* red_all, int f, uint32_t& turn, int lane, float2 (&v)[NT][2]) {
    w.bar(s_addr(&sh->sums[f]), turn);
    __syncwarp();
    turn ^= 1;
#pragma unroll
    for (int nt = 0; nt < NT; ++nt) {
        float2 lo = make_float2(0.f, 0.f), hi = make_float2(0.f, 0.f);
#pragma unroll
        for (int w = 0; w < DD_WARPS; ++w) {
            const float* s = red_all + ((f * DD_WARPS + w) * NT + nt) * 128 + lane * 2;
            const float2 a = *reinterpret_cast<const float2*>(s), b = *reinterpret_cast<const float2*>(s + 64);
            lo.x += a.x; lo.y += a.y;
            hi.x += b.x; hi.y += b.y;
        }
        v[nt][0] = make_float2(lo.x, hi.x);
        v[nt][1] = make_float2(lo.y, hi.y);
    }
    __syncwarp();
    if (lane == 0) mbar_arrive(s_addr(&sh->taken[f]));
}

// 1 / rms of every row, from the owners' sums of squares (Th of them, one per tile); by the finishing warps together
__device__ __forceinline__ void row_norms(const u64* ss, float* out, int M, int Th, int H, float eps, uint32_t num, const Waiter& w, int f, int lane) {
    constexpr int R = 3, B = 2;                   // rows and words on their way at a time
#pragma unroll 1
    for (int m0 = f; m0 < M; m0 += R * DD_FIN) {
        float sum[R] = {0.f, 0.f, 0.f};
#pragma unroll 1
        for (int tb = 0; tb < Th; tb += B * 64) {
            Pair v[R][B];
            auto word = [&](int k, int i) { return ss + (size_t)(m0 + k * DD_FIN < M ? m0 + k * DD_FIN : m0) * Th + min(tb + lane * 2 + i * 64, Th - 2); };
            uint32_t spins = 0;
            u64 since = 0;
#pragma unroll 1
            for (;;) {
                bool done = true;
#pragma unroll
                for (int k = 0; k < R; ++k)
#pragma unroll
                    for (int i = 0; i < B; ++i)
                        v[k][i] = get2(word(k, i));
#pragma unroll
                for (int k = 0; k < R; ++k)
#pragma unroll
                    for (int i = 0; i < B; ++i) done = done && fresh(v[k][i], num);
                const uint32_t who = __ballot_sync(0xffffffffu, !done && w.more(spins, since));
                if (who == 0) break;
                const u64* at = word(0, 0);
#pragma unroll
                for (int k = 0; k < R; ++k)
#pragma unroll
                    for (int i = 0; i < B; ++i) at = fresh(v[k][i], num) ? at : word(k, i);
                w.first(at, num, lane - (__ffs(who) - 1));
            }
#pragma unroll
            for (int k = 0; k < R; ++k)
#pragma unroll
                for (int i = 0; i < B; ++i)
                    sum[k] += tb + lane * 2 + i * 64 < Th ? __uint_as_float((uint32_t)v[k][i].a) + __uint_as_float((uint32_t)v[k][i].b) : 0.f;
        }
        __syncwarp();
#pragma unroll
        for (int k = 0; k < R; ++k) {
            const float t = warp_sum(sum[k]);
            if (lane == 0 && m0 + k * DD_FIN < M) out[m0 + k * DD_FIN] = rsqrtf(t / H + eps);
        }
    }
    asm volatile("bar.sync 2, %0;" ::"n"(DD_FIN * 32) : "memory");
}

// Of two threads with neighbouring rows (lanes 4 apart) the even one gets both rows' .x as a word, the odd one both rows' .y.
__device__ __forceinline__ uint32_t pair_words(float2 v, int r) {
    const float give = (r & 1) ? v.x : v.y;
    const float got = __shfl_xor_sync(0xffffffffu, give, 4);
    return (r & 1) ? pack_bf16(got, v.y) : pack_bf16(v.x, got);
}

// Which keys each row sees in a layer, and how they are cut: into at the most p.splits splits of 128 keys and more, in steps of 64.  That
// follows from the row's own length and the number of rows, not from the other rows' lengths, and so does every bit of its result.
// By one warp.
__device__ __forceinline__ void cut_keys(const DdParams& p, DdShared* sh, int window, int chunk, int lane) {
    const bool live = lane < p.M && sh->slot[lane] >= 0;
    int lo = 0, len = 0;
    if (live) {
        const int ctx = sh->ctx[lane];
        lo = window > 0 ? max(0, ctx - window + 1) : 0;
        if (chunk > 0) lo = max(lo, ctx / chunk * chunk);
        len = ctx + 1 - lo;
    }
    const int cut = max(128, ((len + p.splits - 1) / p.splits + 63) / 64 * 64), ns = (len + cut - 1) / cut;
    int inc = ns;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const int t = __shfl_up_sync(0xffffffffu, inc, o);
        if (lane >= o) inc += t;
    }
    if (lane < DD_ROWS) {
        sh->lo[lane] = lo;
        sh->ns[lane] = ns;
        sh->cut[lane] = cut;
        sh->before[lane + 1] = inc;
        if (lane == 0) sh->before[0] = 0;
    }
}

__device__ __forceinline__ uint32_t transpose8(uint32_t a) {
    uint32_t d;
    asm volatile("movmatrix.sync.aligned.m8n8.trans.b16 %0, %1;" : "=r"(d) : "r"(a));
    return d;
}
__device__ __forceinline__ float ex2(float x) {
    float y;
    asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
}

// C times 32 bytes of packets (4 words = 8 bfloat16), 16 packets apart, awaited together
template <int C>
__device__ __forceinline__ void wait_words(const u64* p, uint32_t num, const Waiter& w, uint4 (&out)[C], int lane) {
    Pair v[C][2];
    uint32_t spins = 0;
    u64 since = 0;
    bool done;
    do {
#pragma unroll
        for (int j = 0; j < C; ++j)
#pragma unroll
            for (int h = 0; h < 2; ++h) v[j][h] = get2(p + j * 16 + h * 2);
        done = true;
#pragma unroll
        for (int j = 0; j < C; ++j) done = done && fresh(v[j][0], num) && fresh(v[j][1], num);
        const uint32_t who = __ballot_sync(0xffffffffu, !done && w.more(spins, since));
        if (who == 0) break;
        const u64* at = p;
#pragma unroll
        for (int j = 0; j < C; ++j) at = fresh(v[j][0], num) && fresh(v[j][1], num) ? at : p + j * 16 + (fresh(v[j][0], num) ? 2 : 0);
        w.first(at, num, lane - (__ffs(who) - 1));
    } while (true);
#pragma unroll
    for (int j = 0; j < C; ++j) out[j] = make_uint4((uint32_t)v[j][0].a, (uint32_t)v[j][0].b, (uint32_t)v[j][1].a, (uint32_t)v[j][1].b);
}

// Attention of one (row b, KV head, split) by the consumer warps.  Tiles of 16 keys, dealt to the warps in turn; the 16 keys are the M rows
// of the MMAs and the group's (up to 8) heads their columns, S^T = K Q^T and O^T += V^T P^T.  Keys and values go to registers in
// the order in which 16-byte loads bring them: a thread's eight dimensions are those of four (K) or, through `movmatrix`, of
// eight (V) fragment places, the same for Q, and the output's dimensions are put right when it is written.
template <int D>
__device__ __forceinline__ void attend(const DdParams& p, const DdLayer& L, DdShared* sh, unsigned char* xs, int b, int kvh, int split, uint32_t num,
                                       const Waiter& w, int tid) {
    constexpr int C = D / 32, OS = D + 1;
    const int warp = tid >> 5, lane = tid & 31, r = lane >> 2, q = lane & 3;
    const int G = p.n_q / p.n_kv, ctx = sh->ctx[b], slot = sh->slot[b];
    const int k0 = sh->lo[b] + split * sh->cut[b], k1 = min(k0 + sh->cut[b], ctx + 1);
    const int bs = p.block_size;
    auto column = [&](int key) -> int { return (int)((u64)key * p.bs_inv >> 32); };           // key / bs
    const int* table = L.table + (size_t)slot * L.max_blocks;
    // a key's block number as the table has it (-1: the key is not read), and whether it is one
    auto entry = [&](int key) -> int { return key < k1 && key != ctx ? table[column(key)] : -1; };
    auto block_of = [&](int key, int e) -> int {
        if (e >= 0 && e < p.num_blocks) return e;
        if (key < k1 && key != ctx) set_status(p.status, STATUS_BAD_BLOCK);
        return -1;
    };
    uint4 ka[C], kb[C], va[C], vb[C];
    auto load = [&](const __nv_bfloat16* pool, int key, int blk, uint4 (&v)[C]) {
        const int in = key - column(key) * bs;
        const uint4* s = reinterpret_cast<const uint4*>(pool + (((size_t)blk * p.n_kv + kvh) * bs + in) * D) + q;
#pragma unroll
        for (int j = 0; j < C; ++j) v[j] = blk >= 0 ? load16(s + j * 4) : make_uint4(0, 0, 0, 0);
    };
    int t = k0 + warp * 16;
    const int step = DD_WARPS * 16;
    int ea = entry(t + step + r), eb = entry(t + step + r + 8);           // of the tile after this one
    const int ba = block_of(t + r, entry(t + r)), bb = block_of(t + r + 8, entry(t + r + 8));
    load(L.kp, t + r, ba, ka);
    load(L.kp, t + r + 8, bb, kb);
    load(L.vp, t + r, ba, va);
    load(L.vp, t + r + 8, bb, vb);

    // queries: this thread's head is r, its dimensions 32 j + 8 q ..
    uint4 qf[C];
    if (t < k1) {
        const u64* qs = p.q + ((size_t)b * p.n_q + kvh * G + min(r, G - 1)) * (D / 2) + q * 4;
        wait_words<C>(qs, num, w, qf, lane);
#pragma unroll
        for (int j = 0; j < C; ++j)
            if (r >= G) qf[j] = make_uint4(0, 0, 0, 0);
    }
    float o[C * 2][4];
#pragma unroll
    for (int i = 0; i < C * 2; ++i) o[i][0] = o[i][1] = o[i][2] = o[i][3] = 0.f;
    float m_run[2] = {-INFINITY, -INFINITY}, l_run[2] = {0.f, 0.f};
    const float scale_log2 = L.scale * 1.4426950408889634f;

#pragma unroll 1
    for (; t < k1; t += step) {
        const int na = t + step + r, nba = block_of(na, ea), nbb = block_of(na + 8, eb);
        ea = entry(na + step);
        eb = entry(na + step + 8);
        if (ctx >= t && ctx < t + 16) {           // the new token's own key and value come from the projection's packets
            // (each lane fetches four elements of both, and passes them to the lanes of that key's row)
            const u64* ks = p.kv + ((size_t)b * 2 * p.n_kv + kvh) * (D / 2) + min(lane, D / 4 - 1) * 2;
            const u64* vs = ks + (size_t)p.n_kv * (D / 2);
            Pair k1_ = get2(ks), v1_ = get2(vs);
            if (!fresh(k1_, num)) k1_ = w.wait2(ks, num);
            if (!fresh(v1_, num)) v1_ = w.wait2(vs, num);
            __syncwarp();
            const bool first = t + r == ctx, second = t + r + 8 == ctx;
            auto pass = [&](const Pair& x, uint4& lo, uint4& hi, int j) {
                const int at = 8 * j + 2 * q;
                const uint4 y = make_uint4(__shfl_sync(0xffffffffu, (uint32_t)x.a, at), __shfl_sync(0xffffffffu, (uint32_t)x.b, at),
                                           __shfl_sync(0xffffffffu, (uint32_t)x.a, at + 1), __shfl_sync(0xffffffffu, (uint32_t)x.b, at + 1));
                if (first) lo = y;
                if (second) hi = y;
            };
#pragma unroll
            for (int j = 0; j < C; ++j) {
                pass(k1_, ka[j], kb[j], j);
                pass(v1_, va[j], vb[j], j);
            }
        }
        float s[4] = {0.f, 0.f, 0.f, 0.f}, s2[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
        for (int j = 0; j < C; ++j) {
            mma_bf16(s, ka[j].x, kb[j].x, ka[j].y, kb[j].y, qf[j].x, qf[j].y);
            mma_bf16(s2, ka[j].z, kb[j].z, ka[j].w, kb[j].w, qf[j].z, qf[j].w);
        }
        load(L.kp, na, nba, ka);
        load(L.kp, na + 8, nbb, kb);
#pragma unroll
        for (int e = 0; e < 4; ++e) s[e] += s2[e];
        if (t + r >= k1) s[0] = s[1] = -INFINITY;
        if (t + r + 8 >= k1) s[2] = s[3] = -INFINITY;
        float alpha[2], m_off[2];
#pragma unroll
        for (int h = 0; h < 2; ++h) {
            float mx = fmaxf(s[h], s[2 + h]);
            mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, 4));
            mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, 8));
            mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, 16));
            const float m_new = fmaxf(m_run[h], mx);
            alpha[h] = m_new == -INFINITY ? 1.f : ex2((m_run[h] - m_new) * scale_log2);
            m_run[h] = m_new;
            m_off[h] = m_new == -INFINITY ? 0.f : m_new * scale_log2;
        }
#pragma unroll
        for (int e = 0; e < 4; ++e) s[e] = ex2(fmaf(s[e], scale_log2, -m_off[e & 1]));
        l_run[0] = l_run[0] * alpha[0] + s[0] + s[2];
        l_run[1] = l_run[1] * alpha[1] + s[1] + s[3];
        const uint32_t pb0 = transpose8(pack_bf16(s[0], s[1])), pb1 = transpose8(pack_bf16(s[2], s[3]));
#pragma unroll
        for (int i = 0; i < C * 2; ++i) {
            o[i][0] *= alpha[0]; o[i][1] *= alpha[1]; o[i][2] *= alpha[0]; o[i][3] *= alpha[1];
        }
#pragma unroll
        for (int j = 0; j < C; ++j) {
            mma_bf16(o[2 * j], transpose8(va[j].x), transpose8(va[j].y), transpose8(vb[j].x), transpose8(vb[j].y), pb0, pb1);
            mma_bf16(o[2 * j + 1], transpose8(va[j].z), transpose8(va[j].w), transpose8(vb[j].z), transpose8(vb[j].w), pb0, pb1);
        }
        load(L.vp, na, nba, va);
        load(L.vp, na + 8, nbb, vb);
    }
    // the warps' results to shared memory
#pragma unroll
    for (int h = 0; h < 2; ++h) {
        l_run[h] += __shfl_xor_sync(0xffffffffu, l_run[h], 4);
        l_run[h] += __shfl_xor_sync(0xffffffffu, l_run[h], 8);
        l_run[h] += __shfl_xor_sync(0xffffffffu, l_run[h], 16);
        if (r == 0) { sh->m[warp][2 * q + h] = m_run[h]; sh->l[warp][2 * q + h] = l_run[h]; }
    }
    float* ow = reinterpret_cast<float*>(xs) + warp * 8 * OS;
#pragma unroll
    for (int j = 0; j < C; ++j)
#pragma unroll
        for (int i = 0; i < 2; ++i) {
            float* at = ow + 2 * q * OS + j * 32 + (r >> 1) * 8 + 4 * i + (r & 1);
            at[0] = o[2 * j + i][0];
            at[OS] = o[2 * j + i][1];
            at[2] = o[2 * j + i][2];
            at[OS + 2] = o[2 * j + i][3];
        }
    cons_sync();
    // one warp per head; a lane has every 32nd dimension
    if (warp >= G) return;
    const int h = warp;
    const float mi = lane < DD_WARPS ? sh->m[lane][h] : -INFINITY, m = warp_max(mi);
    const float f = mi == -INFINITY ? 0.f : exp2f((mi - m) * scale_log2);
    const float l = warp_sum(lane < DD_WARPS ? sh->l[lane][h] * f : 0.f);
    float a[C];
#pragma unroll
    for (int k = 0; k < C; ++k) a[k] = 0.f;
#pragma unroll
    for (int i = 0; i < DD_WARPS; ++i) {
        const float fi = __shfl_sync(0xffffffffu, f, i);
        const float* from = reinterpret_cast<const float*>(xs) + (i * 8 + h) * OS + lane;
#pragma unroll
        for (int k = 0; k < C; ++k) a[k] = fmaf(from[k * 32], fi, a[k]);
    }
    const size_t row = (size_t)b * p.n_q + kvh * G + h;
    if (p.skip == 3 && &L == &p.layer[p.n_layers - 1] && blockIdx.x == gridDim.x - 1) return;
    if (sh->ns[b] > 1) {
        u64* out = p.part + (uint32_t)(((int)row * p.splits + split) * (D + 2));
#pragma unroll
        for (int k = 0; k < C; ++k) put(out + 2 + k * 32 + lane, __float_as_uint(a[k]), num);
        if (lane == 0) put2(out, __float_as_uint(m * scale_log2), __float_as_uint(l), num);
        return;
    }
    const float to = l > 0.f ? 1.f / l : (l == 0.f ? 0.f : l);           // (a NaN stays one)
#pragma unroll
    for (int k = 0; k < C; ++k) {
        const float x = a[k] * to, y = __shfl_down_sync(0xffffffffu, x, 1);
        if ((lane & 1) == 0) put(p.attn + row * (D / 2) + (k * 32 + lane) / 2, pack_bf16(x, y), num);
    }
}

// The splits' outputs of the step's heads added up: a head of a row by `wpi` warps, each of which takes every wpi-th split.
template <int D>
__device__ __forceinline__ void merge_splits(const DdParams& p, DdShared* sh, uint32_t num, const Waiter& w, int c, int n, int tid) {
    constexpr int W = D / 32, B = 4;              // dims per lane; splits in flight
    const int warp = tid >> 5, lane = tid & 31, items = p.M * p.n_q;
    const int wpi = items <= n ? 8 : items <= 2 * n ? 4 : items <= 4 * n ? 2 : 1, sub = warp % wpi, per = n * (DD_WARPS / wpi);
#pragma unroll 1
    for (int i0 = c; i0 < items; i0 += per) {
        const int item = i0 + n * (warp / wpi), b = item / p.n_q;
        const bool live = item < items && sh->slot[b] >= 0;
        const int ns = live ? sh->ns[b] : 0;
        u64* out = p.attn + (size_t)item * (D / 2) + lane * (W / 2);
        if (item < items && !live && sub == 0) {      // padding row: zeros; not before this layer's queries, when the layer before has been read
            w.first(p.q + (size_t)item * (D / 2), num, lane);
#pragma unroll
            for (int i = 0; i < W / 2; ++i) put(out + i, 0u, num);
        }
        const u64* src = p.part + (uint32_t)(item * p.splits * (D + 2));
        float m = -INFINITY, l = 0.f, a[W];
#pragma unroll
        for (int i = 0; i < W; ++i) a[i] = 0.f;
#pragma unroll 1
        for (int s0 = sub; s0 < ns && ns > 1; s0 += B * wpi) {
            Pair ml[B], v[B][W / 2];
            uint32_t spins = 0;
            u64 t0 = 0;
            bool all;
            do {
                all = true;
#pragma unroll
                for (int i = 0; i < B; ++i) {
                    const u64* s = src + (size_t)(s0 + i * wpi < ns ? s0 + i * wpi : s0) * (D + 2);
                    ml[i] = get2(s);
#pragma unroll
                    for (int k = 0; k < W / 2; ++k) v[i][k] = get2(s + 2 + lane * W + 2 * k);
                }
#pragma unroll
                for (int i = 0; i < B; ++i) {
                    all = all && fresh(ml[i], num);
#pragma unroll
                    for (int k = 0; k < W / 2; ++k) all = all && fresh(v[i][k], num);
                }
                if (!__any_sync(0xffffffffu, !all && w.more(spins, t0))) break;
                int late = 0;                     // the last split that is not there
#pragma unroll
                for (int i = 1; i < B; ++i) late = fresh(ml[i], num) ? late : i;
                w.first(src + (size_t)(s0 + late * wpi < ns ? s0 + late * wpi : s0) * (D + 2), num, lane);
            } while (true);
            float m_new = m;
#pragma unroll
            for (int i = 0; i < B; ++i)
                if (s0 + i * wpi < ns) m_new = fmaxf(m_new, __uint_as_float((uint32_t)ml[i].a));
            const float keep = m == -INFINITY ? 0.f : exp2f(m - m_new);
            m = m_new;
            l *= keep;
#pragma unroll
            for (int i = 0; i < W; ++i) a[i] *= keep;
#pragma unroll
            for (int i = 0; i < B; ++i) {
                if (s0 + i * wpi >= ns) continue;
                const float mi = __uint_as_float((uint32_t)ml[i].a);
                const float f = mi == -INFINITY ? 0.f : exp2f(mi - m);
                l = fmaf(__uint_as_float((uint32_t)ml[i].b), f, l);
#pragma unroll
                for (int k = 0; k < W / 2; ++k) {
                    a[2 * k] = fmaf(__uint_as_float((uint32_t)v[i][k].a), f, a[2 * k]);
                    a[2 * k + 1] = fmaf(__uint_as_float((uint32_t)v[i][k].b), f, a[2 * k + 1]);
                }
            }
        }
        __syncwarp();
        if (wpi > 1) {
            float* mine = sh->merge[warp];
#pragma unroll
            for (int i = 0; i < W; ++i) mine[lane * W + i] = a[i];
            if (lane == 0) { mine[D] = m; mine[D + 1] = l; }
            cons_sync();
            if (sub == 0 && ns > 1) {
                float top = m;
#pragma unroll 1
                for (int i = 1; i < wpi; ++i) top = fmaxf(top, sh->merge[warp + i][D]);
                float f = m == -INFINITY ? 0.f : exp2f(m - top);
                l *= f;
#pragma unroll
                for (int k = 0; k < W; ++k) a[k] *= f;
#pragma unroll 1
                for (int i = 1; i < wpi; ++i) {
                    const float* o = sh->merge[warp + i];
                    f = o[D] == -INFINITY ? 0.f : exp2f(o[D] - top);
                    l = fmaf(o[D + 1], f, l);
#pragma unroll
                    for (int k = 0; k < W; ++k) a[k] = fmaf(o[lane * W + k], f, a[k]);
                }
            }
        }
        if (sub == 0 && ns > 1) {
            const float f = l > 0.f ? 1.f / l : (l == 0.f ? 0.f : l);
            if constexpr (W == 4) put2(out, pack_bf16(a[0] * f, a[1] * f), pack_bf16(a[2] * f, a[3] * f), num);
            else put(out, pack_bf16(a[0] * f, a[1] * f), num);
        }
        if (i0 + per < items) cons_sync();
    }
}

template <int D, int NT>
__global__ void __launch_bounds__(DD_THREADS, 1) dense_decode_kernel(const __grid_constant__ DdParams p) {
    extern __shared__ __align__(1024) unsigned char smem[];
    unsigned char* ring = smem;
    unsigned char* xs = smem + p.n_stages * p.kbs * DD_BLOCK;
    float* red_all = reinterpret_cast<float*>(xs + p.x_bytes);
    float* own_r = red_all + dd_red_bytes(NT) / 4;
    __shared__ DdShared sh_mem;
    DdShared* sh = &sh_mem;
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, c = blockIdx.x, n = gridDim.x;
    const int M = p.M, H = p.H, Q = p.n_q * D;

    if (tid == 0) {
#pragma unroll 1
        for (int i = 0; i < p.n_stages; ++i) {
            mbar_init(s_addr(&sh->full[i]), 1);
            mbar_init(s_addr(&sh->empty[i]), DD_WARPS);
        }
#pragma unroll 1
        for (int i = 0; i < DD_FIN; ++i) {
            mbar_init(s_addr(&sh->sums[i]), DD_WARPS);
            mbar_init(s_addr(&sh->taken[i]), 1);
        }
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        sh->abort = 0;
        sh->base = *(volatile unsigned*)p.ctrl;
    }
    if (tid < M) {
        sh->slot[tid] = p.row_slot[tid];
        sh->pos[tid] = p.tok_pos[tid];
        sh->ctx[tid] = p.row_ctx[tid];
    }
    __syncthreads();
    bool any = false;
#pragma unroll 1
    for (int m = 0; m < M; ++m) any = any || sh->slot[m] >= 0;
    if (!any) return;                             // padding rows only (the same for every CTA)

    const Waiter w{&sh->abort, p.status, p.wait_ns};
    const uint32_t base = sh->base;
    // this CTA's work: q/k/v tiles c, c + n, ..; the tiles j = member, member + S, .. of its group (whose part of the stream it
    // owns: o and the end of down); gate/up tiles; all tiles of its group over slice `member` of down's k
    const int Tq = (p.n_q + 2 * p.n_kv) * D / 16, Th = H / 16;
    const int SK = p.kbs * 64, KH = (H + SK - 1) / SK, KQ = (Q + SK - 1) / SK, KI = (p.I + SK - 1) / SK;
    const int grp = c / p.S, member = c - grp * p.S;
    const int g0 = grp * p.tp, g_n = grp < p.n_groups ? min(p.tp, Th - g0) : 0;
    const int gu0 = p.gu[c], gu1 = p.gu[c + 1];
    const int sl0 = member * KI / p.S, sl1 = (member + 1) * KI / p.S;

    if (warp == DD_WARPS) {
        // ---- producer: every stage of every tile, in the order in which the consumers take them
        if (lane != 0) return;
        struct Walk {
            int l = 0, job = -1, i = 0, k = 0, end = 0;
        };
        const int cnt[4] = {c < Tq ? (Tq - c + n - 1) / n : 0, member < g_n ? (g_n - member + p.S - 1) / p.S : 0, gu1 - gu0, g_n};
        auto next = [&](Walk& x) -> bool {
            if (++x.k < x.end) return true;
            if (x.job < 0 || ++x.i >= (x.job == 0 ? cnt[0] : x.job == 1 ? cnt[1] : x.job == 2 ? cnt[2] : cnt[3])) {
                x.i = 0;
                do {
                    if (++x.job == 4) { x.job = 0; ++x.l; }
                    if (x.l >= p.n_layers) return false;
                } while ((x.job == 0 ? cnt[0] : x.job == 1 ? cnt[1] : x.job == 2 ? cnt[2] : cnt[3]) == 0);
            }
            x.k = x.job == 3 ? sl0 : 0;
            x.end = x.job == 3 ? sl1 : x.job == 1 ? KQ : KH;
            return true;
        };
        auto row_of = [&](const Walk& x) {
            return 16 * (x.job == 0 ? c + x.i * n : x.job == 1 ? g0 + member + x.i * p.S : x.job == 2 ? gu0 + x.i : g0 + x.i);
        };
        Place at, landed;                         // the next copy; the oldest of those that may still be under way
        Walk now;
        int issued = 0;
        const int bytes = p.kbs * DD_BLOCK;
#pragma unroll 1
        while (next(now)) {
            // (a CTA that has given up a wait goes on to its end, and so does the ring: it never waits for another CTA)
            if (issued >= p.n_stages && !w.bar(s_addr(&sh->empty[at.slot]), at.phase ^ 1)) break;
            if (issued >= p.flying) {
                if (!w.bar(s_addr(&sh->full[landed.slot]), landed.phase)) break;
                landed.next(p.n_stages);
            }
            const uint32_t bar = s_addr(&sh->full[at.slot]);
            mbar_expect_tx(bar, bytes);
            tma_load_3d(smem_u32(ring) + at.slot * bytes, &p.layer[now.l].map[now.job], bar, 0, row_of(now), now.k * p.kbs);
            at.next(p.n_stages);
            ++issued;
        }
        if (p.pf_bytes != 0) l2_prefetch_share(p.pf_ptr, p.pf_bytes);
        // no copy may be under way when the block's shared memory goes (the limit starts anew: copies do end)
        volatile int never = 0;
        if (issued < p.n_stages) at.slot = 0;
        else at.phase ^= 1;                       // the oldest of the last n_stages copies
#pragma unroll 1
        for (int i = min(issued, p.n_stages); i > 0; --i) {
            Waiter{&never, p.status, DD_WAIT_NS}.bar(s_addr(&sh->full[at.slot]), at.phase);
            at.next(p.n_stages);
        }
        return;
    }
    if (warp > DD_WARPS) {
        // ---- finishing: what becomes of the tiles' sums.  Tile by tile one of the three warps; an own tile of the stream stays with one warp
        const int f = warp - DD_WARPS - 1, r = lane >> 2, cq = (lane & 3) * 2;
        uint32_t taken = 0;
        // a finished piece of the stream: its normed words and the tile's sums of squares
        auto hand_out = [&](int ph, float w0, float w1, int row0, const float2 (&v)[NT][2], uint32_t num) {
#pragma unroll
            for (int nt = 0; nt < NT; ++nt)
#pragma unroll
                for (int e = 0; e < 2; ++e) {
                    const int m = nt * 8 + cq + e;
                    const float2 x = v[nt][e];
                    const uint32_t word = pair_words(make_float2(x.x * w0, x.y * w1), r);
                    if (m < M) put(p.x[ph] + ((size_t)m * H + row0 + ((r & 1) ? 8 : 0) + (r & ~1)) / 2, word, num);
                    float sq = x.x * x.x + x.y * x.y;
                    sq += __shfl_xor_sync(0xffffffffu, sq, 4);
                    sq += __shfl_xor_sync(0xffffffffu, sq, 8);
                    sq += __shfl_xor_sync(0xffffffffu, sq, 16);
                    if (r == 0 && m < M) put(p.ss[ph] + (size_t)m * Th + row0 / 16, __float_as_uint(sq), num);
                }
        };
        auto own_at = [&](int i, int nt) { return reinterpret_cast<float4*>(own_r + ((i * NT + nt) * 32 + lane) * 4); };
        auto norms = [&](int ph, float eps, uint32_t num) { row_norms(p.ss[ph], sh->inv[ph], M, Th, H, eps, num, w, f, lane); };
#pragma unroll 1
        for (int i = f; member + i * p.S < g_n; i += DD_FIN) {
            const int row0 = (g0 + member + i * p.S) * 16;
            float2 v[NT][2];
#pragma unroll
            for (int nt = 0; nt < NT; ++nt) {
#pragma unroll
                for (int e = 0; e < 2; ++e) {
                    const int m = nt * 8 + cq + e;
                    v[nt][e] = m < M ? make_float2(p.resid[(size_t)m * H + row0 + r], p.resid[(size_t)m * H + row0 + r + 8]) : make_float2(0.f, 0.f);
                }
                *own_at(i, nt) = make_float4(v[nt][0].x, v[nt][1].x, v[nt][0].y, v[nt][1].y);
            }
            hand_out(0, vec_at(p.layer[0].norm1, row0 + r, p.layer[0].f32 & 1), vec_at(p.layer[0].norm1, row0 + r + 8, p.layer[0].f32 & 1), row0, v, base + 1);
        }
#pragma unroll 1
        for (int l = 0; l < p.n_layers; ++l) {
            const DdLayer& L = p.layer[l];
            const uint32_t num = base + l + 1;
            // ---- q, k, v: norm, bias, rotation, append
            if (c < Tq) {
                int turn = 0;
                bool normed = false;
#pragma unroll 1
                for (int t = c; t < Tq; t += n, ++turn) {
                    const bool mine = turn % DD_FIN == f;
                    const int head = t / (D / 16), t_in = t % (D / 16);
                    const bool is_v = head >= p.n_q + p.n_kv;
                    const int j0 = is_v ? t_in * 16 + r : t_in * 8 + r;
                    float cs[NT][2], sn[NT][2], b0 = 0.f, b1 = 0.f;
                    int blk[NT][2];
                    if (mine) {                   // everything the end needs, asked for before the sums are there
#pragma unroll
                        for (int nt = 0; nt < NT; ++nt)
#pragma unroll
                            for (int e = 0; e < 2; ++e) {
                                const int m = nt * 8 + cq + e;
                                cs[nt][e] = 1.f; sn[nt][e] = 0.f; blk[nt][e] = -1;
                                if (m >= M || sh->slot[m] < 0) continue;
                                const int slot = sh->slot[m], pos = sh->pos[m];
                                if (pos < 0 || pos >= L.table_len) { set_status(p.status, STATUS_BAD_POSITION); continue; }
                                if (!is_v) {
                                    cs[nt][e] = L.cos_t[(size_t)pos * (D / 2) + j0];
                                    sn[nt][e] = L.sin_t[(size_t)pos * (D / 2) + j0];
                                }
                                if (head >= p.n_q) blk[nt][e] = L.table[(size_t)slot * L.max_blocks + pos / p.block_size];
                            }
                        if (L.bias != nullptr) {
                            b0 = vec_at(L.bias, t * 16 + r, L.f32 & 4);
                            b1 = vec_at(L.bias, t * 16 + r + 8, L.f32 & 4);
                        }
                    }
                    if (!normed) { norms(0, L.eps1, num); normed = true; }
                    if (!mine) continue;
                    float2 v[NT][2];
                    take_sums<NT>(w, sh, red_all, f, taken, lane, v);
                    // the even thread has the first of its two rows' dimensions, the odd one the second
                    const int dim = (is_v ? t_in * 16 : t_in * 8) + (r & ~1) + ((r & 1) ? (is_v ? 8 : D / 2) : 0);
                    const int kvh = is_v ? head - p.n_q - p.n_kv : head - p.n_q;
#pragma unroll
                    for (int nt = 0; nt < NT; ++nt)
#pragma unroll
                        for (int e = 0; e < 2; ++e) {
                            const int m = nt * 8 + cq + e;
                            const float inv = m < M ? sh->inv[0][m] : 0.f;
                            float2 x = make_float2(fmaf(v[nt][e].x, inv, b0), fmaf(v[nt][e].y, inv, b1));
                            if (!is_v) x = make_float2(x.x * cs[nt][e] - x.y * sn[nt][e], x.y * cs[nt][e] + x.x * sn[nt][e]);
                            const uint32_t word = pair_words(x, r);
                            if (m >= M) continue;
                            if (head < p.n_q) {
                                if (p.skip == 2 && l == p.n_layers - 1 && c == 0) continue;
                                put(p.q + ((size_t)m * p.n_q + head) * (D / 2) + dim / 2, word, num);
                                continue;
                            }
                            put(p.kv + ((size_t)m * 2 * p.n_kv + head - p.n_q) * (D / 2) + dim / 2, word, num);
                            const int pos = sh->pos[m];
                            if (sh->slot[m] < 0 || pos < 0 || pos >= L.table_len) continue;
                            if (blk[nt][e] < 0 || blk[nt][e] >= p.num_blocks) { set_status(p.status, STATUS_BAD_BLOCK); continue; }
                            *reinterpret_cast<uint32_t*>((is_v ? L.vp : L.kp) + (((size_t)blk[nt][e] * p.n_kv + kvh) * p.block_size + pos % p.block_size) * D + dim) = word;
                        }
                    __syncwarp();
                }
            }
            // ---- output projection: into the stream
#pragma unroll 1
            for (int i = 0; member + i * p.S < g_n; ++i) {
                if (i % DD_FIN != f) continue;
                const int row0 = (g0 + member + i * p.S) * 16;
                const float w0 = vec_at(L.norm2, row0 + r, L.f32 & 2), w1 = vec_at(L.norm2, row0 + r + 8, L.f32 & 2);
                float2 v[NT][2];
                take_sums<NT>(w, sh, red_all, f, taken, lane, v);
#pragma unroll
                for (int nt = 0; nt < NT; ++nt) {
                    float4* own = own_at(i, nt);
                    const float4 o = *own;
                    v[nt][0] = make_float2(o.x + v[nt][0].x, o.z + v[nt][0].y);
                    v[nt][1] = make_float2(o.y + v[nt][1].x, o.w + v[nt][1].y);
                    *own = make_float4(v[nt][0].x, v[nt][1].x, v[nt][0].y, v[nt][1].y);
                }
                if (p.skip == 1 && l == p.n_layers - 1 && c == 0) continue;
                hand_out(1, w0, w1, row0, v, num);
            }
            // ---- gate and up: norm, activation
            if (gu0 < gu1) {
                norms(1, L.eps2, num);
#pragma unroll 1
                for (int t = gu0; t < gu1; ++t) {
                    if ((t - gu0) % DD_FIN != f) continue;
                    float2 v[NT][2];
                    take_sums<NT>(w, sh, red_all, f, taken, lane, v);
#pragma unroll
                    for (int nt = 0; nt < NT; ++nt)
#pragma unroll
                        for (int e = 0; e < 2; ++e) {
                            const int m = nt * 8 + cq + e;
                            const float inv = m < M ? sh->inv[1][m] : 0.f;
                            const float a = gated_value(0, v[nt][e].x * inv, v[nt][e].y * inv, 0.f);
                            const float a2 = __shfl_xor_sync(0xffffffffu, a, 4);
                            if (m < M && (r & 1) == 0) put(p.act + ((size_t)m * p.I + t * 8 + r) / 2, pack_bf16(a, a2), num);
                        }
                }
            }
            // ---- down: own tiles into the stream, the others' sums to their owners
#pragma unroll 1
            for (int j = 0; j < g_n; ++j) {
                const bool own_tile = j % p.S == member;
                if ((own_tile ? j / p.S : j) % DD_FIN != f) continue;
                float2 v[NT][2];
                take_sums<NT>(w, sh, red_all, f, taken, lane, v);
#pragma unroll
                for (int nt = 0; nt < NT; ++nt) {
                    if (own_tile) {
                        float4* own = own_at(j / p.S, nt);
                        const float4 o = *own;
                        *own = make_float4(o.x + v[nt][0].x, o.y + v[nt][1].x, o.z + v[nt][0].y, o.w + v[nt][1].y);
                        continue;
                    }
#pragma unroll
                    for (int e = 0; e < 2; ++e) {
                        const int m = nt * 8 + cq + e;
                        if (m < M && !(p.skip == 4 && l == p.n_layers - 1 && c == 0))
                            put2(p.dpart + ((((size_t)(g0 + j) * p.S + member) * M + m) * 8 + r) * 2, __float_as_uint(v[nt][e].x), __float_as_uint(v[nt][e].y), num);
                    }
                }
            }
#pragma unroll 1
            for (int i = f; member + i * p.S < g_n; i += DD_FIN) {
                const int tile = g0 + member + i * p.S;
                const DdLayer& N = p.layer[min(l + 1, p.n_layers - 1)];
                const float w0 = vec_at(N.norm1, tile * 16 + r, N.f32 & 1), w1 = vec_at(N.norm1, tile * 16 + r + 8, N.f32 & 1);
                float2 v[NT][2];
#pragma unroll
                for (int nt = 0; nt < NT; ++nt) {
                    const float4 o = *own_at(i, nt);
                    v[nt][0] = make_float2(o.x, o.z);
                    v[nt][1] = make_float2(o.y, o.w);
                }
#pragma unroll 1
                for (int s0 = 0; s0 < p.S; s0 += 2) {         // the other slices' sums, two on their way at a time, added in order
                    Pair d[2][2 * NT];
                    auto word = [&](int k, int e) {
                        const int sl = min(s0 + k, p.S - 1), m = min((e >> 1) * 8 + cq + (e & 1), M - 1);
                        return p.dpart + ((((size_t)tile * p.S + sl) * M + m) * 8 + r) * 2;
                    };
                    uint32_t spins = 0;
                    u64 since = 0;
                    bool done;
                    do {
                        done = true;
#pragma unroll
                        for (int k = 0; k < 2; ++k)
#pragma unroll
                            for (int e = 0; e < 2 * NT; ++e) d[k][e] = get2(word(k, e));
#pragma unroll
                        for (int k = 0; k < 2; ++k)
#pragma unroll
                            for (int e = 0; e < 2 * NT; ++e) done = done && (min(s0 + k, p.S - 1) == member || fresh(d[k][e], num));
                    } while (!done && w.more(spins, since));
#pragma unroll
                    for (int k = 0; k < 2; ++k)
#pragma unroll
                        for (int e = 0; e < 2 * NT; ++e) {
                            const bool used = s0 + k < p.S && s0 + k != member;
                            v[e >> 1][e & 1].x += used ? __uint_as_float((uint32_t)d[k][e].a) : 0.f;
                            v[e >> 1][e & 1].y += used ? __uint_as_float((uint32_t)d[k][e].b) : 0.f;
                        }
                }
                __syncwarp();
#pragma unroll
                for (int nt = 0; nt < NT; ++nt) {
                    *own_at(i, nt) = make_float4(v[nt][0].x, v[nt][1].x, v[nt][0].y, v[nt][1].y);
                    if (l + 1 < p.n_layers) continue;
#pragma unroll
                    for (int e = 0; e < 2; ++e) {
                        const int m = nt * 8 + cq + e;
                        if (m >= M) continue;
                        p.resid[(size_t)m * H + tile * 16 + r] = v[nt][e].x;
                        p.resid[(size_t)m * H + tile * 16 + r + 8] = v[nt][e].y;
                    }
                }
                if (l + 1 < p.n_layers) hand_out(0, w0, w1, tile * 16, v, num + 1);
            }
        }
        return;
    }

    // ---- consumers: rows of x to shared memory, the tiles' sums; attention
    const uint32_t x_s = smem_u32(xs);
    Place at;
    uint32_t turns = 0;
#pragma unroll 1
    for (int l = 0; l < p.n_layers; ++l) {
        const DdLayer& L = p.layer[l];
        const uint32_t num = base + l + 1;
        if (l == 0 || L.window != p.layer[l - 1].window || L.chunk != p.layer[l - 1].chunk) {
            cons_sync();                          // the layer before is through with the old cut
            if (warp == 0) cut_keys(p, sh, L.window, L.chunk, lane);
        }
        cons_sync();                              // x's memory is free, the cut is known

        const int items = sh->before[M] * p.n_kv;
#pragma unroll 1
        for (int i = n - 1 - c; i < items; i += n) {          // the keys and values of this layer's attention, asked of L2
            const int place = i / p.n_kv, kvh = i - place * p.n_kv;
            int b = 0;
#pragma unroll 1
            while (sh->before[b + 1] <= place) ++b;
            const int k0 = sh->lo[b] + (place - sh->before[b]) * sh->cut[b], k1 = min(k0 + sh->cut[b], sh->ctx[b]);
#pragma unroll 1
            for (int key = k0 + (tid >> 1); key < k1; key += DD_CONS / 2) {
                const int col = (int)((u64)key * p.bs_inv >> 32), blk = L.table[(size_t)sh->slot[b] * L.max_blocks + col];
                if (blk < 0 || blk >= p.num_blocks) continue;
                const char* a = reinterpret_cast<const char*>(((tid & 1) ? L.vp : L.kp) + (((size_t)blk * p.n_kv + kvh) * p.block_size + key - col * p.block_size) * D);
                asm volatile("prefetch.global.L2 [%0];" ::"l"(a));
                if (D > 64) asm volatile("prefetch.global.L2 [%0];" ::"l"(a + 128));
            }
        }
        // ---- the four products, in one copy of the code; the attention after the first
#pragma unroll 1
        for (int ph = 0; ph < 4; ++ph) {
            const int tiles = ph == 0 ? (c < Tq ? (Tq - c + n - 1) / n : 0) : ph == 1 ? (member < g_n ? (g_n - member + p.S - 1) / p.S : 0) : ph == 2 ? gu1 - gu0 : g_n;
            if (tiles > 0) {
                const int cols = ph == 1 ? Q : ph == 3 ? min(sl1 * SK, p.I) - sl0 * SK : H;
                const int row = ph == 1 ? Q : ph == 3 ? p.I : H, stages = ph == 1 ? KQ : ph == 3 ? sl1 - sl0 : KH;
                const u64* src = ph == 0 ? p.x[0] : ph == 1 ? p.attn : ph == 2 ? p.x[1] : p.act + sl0 * SK / 2;
                const int stride = (ph == 3 ? stages * SK : cols) * 2 + 16;
                load_rows(src, row / 2, cols / 4, M, xs, stride, num, w, tid);
                cons_sync();
#pragma unroll 1
                for (int i = 0; i < tiles; ++i) {
                    const int f = (ph == 3 && i % p.S == member ? i / p.S : i) % DD_FIN;
                    tile_sums<NT>(p, w, sh, ring, at, f, turns, stages, cols / 64, x_s, stride, red_all, warp, lane);
                }
                cons_sync();                      // x's memory is free again
            }
            if (ph != 0) continue;
            // ---- attention
#pragma unroll 1
            for (int i = n - 1 - c; i < items; i += n) {      // from the last CTA on: those have no q/k/v tile
                const int place = i / p.n_kv, kvh = i - place * p.n_kv;
                int b = 0;
#pragma unroll 1
                while (sh->before[b + 1] <= place) ++b;
                attend<D>(p, L, sh, xs, b, kvh, place - sh->before[b], num, w, tid);
                cons_sync();
            }
            merge_splits<D>(p, sh, num, w, c, n, tid);
        }
    }
    if (tid == 0) {
        // the last CTA leaves the number for the next launch: every other one has read this launch's
        __threadfence();
        if (atomicAdd(p.ctrl + 1, 1u) == (unsigned)n - 1) {
            p.ctrl[1] = 0;
            p.ctrl[0] = base + p.n_layers + 1;
        }
    }
}

// How a step of these sizes is dealt to the CTAs, and the shared memory it takes.  False: the sizes are not taken.
struct DdPlan {
    int n, S, tp, n_groups, n_stages, kbs, x_bytes, own, NT;
    size_t smem;
    short gu[DD_CTAS + 1];
};

static bool dd_plan(int M, int H, int I, int n_q, int n_kv, int D, int sms, int smem_max, DdPlan* out) {
    if (M < 1 || M > DD_ROWS || (D != 64 && D != 128) || n_kv < 1 || n_q % n_kv != 0 || n_q / n_kv > 8) return false;
    if (H % 64 != 0 || I % 64 != 0 || H < 64 || I < 64 || sms < 1) return false;
    const int n = sms < DD_CTAS ? sms : DD_CTAS, NT = (M + 7) / 8;
    const int Q = n_q * D, Tq = (n_q + 2 * n_kv) * D / 16, Th = H / 16, Tg = I / 8;
    const int wide = H > Q ? H : Q;
    const int merge = DD_WARPS * 8 * (D + 1) * 4;
    // The stage (24 or 32 KB: an SM keeps about five bulk copies in flight, whatever their size, and with 16 KB copies that was 32
    // GB/s of the 44 that are an SM's share of HBM) and down's tp row tiles x S slices of k per group of S CTAs: the fewest blocks
    // on a CTA (an exchange of partial sums counts twelve per other slice), with room for at least four stages beside the rows of x (three from
    // 17 rows on: 24 rows of 300 tokens 51.0 us per layer against 59.3 in the kernels of their own; 32 rows, 66.4 against 60.4).
    long best = -1;
    for (int kbs = 16; kbs >= 12; kbs -= 4)
        for (int tp = 1; tp <= DD_OWN; ++tp) {
            const int KI = (I / 64 + kbs - 1) / kbs, KQ = (Q / 64 + kbs - 1) / kbs, KH = (H / 64 + kbs - 1) / kbs;
            for (int S = 1; S <= KI && S <= 16; ++S) {
                const int groups = (Th + tp - 1) / tp, own = (tp + S - 1) / S;
                if (groups * S > n) continue;
                int x = M * (wide * 2 + 16);
                const int slice = M * (((KI + S - 1) / S) * kbs * 128 + 16);
                if (slice > x) x = slice;
                if (merge > x) x = merge;
                x = (x + 127) / 128 * 128;
                const long rest = (long)x + dd_red_bytes(NT) + dd_own_bytes(NT, own);
                long stages = (smem_max - rest) / (kbs * DD_BLOCK);
                if (stages < (NT == 3 ? 3 : 4)) continue;
                if (stages > DD_MAX_STAGES) stages = DD_MAX_STAGES;
                const long cost = (long)kbs * (tp * ((KI + S - 1) / S) + own * KQ + (long)(Tg + n - 1) / n * KH) + 12l * (S - 1);
                if (best >= 0 && cost >= best) continue;
                best = cost;
                out->n = n; out->S = S; out->tp = tp; out->n_groups = groups; out->n_stages = (int)stages; out->kbs = kbs;
                out->x_bytes = x; out->own = own; out->NT = NT;
                out->smem = (size_t)stages * kbs * DD_BLOCK + rest;
            }
        }
    if (best < 0) return false;
    // gate/up: whoever has less of the rest takes more, up to two tiles above the average
    const int S = out->S, tp = out->tp, SK = out->kbs * 64, KH = (H + SK - 1) / SK, KQ = (Q + SK - 1) / SK, KI = (I + SK - 1) / SK;
    int load[DD_CTAS], take[DD_CTAS];
    for (int c = 0; c < n; ++c) {
        const int grp = c / S, mem = c % S, g0 = grp * tp;
        const int g_n = grp < out->n_groups ? (tp < Th - g0 ? tp : Th - g0) : 0;
        load[c] = (c < Tq ? (Tq - c + n - 1) / n * KH : 0) + (mem < g_n ? (g_n - mem + S - 1) / S * KQ : 0) +
                  g_n * ((mem + 1) * KI / S - mem * KI / S);
        take[c] = 0;
    }
    const int most = (Tg + n - 1) / n;
    for (int t = 0; t < Tg; ++t) {
        int at = -1;
        for (int c = 0; c < n; ++c)
            if (take[c] < most && (at < 0 || load[c] < load[at])) at = c;
        load[at] += KH;
        ++take[at];
    }
    out->gu[0] = 0;
    for (int c = 0; c < n; ++c) out->gu[c + 1] = (short)(out->gu[c] + take[c]);
    return Tg <= 32767;
}

// The splits of a row's keys at the most: its share of a grid in which every CTA takes one (row, KV head, split).  A CTA that takes two is
// some 2.7 us later than one with a single one of the same keys, so shares are rounded down.  What it costs that rows of unequal lengths get equal
// shares, us per layer, keys cut by the batch's mean length / by the row's own: 1.5B sizes, 8 rows of 2,200 tokens 41.0 / 40.4, of 1,500 to 3,000
// 42.4 / 42.4, 12 of 500 to 900 45.8 / 46.8, 16 of 600 47.1 / 46.9, 24 of 400 to 1,800 58.1 / 58.9; 7B 8 of 1,800 105.8 / 106.3, of 1,100 to
// 2,600 105.7 / 109.5.  In steps of 128 keys the last is 110.5, in steps of 16 108.8 (and the second 42.6).  Cut by the step's length bound, 0.6
// of which a row has on average, 8 of 1,800 take 108.7 at 7B and 8 of 1,000 126.7 at 14B sizes (124.3): two splits for most CTAs.
static int dd_splits(int M, int n_kv, int n) {
    const int share = n / (M * n_kv);
    return share < 1 ? 1 : share > DD_SPLITS ? DD_SPLITS : share;
}

// The exchange memory, in packets: where each buffer starts, and the whole.  The control words come first for all sizes: steps of
// different ones may share the memory, as what an earlier step left anywhere has another number than any that is awaited (numbers come
// round after 2^32: a word would have to lie unwritten for all of them).  At 24 rows of the 1.5B sizes 3.5 MB, at 8 of 7B 3.1.
struct DdBuffers {
    size_t x[2], ss[2], q, kv, part, attn, act, dpart, all;
};
static DdBuffers dd_buffers(int M, int H, int I, int n_q, int n_kv, int D, const DdPlan& plan) {
    DdBuffers b;
    size_t at = 16;                               // the control words
    auto take = [&](size_t packets) { const size_t o = at; at += (packets + 15) / 16 * 16; return o; };
    const size_t m = M;
    b.x[0] = take(m * H / 2);
    b.x[1] = take(m * H / 2);
    b.ss[0] = take(m * H / 16);
    b.ss[1] = take(m * H / 16);
    b.q = take(m * n_q * D / 2);
    b.kv = take(m * n_kv * D);
    b.attn = take(m * n_q * D / 2);
    b.act = take(m * I / 2);
    b.dpart = take(m * H * plan.S);
    b.part = take(m * n_q * dd_splits(M, n_kv, plan.n) * (D + 2));
    b.all = at;
    return b;
}

static int dd_device(int* sms, int* smem) {
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || cudaDeviceGetAttribute(sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess ||
        cudaDeviceGetAttribute(smem, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev) != cudaSuccess)
        return fail(-1, "dense_decode: no CUDA device");
    *smem -= (int)sizeof(DdShared) + 1024;        // the static part, and the ring's alignment
    return 0;
}

template <int D, int NT>
static int dd_launch(const DdParams& p, const DdPlan& plan, cudaStream_t stream) {
    auto k = dense_decode_kernel<D, NT>;
    cudaError_t e = cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)plan.smem);
    if (e != cudaSuccess) return fail(-3, "dense_decode: cannot get %zu bytes of shared memory: %s", plan.smem, cudaGetErrorString(e));
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(plan.n);
    cfg.blockDim = dim3(DD_THREADS);
    cfg.dynamicSmemBytes = plan.smem;
    cfg.stream = stream;
    cudaLaunchAttribute attr;
    attr.id = cudaLaunchAttributeCooperative;
    attr.val.cooperative = 1;
    cfg.attrs = &attr;
    cfg.numAttrs = 1;
    e = cudaLaunchKernelEx(&cfg, k, p);
    if (e != cudaSuccess) return fail(-100, "dense_decode: launch failed: %s", cudaGetErrorString(e));
    ++g_launches;
    return 0;
}

}  // namespace fd

// 8-byte words of exchange memory (zeroed once, then the kernel's own) for a step of M sequences of such a model; 0: not taken.
// info, if not null, gets {slices of down's k, row tiles per group, ring stages, bytes of shared memory, most gate/up tiles of a CTA}.
extern "C" long long fd_dense_decode_plan(int M, int H, int I, int n_q, int n_kv, int D, int sms, int smem_max, long long* info) {
    if (sms <= 0 && fd::dd_device(&sms, &smem_max) != 0) return 0;
    fd::DdPlan plan;
    if (!fd::dd_plan(M, H, I, n_q, n_kv, D, sms, smem_max, &plan)) return 0;
    if (info != nullptr) {
        info[0] = plan.S; info[1] = plan.tp; info[2] = plan.n_stages * 100 + plan.kbs; info[3] = (long long)plan.smem;
        info[4] = 0;
        for (int c = 0; c < plan.n; ++c)
            if (plan.gu[c + 1] - plan.gu[c] > info[4]) info[4] = plan.gu[c + 1] - plan.gu[c];
    }
    return (long long)fd::dd_buffers(M, H, I, n_q, n_kv, D, plan).all;
}

// All `count` entries of a decode step; the finished stream is left in resid.
extern "C" int fd_dense_decode(const FdDenseDecode* s, const FdDenseLayer* layers, int count) {
    using namespace fd;
    const FdDenseLayer& first = layers[0];
    const int M = (int)s->M, H = (int)first.hidden, I = (int)first.inter, n_q = (int)first.n_q, n_kv = (int)first.n_kv, D = (int)first.d;
    int sms = 0, smem = 0;
    int rc = dd_device(&sms, &smem);
    if (rc != 0) return rc;
    DdPlan plan;
    FD_REQUIRE(dd_plan(M, H, I, n_q, n_kv, D, sms, smem, &plan), -2, "dense_decode: sizes not taken");
    FD_REQUIRE((uintptr_t)s->next % 16 == 0, -2, "dense_decode: the memory to prefetch must be 16-byte aligned");
    const DdBuffers buf = dd_buffers(M, H, I, n_q, n_kv, D, plan);
    static thread_local DdParams p;               // (26 KB: not on the caller's stack)
    u64* at = static_cast<u64*>(s->exchange);
    p.resid = s->resid;
    p.tok_pos = s->tok_pos; p.row_slot = s->row_slot; p.row_ctx = s->row_ctx_len;
    p.status = s->status;
    p.ctrl = reinterpret_cast<unsigned*>(at);
    for (int i = 0; i < 2; ++i) { p.x[i] = at + buf.x[i]; p.ss[i] = at + buf.ss[i]; }
    p.q = at + buf.q; p.kv = at + buf.kv; p.part = at + buf.part; p.attn = at + buf.attn; p.act = at + buf.act; p.dpart = at + buf.dpart;
    p.wait_ns = g_tc_wait_ns == TC_WAIT_NS ? DD_WAIT_NS : g_tc_wait_ns;
    p.skip = g_tc_skip_last;
    p.M = M; p.H = H; p.I = I; p.n_q = n_q; p.n_kv = n_kv;
    p.num_blocks = (int)s->num_blocks; p.block_size = (int)s->block_size;
    p.bs_inv = (0x100000000ull + p.block_size - 1) / p.block_size;
    p.S = plan.S; p.tp = plan.tp; p.n_groups = plan.n_groups; p.n_stages = plan.n_stages; p.kbs = plan.kbs; p.flying = plan.n_stages - 1 < DD_FLYING ? plan.n_stages - 1 : DD_FLYING; p.x_bytes = plan.x_bytes;
    p.splits = dd_splits(M, n_kv, plan.n);
    memcpy(p.gu, plan.gu, sizeof(p.gu));
    for (int l0 = 0; l0 < count; l0 += DD_LAYERS) {
        p.pf_ptr = static_cast<const unsigned char*>(s->next);
        p.pf_bytes = s->next != nullptr && l0 + DD_LAYERS >= count ? (u64)s->next_bytes & ~15ull : 0;
        p.n_layers = count - l0 < DD_LAYERS ? count - l0 : DD_LAYERS;
        for (int i = 0; i < p.n_layers; ++i) {
            const FdDenseLayer& L = layers[l0 + i];
            DdLayer& o = p.layer[i];
            const int g = (int)L.group, r = (int)L.position, qkv = (n_q + 2 * n_kv) * D;
            const struct { const void* w; int rows, cols; } mats[4] = {
                {L.w_qkv, qkv, H}, {L.w_o, H, n_q * D}, {L.w_gate_up, 2 * I, H}, {L.w_down, H, I}};
            for (int k = 0; k < 4; ++k)
                FD_REQUIRE(tensor_map_blocks(mats[k].w, mats[k].rows, mats[k].cols, &o.map[k], 16, plan.kbs) == 0, -4,
                           "dense_decode: no tensor map for a %d x %d matrix", mats[k].rows, mats[k].cols);
            o.norm1 = L.norm1; o.norm2 = L.norm2; o.bias = L.b_qkv;
            o.kp = reinterpret_cast<__nv_bfloat16*>(s->k_base[g] + L.index * s->k_stride[g]);
            o.vp = reinterpret_cast<__nv_bfloat16*>(s->v_base[g] + L.index * s->v_stride[g]);
            o.table = s->table[g]; o.max_blocks = (int)s->max_blocks[g];
            o.cos_t = s->cos_t[r]; o.sin_t = s->sin_t[r]; o.table_len = (int)s->table_len[r];
            o.eps1 = (float)L.eps1; o.eps2 = (float)L.eps2; o.scale = (float)L.scale;
            o.window = (int)L.window; o.chunk = (int)L.chunk;
            o.f32 = (L.norm1_f32 ? 1 : 0) | (L.norm2_f32 ? 2 : 0) | (L.bias_f32 ? 4 : 0);
        }
        switch (plan.NT * 1000 + D) {
            case 1128: rc = dd_launch<128, 1>(p, plan, s->stream); break;
            case 2128: rc = dd_launch<128, 2>(p, plan, s->stream); break;
            case 3128: rc = dd_launch<128, 3>(p, plan, s->stream); break;
            case 1064: rc = dd_launch<64, 1>(p, plan, s->stream); break;
            case 2064: rc = dd_launch<64, 2>(p, plan, s->stream); break;
            default: rc = dd_launch<64, 3>(p, plan, s->stream); break;
        }
        if (rc != 0) return rc;
    }
    return 0;
}
