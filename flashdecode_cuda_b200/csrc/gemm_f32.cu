// C[M, N] = A[M, K] * W[N, K]^T (+ bias[N]) in float32 on the CUDA cores: the matrix product of the true 32-bit path
// (rows that are not 16-byte aligned go to gemm_simt.cu, but for up to 16 rows of A and W of few rows).
//
// Every output element is one fmaf chain over k = 0 .. K-1 in that order, in every kernel and tiling of this file and in
// the general kernel, so a token gives the same bits alone, in a prompt and in any batch; nothing is split over K.  What is
// left to choose is who computes which output and how the operands get there.
#include "common.cuh"

namespace fd {

__device__ __forceinline__ void cp_async16(void* dst, const void* src, bool on) {
    const unsigned d = (unsigned)__cvta_generic_to_shared(dst);
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" :: "r"(d), "l"(src), "r"(on ? 16 : 0) : "memory");
}
__device__ __forceinline__ void cp_async4(void* dst, const void* src, bool on) {
    const unsigned d = (unsigned)__cvta_generic_to_shared(dst);
    asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;" :: "r"(d), "l"(src), "r"(on ? 4 : 0) : "memory");
}
__device__ __forceinline__ void cp_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N> __device__ __forceinline__ void cp_wait() { asm volatile("cp.async.wait_group %0;" :: "n"(N) : "memory"); }

// Two fmaf in one instruction: (c0, c1) <- (a * b0 + c0, a * b1 + c1), each rounded as fmaf rounds.
__device__ __forceinline__ void fma2(unsigned long long& c, unsigned long long aa, unsigned long long b) {
    asm("fma.rn.f32x2 %0, %1, %2, %0;" : "+l"(c) : "l"(aa), "l"(b));
}
__device__ __forceinline__ unsigned long long twice(float a) {
    unsigned long long r;
    asm("mov.b64 %0, {%1, %1};" : "=l"(r) : "f"(a));
    return r;
}
__device__ __forceinline__ float2 halves(unsigned long long v) {
    float2 r;
    asm("mov.b64 {%0, %1}, %2;" : "=f"(r.x), "=f"(r.y) : "l"(v));
    return r;
}

// ---------------------------------------------------------------------------
// more than 16 rows: register tiles
// ---------------------------------------------------------------------------
// A CTA computes BM x BN outputs, a thread TM x TN of them, k in steps of BK.  A thread brings its 16-byte pieces of the
// operands by cp.async into slots of its own, S steps ahead (one step ahead, in registers, a small tile's step was as long
// as a trip to memory: 60 cycles per k with tiles of 32 x 32), and lays them out as [k][row] in one of two buffers, so that the
// rows a thread multiplies are whole float4s.  A warp's pieces are whole rows of BK values (BK / 4 lanes a row, RW rows); row r of
// k is stored at column r + RW * (k / 4), wrapped, so that a warp's 32 values of one store fall into 32 banks.
// Bound by the FMA pipes, and by what shared memory delivers (128 bytes a cycle to all lanes together, read alike or not).  The inner
// loop alone, from shared memory, on all SMs: 63 TFLOP/s in this form (two fmaf per instruction, A's value doubled in a
// register) with 8 x 16 per thread, 62 with 8 x 8, 58 with 8 x 4, 46 with 4 x 4; with single fmaf 59 (8 x 8), with A stored twice 56, with
// both operands left as rows of k 44.  Measured: 2,048 rows of gate/up (17,920 x 1,536) 2.06 ms = 55 TFLOP/s, 400 rows
// 0.53 ms = 42; in the general kernel (gemm_simt.cu) 27.
template <int BM, int BN, int TM, int TN, int BK, int S>
__global__ void __launch_bounds__((BM / TM) * (BN / TN), TM * TN >= 64 ? 2 : 4)
gemm_f32_tile_kernel(const float* __restrict__ A, const float* __restrict__ W, const float* __restrict__ bias,
                     float* __restrict__ C, int M, int N, int K) {
    constexpr int THREADS = (BM / TM) * (BN / TN), KQ = BK / 4, RW = 32 / KQ, RT = THREADS / KQ;
    constexpr int NA = BM / RT, NL = (BM + BN) / RT;                         // 16-byte pieces of a thread per step: of A, of both
    static_assert(BM % RT == 0 && BN % RT == 0 && (BM & (BM - 1)) == 0 && (BN & (BN - 1)) == 0, "whole pieces per thread");
    extern __shared__ __align__(16) float tile_smem[];
    float4* slots = reinterpret_cast<float4*>(tile_smem);                    // [S][NL][THREADS]
    float* As = tile_smem + S * NL * THREADS * 4;                            // [2][BK][BM]
    float* Bs = As + 2 * BK * BM;                                            // [2][BK][BN]
    const int tid = threadIdx.x;
    // 8 x 4 threads of a warp: their reads of a row of B are 128 bytes, of A four groups
    constexpr int TX = BN / TN, WX = TX < 8 ? TX : 8, WY = 32 / WX;
    const int lane = tid & 31, warp = tid >> 5;
    const int tx = (warp % (TX / WX)) * WX + lane % WX, ty = (warp / (TX / WX)) * WY + lane / WX;
    const int m0 = blockIdx.y * BM, n0 = blockIdx.x * BN;
    const int steps = (K + BK - 1) / BK;

    const int prow = tid / KQ, pk = (tid % KQ) * 4;                          // a thread's pieces: rows prow + i * RT, four k from pk on
    const float* src[NL];
    bool on[NL];
#pragma unroll
    for (int i = 0; i < NL; ++i) {
        const int at = i < NA ? m0 + prow + i * RT : n0 + prow + (i - NA) * RT;
        on[i] = at < (i < NA ? M : N);
        src[i] = (i < NA ? A : W) + (on[i] ? (size_t)at * K : 0) + pk;
    }
    auto fetch = [&](int step) {
        if (step < steps) {
            float4* sl = slots + (step % S) * NL * THREADS + tid;
            const int k0 = step * BK;
            const bool in_k = k0 + pk < K;
#pragma unroll
            for (int i = 0; i < NL; ++i) {
                const bool ok = on[i] && in_k;
                cp_async16(sl + i * THREADS, ok ? src[i] + k0 : A, ok);      // zeros beyond K, M and N
            }
        }
        cp_commit();
    };
    float4 held[NL];
    auto take = [&](int step) {
        const float4* sl = slots + (step % S) * NL * THREADS + tid;
#pragma unroll
        for (int i = 0; i < NL; ++i) held[i] = sl[i * THREADS];
    };
    const int shift = RW * (tid % KQ);
    auto spread = [&](int buf) {
#pragma unroll
        for (int i = 0; i < NL; ++i) {
            const int B = i < NA ? BM : BN;
            const int col = (prow + (i < NA ? i : i - NA) * RT + shift) & (B - 1);
            float* d = (i < NA ? As : Bs) + (buf * BK + pk) * B + col;
            d[0] = held[i].x; d[B] = held[i].y; d[2 * B] = held[i].z; d[3 * B] = held[i].w;
        }
    };

    unsigned long long acc[TM][TN / 2];
#pragma unroll
    for (int i = 0; i < TM; ++i)
#pragma unroll
        for (int j = 0; j < TN / 2; ++j) acc[i][j] = 0ull;

    for (int s = 0; s < S; ++s) fetch(s);
    cp_wait<S - 1>();
    take(0);
    spread(0);
    __syncthreads();
    for (int step = 0; step < steps; ++step) {
        const int buf = step & 1;
        const float* as = As + buf * BK * BM;
        const float* bs = Bs + buf * BK * BN;
        const bool more = step + 1 < steps;
        if (more) {
            cp_wait<S - 2>();                     // its pieces of the next step, which go to the other buffer under the products
            take(step + 1);
        }
#pragma unroll
        for (int k = 0; k < BK; ++k) {
            if (k == BK / 2) {
                if (more) spread(buf ^ 1);
                fetch(step + S);                  // into the slots that this thread has spread already
            }
            float a[TM];
            unsigned long long b[TN / 2];
            // a thread's rows (columns) come as groups of four, a quarter or half of the tile apart
#pragma unroll
            for (int i = 0; i < TM; i += 4)
                *reinterpret_cast<float4*>(a + i) =
                    *reinterpret_cast<const float4*>(as + k * BM + ((ty * 4 + (i / 4) * (BM / (TM / 4)) + RW * (k / 4)) & (BM - 1)));
#pragma unroll
            for (int j = 0; j < TN; j += 4)
                *reinterpret_cast<ulonglong2*>(b + j / 2) =
                    *reinterpret_cast<const ulonglong2*>(bs + k * BN + ((tx * 4 + (j / 4) * (BN / (TN / 4)) + RW * (k / 4)) & (BN - 1)));
#pragma unroll
            for (int i = 0; i < TM; ++i) {
                const unsigned long long aa = twice(a[i]);
#pragma unroll
                for (int j = 0; j < TN / 2; ++j) fma2(acc[i][j], aa, b[j]);
            }
        }
        __syncthreads();
    }
    const bool vec = (N & 3) == 0 && (reinterpret_cast<uintptr_t>(C) & 15) == 0;
#pragma unroll
    for (int i = 0; i < TM; ++i) {
        const int m = m0 + (i / 4) * (BM / (TM / 4)) + ty * 4 + (i & 3);
        if (m >= M) continue;
#pragma unroll
        for (int j = 0; j < TN; j += 4) {
            const int n = n0 + (j / 4) * (BN / (TN / 4)) + tx * 4;
            const float2 u = halves(acc[i][j / 2]), v = halves(acc[i][j / 2 + 1]);
            float o[4] = {u.x, u.y, v.x, v.y};
            float* c = C + (size_t)m * N + n;
            if (bias != nullptr) {
#pragma unroll
                for (int e = 0; e < 4; ++e) if (n + e < N) o[e] += bias[n + e];
            }
            if (vec && n < N) *reinterpret_cast<float4*>(c) = make_float4(o[0], o[1], o[2], o[3]);
            else {
#pragma unroll
                for (int e = 0; e < 4; ++e) if (n + e < N) c[e] = o[e];
            }
        }
    }
}

// ---------------------------------------------------------------------------
// few rows: W streamed
// ---------------------------------------------------------------------------
// The decode steps of the 32-bit path.  A CTA takes NT rows of W and MP rows of A; both come in steps of KT through a ring
// of S shared-memory stages (row by row as they lie in memory, rows padded by 16 bytes: eight lanes' float4 reads of eight
// rows then cover all banks).  Four warps fill the ring by cp.async (in the same warps as the chains it took as long as they
// did); a thread of the others runs the chains of TN rows of W with TM rows of A.  Three bounds: HBM for the wide
// matrices; for those with few rows the chain itself, K dependent fmaf of four cycles each; and what shared memory delivers,
// 128 bytes a cycle to all lanes together whether they read the same value or not, which larger TM x TN need less of - but
// then fewer warps are there to hide its latency.  The sizes below are the fastest of those tried at the widths of
// Qwen2.5-1.5B (the tiles of 12 rows: 128 CTAs for its 1,536 columns, of 14: 147 for 2,048); at 8 to 37,888 columns and 64 to 8,960 k none was slower than the
// register-fed kernels before them.  Measured (M rows; us, and before with the loads of
// one step ahead in registers): M 8: 1,536 x 8,960 39 (81), 17,920 x 1,536 31 (73), the head of 151,936
// rows 0.24 ms; M 1: 31 and 23; M 16: 51 and 39.  Two rows of A to a thread instead of one took the first from 43 to 39 (and M 16 with 12
// instead of 16 rows of W from 60 to 51); four, or two rows of W, 52 and more: too few threads.  V16: rows are 16-byte aligned.  G: float4s of k read ahead of the multiplications.
template <int NT, int KT, int S, int MP, int TM, int TN, int G, bool V16>
__global__ void __launch_bounds__(256)
gemm_f32_rows_kernel(const float* __restrict__ A, const float* __restrict__ W, const float* __restrict__ bias,
                     float* __restrict__ C, int M, int N, int K) {
    constexpr int LD = KT + 4, ROWS = NT + MP, E = V16 ? 4 : 1, CH = KT / E;
    extern __shared__ __align__(16) float ring[];                // [S][NT rows of W, MP rows of A][LD]
    const int tid = threadIdx.x;
    const int n0 = blockIdx.x * NT, m0 = blockIdx.y * MP;
    const int steps = (K + KT - 1) / KT;
    if (tid >= 128) {
        // piece c of a step: E floats of row c / CH; a thread's pieces lie in the same columns when CH divides 128
        const int t = tid - 128;
        auto fetch = [&](int step) {
            if (step < steps) {
                float* st = ring + (size_t)(step % S) * ROWS * LD;
                const int k0 = step * KT;
#pragma unroll 4
                for (int c = t; c < ROWS * CH; c += 128) {
                    const int row = c / CH, col = (c % CH) * E;
                    const bool is_w = row < NT;
                    const bool on = k0 + col < K && (is_w ? n0 + row < N : m0 + row - NT < M);
                    const float* src = (is_w ? W + (size_t)(n0 + row) * K : A + (size_t)(m0 + row - NT) * K) + k0 + col;
                    if (V16) cp_async16(st + row * LD + col, on ? src : A, on);      // zeros beyond K, N and M
                    else cp_async4(st + row * LD + col, on ? src : A, on);
                }
            }
            cp_commit();
        };
        for (int s = 0; s < S - 1; ++s) fetch(s);
        for (int step = 0; step < steps; ++step) {
            cp_wait<S - 2>();
            __syncthreads();                     // this step's stage is there, and the stage of the step before is consumed
            fetch(step + S - 1);
        }
        cp_wait<0>();
        return;
    }
    constexpr int NL = NT / TN;                                  // a thread's rows of W are NL apart: neighbouring lanes, neighbouring rows
    const int nl = tid % NL, mg = tid / NL;
    const bool works = mg < MP / TM;
    float acc[TM][TN];
#pragma unroll
    for (int i = 0; i < TM; ++i)
#pragma unroll
        for (int j = 0; j < TN; ++j) acc[i][j] = 0.f;
    for (int step = 0; step < steps; ++step) {
        __syncthreads();
        if (!works) continue;
        const float* st = ring + (size_t)(step % S) * ROWS * LD;
        const float* wr = st + nl * LD;
        const float* ar = st + (NT + mg * TM) * LD;
        float4 w[2][G][TN], a[2][G][TM];
        auto load = [&](int b, int k) {
#pragma unroll
            for (int g = 0; g < G; ++g) {
#pragma unroll
                for (int j = 0; j < TN; ++j) w[b][g][j] = *reinterpret_cast<const float4*>(wr + j * NL * LD + k + g * 4);
#pragma unroll
                for (int i = 0; i < TM; ++i) a[b][g][i] = *reinterpret_cast<const float4*>(ar + i * LD + k + g * 4);
            }
        };
        auto chain = [&](int b) {
#pragma unroll
            for (int g = 0; g < G; ++g) {
#pragma unroll
                for (int i = 0; i < TM; ++i)
#pragma unroll
                    for (int j = 0; j < TN; ++j) acc[i][j] = fmaf(a[b][g][i].x, w[b][g][j].x, acc[i][j]);
#pragma unroll
                for (int i = 0; i < TM; ++i)
#pragma unroll
                    for (int j = 0; j < TN; ++j) acc[i][j] = fmaf(a[b][g][i].y, w[b][g][j].y, acc[i][j]);
#pragma unroll
                for (int i = 0; i < TM; ++i)
#pragma unroll
                    for (int j = 0; j < TN; ++j) acc[i][j] = fmaf(a[b][g][i].z, w[b][g][j].z, acc[i][j]);
#pragma unroll
                for (int i = 0; i < TM; ++i)
#pragma unroll
                    for (int j = 0; j < TN; ++j) acc[i][j] = fmaf(a[b][g][i].w, w[b][g][j].w, acc[i][j]);
            }
        };
        static_assert(KT % (8 * G) == 0, "whole pairs of groups");
        load(0, 0);
#pragma unroll 2
        for (int k = 0; k < KT; k += 8 * G) {
            load(1, k + 4 * G);
            chain(0);
            if (k + 8 * G < KT) load(0, k + 8 * G);
            chain(1);
        }
    }
    if (!works) return;
#pragma unroll
    for (int i = 0; i < TM; ++i) {
        const int m = m0 + mg * TM + i;
        if (m >= M) break;
#pragma unroll
        for (int j = 0; j < TN; ++j) {
            const int n = n0 + j * NL + nl;
            if (n < N) C[(size_t)m * N + n] = bias != nullptr ? acc[i][j] + bias[n] : acc[i][j];
        }
    }
}

template <int NT, int KT, int S, int MP, int TM, int TN, int G, bool V16 = true>
static int launch_rows(const float* A, const float* W, const float* bias, float* C, int M, int N, int K, cudaStream_t stream) {
    static_assert((NT / TN) * (MP / TM) <= 128, "one thread per group of rows of W and of A");
    auto k = gemm_f32_rows_kernel<NT, KT, S, MP, TM, TN, G, V16>;
    constexpr int smem = S * (NT + MP) * (KT + 4) * (int)sizeof(float);
    static_assert(smem <= 227 * 1024, "shared memory of an SM");
    static bool configured = false;
    if (!configured) {
        const cudaError_t e = cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
        if (e != cudaSuccess) return fail(-3, "gemm_f32: cannot get %d bytes of shared memory: %s", smem, cudaGetErrorString(e));
        configured = true;
    }
    k<<<dim3((N + NT - 1) / NT, (M + MP - 1) / MP), 256, smem, stream>>>(A, W, bias, C, M, N, K);
    return check_launch("gemm_f32_rows");
}

template <int BM, int BN, int TM, int TN, int BK, int S>
static int launch_tile(const float* A, const float* W, const float* bias, float* C, int M, int N, int K, cudaStream_t stream) {
    constexpr int threads = (BM / TM) * (BN / TN);
    constexpr int smem = (S + 2) * BK * (BM + BN) * (int)sizeof(float);
    auto k = gemm_f32_tile_kernel<BM, BN, TM, TN, BK, S>;
    static bool configured = false;
    if (!configured) {
        const cudaError_t e = cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
        if (e != cudaSuccess) return fail(-3, "gemm_f32: cannot get %d bytes of shared memory: %s", smem, cudaGetErrorString(e));
        configured = true;
    }
    k<<<dim3((N + BN - 1) / BN, (M + BM - 1) / BM), threads, smem, stream>>>(A, W, bias, C, M, N, K);
    return check_launch("gemm_f32_tile");
}

static int f32_sm_count() {
    static int sms = 0;
    if (sms == 0) {
        int dev = 0;
        cudaGetDevice(&dev);
        cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    }
    return sms > 0 ? sms : 1;      // (no device: the launch says so)
}

static int g_f32_form = 0;       // 0: by the rule below; 1 + i: form i (tests and measurements)

// aligned: A and W 16-byte aligned and K a multiple of 4.  Returns 1 if it does not take the sizes.
int launch_gemm_f32(const float* A, const float* W, const float* bias, float* C, int M, int N, int K, bool aligned,
                    cudaStream_t stream) {
    const int sms = f32_sm_count();
    if (M <= 16) {
        const bool wide = N >= 64 * sms;         // 64 rows of W per CTA still give every SM one
        // rows that are not 16-byte aligned come four bytes a copy: short steps and many CTAs (8 x 333 x 1,537 15 us, 8 x 64 x 65 2.8; with steps
        // of 256 k and 16 rows 39 and 8.0), and the caller's kernel where W has many rows
        if (!aligned) return wide ? 1 : launch_rows<8, 32, 6, 16, 1, 1, 1, false>(A, W, bias, C, M, N, K, stream);
        if (wide) {
            if (M <= 1) return launch_rows<64, 128, 3, 1, 1, 1, 4>(A, W, bias, C, M, N, K, stream);
            if (M <= 2) return launch_rows<64, 128, 3, 2, 1, 1, 4>(A, W, bias, C, M, N, K, stream);
            if (M <= 4) return launch_rows<64, 128, 3, 4, 2, 1, 4>(A, W, bias, C, M, N, K, stream);
            if (M <= 8 && K > 64) return launch_rows<64, 128, 3, 8, 2, 2, 1>(A, W, bias, C, M, N, K, stream);
            return launch_rows<64, 64, 5, 16, 4, 2, 1>(A, W, bias, C, M, N, K, stream);
        }
        // a short chain is not worth a ring of long steps, most of which may lie beyond K (16 x 8 x 64 4.6 us in those, 2.2 here; 16 x 1,536 x 384 6.4 and 4.3)
        if (K <= 384) return launch_rows<16, 64, 4, 16, 2, 1, 4>(A, W, bias, C, M, N, K, stream);
        // Rows of W per CTA: where CTAs outnumber the SMs, some SM has two, which share what its shared memory delivers (rings of up to 114
        // KB: M 8, 2,048 x 1,536 12.9 us in 171 CTAs of 12 rows, 10.0 in 147 of 14) or, where two rings do not fit, follow one another (12 rows
        // at M 16, 117 KB: 22.2 against 12.0 us).  So the fewest of 12, 14 and 16 rows with a CTA per SM; fewer are faster where all have
        // one (M 8, 1,536 columns 9.5, 9.9, 10.8 us).  Where none has: for M of 5 to 8 twelve rows, whose rings fit twice (2,560 columns 13.2 us,
        // with 16 rows, 125 KB, 20.3), for more 16 (18.5, with 12 rows 22.4).  M of 2 to 4 always 16: 12 rows take as long at M 2 (8.8 us for 2,048
        // columns) and longer at M 4 (10.7 against 8.9).  M 1 has no form of 14 (its 12 rows 7.4 us up to 1,776 columns, 16 8.6).
        const int rows = N <= 12 * sms ? 12 : N <= 14 * sms ? 14 : 16;
        if (M <= 1) {
            if (rows == 12) return launch_rows<12, 256, 5, 1, 1, 1, 8>(A, W, bias, C, M, N, K, stream);
            return launch_rows<16, 256, 5, 1, 1, 1, 8>(A, W, bias, C, M, N, K, stream);
        }
        if (M <= 2) return launch_rows<16, 256, 5, 2, 1, 1, 4>(A, W, bias, C, M, N, K, stream);
        if (M <= 4) return launch_rows<16, 256, 5, 4, 1, 1, 4>(A, W, bias, C, M, N, K, stream);
        if (M <= 8) {
            if (rows == 14) return launch_rows<14, 256, 5, 8, 2, 1, 4>(A, W, bias, C, M, N, K, stream);
            if (N > 14 * sms && N <= 16 * sms) return launch_rows<16, 256, 5, 8, 2, 1, 4>(A, W, bias, C, M, N, K, stream);
            return launch_rows<12, 256, 5, 8, 2, 1, 4>(A, W, bias, C, M, N, K, stream);
        }
        if (rows == 12) return launch_rows<12, 256, 4, 16, 2, 1, 4>(A, W, bias, C, M, N, K, stream);
        if (rows == 14) return launch_rows<14, 256, 3, 16, 2, 1, 4>(A, W, bias, C, M, N, K, stream);
        return launch_rows<16, 256, 3, 16, 2, 1, 4>(A, W, bias, C, M, N, K, stream);
    }
    if (!aligned) return 1;
    // The tiling whose fullest SM is through first.  Measured cycles per k (products with 40 to 2,048 rows of 17,920 x 1,536 and
    // 1,536 x 8,960 matrices): of a CTA that has an SM to itself, and per CTA where several share it.  Large tiles feed the FMA pipes
    // best, small ones spread a product of few outputs over more SMs, and the smallest are bound by the chains.
    static const int bm[6] = {128, 64, 64, 32, 32, 32}, bn[6] = {128, 128, 64, 64, 32, 16};
    static const float alone[6] = {185.f, 112.f, 77.f, 44.f, 37.f, 21.f}, shared[6] = {165.f, 107.f, 55.f, 34.f, 22.f, 16.5f};
    int form = g_f32_form - 1;
    if (form < 0) {
        float best = 0.f;
        for (int i = 0; i < 6; ++i) {
            if ((M + bm[i] - 1) / bm[i] > 65535) continue;           // more rows of tiles than a grid has
            const long long tiles = (long long)((M + bm[i] - 1) / bm[i]) * ((N + bn[i] - 1) / bn[i]);
            const float per_sm = (float)((tiles + sms - 1) / sms) * shared[i], t = per_sm > alone[i] ? per_sm : alone[i];
            if (form < 0 || t < best) { form = i; best = t; }
        }
    }
    FD_REQUIRE(form >= 0 && (M + bm[form] - 1) / bm[form] <= 65535, -2, "gemm_f32: M=%d too large for one launch", M);
    switch (form) {
        case 0: return launch_tile<128, 128, 8, 16, 16, 3>(A, W, bias, C, M, N, K, stream);
        case 1: return launch_tile<64, 128, 8, 8, 32, 3>(A, W, bias, C, M, N, K, stream);
        case 2: return launch_tile<64, 64, 8, 4, 32, 3>(A, W, bias, C, M, N, K, stream);
        case 3: return launch_tile<32, 64, 4, 4, 32, 3>(A, W, bias, C, M, N, K, stream);
        case 4: return launch_tile<32, 32, 4, 4, 32, 4>(A, W, bias, C, M, N, K, stream);
        default: return launch_rows<16, 128, 4, 32, 4, 1, 2>(A, W, bias, C, M, N, K, stream);
    }
}

}  // namespace fd

// 0: the rule; 1..6: one of the tilings of the float32 product for more than 16 rows (all give the same bits).
extern "C" int fd_gemm_f32_set_form(int form) {
    FD_REQUIRE(form >= 0 && form <= 6, -2, "gemm_f32: no tiling %d", form);
    fd::g_f32_form = form;
    return 0;
}
