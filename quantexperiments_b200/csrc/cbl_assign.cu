// Encoder side of the format: nearest codeword of every 8-wide chunk (the "snap" that produces the tags) and the
// little-endian bit packing of the tags.
//
// k_assign     each thread keeps CH chunks in registers and scans the whole book from shared memory (fp32, read as
//              warp-wide broadcasts): 8 fp32 FMAs per (chunk, codeword) starting from |c|^2, i.e. c_sq - 2 x.c in fp32
//              exactly as the reference states it.  The minimum is tracked per group of eight codewords (one min per
//              codeword and one compare per group instead of a compare and two selects per codeword); the winning
//              group is evaluated once more at the end to name the first codeword that reaches the minimum.
//              Bound by the fp32 FMA rate, not by memory: 65 kflop per 44 bytes of traffic.
// k_pack_tags  one thread per 32-bit word of the stream.
#include "cbl_tc.cuh"
#include <cmath>
#include <type_traits>

constexpr int AS_THREADS = 256, AS_GROUP = 8;

// Three-input minimum (one instruction on sm_100).
__device__ __forceinline__ float as_min3(float a, float b, float c) {
    float r;
    asm("min.f32 %0, %1, %2, %3;" : "=f"(r) : "f"(a), "f"(b), "f"(c));
    return r;
}

template <int CH, bool WT>
__global__ void __launch_bounds__(AS_THREADS, 1)
k_assign(const float* __restrict__ x, const float* __restrict__ wt, int64_t n, const void* __restrict__ book, int bdtype, int K, int Kpad,
         int64_t* __restrict__ idx, float* __restrict__ err) {
    extern __shared__ __align__(16) unsigned char as_smem[];
    float4* s_book = (float4*)as_smem;                       // [Kpad][2]
    float* s_init = (float*)(as_smem + (size_t)Kpad * 32);   // |c|^2 (0 when weighted); +inf for the padding
    const int tid = threadIdx.x;
    for (int k = tid; k < Kpad; k += AS_THREADS) {
        float c[8], sq = 0.f;
#pragma unroll
        for (int i = 0; i < 8; i++) {
            c[i] = k < K ? cbl_load_in(book, bdtype, (int64_t)k * 8 + i) : 0.f;
            sq += c[i] * c[i];
        }
        s_book[2 * k] = make_float4(c[0], c[1], c[2], c[3]);
        s_book[2 * k + 1] = make_float4(c[4], c[5], c[6], c[7]);
        s_init[k] = k < K ? (WT ? 0.f : sq) : INFINITY;
    }
    __syncthreads();
    const int64_t per_block = (int64_t)AS_THREADS * CH;
    for (int64_t base = (int64_t)blockIdx.x * per_block; base < n; base += (int64_t)gridDim.x * per_block) {
        float a[CH][8], w[WT ? CH : 1][8], xx[CH], best[CH];
        int bg[CH];
#pragma unroll
        for (int j = 0; j < CH; j++) {
            const int64_t ci = base + (int64_t)j * AS_THREADS + tid;
            float4 lo = make_float4(0, 0, 0, 0), hi = lo, wl = lo, wh = lo;
            if (ci < n) {
                lo = __ldg((const float4*)x + 2 * ci);
                hi = __ldg((const float4*)x + 2 * ci + 1);
                if (WT) { wl = __ldg((const float4*)wt + 2 * ci); wh = __ldg((const float4*)wt + 2 * ci + 1); }
            }
            const float xv[8] = {lo.x, lo.y, lo.z, lo.w, hi.x, hi.y, hi.z, hi.w};
            const float wv[8] = {wl.x, wl.y, wl.z, wl.w, wh.x, wh.y, wh.z, wh.w};
            float s = 0.f;
#pragma unroll
            for (int i = 0; i < 8; i++) {
                if (WT) {
                    w[j][i] = wv[i];
                    a[j][i] = (-2.0f * wv[i]) * xv[i];
                    s += (wv[i] * xv[i]) * xv[i];
                } else {
                    a[j][i] = -2.0f * xv[i];
                    s += xv[i] * xv[i];
                }
            }
            xx[j] = s;
            best[j] = INFINITY;
            bg[j] = 0;
        }
        auto dist = [&](int j, const float4& c0, const float4& c1, float init) -> float {
            const float c[8] = {c0.x, c0.y, c0.z, c0.w, c1.x, c1.y, c1.z, c1.w};
            float d = init;
#pragma unroll
            for (int i = 0; i < 8; i++) {
                if (WT) d = fmaf(c[i], fmaf(w[j][i], c[i], a[j][i]), d);
                else d = fmaf(a[j][i], c[i], d);
            }
            return d;
        };
        for (int k0 = 0; k0 < Kpad; k0 += AS_GROUP) {
            float gm[CH];
#pragma unroll
            for (int j = 0; j < CH; j++) gm[j] = INFINITY;
#pragma unroll
            for (int q = 0; q < AS_GROUP; q += 2) {
                const float4 c0 = s_book[2 * (k0 + q)], c1 = s_book[2 * (k0 + q) + 1];
                const float4 e0 = s_book[2 * (k0 + q) + 2], e1 = s_book[2 * (k0 + q) + 3];
                const float2 init = *(const float2*)(s_init + k0 + q);
#pragma unroll
                for (int j = 0; j < CH; j++) gm[j] = as_min3(gm[j], dist(j, c0, c1, init.x), dist(j, e0, e1, init.y));
            }
#pragma unroll
            for (int j = 0; j < CH; j++)
                if (gm[j] < best[j]) { best[j] = gm[j]; bg[j] = k0; }
        }
#pragma unroll
        for (int j = 0; j < CH; j++) {
            const int64_t ci = base + (int64_t)j * AS_THREADS + tid;
            if (ci >= n) continue;
            int bi = bg[j];
            float bd = INFINITY;
#pragma unroll
            for (int q = 0; q < AS_GROUP; q++) {
                const int k = bg[j] + q;
                const float dq = dist(j, s_book[2 * k], s_book[2 * k + 1], s_init[k]);
                if (dq < bd) { bd = dq; bi = k; }
            }
            idx[ci] = bi < K ? bi : 0;
            err[ci] = fmaxf(bd + xx[j], 0.f);
        }
    }
}

// ------------------------------------------------------------------------------------ unweighted snap on the tensor cores
//
// The same minimum with the distances of a tile of 128 chunks to all codewords on tcgen05.mma, for fp16 books of a multiple
// of 256 words.  A chunk's -2 x is split into two fp16 parts (22 bits; the book is fp16 as it is), |c|^2 into three that
// ride along in the unused half of K = 16:
//     A1 = [hi(-2 x) | f f f 0 0 0 0 0]   A2 = [lo(-2 x) | 0]   B = [c | hi, mid, lo of |c|^2 | 0]
// so A1 B + A2 B = f |c|^2 - 2 x.c in fp32 (f: a power of two per chunk that keeps large chunks inside fp16; 1 otherwise).
// Book and chunks are scaled by one more power of two when the book's largest value is not within 2 .. 64.
// Twelve warps read the distances out of tensor memory (four accumulators of 128 words, taken in turn by three warpgroups) and keep
// the smallest values of the two best groups of 32 words per chunk and warpgroup, the group's number in the value's last six bits.
// Four other warps evaluate the words of the best group - and of every group that is closer than the arithmetic above can tell -
// in fp32 exactly as k_assign does, so that index and error are k_assign's, bit for bit, while the twelve read the next tile.
//
// 8.49 M chunks x 4096 words: 11.1 ms by k_assign (0.65 of the fp32 FMA rate), 2.42 ms here.  The ALU pipe bounds it (77 % busy): a
// three-input minimum takes it two clocks per two values, and the groups' numbers, the two smallest and the exact evaluation
// make 0.9 instructions per value.  With 512 threads that met at a barrier after every tile, a branch per group of 16 and one
// warp that issued all products it took 3.6 ms; four warpgroups of 64 values at a time take 2.5.
constexpr int AT_TILE = 128, AT_N = 128, AT_GROUP = 32, AT_WG = 3, AT_EPI = AT_WG * 128, AT_THREADS = AT_EPI + 256;
constexpr int AT_AUX_WARP = AT_EPI / 32, AT_MMA_WARP = AT_AUX_WARP + 4;
constexpr int AT_A_BYTES = 4096;                 // 128 rows x 16 fp16
constexpr int AT_SQ = 131072;                    // behind the book in MMA order: |c|^2 of every word, as k_assign adds it up
constexpr int AT_BOOK = AT_SQ + 16384;
constexpr int AT_STAGE = 2 * AT_A_BYTES + AT_TILE * 36;         // A1 | A2 | the chunks in fp32 | the scales f
constexpr int AT_SMEM = AT_BOOK + 2 * AT_STAGE + 2 * AT_WG * AT_TILE * 12;
constexpr uint32_t AT_ID = 63;                   // a warpgroup sees a third of 4096 words: 44 groups
constexpr uint32_t AT_WAIT_LIMIT = 1u << 20;

// Bounded wait.  One that expires is remembered (the errors of the block become NaN) and ends the waits after it at once; the roles
// keep their step.
__device__ __forceinline__ void at_wait(uint32_t bar, uint32_t parity, volatile int* abort) {
    for (uint32_t i = 1; i <= AT_WAIT_LIMIT; i++) {
        uint32_t ok;
        asm volatile("{ .reg .pred p; mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2; selp.u32 %0, 1, 0, p; }"
                     : "=r"(ok)
                     : "r"(bar), "r"(parity)
                     : "memory");
        if (ok || ((i & 255u) == 0 && *abort)) return;
    }
    *abort = 1;
}
__device__ __forceinline__ void at_umma(uint32_t d, uint64_t a, uint64_t b, uint32_t idesc, uint32_t accumulate) {
    asm volatile(
        "{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, {%5, %5, %5, %5}, p;\n\t}"
        ::"r"(d), "l"(a), "l"(b), "r"(idesc), "r"(accumulate), "r"(0u)
        : "memory");
}
// K-major without swizzle, K = 16: core matrices of 8 rows x 16 bytes; the two of a row group are 128 bytes apart (leading
// byte offset), row groups 256 (stride byte offset).
__device__ __forceinline__ uint64_t at_desc(uint32_t addr) {
    return (uint64_t)((addr >> 4) & 0x3FFF) | (uint64_t)(128 >> 4) << 16 | (uint64_t)(256 >> 4) << 32 | (uint64_t)1 << 46;
}
__device__ __forceinline__ uint32_t at_row(int r) { return (uint32_t)((r >> 3) * 256 + (r & 7) * 16); }      // first half; the second 128 bytes on
// 64 columns, landed: load and wait are one statement, so that the values are not copied to be tied to the wait.
__device__ __forceinline__ void at_ld64(uint32_t taddr, uint32_t (&v)[32], uint32_t (&u)[32]) {
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x32.b32 {%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, %16, %17, %18, %19, "
        "%20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31}, [%64];\n\t"
        "tcgen05.ld.sync.aligned.32x32b.x32.b32 {%32, %33, %34, %35, %36, %37, %38, %39, %40, %41, %42, %43, %44, %45, %46, %47, %48, %49, %50, %51, "
        "%52, %53, %54, %55, %56, %57, %58, %59, %60, %61, %62, %63}, [%65];\n\t"
        "tcgen05.wait::ld.sync.aligned;"
        : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]), "=r"(v[7]), "=r"(v[8]), "=r"(v[9]),
          "=r"(v[10]), "=r"(v[11]), "=r"(v[12]), "=r"(v[13]), "=r"(v[14]), "=r"(v[15]), "=r"(v[16]), "=r"(v[17]), "=r"(v[18]),
          "=r"(v[19]), "=r"(v[20]), "=r"(v[21]), "=r"(v[22]), "=r"(v[23]), "=r"(v[24]), "=r"(v[25]), "=r"(v[26]), "=r"(v[27]),
          "=r"(v[28]), "=r"(v[29]), "=r"(v[30]), "=r"(v[31]), "=r"(u[0]), "=r"(u[1]), "=r"(u[2]), "=r"(u[3]), "=r"(u[4]),
          "=r"(u[5]), "=r"(u[6]), "=r"(u[7]), "=r"(u[8]), "=r"(u[9]), "=r"(u[10]), "=r"(u[11]), "=r"(u[12]), "=r"(u[13]),
          "=r"(u[14]), "=r"(u[15]), "=r"(u[16]), "=r"(u[17]), "=r"(u[18]), "=r"(u[19]), "=r"(u[20]), "=r"(u[21]), "=r"(u[22]),
          "=r"(u[23]), "=r"(u[24]), "=r"(u[25]), "=r"(u[26]), "=r"(u[27]), "=r"(u[28]), "=r"(u[29]), "=r"(u[30]), "=r"(u[31])
        : "r"(taddr), "r"(taddr + 32)
        : "memory");
}

// Where the chunks come from: an array of them, or rows of a matrix divided by their fp16 scale (zero columns appended).
struct AtSource {
    const float* x;
    const __half* scale;                         // NULL: x is [n][8]
    int C, nch;                                  // columns and chunks of a row
    int64_t ld;
};
__device__ __forceinline__ void at_chunk(const AtSource& s, int64_t ci, float (&v)[8]) {
    if (!s.scale) {
        const float4 lo = __ldg((const float4*)s.x + 2 * ci), hi = __ldg((const float4*)s.x + 2 * ci + 1);
        v[0] = lo.x; v[1] = lo.y; v[2] = lo.z; v[3] = lo.w; v[4] = hi.x; v[5] = hi.y; v[6] = hi.z; v[7] = hi.w;
        return;
    }
    const int64_t r = ci / s.nch;
    const int c = (int)(ci - r * s.nch) * 8;
    const float* p = s.x + r * s.ld + c;
    const float sc = __half2float(s.scale[r]);
    if (c + 8 <= s.C && ((uintptr_t)p & 15) == 0) {
        const float4 lo = __ldg((const float4*)p), hi = __ldg((const float4*)p + 1);
        v[0] = lo.x; v[1] = lo.y; v[2] = lo.z; v[3] = lo.w; v[4] = hi.x; v[5] = hi.y; v[6] = hi.z; v[7] = hi.w;
    } else {
#pragma unroll
        for (int i = 0; i < 8; i++) v[i] = c + i < s.C ? __ldg(p + i) : 0.f;
    }
#pragma unroll
    for (int i = 0; i < 8; i++) v[i] = __fdiv_rn(v[i], sc);
}

struct AtPart { float best; int bg; float second; };           // bg: the best value's group of 32 words

// Word k in fp32.  HOW: 0 as it lies in shared memory, 1 there scaled up, 2 from the book itself (scaled down it may have lost bits).
template <int HOW>
__device__ __forceinline__ void at_word(const unsigned char* smem, const __half* __restrict__ book, float ibs, int k, float (&c)[8]) {
    const uint4 cw = HOW < 2 ? *(const uint4*)(smem + at_row(k)) : __ldg((const uint4*)book + k);
    const __half2* h = (const __half2*)&cw;
#pragma unroll
    for (int i = 0; i < 4; i++) {
        const float2 p = __half22float2(h[i]);
        c[2 * i] = HOW == 1 ? p.x * ibs : p.x;
        c[2 * i + 1] = HOW == 1 ? p.y * ibs : p.y;
    }
}
__device__ __forceinline__ uint64_t at_pair(float lo, float hi) { return (uint64_t)__float_as_uint(hi) << 32 | __float_as_uint(lo); }

// |c_k|^2 - 2 x.c_k of word k, added up as k_assign does.
__device__ __forceinline__ float at_dist(const unsigned char* smem, const __half* __restrict__ book, int q2, float ibs, const float (&x)[8], int k) {
    float c[8];
    if (q2 >= 0) at_word<1>(smem, book, ibs, k, c);
    else at_word<2>(smem, book, ibs, k, c);
    float d = *(const float*)(smem + AT_SQ + 4 * k);
#pragma unroll
    for (int i = 0; i < 8; i++) d = fmaf(-2.0f * x[i], c[i], d);
    return d;
}

// The nearest of words k0 .. k0 + 127, k0 + step .. k0 + step + 127 and so on below k1 to one chunk, for a warp: {distance, index}, the
// first index that reaches the minimum.
__device__ __forceinline__ float2 at_nearest(const unsigned char* words, const __half* __restrict__ book, int q2, float ibs, float4 x0, float4 x1, int k0, int k1, int step) {
    const float xs[8] = {x0.x, x0.y, x0.z, x0.w, x1.x, x1.y, x1.z, x1.w};
    float d0 = INFINITY;
    int i0 = 0;
#pragma unroll 1
    for (; k0 < k1; k0 += step) {
#pragma unroll
        for (int h = 0; h < AT_N; h += 32) {
            const int k = k0 + h + (threadIdx.x & 31);
            const float d = at_dist(words, book, q2, ibs, xs, k);
            if (d < d0 || (d == d0 && k < i0)) { d0 = d; i0 = k; }
        }
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        const float d1 = __shfl_xor_sync(0xffffffffu, d0, o);
        const int i1 = __shfl_xor_sync(0xffffffffu, i0, o);
        if (d1 < d0 || (d1 == d0 && i1 < i0)) { d0 = d1; i0 = i1; }
    }
    return make_float2(d0, __int_as_float(i0));
}

__global__ void __launch_bounds__(AT_THREADS, 1)
k_assign_tc(AtSource src, int64_t n, const __half* __restrict__ book, int K, int64_t* __restrict__ idx, float* __restrict__ err,
            unsigned char* __restrict__ used) {
    extern __shared__ __align__(1024) unsigned char at_smem[];
    __shared__ __align__(8) unsigned long long s_bar[22];
    __shared__ uint32_t s_tmem;
    __shared__ int s_abort;
    __shared__ unsigned int s_max;
    const int tid = threadIdx.x, warp = uniform_warp(tid), lane = tid & 31;
    const uint32_t sb = cbl_smem_u32(at_smem), bar0 = cbl_smem_u32(s_bar);
    auto full_a = [&](int s) { return bar0 + 8u * s; };
    auto acc_empty = [&](int b) { return bar0 + 16u + 8u * b; };
    auto part_full = [&](int s) { return bar0 + 48u + 8u * s; };
    auto part_empty = [&](int s) { return bar0 + 64u + 8u * s; };
    // use u is announced at barrier u % 12: that one is waited for by one warpgroup only (the four accumulators' uses are finished in
    // no certain order, so a barrier per accumulator could be two phases behind the one that looks at its parity)
    auto use_full = [&](uint32_t i) { return bar0 + 80u + 8u * i; };
    AtPart* s_part = (AtPart*)(at_smem + AT_BOOK + 2 * AT_STAGE);      // [2 tiles][3 warpgroups][128 chunks]
    const int64_t ntile = (n + AT_TILE - 1) / AT_TILE;
    // A use of an accumulator: 128 words of a tile; uses are numbered over all of the block's tiles, use u is one of accumulator u & 3.
    const uint32_t nuse = K / AT_N, uses = blockIdx.x < ntile ? (uint32_t)((ntile - blockIdx.x + gridDim.x - 1) / gridDim.x) * nuse : 0u;
    if (tid == 0) {
        s_abort = 0;
        s_max = 0u;
        for (int s = 0; s < 2; s++) {
            mbar_init(full_a(s), 4);
            mbar_init(part_full(s), AT_EPI / 32);
            mbar_init(part_empty(s), 4);
        }
        for (int b = 0; b < 4; b++) mbar_init(acc_empty(b), 4);
        for (int i = 0; i < 12; i++) mbar_init(use_full(i), 1);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == AT_MMA_WARP) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(cbl_smem_u32(&s_tmem)), "r"(512u) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    __syncthreads();
    {
        float mx = 0.f;
        for (int k = tid; k < K * 4; k += AT_THREADS) {
            const uint32_t w = __ldg((const uint32_t*)book + k) & 0x7FFF7FFFu;
            const float2 f = __half22float2(*(const __half2*)&w);
            mx = fmaxf(mx, fmaxf(f.x, f.y));
        }
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, o));
        if (lane == 0) atomicMax(&s_max, __float_as_uint(mx));
    }
    __syncthreads();
    const float top = __uint_as_float(s_max);
    const int q2 = top > 0.f && top < 3.0e38f && (top < 2.f || top >= 64.f) ? (top < 2.f ? 1 : 5) - ilogbf(top) : 0;
    const float bs = ldexpf(1.f, q2);                          // scale of book and chunks
    for (int k = tid; k < K; k += AT_THREADS) {
        const uint4 w = __ldg((const uint4*)book + k);
        const __half2* h = (const __half2*)&w;
        uint4 scaled;
        __half2* g = (__half2*)&scaled;
        float sq = 0.f;
#pragma unroll
        for (int i = 0; i < 4; i++) {
            const float2 f = __half22float2(h[i]);
            g[i] = __floats2half2_rn(f.x * bs, f.y * bs);
            sq += f.x * f.x;
            sq += f.y * f.y;
        }
        ((float*)(at_smem + AT_SQ))[k] = sq;
        sq = sq * bs * bs;
        __align__(16) __half part[8];
#pragma unroll
        for (int i = 0; i < 8; i++) part[i] = __float2half_rn(0.f);
#pragma unroll
        for (int i = 0; i < 3; i++) {
            part[i] = __float2half_rn(sq);
            sq -= __half2float(part[i]);
        }
        unsigned char* row = at_smem + at_row(k);
        *(uint4*)row = scaled;
        *(uint4*)(row + 128) = *(const uint4*)part;
    }
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    const uint32_t tmem = s_tmem;
    auto wait = [&](uint32_t bar, uint32_t parity) {
        at_wait(bar, parity, &s_abort);
        __syncwarp();
    };

    if (warp >= AT_MMA_WARP) {
        // ---------------- MMA issue: a warp per accumulator (one warp for all of them needs some 200 clocks per use, wait and commit
        // included; the products take 128)
        const uint32_t idesc = (1u << 4) | ((uint32_t)(AT_N >> 3) << 17) | ((uint32_t)(AT_TILE >> 4) << 24);
        const int b = warp - AT_MMA_WARP;
        // descriptors hold addresses / 16, in their lowest bits
        const uint64_t stage0 = at_desc(sb + AT_BOOK), book0 = at_desc(sb);
        uint32_t it = 0, j = b, i12 = b, par = 1;
        for (uint32_t use = b; use < uses; use += 4, j += 4, par ^= 1u) {
            for (; j >= nuse; j -= nuse) it++;
            wait(full_a(it & 1), (it >> 1) & 1);
            wait(acc_empty(b), par);
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
            const uint64_t a1 = stage0 + (it & 1) * (AT_STAGE / 16), bd = book0 + j * (AT_N * 32 / 16);
            if (elect_one()) {
                at_umma(tmem + b * AT_N, a1, bd, idesc, 0u);
                at_umma(tmem + b * AT_N, a1 + AT_A_BYTES / 16, bd, idesc, 1u);
                umma_commit(use_full(i12));
            }
            __syncwarp();
            i12 = i12 == b + 8u ? b : i12 + 4u;
        }
    } else if (warp >= AT_AUX_WARP) {
        // ---------------- a thread a chunk of the tile: stages the next tile, then names the nearest words of this one.  A stage
        // is free when its tile is finished (its products were complete before the epilogue's results were).
        const int row = tid - AT_EPI;
        const float ibs = ldexpf(1.f, -q2);
        auto stage = [&](int64_t t, int ab) {
            float v[8];
            const int64_t ci = t * AT_TILE + row;
#pragma unroll
            for (int i = 0; i < 8; i++) v[i] = 0.f;
            if (ci < n) at_chunk(src, ci, v);
            unsigned char* st = at_smem + AT_BOOK + ab * AT_STAGE;
            float mx = 0.f;
#pragma unroll
            for (int i = 0; i < 8; i++) mx = fmaxf(mx, fabsf(v[i]));
            mx *= bs;
            const int e = mx > 8192.f && mx < 3.0e38f ? ilogbf(mx) - 12 : 0;      // |2 x| f < 2^14 (f only shrinks)
            const float f = ldexpf(1.f, -e), fs = -2.0f * f * bs;
            __align__(16) __half hi[8], lo[8], ff[8];
#pragma unroll
            for (int i = 0; i < 8; i++) {
                const float a = fs * v[i];
                hi[i] = __float2half_rn(a);
                lo[i] = __float2half_rn(a - __half2float(hi[i]));
                ff[i] = __float2half_rn(i < 3 ? f : 0.f);
            }
            const uint32_t o = at_row(row);
            *(uint4*)(st + o) = *(const uint4*)hi;
            *(uint4*)(st + o + 128) = *(const uint4*)ff;
            *(uint4*)(st + AT_A_BYTES + o) = *(const uint4*)lo;
            *(uint4*)(st + AT_A_BYTES + o + 128) = make_uint4(0, 0, 0, 0);
            float4* xs = (float4*)(st + 2 * AT_A_BYTES) + row;         // [2][128]: the two halves of the chunks
            xs[0] = make_float4(v[0], v[1], v[2], v[3]);
            xs[AT_TILE] = make_float4(v[4], v[5], v[6], v[7]);
            ((float*)(st + 2 * AT_A_BYTES + AT_TILE * 32))[row] = f;
            asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
            __syncwarp();
            if (lane == 0) mbar_arrive(full_a(ab));
        };
        if (blockIdx.x < ntile) stage(blockIdx.x, 0);
        int it = 0;
        uint32_t base = 0;                                     // number of the tile's first use
        for (int64_t t = blockIdx.x; t < ntile; t += gridDim.x, it++, base += nuse) {
            if (t + gridDim.x < ntile) stage(t + gridDim.x, (it + 1) & 1);
            wait(part_full(it & 1), (it >> 1) & 1);
            const AtPart* const part = s_part + (it & 1) * AT_WG * AT_TILE;
            // the two best groups that each warpgroup has seen
            float best = INFINITY;
            int bg = 0;
#pragma unroll
            for (int q = 0; q < AT_WG; q++) {
                const AtPart p = part[q * AT_TILE + row];
                if (q == 0 || p.best < best) { best = p.best; bg = p.bg; }
            }
            const unsigned char* st = at_smem + AT_BOOK + (it & 1) * AT_STAGE;
            const float4 x0 = ((const float4*)(st + 2 * AT_A_BYTES))[row], x1 = ((const float4*)(st + 2 * AT_A_BYTES))[AT_TILE + row];
            const float f = ((const float*)(st + 2 * AT_A_BYTES + AT_TILE * 32))[row];
            const float xv[8] = {x0.x, x0.y, x0.z, x0.w, x1.x, x1.y, x1.z, x1.w};
            float xx = 0.f;
#pragma unroll
            for (int i = 0; i < 8; i++) xx += xv[i] * xv[i];
            float bd = INFINITY;
            int bi = 0;
            // two words at a time, every lane at another place of its group (a group is 32 x 16 bytes: at the same place, all lanes
            // would read the same four banks)
            auto words = [&](auto how) {
                uint64_t m2x[8];
#pragma unroll
                for (int i = 0; i < 8; i++) m2x[i] = at_pair(-2.0f * xv[i], -2.0f * xv[i]);
#pragma unroll 2
                for (int q = 0; q < AT_GROUP / 2; q++) {
                    const int k0 = bg * AT_GROUP + ((q + lane) & (AT_GROUP / 2 - 1)), k1 = k0 + AT_GROUP / 2;
                    float c0[8], c1[8];
                    at_word<decltype(how)::value>(at_smem, book, ibs, k0, c0);
                    at_word<decltype(how)::value>(at_smem, book, ibs, k1, c1);
                    uint64_t d = at_pair(*(const float*)(at_smem + AT_SQ + 4 * k0), *(const float*)(at_smem + AT_SQ + 4 * k1));
#pragma unroll
                    for (int i = 0; i < 8; i++) asm("fma.rn.f32x2 %0, %1, %2, %0;" : "+l"(d) : "l"(m2x[i]), "l"(at_pair(c0[i], c1[i])));
                    const float d0 = __uint_as_float((uint32_t)d), d1 = __uint_as_float((uint32_t)(d >> 32));
                    if (d0 < bd || (d0 == bd && k0 < bi)) { bd = d0; bi = k0; }
                    if (d1 < bd || (d1 == bd && k1 < bi)) { bd = d1; bi = k1; }
                }
            };
            if (q2 == 0) words(std::integral_constant<int, 0>());
            else if (q2 > 0) words(std::integral_constant<int, 1>());
            else words(std::integral_constant<int, 2>());
            // What two groups' values can be off by against each other.  Relative to the largest term or sum, 2^-24 for each of the 17
            // addends of an MMA, two MMAs, and 2^-23 of the products for the split; of two groups near the minimum d that is at
            // most 2e-5 of |d| + |x|^2.  The group's number in place of the last six bits: 2 x 63 x 2^-23 of |d|.  And the last
            // place of the parts in fp16, 2^-25, times the sizes of a word's eight values.
            // Every group that is no further from the best is evaluated; a warpgroup knows two, so where its second is among them
            // (or the values are not finite) all words that it has seen are, a chunk at a time.
            const float margin = 2e-5f * (fabsf(best) + f * (bs * bs) * xx) + 1.6e-5f * fabsf(best) + 0x1p-23f * (4.f * top * bs + 1.f);
            bool close = false;
#pragma unroll
            for (int q = 0; q < AT_WG; q++) {
                const AtPart p = part[q * AT_TILE + row];
                close |= !((p.bg == bg ? p.second : p.best) - best > margin);
            }
            for (uint32_t todo = __ballot_sync(0xffffffffu, close); todo; todo &= todo - 1) {
                const int who = __ffs(todo) - 1, rw = (warp - AT_AUX_WARP) * 32 + who;
                const float bw = __shfl_sync(0xffffffffu, best, who), mw = __shfl_sync(0xffffffffu, margin, who);
                const float4* xw = (const float4*)(st + 2 * AT_A_BYTES) + rw;
#pragma unroll 1
                for (int q = 0; q < AT_WG; q++) {
                    const AtPart p = part[q * AT_TILE + rw];
                    const bool all = !(p.second - bw > mw);
                    if (!all && !(p.best - bw <= mw)) continue;
                    // its steps of 128 words, or the one that its best group lies in
                    const uint32_t mine = (uint32_t)(q + AT_WG - base % AT_WG) % AT_WG;
                    const int k0 = all ? (int)mine * AT_N : p.bg * AT_GROUP / AT_N * AT_N;
                    const float2 r = at_nearest(at_smem, book, q2, ibs, xw[0], xw[AT_TILE], k0, all ? K : k0 + 1, AT_WG * AT_N);
                    const int i = __float_as_int(r.y);
                    if (lane == who && (r.x < bd || (r.x == bd && i < bi))) { bd = r.x; bi = i; }
                }
            }
            const int64_t ci = t * AT_TILE + row;
            if (ci < n) {
                idx[ci] = bi;
                err[ci] = s_abort ? __int_as_float(0x7fc00000) : fmaxf(bd + xx, 0.f);          // an expired wait shows as NaN
                if (used) used[bi] = 1;
            }
            __syncwarp();
            if (lane == 0) mbar_arrive(part_empty(it & 1));
        }
    } else {
        // ---------------- epilogue: warpgroup w takes every third use; a thread's lane is a chunk of the tile
        const int w = warp >> 2, row = (warp & 3) * 32 + lane;
        const uint32_t t0 = tmem + ((uint32_t)((warp & 3) * 32) << 16);
        const uint32_t zero = (uint32_t)K & 255u;              // orders a load behind the values before it: started early, it would take their registers
        uint32_t use = w, base = 0, i12 = w, par = 0;
        for (int it = 0; base < uses; it++, base += nuse) {
            float best = INFINITY, second = INFINITY;
            const uint32_t j0 = use - base;                    // this warpgroup's first step of the tile
            for (uint32_t g0 = 0; use < base + nuse; use += AT_WG, g0 += 4) {
                const uint32_t ta = t0 + (use & 3) * AT_N;
                wait(use_full(i12), par);
                if ((i12 += AT_WG) >= 12) { i12 -= 12; par ^= 1u; }
                asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                uint32_t va[32], vb[32];
                // minima of two groups with the groups' numbers in their last bits, and the two smallest of all so far: no branch (in some
                // of a warp's lanes nearly every group is among the best two so far)
                auto least = [&](const uint32_t (&v)[32], uint32_t g) {
                    float m = as_min3(__uint_as_float(v[0]), __uint_as_float(v[1]), __uint_as_float(v[2])),
                          o = as_min3(__uint_as_float(v[16]), __uint_as_float(v[17]), __uint_as_float(v[18]));
#pragma unroll
                    for (int q = 3; q < 15; q += 2) {
                        m = as_min3(m, __uint_as_float(v[q]), __uint_as_float(v[q + 1]));
                        o = as_min3(o, __uint_as_float(v[16 + q]), __uint_as_float(v[17 + q]));
                    }
                    m = fminf(as_min3(m, __uint_as_float(v[15]), __uint_as_float(v[31])), o);
                    return __uint_as_float((__float_as_uint(m) & ~AT_ID) | g);
                };
                auto look = [&](uint32_t g) {
                    const float m0 = least(va, g), m1 = least(vb, g + 1), lo = fminf(m0, m1);
                    second = as_min3(second, fmaxf(m0, m1), fmaxf(best, lo));
                    best = fminf(best, lo);
                };
                at_ld64((__float_as_uint(best) & zero) | ta, va, vb);
                look(g0);
                at_ld64((__float_as_uint(best) & zero) | (ta + 64), va, vb);
                asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
                __syncwarp();
                if (lane == 0) mbar_arrive(acc_empty(use & 3));
                look(g0 + 2);
            }
            wait(part_empty(it & 1), ((it >> 1) & 1) ^ 1);
            const uint32_t id = __float_as_uint(best) & AT_ID;
            // the group's number among all words; 0 where no value was finite
            const AtPart mine = {best, best < INFINITY ? (int)((j0 + AT_WG * (id >> 2)) * (AT_N / AT_GROUP) + (id & 3)) : 0, second};
            s_part[((it & 1) * AT_WG + w) * AT_TILE + row] = mine;
            __syncwarp();
            if (lane == 0) mbar_arrive(part_full(it & 1));
        }
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    if (warp == AT_MMA_WARP) {
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(512u) : "memory");
    }
}

static int launch_assign_tc(const AtSource& src, int64_t n, const void* book, int K, int64_t* idx, float* err, unsigned char* used, cudaStream_t st) {
    static bool attr_set[64] = {};
    int dev = 0;
    CBL_CUDA(cudaGetDevice(&dev));
    if (dev >= 0 && dev < 64 && !attr_set[dev]) {
        CBL_CUDA(cudaFuncSetAttribute(k_assign_tc, cudaFuncAttributeMaxDynamicSharedMemorySize, AT_SMEM));
        attr_set[dev] = true;
    }
    const int64_t tiles = (n + AT_TILE - 1) / AT_TILE;
    const int grid = (int)(tiles < cbl_sm_count() ? tiles : cbl_sm_count());
    k_assign_tc<<<grid, AT_THREADS, AT_SMEM, st>>>(src, n, (const __half*)book, K, idx, err, used);
    return cbl_check_launch();
}

extern "C" int cbl_assign_max_codewords() { return 4096; }

extern "C" int cbl_assign(const float* x, const float* wt, int64_t n, int32_t d, const void* book, int bdtype, int32_t K, int64_t* idx,
                          float* err, cbl_stream s) {
    if (!book || n < 0 || K < 1 || (n > 0 && (!x || !idx || !err))) return CBL_EINVAL;
    if (bdtype != CBL_F16 && bdtype != CBL_BF16 && bdtype != CBL_F32) return CBL_EINVAL;
    if (d != 8 || K > 4096) return CBL_EUNSUPPORTED;
    if (((uintptr_t)x % 16) || (wt && ((uintptr_t)wt % 16))) return CBL_EINVAL;
    if (n == 0) return CBL_OK;
    // fp16 books of whole MMA tiles, unweighted, at least a few tiles of chunks: the tensor cores find the candidates
    if (!wt && bdtype == CBL_F16 && K % 256 == 0 && (uintptr_t)book % 16 == 0 && n >= 4 * AT_TILE)
        return launch_assign_tc(AtSource{x, nullptr, 0, 0, 0}, n, book, K, idx, err, nullptr, (cudaStream_t)s);
    const int Kpad = (K + AS_GROUP - 1) / AS_GROUP * AS_GROUP;
    const size_t smem = (size_t)Kpad * 36;
    static bool attr_set[64][2] = {};
    int dev = 0;
    CBL_CUDA(cudaGetDevice(&dev));
    if (dev >= 0 && dev < 64 && !attr_set[dev][wt ? 1 : 0]) {
        if (wt) CBL_CUDA(cudaFuncSetAttribute(k_assign<4, true>, cudaFuncAttributeMaxDynamicSharedMemorySize, 4096 * 36));
        else CBL_CUDA(cudaFuncSetAttribute(k_assign<8, false>, cudaFuncAttributeMaxDynamicSharedMemorySize, 4096 * 36));
        attr_set[dev][wt ? 1 : 0] = true;
    }
    const int ch = wt ? 4 : 8;
    int64_t blocks = (n + (int64_t)AS_THREADS * ch - 1) / ((int64_t)AS_THREADS * ch);
    const int sms = cbl_sm_count();
    // whole waves: every block scans the same number of chunk batches (the last may be short)
    if (blocks > sms) blocks = sms;
    if (wt) k_assign<4, true><<<(unsigned)blocks, AS_THREADS, smem, (cudaStream_t)s>>>(x, wt, n, book, bdtype, K, Kpad, idx, err);
    else k_assign<8, false><<<(unsigned)blocks, AS_THREADS, smem, (cudaStream_t)s>>>(x, wt, n, book, bdtype, K, Kpad, idx, err);
    return cbl_check_launch();
}

// The chunks of w / scale: rows of a matrix divided by their fp16 scale, cut into chunks of 8, zeros appended to the last.
extern "C" int cbl_snap_rows(const float* w, int64_t R, int32_t C, int64_t ld, const void* scale, const void* book, int32_t K, int64_t* idx, float* err,
                             unsigned char* used, cbl_stream s) {
    if (!w || !scale || !book || !idx || !err || R < 0 || C < 1 || ld < C) return CBL_EINVAL;
    if (K < 256 || K > 4096 || K % 256 || (uintptr_t)book % 16) return CBL_EUNSUPPORTED;
    if (R == 0) return CBL_OK;
    const int nch = cbl_ceil_div(C, 8);
    return launch_assign_tc(AtSource{w, (const __half*)scale, C, nch, ld}, R * nch, book, K, idx, err, used, (cudaStream_t)s);
}

// ------------------------------------------------------------------------------------ bit packing
__global__ void __launch_bounds__(256) k_pack_tags(const int64_t* __restrict__ vals, int64_t R, int n, int bits, int W, int32_t* __restrict__ words,
                                                   int* __restrict__ bad) {
    const int64_t gi = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (gi >= R * W) return;
    const int64_t r = gi / W;
    const int wi = (int)(gi % W);
    const int64_t b0 = (int64_t)wi * 32;
    const unsigned long long mask = (1ull << bits) - 1ull;
    unsigned int out = 0;
    for (int t = (int)(b0 / bits); t < n && (int64_t)t * bits < b0 + 32; t++) {
        const unsigned long long full = (unsigned long long)vals[r * n + t], v = full & mask;
        if (bad && full != v) *bad = 1;
        const int64_t sh = (int64_t)t * bits - b0;          // position of the tag's bit 0 relative to the word
        out |= sh >= 0 ? (unsigned int)(v << sh) : (unsigned int)(v >> (-sh));
    }
    words[gi] = (int32_t)out;
}

extern "C" int cbl_pack_tags(const int64_t* vals, int64_t R, int32_t n, int32_t bits, int32_t* words, cbl_stream s) {
    return cbl_pack_tags_checked(vals, R, n, bits, words, nullptr, s);
}

extern "C" int cbl_pack_tags_checked(const int64_t* vals, int64_t R, int32_t n, int32_t bits, int32_t* words, int32_t* bad, cbl_stream s) {
    if (!vals || !words || R < 0 || n < 1 || bits < 1 || bits > 16) return CBL_EINVAL;
    const int W = (int)(((int64_t)n * bits + 31) / 32);
    const int64_t total = R * W;
    if (total == 0) return CBL_OK;
    k_pack_tags<<<(unsigned)((total + 255) / 256), 256, 0, (cudaStream_t)s>>>(vals, R, n, bits, W, words, bad);
    return cbl_check_launch();
}
