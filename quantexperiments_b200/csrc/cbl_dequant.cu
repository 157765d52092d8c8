// Dense decode, tag unpacking and the load-time re-layouts (file layout -> kernel layouts).
#include <cstdlib>
#include <type_traits>
#include "cbl_common.cuh"

int g_cbl_last_cuda_error = 0;

extern "C" int cbl_version(void) { return 100; }
extern "C" int cbl_built_for_sm(void) { return 100; }
extern "C" int cbl_last_cuda_error(void) { return g_cbl_last_cuda_error; }
extern "C" const char* cbl_status_string(int status) {
    switch (status) {
        case CBL_OK: return "ok";
        case CBL_EINVAL: return "invalid argument";
        case CBL_EUNSUPPORTED: return "unsupported shape or format variant";
        case CBL_ECUDA: return "CUDA runtime error";
        case CBL_ETIMEOUT: return "bounded device-side wait expired";
        default: return "unknown status";
    }
}

int cbl_sm_count() {
    static int cached[64];
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) return 148;
    if (cached[dev] == 0) {
        int n = 0;
        if (cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess || n <= 0) n = 148;
        cached[dev] = n;
    }
    return cached[dev];
}

// A kernel launched without early start waits for everything before it, and an early one after it reaches back no further than to it.
__global__ void k_order() {}
extern "C" int cbl_order(cbl_stream s) {
    k_order<<<1, 32, 0, (cudaStream_t)s>>>();
    return cbl_check_launch();
}

static int check_packed(const cbl_packed* m) {
    if (!m || !m->tags || !m->table || !m->row_scale) return CBL_EINVAL;
    if (m->R < 0 || m->C <= 0 || m->d < 1 || m->d > 16 || m->bits < 1 || m->bits > 16) return CBL_EINVAL;
    if (m->C % m->d) return CBL_EINVAL;
    if (m->G < 1 || m->M < 1 || (m->books != 1 && m->books != 2)) return CBL_EINVAL;
    if ((int64_t)m->W * 32 < (int64_t)(m->C / m->d) * m->bits) return CBL_EINVAL;
    if (m->books == 2 && (!m->tags2 || !m->table2 || m->G != 1)) return CBL_EINVAL;
    if (m->G > 1 && !m->row_book) return CBL_EINVAL;
    if (m->M > 1 && (!m->row_mask || !m->perms)) return CBL_EINVAL;
    return CBL_OK;
}

// ------------------------------------------------------------------------------------ dense decode
//
// One thread per chunk.  u = fp32(cw) [+ fp32(cw2)] rounded, then u * fp32(row_scale) rounded, then
// one rounding to the output type: the order of shapequant/packed.py:266 and masks.py:193-200.
template <typename OutT, int D, bool VEC>
__global__ void __launch_bounds__(256) k_dequant(cbl_packed m, OutT* __restrict__ out, int64_t ld, int r0, int64_t nchunks_total) {
    int64_t gi = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (gi >= nchunks_total) return;
    const int d = (D > 0) ? D : m.d;
    const int nch = m.C / d;
    int rr = (int)(gi / nch);
    int j = (int)(gi - (int64_t)rr * nch);
    int r = r0 + rr;
    const uint32_t K = 1u << m.bits;
    uint32_t tag = cbl_read_tag(m.tags + (int64_t)r * m.W, m.W, j, m.bits);
    if (m.row_book) tag += (uint32_t)m.row_book[r] * K;
    const __half* cw = (const __half*)m.table + (int64_t)tag * d;
    const __half* cw2 = nullptr;
    if (m.books == 2) cw2 = (const __half*)m.table2 + (int64_t)cbl_read_tag(m.tags2 + (int64_t)r * m.W, m.W, j, m.bits) * d;
    const float rs = __half2float(((const __half*)m.row_scale)[r]);
    const int32_t* perm = (m.M > 1) ? m.perms + (int64_t)m.row_mask[r] * m.C : nullptr;
    OutT* orow = out + (int64_t)rr * ld;
    if (VEC && D == 8) {
        // M == 1, 8 values per chunk: one 16-byte table read, contiguous aligned stores
        uint4 q = __ldg((const uint4*)cw);
        const __half2* h = (const __half2*)&q;
        float v[8];
#pragma unroll
        for (int i = 0; i < 4; i++) {
            float2 f = __half22float2(h[i]);
            v[2 * i] = f.x;
            v[2 * i + 1] = f.y;
        }
        if (cw2) {
            uint4 q2 = __ldg((const uint4*)cw2);
            const __half2* h2 = (const __half2*)&q2;
#pragma unroll
            for (int i = 0; i < 4; i++) {
                float2 f = __half22float2(h2[i]);
                v[2 * i] = __fadd_rn(v[2 * i], f.x);
                v[2 * i + 1] = __fadd_rn(v[2 * i + 1], f.y);
            }
        }
#pragma unroll
        for (int i = 0; i < 8; i++) v[i] = __fmul_rn(v[i], rs);
        OutT* o = orow + j * 8;
        if (sizeof(OutT) == 4) {
            float4* o4 = (float4*)o;
            o4[0] = make_float4(v[0], v[1], v[2], v[3]);
            o4[1] = make_float4(v[4], v[5], v[6], v[7]);
        } else {
            union { uint4 u; OutT t[8]; } pk;
#pragma unroll
            for (int i = 0; i < 8; i++) pk.t[i] = cbl_cvt_out<OutT>(v[i]);
            *(uint4*)o = pk.u;
        }
    } else {
        for (int i = 0; i < d; i++) {
            float u = __half2float(cw[i]);
            if (cw2) u = __fadd_rn(u, __half2float(cw2[i]));
            u = __fmul_rn(u, rs);
            int c = j * d + i;
            if (perm) c = perm[c];
            orow[c] = cbl_cvt_out<OutT>(u);
        }
    }
}

// The benchmark format (d = 8, 12-bit tags, one table per book): the book(s) live in shared memory and a warp decodes 128
// chunks of a row at a time, lane l chunks l, l + 32, ...: one 16-byte codeword read per chunk and book, stores of a warp
// contiguous.  32 chunks are 12 words of tags, so a lane's word offset and shift are the same in every group of 32 and its
// loads differ by immediates; the next unit's tags are on their way while one is decoded.
//
// HBM-write bound: 18944 x 3584 to fp16 takes 30 us (4.5 TB/s written; 48 us when a tag was located and its bounds were
// checked one by one), 27 us without the scale.  RAW: the codewords
// as they are (two books: the fp16 rounding of their sum), no row scale, for the GEMM that follows.  Otherwise the
// arithmetic of k_dequant; an fp16 result of one book is one fp16 multiplication (the fp32 product of two fp16 values is exact).
constexpr int DQ_THREADS = 512;
// weights from which staging the book(s) in every block pays; with column orders the alternative is scattered stores
constexpr int64_t DQ_MIN_WEIGHTS = 1 << 20, DQ_MIN_WEIGHTS_ORDERS = 1 << 17;
template <typename OutT, int BOOKS, bool RAW>
__device__ __forceinline__ void dq_chunk(const uint4& a, const uint4& b, float rs, __half2 rsh, OutT* __restrict__ o) {
    const __half2* h = (const __half2*)&a;
    const __half2* h2 = (const __half2*)&b;
    if constexpr (sizeof(OutT) == 2) {
        uint4 pk;
        uint32_t* pw = (uint32_t*)&pk;
        if constexpr (RAW && BOOKS == 1) {
            pk = a;
        } else if constexpr (std::is_same<OutT, __half>::value && BOOKS == 1) {
#pragma unroll
            for (int e = 0; e < 4; e++) {
                const __half2 v = __hmul2_rn(h[e], rsh);
                pw[e] = *(const uint32_t*)&v;
            }
        } else {
#pragma unroll
            for (int e = 0; e < 4; e++) {
                float2 f = __half22float2(h[e]);
                if (BOOKS == 2) {
                    const float2 f2 = __half22float2(h2[e]);
                    f.x = __fadd_rn(f.x, f2.x);
                    f.y = __fadd_rn(f.y, f2.y);
                }
                if (!RAW) {
                    f.x = __fmul_rn(f.x, rs);
                    f.y = __fmul_rn(f.y, rs);
                }
                if (std::is_same<OutT, __half>::value) {
                    const __half2 v = __floats2half2_rn(f.x, f.y);
                    pw[e] = *(const uint32_t*)&v;
                } else {
                    const __nv_bfloat162 v = __floats2bfloat162_rn(f.x, f.y);
                    pw[e] = *(const uint32_t*)&v;
                }
            }
        }
        *(uint4*)o = pk;
    } else {
        float v[8];
#pragma unroll
        for (int e = 0; e < 4; e++) {
            float2 f = __half22float2(h[e]);
            if (BOOKS == 2) {
                const float2 f2 = __half22float2(h2[e]);
                f.x = __fadd_rn(f.x, f2.x);
                f.y = __fadd_rn(f.y, f2.y);
            }
            v[2 * e] = __fmul_rn(f.x, rs);
            v[2 * e + 1] = __fmul_rn(f.y, rs);
        }
        ((float4*)o)[0] = make_float4(v[0], v[1], v[2], v[3]);
        ((float4*)o)[1] = make_float4(v[4], v[5], v[6], v[7]);
    }
}

// fp32 results: half a chunk per lane, so that a warp-wide store is contiguous here too.
template <int BOOKS>
__device__ __forceinline__ float4 dq_half(const uint2& a, const uint2& b, float rs) {
    float v[4];
#pragma unroll
    for (int e = 0; e < 2; e++) {
        float2 f = __half22float2(*(const __half2*)(e ? &a.y : &a.x));
        if (BOOKS == 2) {
            const float2 f2 = __half22float2(*(const __half2*)(e ? &b.y : &b.x));
            f.x = __fadd_rn(f.x, f2.x);
            f.y = __fadd_rn(f.y, f2.y);
        }
        v[2 * e] = __fmul_rn(f.x, rs);
        v[2 * e + 1] = __fmul_rn(f.y, rs);
    }
    return make_float4(v[0], v[1], v[2], v[3]);
}
__device__ __forceinline__ uint2 dq_lds64(uint32_t addr) {
    uint2 v;
    asm volatile("ld.shared.v2.u32 {%0,%1}, [%2];" : "=r"(v.x), "=r"(v.y) : "r"(addr));
    return v;
}

// A lane's tag words of one unit of 4 x 32 / LPC chunks from c0 on (LPC lanes per chunk): chunk i x 32 / LPC + lane / LPC, i = 0..3.
// hi is the word that a tag may run into.
struct DqTags { uint32_t lo[4], hi[4]; };
template <int LPC>
__device__ __forceinline__ void dq_fetch(DqTags& t, const int32_t* __restrict__ row, int c0, int nch, int lane, uint32_t sh) {
    constexpr int N = 32 / LPC, W = 12 / LPC;              // chunks and words of a group
    const uint32_t* p = (const uint32_t*)row + (c0 >> 5) * 12 + ((c0 & 31) * 12 >> 5) + ((3 * (lane / LPC)) >> 3);
    const uint32_t* q = p + (sh > 20u ? 1 : 0);
    if (c0 + 4 * N <= nch) {
#pragma unroll
        for (int i = 0; i < 4; i++) {
            t.lo[i] = __ldg(p + W * i);
            t.hi[i] = __ldg(q + W * i);
        }
    } else {
#pragma unroll
        for (int i = 0; i < 4; i++) {
            const bool in = c0 + N * i + lane / LPC < nch;
            t.lo[i] = in ? __ldg(p + W * i) : 0u;
            t.hi[i] = in ? __ldg(q + W * i) : 0u;
        }
    }
}

template <typename OutT, int BOOKS, bool RAW>
__global__ void __launch_bounds__(DQ_THREADS, BOOKS == 1 ? 2 : 1) k_decode_rows(cbl_packed m, OutT* __restrict__ out, int64_t ld, int r0, int r1) {
    extern __shared__ __align__(16) unsigned char dq_smem[];
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    if (RAW) asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
    {
        uint4* dst = (uint4*)dq_smem;
        const uint4* t0 = (const uint4*)m.table;
        for (int i = tid; i < 4096; i += DQ_THREADS) dst[i] = __ldg(t0 + i);
        if (BOOKS == 2) {
            const uint4* t1 = (const uint4*)m.table2;
            for (int i = tid; i < 4096; i += DQ_THREADS) dst[4096 + i] = __ldg(t1 + i);
        }
    }
    constexpr int LPC = sizeof(OutT) == 4 ? 2 : 1, N = 32 / LPC, UC = 4 * N;      // lanes per chunk, chunks of a group and of a unit
    const uint32_t sb = cbl_smem_u32(dq_smem), sh = (12u * (uint32_t)(lane / LPC)) & 31u;
    const int nch = m.C >> 3, nseg = (nch + UC - 1) / UC;
    // units (row, segment) in order, consecutive warps on consecutive segments
    const int stride = gridDim.x * (DQ_THREADS / 32), dr = stride / nseg, ds = stride % nseg;
    const int first = blockIdx.x * (DQ_THREADS / 32) + warp;
    int r = r0 + first / nseg, seg = first % nseg;
    DqTags cur[BOOKS], nxt[BOOKS];
    auto fetch = [&](DqTags (&t)[BOOKS], int row, int sg) {
        if (row < r1) {
            dq_fetch<LPC>(t[0], m.tags + (int64_t)row * m.W, sg * UC, nch, lane, sh);
            if (BOOKS == 2) dq_fetch<LPC>(t[BOOKS - 1], m.tags2 + (int64_t)row * m.W, sg * UC, nch, lane, sh);
        }
    };
    fetch(cur, r, seg);
    __syncthreads();
    while (r < r1) {
        int rn = r + dr, sn = seg + ds;
        if (sn >= nseg) { sn -= nseg; rn++; }
        fetch(nxt, rn, sn);
        const __half rh = RAW ? __half() : ((const __half*)m.row_scale)[r];
        const float rs = RAW ? 0.f : __half2float(rh);
        const __half2 rsh = __half2(rh, rh);
        const int left = nch - seg * UC - lane / LPC;          // this lane's groups that exist: N i < left
        auto slot = [&](int k, int i) { return sb + k * 65536u + ((__funnelshift_r(cur[k].lo[i], cur[k].hi[i], sh) & 0xFFFu) << 4); };
        if constexpr (LPC == 2) {
            uint2 cw[BOOKS][4];
#pragma unroll
            for (int k = 0; k < BOOKS; k++)
#pragma unroll
                for (int i = 0; i < 4; i++) cw[k][i] = dq_lds64(slot(k, i) + (lane & 1) * 8);
            float4* o = (float4*)(out + (int64_t)(r - r0) * ld + seg * UC * 8) + lane;
#pragma unroll
            for (int i = 0; i < 4; i++)
                if (N * i < left) o[i * 32] = dq_half<BOOKS>(cw[0][i], cw[BOOKS - 1][i], rs);
        } else {
            uint4 cw[BOOKS][4];
#pragma unroll
            for (int k = 0; k < BOOKS; k++)
#pragma unroll
                for (int i = 0; i < 4; i++) cw[k][i] = cbl_lds128(slot(k, i));
            OutT* o = out + (int64_t)(r - r0) * ld + seg * UC * 8 + lane * 8;
#pragma unroll
            for (int i = 0; i < 4; i++)
                if (N * i < left) dq_chunk<OutT, BOOKS, RAW>(cw[0][i], cw[BOOKS - 1][i], rs, rsh, o + i * 256);
        }
#pragma unroll
        for (int k = 0; k < BOOKS; k++) cur[k] = nxt[k];
        r = rn;
        seg = sn;
    }
    // RAW runs beside the kernels before it; later kernels that wait for this one also wait for those
    if (RAW) asm volatile("griddepcontrol.wait;" ::: "memory");
}

// The same with column orders: the values of a row go to their columns in a shared-memory copy of the row, which is then
// written out whole (scattered 2-byte stores to global memory cost a sector each).  512 / GR threads per row.
template <typename OutT, int BOOKS, bool RAW>
__global__ void __launch_bounds__(DQ_THREADS, 1) k_decode_rows_perm(cbl_packed m, OutT* __restrict__ out, int64_t ld, int C_out, int GR, int r0, int r1) {
    extern __shared__ __align__(16) unsigned char dq_smem[];
    const int tid = threadIdx.x;
    if (RAW) asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
    {
        uint4* dst = (uint4*)dq_smem;
        const uint4* t0 = (const uint4*)m.table;
        for (int i = tid; i < 4096; i += DQ_THREADS) dst[i] = __ldg(t0 + i);
        if (BOOKS == 2) {
            const uint4* t1 = (const uint4*)m.table2;
            for (int i = tid; i < 4096; i += DQ_THREADS) dst[4096 + i] = __ldg(t1 + i);
        }
    }
    const int nt = DQ_THREADS / GR, grp = tid / nt, t = tid % nt, lane = tid & 31, w = t >> 5;
    const int row_bytes = (C_out * (int)sizeof(OutT) + 15) & ~15;
    unsigned char* buf = dq_smem + BOOKS * 65536 + grp * row_bytes;
    OutT* row = (OutT*)buf;
    const uint32_t sb = cbl_smem_u32(dq_smem), sh = (12u * (uint32_t)lane) & 31u;
    const int nch = m.C >> 3;
    __syncthreads();
    auto meet = [&]() { asm volatile("bar.sync %0, %1;" ::"r"(1 + grp), "r"(nt) : "memory"); };
    for (int r = r0 + blockIdx.x * GR + grp; r < r1; r += gridDim.x * GR) {
        const int32_t* perm = m.perms + (int64_t)m.row_mask[r] * m.C;
        const __half rh = RAW ? __half() : ((const __half*)m.row_scale)[r];
        const float rs = RAW ? 0.f : __half2float(rh);
        const __half2 rsh = __half2(rh, rh);
        if (C_out > m.C) {                                 // a column shard: the columns it does not have are zero
            for (int i = t; i < row_bytes / 16; i += nt) ((uint4*)buf)[i] = make_uint4(0, 0, 0, 0);
            meet();
        }
        for (int c0 = w * 128; c0 < nch; c0 += nt * 4) {
            DqTags tg[BOOKS];
            dq_fetch<1>(tg[0], m.tags + (int64_t)r * m.W, c0, nch, lane, sh);
            if (BOOKS == 2) dq_fetch<1>(tg[BOOKS - 1], m.tags2 + (int64_t)r * m.W, c0, nch, lane, sh);
            int4 pa[4], pb[4];
#pragma unroll
            for (int i = 0; i < 4; i++) {
                const int c = c0 + 32 * i + lane;
                if (c < nch) {
                    pa[i] = __ldg((const int4*)(perm + c * 8));
                    pb[i] = __ldg((const int4*)(perm + c * 8) + 1);
                }
            }
#pragma unroll
            for (int i = 0; i < 4; i++) {
                if (c0 + 32 * i + lane >= nch) continue;
                uint4 cw[BOOKS];
#pragma unroll
                for (int k = 0; k < BOOKS; k++) cw[k] = cbl_lds128(sb + k * 65536u + ((__funnelshift_r(tg[k].lo[i], tg[k].hi[i], sh) & 0xFFFu) << 4));
                __align__(16) OutT v[8];
                dq_chunk<OutT, BOOKS, RAW>(cw[0], cw[BOOKS - 1], rs, rsh, v);
                const int p[8] = {pa[i].x, pa[i].y, pa[i].z, pa[i].w, pb[i].x, pb[i].y, pb[i].z, pb[i].w};
#pragma unroll
                for (int e = 0; e < 8; e++) row[p[e]] = v[e];
            }
        }
        meet();
        OutT* o = out + (int64_t)(r - r0) * ld;
        constexpr int V = 16 / (int)sizeof(OutT);
        const bool vec = ((uintptr_t)o % 16) == 0;
        for (int i = t; i < (vec ? C_out / V : 0); i += nt) ((uint4*)o)[i] = ((const uint4*)buf)[i];
        for (int i = (vec ? C_out / V * V : 0) + t; i < C_out; i += nt) o[i] = row[i];
        meet();
    }
    if (RAW) asm volatile("griddepcontrol.wait;" ::: "memory");
}

// 0 when the fast kernels do not take the matrix; else launches one of them.
template <typename OutT, int BOOKS, bool RAW>
static int launch_decode_rows(const cbl_packed* m, OutT* out, int64_t ld, int C_out, int r0, int r1, cudaStream_t st, bool* taken) {
    constexpr int MAX_SMEM = 227 * 1024;
    const int row_bytes = (C_out * (int)sizeof(OutT) + 15) & ~15;
    const bool perm = m->M > 1;
    int GR = 4;
    while (perm && GR > 0 && BOOKS * 65536 + GR * row_bytes > MAX_SMEM) GR >>= 1;
    *taken = !perm || GR > 0;
    if (!*taken) return CBL_OK;
    const int smem = BOOKS * 65536 + (perm ? GR * row_bytes : 0);
    static bool attr_set[64] = {};
    int dev = 0;
    CBL_CUDA(cudaGetDevice(&dev));
    if (dev >= 0 && dev < 64 && !attr_set[dev]) {
        CBL_CUDA(cudaFuncSetAttribute(k_decode_rows<OutT, BOOKS, RAW>, cudaFuncAttributeMaxDynamicSharedMemorySize, BOOKS * 65536));
        CBL_CUDA(cudaFuncSetAttribute(k_decode_rows_perm<OutT, BOOKS, RAW>, cudaFuncAttributeMaxDynamicSharedMemorySize, MAX_SMEM));
        attr_set[dev] = true;
    }
    const int64_t units = perm ? (int64_t)(r1 - r0 + GR - 1) / GR : ((int64_t)(r1 - r0) * cbl_ceil_div(m->C / 8, sizeof(OutT) == 4 ? 64 : 128) + DQ_THREADS / 32 - 1) / (DQ_THREADS / 32);
    int grid = cbl_sm_count() * (!perm && BOOKS == 1 ? 2 : 1);
    if (grid > units) grid = (int)units;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    cudaLaunchConfig_t cfg = {};
    cfg.stream = st;
    cfg.attrs = attr;
    cfg.numAttrs = RAW ? 1 : 0;
    cfg.gridDim = dim3(grid);
    cfg.blockDim = dim3(DQ_THREADS);
    cfg.dynamicSmemBytes = smem;
    if (perm) CBL_CUDA(cudaLaunchKernelEx(&cfg, k_decode_rows_perm<OutT, BOOKS, RAW>, *m, out, ld, C_out, GR, r0, r1));
    else CBL_CUDA(cudaLaunchKernelEx(&cfg, k_decode_rows<OutT, BOOKS, RAW>, *m, out, ld, r0, r1));
    return cbl_check_launch();
}

template <typename OutT>
static int launch_dequant(const cbl_packed* m, void* out, int64_t ld, int r0, int r1, cudaStream_t st) {
    int64_t n = (int64_t)(r1 - r0) * (m->C / m->d);
    if (n == 0) return CBL_OK;
    int64_t blocks = (n + 255) / 256;
    if (blocks > 0x7fffffffLL) return CBL_EUNSUPPORTED;
    const bool aligned = m->d == 8 && (uintptr_t)m->table % 16 == 0 && (m->books == 1 || (uintptr_t)m->table2 % 16 == 0) && (uintptr_t)out % 16 == 0;
    const bool vec = m->M == 1 && aligned && ld % 8 == 0;
    // enough weights to pay for staging the book(s) in every block: the shared-memory kernels
    if (aligned && (m->M > 1 || vec) && m->bits == 12 && m->G == 1 && !m->row_book && (m->M == 1 || (uintptr_t)m->perms % 16 == 0) &&
        (int64_t)(r1 - r0) * m->C >= (m->M > 1 ? DQ_MIN_WEIGHTS_ORDERS : DQ_MIN_WEIGHTS)) {
        bool taken;
        const int rc = m->books == 1 ? launch_decode_rows<OutT, 1, false>(m, (OutT*)out, ld, m->C, r0, r1, st, &taken)
                                     : launch_decode_rows<OutT, 2, false>(m, (OutT*)out, ld, m->C, r0, r1, st, &taken);
        if (rc || taken) return rc;
    }
    if (vec) k_dequant<OutT, 8, true><<<(unsigned)blocks, 256, 0, st>>>(*m, (OutT*)out, ld, r0, n);
    else k_dequant<OutT, 0, false><<<(unsigned)blocks, 256, 0, st>>>(*m, (OutT*)out, ld, r0, n);
    return cbl_check_launch();
}

extern "C" int cbl_dequant(const cbl_packed* m, void* out, int dtype, int64_t ld, int32_t r0, int32_t r1, cbl_stream s) {
    int rc = check_packed(m);
    if (rc) return rc;
    if (r0 < 0 || r1 < r0 || r1 > m->R || ld < m->C) return CBL_EINVAL;
    if (r0 == r1) return CBL_OK;
    if (!out) return CBL_EINVAL;
    cudaStream_t st = (cudaStream_t)s;
    switch (dtype) {
        case CBL_F32: return launch_dequant<float>(m, out, ld, r0, r1, st);
        case CBL_F16: return launch_dequant<__half>(m, out, ld, r0, r1, st);
        case CBL_BF16: return launch_dequant<__nv_bfloat16>(m, out, ld, r0, r1, st);
        default: return CBL_EINVAL;
    }
}

// ------------------------------------------------------------------------------------ 16-bit decode for the two-phase GEMM
extern "C" size_t cbl_dense_scratch_bytes(int32_t R, int32_t C) {
    if (R < 0 || C < 0) return 0;
    return (size_t)R * ((size_t)(C + 7) / 8 * 8) * 2;
}

// Rows too long for shared memory, with column orders: one thread per chunk, scattered stores.
template <int BOOKS>
__global__ void __launch_bounds__(256) k_decode_raw_scatter(cbl_packed m, __half* __restrict__ out, int64_t ld, int64_t n) {
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
    const int nch = m.C / 8;
    for (int64_t gi = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; gi < n; gi += (int64_t)gridDim.x * blockDim.x) {
        const int r = (int)(gi / nch), j = (int)(gi - (int64_t)r * nch);
        const uint4 a = __ldg((const uint4*)m.table + cbl_read_tag(m.tags + (int64_t)r * m.W, m.W, j, 12));
        uint4 b = a;
        if (BOOKS == 2) b = __ldg((const uint4*)m.table2 + cbl_read_tag(m.tags2 + (int64_t)r * m.W, m.W, j, 12));
        __align__(16) __half v[8];
        dq_chunk<__half, BOOKS, true>(a, b, 0.f, __half2(), v);
        const int32_t* perm = m.perms + (int64_t)m.row_mask[r] * m.C + j * 8;
#pragma unroll
        for (int e = 0; e < 8; e++) out[(int64_t)r * ld + __ldg(perm + e)] = v[e];
    }
    asm volatile("griddepcontrol.wait;" ::: "memory");
}

static int decode_raw_impl(const cbl_packed* m, void* out, int32_t C_out, cbl_stream s) {
    if (!m || !m->tags || !m->table || !out || ((uintptr_t)out % 16) || ((uintptr_t)m->table % 16)) return CBL_EINVAL;
    if (C_out < m->C || (C_out > m->C && m->M <= 1)) return CBL_EINVAL;      // a wider output only makes sense with column orders
    if (m->d != 8 || m->bits != 12 || m->G != 1) return CBL_EUNSUPPORTED;
    if (m->R < 0 || m->C <= 0 || m->C % 8 || (int64_t)m->W * 32 < (int64_t)(m->C / 8) * 12) return CBL_EINVAL;
    if (m->books != 1 && m->books != 2) return CBL_EINVAL;
    if (m->books == 2 && (!m->tags2 || !m->table2 || ((uintptr_t)m->table2 % 16))) return CBL_EINVAL;
    if (m->M > 1 && (!m->row_mask || !m->perms)) return CBL_EINVAL;
    if (m->R == 0) return CBL_OK;
    const int64_t ld = ((int64_t)C_out + 7) / 8 * 8;
    const cudaStream_t st = (cudaStream_t)s;
    bool taken = false;
    if (m->M == 1 || (uintptr_t)m->perms % 16 == 0) {
        const int rc = m->books == 1 ? launch_decode_rows<__half, 1, true>(m, (__half*)out, ld, C_out, 0, m->R, st, &taken)
                                     : launch_decode_rows<__half, 2, true>(m, (__half*)out, ld, C_out, 0, m->R, st, &taken);
        if (rc || taken) return rc;
    }
    const int64_t n = (int64_t)m->R * (m->C / 8);
    if (C_out > m->C) CBL_CUDA(cudaMemsetAsync(out, 0, (size_t)m->R * ld * 2, st));
    const int grid = (int)((n + 255) / 256 < 32768 ? (n + 255) / 256 : 32768);
    if (m->books == 1) k_decode_raw_scatter<1><<<grid, 256, 0, st>>>(*m, (__half*)out, ld, n);
    else k_decode_raw_scatter<2><<<grid, 256, 0, st>>>(*m, (__half*)out, ld, n);
    return cbl_check_launch();
}

extern "C" int cbl_decode_raw(const cbl_packed* m, void* out, cbl_stream s) { return decode_raw_impl(m, out, m ? m->C : 0, s); }

// The same for a column shard of a matrix with several column orders, whose orders name positions of the FULL
// activation vector (C_out of them): the scratch row is C_out wide and the shard's weights land at their positions.
extern "C" int cbl_decode_raw_wide(const cbl_packed* m, void* out, int32_t C_out, cbl_stream s) { return decode_raw_impl(m, out, C_out, s); }

// ------------------------------------------------------------------------------------ tags
__global__ void __launch_bounds__(256) k_unpack(cbl_packed m, const int32_t* __restrict__ words, int32_t* __restrict__ out, int64_t n) {
    int64_t gi = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (gi >= n) return;
    int nch = m.C / m.d;
    int r = (int)(gi / nch), j = (int)(gi - (int64_t)r * nch);
    out[gi] = (int32_t)cbl_read_tag(words + (int64_t)r * m.W, m.W, j, m.bits);
}

extern "C" int cbl_unpack_tags(const cbl_packed* m, int plane, int32_t* out, cbl_stream s) {
    int rc = check_packed(m);
    if (rc) return rc;
    if (!out || plane < 0 || plane >= m->books) return CBL_EINVAL;
    int64_t n = (int64_t)m->R * (m->C / m->d);
    if (n == 0) return CBL_OK;
    k_unpack<<<(unsigned)((n + 255) / 256), 256, 0, (cudaStream_t)s>>>(*m, plane ? m->tags2 : m->tags, out, n);
    return cbl_check_launch();
}

// ------------------------------------------------------------------------------------ t16 layout
//
// Lane (g = lane >> 2, t = lane & 3) of the warp that owns a 16-row tile multiplies rows g and
// g + 8; in step s of a super-step it takes chunk column (ss*16 + s)*4 + t.  Its 32 tags of one
// super-step (i = 2*s + h, h = 0: row g, h = 1: row g + 8) form a 384-bit little-endian stream
// stored as three uint4 at [book][tile][ss][q][lane].
static int t16_nsuper(int C) { return cbl_ceil_div(C / 8, 64); }

extern "C" size_t cbl_t16_bytes(int32_t ntile, int32_t C, int32_t books) {
    if (ntile < 0 || C <= 0 || books < 1) return 0;
    return (size_t)books * ntile * t16_nsuper(C) * 3 * 32 * 16;
}

__global__ void __launch_bounds__(128) k_repack_t16(cbl_packed m, const int32_t* __restrict__ tile_rows, int ntile, int nsuper,
                                                    uint4* __restrict__ out, int64_t nthreads) {
    int64_t gi = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (gi >= nthreads) return;
    int lane = (int)(gi & 31);
    int64_t rest = gi >> 5;
    int ss = (int)(rest % nsuper);
    rest /= nsuper;
    int tile = (int)(rest % ntile);
    int book = (int)(rest / ntile);
    int g = lane >> 2, t = lane & 3;
    const int nch = m.C / 8;
    const int32_t* words = book ? m.tags2 : m.tags;
    int rows[2] = {tile_rows[tile * 16 + g], tile_rows[tile * 16 + g + 8]};
    uint32_t w[13];
#pragma unroll
    for (int i = 0; i < 13; i++) w[i] = 0;
#pragma unroll
    for (int i = 0; i < 32; i++) {
        int sidx = i >> 1, h = i & 1;
        int chunk = (ss * 16 + sidx) * 4 + t;
        uint32_t tag = 0;
        if (rows[h] >= 0 && chunk < nch) tag = cbl_read_tag(words + (int64_t)rows[h] * m.W, m.W, chunk, 12);
        int bit = 12 * i;
        w[bit >> 5] |= tag << (bit & 31);
        if ((bit & 31) > 20) w[(bit >> 5) + 1] |= tag >> (32 - (bit & 31));
    }
    uint4* o = out + (((int64_t)book * ntile + tile) * nsuper + ss) * 96 + lane;
    o[0] = make_uint4(w[0], w[1], w[2], w[3]);
    o[32] = make_uint4(w[4], w[5], w[6], w[7]);
    o[64] = make_uint4(w[8], w[9], w[10], w[11]);
}

extern "C" int cbl_repack_t16(const cbl_packed* m, const int32_t* tile_rows, int32_t ntile, void* out, cbl_stream s) {
    int rc = check_packed(m);
    if (rc) return rc;
    if (m->d != 8 || m->bits != 12 || m->G != 1) return CBL_EUNSUPPORTED;
    if (!tile_rows || !out || ntile < 0 || ((uintptr_t)out % 16)) return CBL_EINVAL;
    int nsuper = t16_nsuper(m->C);
    int64_t n = (int64_t)m->books * ntile * nsuper * 32;
    if (n == 0) return CBL_OK;
    k_repack_t16<<<(unsigned)((n + 127) / 128), 128, 0, (cudaStream_t)s>>>(*m, tile_rows, ntile, nsuper, (uint4*)out, n);
    return cbl_check_launch();
}

// ------------------------------------------------------------------------------------ x16 layout
//
// Column range kr = chunks 16 kr .. 16 kr + 15, row block rb = rows 64 rb .. 64 rb + 63.  Lane (g, t) of a warp owns,
// for each of the block's 8 row tiles rt, the 4 chunks 16 kr + 4 j + t (j = 0..3) of row 64 rb + 8 rt + g: 32 tags,
// tag index 4 rt + j, packed as a 384-bit little-endian stream = three uint4 at [book][kr][rb][3][32 lanes].
extern "C" size_t cbl_x16_bytes(int32_t R, int32_t C, int32_t books) {
    if (R < 0 || C <= 0 || books < 1) return 0;
    return (size_t)books * cbl_ceil_div(C / 8, 16) * cbl_ceil_div(R, 64) * 96 * 16;
}

__global__ void __launch_bounds__(128) k_repack_x16(cbl_packed m, int nkr, int nrb, uint4* __restrict__ out, int64_t nthreads) {
    int64_t gi = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (gi >= nthreads) return;
    const int lane = (int)(gi & 31);
    int64_t rest = gi >> 5;
    const int rb = (int)(rest % nrb);
    rest /= nrb;
    const int kr = (int)(rest % nkr);
    const int book = (int)(rest / nkr);
    const int g = lane >> 2, t = lane & 3;
    const int nch = m.C / 8;
    const int32_t* words = book ? m.tags2 : m.tags;
    uint32_t w[13];
#pragma unroll
    for (int i = 0; i < 13; i++) w[i] = 0;
#pragma unroll
    for (int i = 0; i < 32; i++) {
        const int rt = i >> 2, j = i & 3;
        const int row = rb * 64 + rt * 8 + g, chunk = kr * 16 + 4 * j + t;
        uint32_t tag = 0;
        if (row < m.R && chunk < nch) tag = cbl_read_tag(words + (int64_t)row * m.W, m.W, chunk, 12);
        const int bit = 12 * i;
        w[bit >> 5] |= tag << (bit & 31);
        if ((bit & 31) > 20) w[(bit >> 5) + 1] |= tag >> (32 - (bit & 31));
    }
    uint4* o = out + (((int64_t)book * nkr + kr) * nrb + rb) * 96 + lane;
    o[0] = make_uint4(w[0], w[1], w[2], w[3]);
    o[32] = make_uint4(w[4], w[5], w[6], w[7]);
    o[64] = make_uint4(w[8], w[9], w[10], w[11]);
}

extern "C" int cbl_repack_x16(const cbl_packed* m, void* out, cbl_stream s) {
    int rc = check_packed(m);
    if (rc) return rc;
    if (m->d != 8 || m->bits != 12 || m->G != 1 || m->M != 1) return CBL_EUNSUPPORTED;
    if (!out || ((uintptr_t)out % 16)) return CBL_EINVAL;
    const int nkr = cbl_ceil_div(m->C / 8, 16), nrb = cbl_ceil_div(m->R, 64);
    const int64_t n = (int64_t)m->books * nkr * nrb * 32;
    if (n == 0) return CBL_OK;
    k_repack_x16<<<(unsigned)((n + 127) / 128), 128, 0, (cudaStream_t)s>>>(*m, nkr, nrb, (uint4*)out, n);
    return cbl_check_launch();
}

// ------------------------------------------------------------------------------------ l8 layout
//
// Tile v covers chunk columns 8*(v % ntile1) .. +7 of book v / ntile1.  Row r's 8 tags of the tile
// form a 96-bit little-endian stream; word k of that stream is stored at [v][k][r], so that four
// consecutive rows' k-th words are one aligned 128-bit load.
extern "C" size_t cbl_l8_bytes(int32_t R, int32_t C, int32_t books) {
    if (R < 0 || C <= 0 || books < 1) return 0;
    size_t Rpad = ((size_t)R + 3) / 4 * 4;
    return (size_t)books * cbl_ceil_div(C / 8, 8) * 3 * Rpad * 4;
}

__global__ void __launch_bounds__(256) k_repack_l8(cbl_packed m, int ntile1, int Rpad, uint32_t* __restrict__ out, int64_t nthreads) {
    int64_t gi = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (gi >= nthreads) return;
    int r = (int)(gi % Rpad);
    int v = (int)(gi / Rpad);
    int book = v / ntile1, tile = v % ntile1;
    const int nch = m.C / 8;
    const int32_t* words = book ? m.tags2 : m.tags;
    uint32_t w[4] = {0, 0, 0, 0};
    if (r < m.R) {
#pragma unroll
        for (int c = 0; c < 8; c++) {
            int chunk = tile * 8 + c;
            uint32_t tag = chunk < nch ? cbl_read_tag(words + (int64_t)r * m.W, m.W, chunk, 12) : 0u;
            int bit = 12 * c;
            w[bit >> 5] |= tag << (bit & 31);
            if ((bit & 31) > 20) w[(bit >> 5) + 1] |= tag >> (32 - (bit & 31));
        }
    }
    uint32_t* o = out + (int64_t)v * 3 * Rpad + r;
    o[0] = w[0];
    o[Rpad] = w[1];
    o[2 * (int64_t)Rpad] = w[2];
}

extern "C" int cbl_repack_l8(const cbl_packed* m, void* out, cbl_stream s) {
    int rc = check_packed(m);
    if (rc) return rc;
    if (m->d != 8 || m->bits != 12 || m->G != 1 || m->M != 1) return CBL_EUNSUPPORTED;
    if (!out || ((uintptr_t)out % 16)) return CBL_EINVAL;
    int ntile1 = cbl_ceil_div(m->C / 8, 8);
    int Rpad = (m->R + 3) / 4 * 4;
    int64_t n = (int64_t)m->books * ntile1 * Rpad;
    if (n == 0) return CBL_OK;
    k_repack_l8<<<(unsigned)((n + 255) / 256), 256, 0, (cudaStream_t)s>>>(*m, ntile1, Rpad, (uint32_t*)out, n);
    return cbl_check_launch();
}

// ------------------------------------------------------------------------------------ product for every format the file layout can hold
//
// y[t, r] = round(row_scale[r] * sum_j <table[row_book[r] * K + tag(r, j)] (+ table2[tag2(r, j)]), x[t, perms[row_mask[r]][j d .. j d + d)]>)
// for any chunk length d <= 16, tag width <= 16 bits, several books per matrix (row_book) and several column orders:
// the formats the reference's generic kernel executes and the table-lookup / tensor-core kernels here do not.  A
// warp per row: its lanes take every 32nd chunk, read the codeword from the L1/L2-resident table and the chunk's
// activations through the row's column order, and accumulate up to GEN_TOK tokens in fp32; shuffles add the lanes.
// Not a bandwidth kernel: correctness for the formats outside the benchmark's.
constexpr int GEN_TOK = 4;
__global__ void __launch_bounds__(256) k_gemv_generic(cbl_packed m, const void* __restrict__ x, int xdtype, int ntok, int64_t ldx,
                                                      void* __restrict__ y, int ydtype, int64_t ldy) {
    const int lane = threadIdx.x & 31, r = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
    if (r >= m.R) return;
    const int d = m.d, nch = m.C / d;
    const uint32_t K = 1u << m.bits, boff = m.row_book ? (uint32_t)m.row_book[r] * K : 0u;
    const int32_t* rw = m.tags + (int64_t)r * m.W;
    const int32_t* rw2 = m.books == 2 ? m.tags2 + (int64_t)r * m.W : nullptr;
    const int32_t* perm = m.M > 1 ? m.perms + (int64_t)m.row_mask[r] * m.C : nullptr;
    const float rs = __half2float(((const __half*)m.row_scale)[r]);
    for (int t0 = 0; t0 < ntok; t0 += GEN_TOK) {
        float acc[GEN_TOK];
#pragma unroll
        for (int t = 0; t < GEN_TOK; t++) acc[t] = 0.f;
        for (int j = lane; j < nch; j += 32) {
            const __half* cw = (const __half*)m.table + (int64_t)(boff + cbl_read_tag(rw, m.W, j, m.bits)) * d;
            const __half* cw2 = rw2 ? (const __half*)m.table2 + (int64_t)cbl_read_tag(rw2, m.W, j, m.bits) * d : nullptr;
            for (int i = 0; i < d; i++) {
                float w = __half2float(cw[i]);
                if (cw2) w = __fadd_rn(w, __half2float(cw2[i]));          // the decode's order: the two codewords are added first
                const int c = perm ? perm[j * d + i] : j * d + i;
#pragma unroll
                for (int t = 0; t < GEN_TOK; t++)
                    if (t0 + t < ntok) acc[t] = fmaf(w, cbl_load_in(x, xdtype, (int64_t)(t0 + t) * ldx + c), acc[t]);
            }
        }
#pragma unroll
        for (int t = 0; t < GEN_TOK; t++) {
            float v = acc[t];
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
            if (lane == 0 && t0 + t < ntok) cbl_store_out(y, ydtype, (int64_t)(t0 + t) * ldy + r, v * rs);
        }
    }
}

extern "C" int cbl_gemv_generic(const cbl_packed* m, const void* x, int xdtype, int32_t ntok, int64_t ldx, void* y, int ydtype, int64_t ldy,
                                cbl_stream s) {
    int rc = check_packed(m);
    if (rc) return rc;
    if (!x || !y || ntok < 0 || ldy < m->R) return CBL_EINVAL;
    if (xdtype != CBL_F32 && xdtype != CBL_F16 && xdtype != CBL_BF16) return CBL_EINVAL;
    if (ydtype != CBL_F32 && ydtype != CBL_F16 && ydtype != CBL_BF16) return CBL_EINVAL;
    if (m->R == 0 || ntok == 0) return CBL_OK;
    k_gemv_generic<<<cbl_ceil_div(m->R, 8), 256, 0, (cudaStream_t)s>>>(*m, x, xdtype, ntok, ldx, y, ydtype, ldy);
    return cbl_check_launch();
}
