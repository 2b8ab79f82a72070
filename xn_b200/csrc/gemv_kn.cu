// 16-bit (bf16 / f16) matmul of a few rows with a row-major right-hand side: dst[m,n] = lhs[m,k] . rhs[k,n], n
// contiguous, m <= 16, any batch count -- `attn.matmul(&v)` of a decode step (xn-moshi/src/batched_transformer.rs:188)
// and a projection stored [in, out] (the reference's own GPU example, xn-core/examples/basic_cuda.rs:35-56; there it
// is cuBLAS's OP_N, xn-core/src/cuda_backend.rs:208-223).
//
// HBM-bound by the rhs.  The rhs rides the 16-row dimension of mma.sync.m16n8k16 (output columns), the lhs rows its 8
// columns.  The A fragment wants pairs of consecutive k, which in a row-major rhs are a row apart, so a lane loads the
// same 8 columns (16 bytes) of the four k rows 4t .. 4t+3 and pairs them with byte permutes: 4 loads + 16 permutes + 4
// MMAs per 16 k x 64 columns (2 KB).  Eight lanes cover 128 contiguous bytes of a row.  No shared-memory pass over the
// rhs, no transposed copy.  In the accumulator a lane ends up with 8 consecutive columns of an output row: one 16-byte
// store.
// A CTA owns 64 or 128 columns of one entry; its 8 (4 per 64 columns) warps split k, KN_DEPTH steps (8 KB per warp) in
// flight each, two CTAs per SM: about twice the bytes in flight that HBM latency asks for.  Narrow outputs (fewer 64-column strips than SMs) are
// also split along k over the CTAs of a cluster, which add their sums through distributed shared memory.  All sums
// run in a fixed order.
// The CUDA-core kernel that took these calls before (gemm_generic.cu: 64 x 64 output tiles, of which one row was
// used) needed 483 us for p.v of 256 (stream, head) pairs x 1501 keys x 128; this one takes 20.1 us = 4.9 TB/s.
#include <cooperative_groups.h>

#include <type_traits>

#include "common.cuh"

namespace xn {
namespace {

namespace cg = cooperative_groups;

constexpr int KN_WARPS = 8;
constexpr int KN_DEPTH = 4;    // 16-k steps in flight per warp (four 128-bit loads per lane each)
constexpr int KN_COLS = 64;    // output columns per warp
constexpr int KN_SMEM = 96 * 1024;

template <typename T> struct MmaKn;
template <> struct MmaKn<__half> {
    static __device__ __forceinline__ void run(float (&d)[4], unsigned a0, unsigned a1, unsigned a2, unsigned a3, unsigned b0, unsigned b1) {
        asm("mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
            : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
            : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
    }
};
template <> struct MmaKn<__nv_bfloat16> {
    static __device__ __forceinline__ void run(float (&d)[4], unsigned a0, unsigned a1, unsigned a2, unsigned a3, unsigned b0, unsigned b1) {
        asm("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
            : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
            : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
    }
};

// Staged lhs row pitch in bytes: 32 past a multiple of 128, so that the 16 lanes of an 8-byte access phase (four rows x
// four 8-byte pieces) cover all banks once.
__host__ __device__ inline int kn_pitch(int kc) { return (kc * 2 + 127) / 128 * 128 + 32; }

// kc: k elements of this CTA's share that are staged at once (a multiple of 16); share: k elements per CTA of the
// cluster (a multiple of 16).
template <typename T, int MT>
__global__ void __launch_bounds__(KN_WARPS * 32, 2)
gemv_kn16_kernel(T *__restrict__ y, const T *__restrict__ x, const T *__restrict__ w, int m, int n, int k, size_t ldy, size_t ldx,
                 size_t ldw, size_t xb, size_t wb, int share, int kc, int strips, int cw, int vec_x, int vec_y) {
    extern __shared__ __align__(16) unsigned char smem[];
    const int RS = kn_pitch(kc);
    unsigned char *sX = smem;
    float *red = reinterpret_cast<float *>(smem + (size_t)m * RS);  // [warp][MT * 16][32 lanes]
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int g = lane >> 2, t = lane & 3;
    cg::cluster_group cluster = cg::this_cluster();
    const int csize = (int)cluster.num_blocks(), crank = (int)cluster.block_rank();
    const long long strip_id = (long long)blockIdx.x / csize;
    // cw (1 or 2) strips of 64 columns per CTA, kw warps along k per strip
    const int kw = KN_WARPS / cw, wk = warp & (kw - 1), wc = warp / kw;
    const int b = (int)(strip_id / strips), j0 = ((int)(strip_id - (long long)b * strips) * cw + wc) * KN_COLS;
    dependent_begin<false>();

    const T *X = x + (size_t)b * xb;
    const int col = j0 + 8 * g;                       // this lane's 8 output columns
    // Lanes beyond a ragged strip's end read its last 16-byte piece again.  (That piece holds at least one element of the
    // row, so the aligned load stays inside the operand's memory pages; columns >= n are dropped at the store.)
    const T *W = w + (size_t)b * wb + min(col, (n - 1) / 8 * 8);
    const bool whole = col + 8 <= n;
    const int k0 = crank * share, k1 = min(k, k0 + share);

    float acc[MT][4][4];
    const unsigned char *xr[MT];  // this lane's lhs row; accumulator columns beyond m repeat the last row and are dropped
#pragma unroll
    for (int mt = 0; mt < MT; ++mt) {
        xr[mt] = sX + (size_t)min(8 * mt + g, m - 1) * RS + 8 * t;
#pragma unroll
        for (int j = 0; j < 4; ++j)
#pragma unroll
            for (int i = 0; i < 4; ++i) acc[mt][j][i] = 0.0f;
    }

    for (int c0 = k0; c0 < k1; c0 += kc) {
        const int cn = min(kc, k1 - c0), nst = (cn + 15) / 16;
        const int s0 = nst * wk / kw, s1 = nst * (wk + 1) / kw;
        const int full = cn / 16;  // steps whose 16 k rows all exist; the rest is one more step of the last warp
        const int f1 = min(s1, full);
        uint4 v[KN_DEPTH][4];
        const T *p = W + (size_t)(c0 + s0 * 16 + 4 * t) * ldw;
        auto load = [&](int i) {
#pragma unroll
            for (int r = 0; r < 4; ++r) v[i][r] = ldg_stream(p + r * ldw);
            p += 16 * ldw;
        };
#pragma unroll
        for (int i = 0; i < KN_DEPTH; ++i)
            if (s0 + i < f1) load(i);

        if (c0 != k0) __syncthreads();  // every warp is done with the previous chunk
        if (vec_x) {  // rows at 16-byte boundaries, k a multiple of 8
            const int cols8 = nst * 2;
            for (int idx = tid; idx < m * cols8; idx += KN_WARPS * 32) {
                const int row = (int)((unsigned)idx / (unsigned)cols8), c = idx - row * cols8;
                uint4 e = make_uint4(0, 0, 0, 0);
                if (c * 8 < cn) e = ld_act128(X + (size_t)row * ldx + c0 + c * 8);
                *reinterpret_cast<uint4 *>(sX + (size_t)row * RS + c * 16) = e;
            }
        } else {  // any row pitch: a context has whatever length it has; eight loads in flight per thread
            const unsigned short *Xe = reinterpret_cast<const unsigned short *>(X) + c0;
            const int cols = nst * 16;
            for (int row = 0; row < m; ++row)
                for (int cb = tid; cb < cols; cb += KN_WARPS * 32 * 8) {
                    unsigned short e[8];
#pragma unroll
                    for (int q = 0; q < 8; ++q) {
                        const int c = cb + q * KN_WARPS * 32;
                        e[q] = c < cn ? ld_act_u16(Xe + (size_t)row * ldx + c) : (unsigned short)0;
                    }
#pragma unroll
                    for (int q = 0; q < 8; ++q) {
                        const int c = cb + q * KN_WARPS * 32;
                        if (c < cols) *reinterpret_cast<unsigned short *>(sX + (size_t)row * RS + c * 2) = e[q];
                    }
                }
        }
        __syncthreads();

        auto mul = [&](const uint4 (&a)[4], int st) {
            uint2 xv[MT];
#pragma unroll
            for (int mt = 0; mt < MT; ++mt) xv[mt] = *reinterpret_cast<const uint2 *>(xr[mt] + (size_t)st * 32);
            const unsigned w0[4] = {a[0].x, a[0].y, a[0].z, a[0].w}, w1[4] = {a[1].x, a[1].y, a[1].z, a[1].w};
            const unsigned w2[4] = {a[2].x, a[2].y, a[2].z, a[2].w}, w3[4] = {a[3].x, a[3].y, a[3].z, a[3].w};
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                const unsigned a0 = __byte_perm(w0[j], w1[j], 0x5410), a1 = __byte_perm(w0[j], w1[j], 0x7632);
                const unsigned a2 = __byte_perm(w2[j], w3[j], 0x5410), a3 = __byte_perm(w2[j], w3[j], 0x7632);
#pragma unroll
                for (int mt = 0; mt < MT; ++mt) MmaKn<T>::run(acc[mt][j], a0, a1, a2, a3, xv[mt].x, xv[mt].y);
            }
        };
        int st = s0;
        for (; st + KN_DEPTH <= f1; st += KN_DEPTH) {
#pragma unroll
            for (int i = 0; i < KN_DEPTH; ++i) {
                mul(v[i], st + i);
                if (st + i + KN_DEPTH < f1) load(i);
            }
        }
#pragma unroll
        for (int i = 0; i < KN_DEPTH; ++i)
            if (st + i < f1) mul(v[i], st + i);
        if (s1 > full) {  // rows beyond the end count as zeros
            uint4 a[4];
#pragma unroll
            for (int r = 0; r < 4; ++r) {
                const int kk = full * 16 + 4 * t + r;
                a[r] = kk < cn ? ldg_stream(W + (size_t)(c0 + kk) * ldw) : make_uint4(0, 0, 0, 0);
            }
            mul(a, full);
        }
    }

    // Sum over a strip's warps in k order: value v = (mt * 4 + j) * 4 + i of every lane.
    constexpr int VALS = MT * 16 * 32;
#pragma unroll
    for (int mt = 0; mt < MT; ++mt)
#pragma unroll
        for (int j = 0; j < 4; ++j)
#pragma unroll
            for (int i = 0; i < 4; ++i) red[warp * VALS + (mt * 16 + j * 4 + i) * 32 + lane] = acc[mt][j][i];
    __syncthreads();
    // the slots of a strip's first warp take its totals
    for (int e = tid; e < cw * VALS; e += KN_WARPS * 32) {
        float *p = red + (e / VALS) * kw * VALS + e % VALS;
        float s = p[0];
        for (int o = 1; o < kw; ++o) s += p[o * VALS];
        p[0] = s;
    }
    if (csize > 1) {
        cluster.sync();  // every CTA's totals are in its shared memory
        if (crank == 0)
            for (int e = tid; e < cw * VALS; e += KN_WARPS * 32) {
                float *p = red + (e / VALS) * kw * VALS + e % VALS;
                float s = p[0];
                for (int r = 1; r < csize; ++r) s += *cluster.map_shared_rank(p, r);
                p[0] = s;
            }
        cluster.sync();  // no CTA leaves while its shared memory is read
        if (crank != 0) return;
    } else {
        __syncthreads();
    }
    // lane (g, t) of tile mt: rows 2t, 2t+1 of the eight, columns 8g .. 8g+7 of the strip; the strip's first warps store
    if (wk < MT * 2) {
        const float *sum = red + wc * kw * VALS;
        const int mt = wk >> 1, h = wk & 1, row = 8 * mt + 2 * t + h;
        if (row < m && col < n) {
            T o[8];
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                o[2 * j] = from_f32<T>(sum[(mt * 16 + j * 4 + h) * 32 + lane]);
                o[2 * j + 1] = from_f32<T>(sum[(mt * 16 + j * 4 + 2 + h) * 32 + lane]);
            }
            T *Y = y + (size_t)b * m * n + (size_t)row * ldy + col;
            if (whole && vec_y) {
                *reinterpret_cast<uint4 *>(Y) = *reinterpret_cast<const uint4 *>(o);
            } else {
#pragma unroll
                for (int q = 0; q < 8; ++q)
                    if (col + q < n) Y[q] = o[q];
            }
        }
    }
}

template <typename T, int MT>
int launch(T *y, const T *x, const T *w, int m, size_t n, size_t k, size_t batch, size_t xb, size_t wb, size_t ldy, size_t ldx,
           size_t ldw, cudaStream_t st) {
    // Two strips per CTA where that still gives every SM one: the lhs rows are staged once for both, and twice as many
    // entries are on the machine at once (256 entries of 128 columns: all of them, instead of 1.7 rounds).
    const int cw = n > KN_COLS && (n + 2 * KN_COLS - 1) / (2 * KN_COLS) * batch >= (size_t)sm_count() ? 2 : 1;
    const size_t strips = (n + cw * KN_COLS - 1) / (cw * KN_COLS), units = strips * batch;
    // A cluster splits k while that still leaves every CTA of it an SM of its own and each warp two steps.
    int csize = 1;
    while (csize < 8 && units * csize * 2 <= (size_t)sm_count() && k / (size_t)(csize * 2) >= (size_t)KN_WARPS * 32) csize *= 2;
    const size_t share = ((k + csize - 1) / csize + 15) / 16 * 16;
    // largest multiple of 16 whose staged rows leave room for the warps' sums
    const size_t red = (size_t)KN_WARPS * MT * 16 * 32 * sizeof(float);
    size_t kc = share;
    while ((size_t)m * kn_pitch((int)kc) + red > (size_t)KN_SMEM) kc = (kc / 2 + 15) / 16 * 16;
    const size_t smem = (size_t)m * kn_pitch((int)kc) + red;
    auto kern = gemv_kn16_kernel<T, MT>;
    XN_ENSURE_SMEM(kern, smem);
    const int vec_x = ldx % 8 == 0 && xb % 8 == 0 && k % 8 == 0 && aligned(x, 16);
    const int vec_y = ldy % 8 == 0 && ((size_t)m * n) % 8 == 0 && aligned(y, 16);
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)(units * csize));
    cfg.blockDim = dim3(KN_WARPS * 32);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = st;
    cudaLaunchAttribute attr[2];
    int na = 0;
    if (pdl_enabled()) {
        attr[na].id = cudaLaunchAttributeProgrammaticStreamSerialization;
        attr[na++].val.programmaticStreamSerializationAllowed = 1;
    }
    if (csize > 1) {
        attr[na].id = cudaLaunchAttributeClusterDimension;
        attr[na].val.clusterDim.x = (unsigned)csize;
        attr[na].val.clusterDim.y = 1;
        attr[na++].val.clusterDim.z = 1;
    }
    cfg.attrs = attr;
    cfg.numAttrs = na;
    XN_CHECK_CUDA(cudaLaunchKernelEx(&cfg, kern, y, x, w, m, (int)n, (int)k, ldy, ldx, ldw, xb, wb, (int)share, (int)kc, (int)strips,
                                     cw, vec_x, vec_y));
    return XN_OK;
}

// dst rows at a pitch of `ldd` elements, the columns [k, ldd) left as they are
__global__ void __launch_bounds__(256)
repitch_rows_kernel(unsigned short *dst, const unsigned short *src, size_t rows, size_t m, int k, int ldd,
                    size_t lds, size_t src_bs) {
    dependent_begin();
    for (size_t r = (size_t)blockIdx.x * 8 + (threadIdx.x >> 5); r < rows; r += (size_t)gridDim.x * 8) {
        const unsigned short *s = src + r / m * src_bs + r % m * lds;
        unsigned short *d = dst + r * ldd;
        for (int c = threadIdx.x & 31; c < k; c += 32) d[c] = ld_act_u16(s + c);
    }
}

}  // namespace

bool gemv_kn16_fits(size_t m, size_t n, size_t k, size_t batch) {
    return m <= 16 && n <= 0x7fffff00 && k <= 0x7fffff00 && batch <= 0x7fffffff &&
           ((n + KN_COLS - 1) / KN_COLS) * batch * 8 <= 0x7fffffff;
}

// Caller guarantees: f16 or bf16, lhs k-contiguous (any pitch), rhs n-contiguous with rows and entries at 16-byte
// boundaries, dst rows contiguous and an entry's rows inside m * n elements, gemv_kn16_fits.
int launch_gemv_kn16(xn_dtype dt, void *dst, const void *lhs, const void *rhs, size_t m, size_t n, size_t k, size_t batch,
                     size_t lhs_bs, size_t rhs_bs, size_t dst_rs, size_t lhs_rs, size_t rhs_rs, cudaStream_t st) {
    auto go = [&](auto *d) {
        using T = std::remove_pointer_t<decltype(d)>;
        const T *l = (const T *)lhs, *r = (const T *)rhs;
        if (m <= 8) return launch<T, 1>(d, l, r, (int)m, n, k, batch, lhs_bs, rhs_bs, dst_rs, lhs_rs, rhs_rs, st);
        return launch<T, 2>(d, l, r, (int)m, n, k, batch, lhs_bs, rhs_bs, dst_rs, lhs_rs, rhs_rs, st);
    };
    return dt == XN_F16 ? go((__half *)dst) : go((__nv_bfloat16 *)dst);
}

// The same product with more rows than the kernel above takes, for an lhs whose rows do not start at 16-byte boundaries
// (attention probabilities over a context of any length): TMA cannot address it, so its rows are copied to a pitch it
// can, which costs one pass over m x k elements, and the tensor-memory kernel takes the product.  The map's k extent
// stays k: what lies between k and the pitch is never read.  *taken = false, with nothing enqueued, where there is no scratch to
// be had -- above REPITCH_MAX_SCRATCH (REPITCH_MAX_CAPTURED for a graph, which keeps its block), or when the allocation fails;
// the caller's any-stride kernel then takes the call (32 x 100 x 128 x 1501 bf16: 202 us against 19).
constexpr size_t REPITCH_MAX_SCRATCH = (size_t)512 << 20, REPITCH_MAX_CAPTURED = (size_t)64 << 20;
int launch_gemm_kn_repitched(xn_dtype dt, void *dst, const void *lhs, const void *rhs, size_t m, size_t n, size_t k, size_t batch,
                             size_t lhs_bs, size_t rhs_bs, size_t dst_rs, size_t lhs_rs, size_t rhs_rs, cudaStream_t st, bool *taken) {
    const size_t lda = (k + 7) / 8 * 8;
    *taken = false;
    cudaStreamCaptureStatus cap = cudaStreamCaptureStatusNone;
    XN_CHECK_CUDA(cudaStreamIsCapturing(st, &cap));
    const size_t most_bytes = cap == cudaStreamCaptureStatusNone ? REPITCH_MAX_SCRATCH : REPITCH_MAX_CAPTURED;
    if (batch > most_bytes / m || batch * m > most_bytes / (lda * 2)) return XN_OK;
    const size_t rows = batch * m;
    void *tmp = nullptr;
    ScratchHold hold(st);
    if (launch_scratch(st, rows * lda * 2, SCRATCH_MAIN, &tmp)) return XN_OK;
    *taken = true;
    const size_t blocks = (rows + 7) / 8, most = (size_t)sm_count() * 8;
    if (int rc = launch_dependent(repitch_rows_kernel, dim3((unsigned)(blocks < most ? blocks : most)), dim3(256), 0, st,
                                  (unsigned short *)tmp, (const unsigned short *)lhs, rows, m, (int)k, (int)lda, lhs_rs, lhs_bs))
        return rc;
    return launch_gemm_kn_16bit(dt, dst, tmp, rhs, m, n, k, lda, rhs_rs, dst_rs, batch, m * lda, rhs_bs, st);
}

}  // namespace xn
