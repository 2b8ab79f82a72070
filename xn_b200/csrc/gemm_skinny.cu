// Matmul of up to 128 activation rows against a weight on the tensor cores: y[M, N] = x[M, K] * W^T with W [N, K]
// (e4m3, bf16, f16) or W [K, N] (16-bit, n contiguous).  The decode-time linear of
// a batch of streams (xn-core/src/nn/linear.rs:56-66), HBM-bound by the weights.
//
// The operands swap roles: the 128 tensor-memory lanes carry 128 output channels and the MMA's N dimension carries the
// activation rows (one or two e4m3 pieces of MB rows each, back to back, so one MMA covers both), so almost all bytes in
// flight are weight bytes.  A CTA is one (128 channels, range of k) unit: TMA fills a ring of 128-byte k stages, one
// thread issues tcgen05.mma, four warps read the accumulator back.
//
// Splitting.  A decode-sized weight has fewer 128-channel tiles than the machine has places for CTAs (two per SM: about
// 110 KB of shared memory and at most 256 tensor-memory columns each), so k is cut into S <= 8 ranges that form a
// thread-block cluster.  Each CTA sends the accumulator columns it does not own to their owner's shared memory
// (column c belongs to rank c mod S), one cluster barrier later every owner adds its S partials in k order and stores
// whole rows.  Nothing goes through global memory and nothing waits for another cluster; the sums run in a fixed order.
// The form this replaces cut the work evenly over all SMs and handed partial tiles over through global scratch (store,
// fence, atomic, reload: about 5 of its 10-17 us).  Two CTAs per SM also overlap one's set-up and epilogue with the
// other's loads, and the next launch's weights are fetched before its dependency wait.
// Measured: see the table at the launcher.
#include "tc05.cuh"

namespace xn {
namespace {

constexpr int SK_THREADS = 192;  // warp 0 TMA, warp 1 MMA and tensor memory, warps 2-5 epilogue
constexpr int SK_MAX_STAGES = 8;

struct SkinnyArgs {
    void *y;                         // [M, ldy] bf16 (e4m3 and bf16 operands) or f16
    const float *x_scale, *w_scale;  // e4m3 operands only
    const void *bias;                // optional, 16-bit operands: added to the rounded product and rounded again
    int ldy, M, N, K;
    int MB;      // M rounded up to 16
    int np;      // pieces per activation (1 or 2)
    int nstage;
    int S;       // CTAs per cluster = ranges of k
    int w_static;  // the weights are a model parameter: they may be fetched before the dependency wait
    WaitCtx wait;
};

__device__ __forceinline__ void cluster_arrive() { asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory"); }
__device__ __forceinline__ void cluster_wait() { asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory"); }

__device__ __forceinline__ void tmem_ld16(uint32_t taddr, uint32_t (&v)[16]) {
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];"
        : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]), "=r"(v[7]), "=r"(v[8]),
          "=r"(v[9]), "=r"(v[10]), "=r"(v[11]), "=r"(v[12]), "=r"(v[13]), "=r"(v[14]), "=r"(v[15])
        : "r"(taddr));
    asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
}

template <int KIND> struct Out { using T = __nv_bfloat16; };
template <> struct Out<2> { using T = __half; };

// KIND: 0 = e4m3 pieces -> bf16 (scaled), 1 = bf16, 2 = f16.  MN: W is [K, N] with n contiguous.
template <int KIND, bool MN>
__global__ void __launch_bounds__(SK_THREADS)
gemm_skinny_kernel(const __grid_constant__ CUtensorMap map_w, const __grid_constant__ CUtensorMap map_x0,
                   const __grid_constant__ CUtensorMap map_x1, const SkinnyArgs args) {
    constexpr bool F8 = KIND == 0;
    constexpr int BK = F8 ? BKB : BKB / 2;  // k elements per stage
    constexpr int W_BYTES = BM * BKB;
    using T = typename Out<KIND>::T;
    const int X_BYTES = args.MB * BKB, STAGE_BYTES = W_BYTES + args.np * X_BYTES, NSTAGE = args.nstage;
    const int NB = args.np * args.MB;  // MMA N dimension; columns [0, MB) are the hi products, [MB, 2 MB) the lo ones
    const uint32_t IDESC = (KIND == 1 ? instr_desc(1, 1, NB) : instr_desc(0, 0, NB)) | (MN ? 1u << 15 : 0u);  // bit 15: A is MN-major
    const int TMEM_COLS = NB <= 32 ? 32 : (NB <= 64 ? 64 : (NB <= 128 ? 128 : 256));

    extern __shared__ unsigned char smem_raw[];
    unsigned char *smem = reinterpret_cast<unsigned char *>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~(uintptr_t)1023);
    // partials received from the cluster, [S][columns per owner][128] f32; a single CTA reuses its drained ring
    float *red = reinterpret_cast<float *>(args.S > 1 ? smem + (size_t)NSTAGE * STAGE_BYTES : smem);
    __shared__ __align__(8) uint64_t full[SK_MAX_STAGES], empty[SK_MAX_STAGES], tmem_full;
    __shared__ uint32_t tmem_slot;

    const int warp = warp_id(), lane = threadIdx.x & 31;
    const int S = args.S;
    const int rank = S > 1 ? (int)(blockIdx.x % (unsigned)S) : 0;  // clusters are runs of S consecutive CTAs
    const int tile = (int)(blockIdx.x / (unsigned)S);
    const int num_kb = (args.K + BK - 1) / BK;
    const int kb0 = num_kb * rank / S, kb1 = num_kb * (rank + 1) / S, nkb = kb1 - kb0;
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
    if (S > 1) cluster_arrive();  // completed by the wait ahead of the first remote store: every CTA has started

    if (threadIdx.x == 0) {
        prefetch_tmap(&map_w);
        prefetch_tmap(&map_x0);
        if (args.np == 2) prefetch_tmap(&map_x1);
        for (int s = 0; s < NSTAGE; ++s) { mbar_init(&full[s], 1); mbar_init(&empty[s], 1); }
        mbar_init(&tmem_full, 1);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    }
    if (warp == 1) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&tmem_slot)), "r"(TMEM_COLS)
                     : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    const uint32_t tmem_base = tmem_slot;

    bool ok = true;
    if (warp == 0) {
        if (elect_one()) {
            auto load_w = [&](int it) {
                unsigned char *st = smem + (size_t)(it % NSTAGE) * STAGE_BYTES;
                uint64_t *bar = &full[it % NSTAGE];
                const int k = (kb0 + it) * BK;
                if (MN) {  // two blocks of 64 channels x 64 k
#pragma unroll
                    for (int i = 0; i < 2; ++i)
                        tma_load_3d(st + i * (64 * BKB), &map_w, tile * BM + 64 * i, k, 0, bar);
                } else {
                    tma_load_3d(st, &map_w, k, tile * BM, 0, bar);
                }
            };
            const int pre = min(NSTAGE, nkb);
            if (!args.w_static) asm volatile("griddepcontrol.wait;" ::: "memory");  // the previous kernel may have written w
            for (int it = 0; it < pre; ++it) {
                mbar_expect_tx_only(&full[it], (unsigned)W_BYTES);
                load_w(it);
            }
            asm volatile("griddepcontrol.wait;" ::: "memory");
            for (int it = 0; it < nkb; ++it) {
                const int s = it % NSTAGE, k = (kb0 + it) * BK;
                unsigned char *st = smem + (size_t)s * STAGE_BYTES;
                if (it < pre) {  // the weights of this stage are already on their way
                    mbar_expect_tx(&full[s], (unsigned)(args.np * X_BYTES));
                } else {
                    if (!mbar_wait(&empty[s], ((unsigned)(it / NSTAGE) & 1u) ^ 1u, args.wait)) break;
                    mbar_expect_tx(&full[s], (unsigned)STAGE_BYTES);
                    load_w(it);
                }
                tma_load_3d(st + W_BYTES, &map_x0, k, 0, 0, &full[s]);
                if (args.np == 2) tma_load_3d(st + W_BYTES + X_BYTES, &map_x1, k, 0, 0, &full[s]);
            }
        }
    } else if (warp == 1) {
        if (elect_one()) {
            for (int it = 0; it < nkb; ++it) {
                const int s = it % NSTAGE;
                if (!mbar_wait(&full[s], (unsigned)(it / NSTAGE) & 1u, args.wait)) { ok = false; break; }
                asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                unsigned char *st = smem + (size_t)s * STAGE_BYTES;
                const uint32_t dw = MN ? smem_desc_mn(st, 64 * BKB) : smem_desc(st), dx = smem_desc(st + W_BYTES);
                // k advance per MMA: 32 bytes inside the swizzled row (K-major), 16 k rows of 128 bytes (MN-major)
                constexpr uint32_t WADV = MN ? (16 * 128) >> 4 : UMMA_KB >> 4;
#pragma unroll
                for (int ks = 0; ks < BKB / UMMA_KB; ++ks)
                    umma<F8>(tmem_base, dw + ks * WADV, dx + (uint32_t)(ks * UMMA_KB >> 4), IDESC, it != 0 || ks != 0);
                umma_commit(&empty[s]);
            }
            if (ok) umma_commit(&tmem_full);
        }
    }
    __syncwarp();
    if (warp >= 2) {
        const int q = warp & 3;  // tensor-memory lane quarter this warp may read
        ok = mbar_wait(&tmem_full, 0u, args.wait);
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    }
    if (S > 1) cluster_wait();  // every CTA of the cluster runs: its shared memory may be written
    if (warp >= 2 && ok) {
        const int q = warp & 3, per = (args.MB + S - 1) / S;
        // word address of red[rank][0][q * 32 + lane] in this CTA; the same offset in every CTA of the cluster
        const unsigned mine = smem_u32(red) + (unsigned)((rank * per * BM + q * 32 + lane) * 4);
#pragma unroll 1
        for (int c = 0; c < args.MB; c += 16) {
            uint32_t v[16];
            tmem_ld16(tmem_base + ((uint32_t)(q * 32) << 16) + (uint32_t)c, v);
            if (args.np == 2) {  // the lo products
                uint32_t w[16];
                tmem_ld16(tmem_base + ((uint32_t)(q * 32) << 16) + (uint32_t)(args.MB + c), w);
#pragma unroll
                for (int j = 0; j < 16; ++j) v[j] = __float_as_uint(__uint_as_float(v[j]) + __uint_as_float(w[j]));
            }
            if (S == 1) {
#pragma unroll
                for (int j = 0; j < 16; ++j) red[(c + j) * BM + q * 32 + lane] = __uint_as_float(v[j]);
            } else {
                int owner = c % S, idx = c / S;
#pragma unroll
                for (int j = 0; j < 16; ++j) {
                    if (c + j < args.M) {
                        unsigned remote;
                        asm("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(remote) : "r"(mine + (unsigned)(idx * BM * 4)), "r"(owner));
                        asm volatile("st.shared::cluster.u32 [%0], %1;" ::"r"(remote), "r"(v[j]) : "memory");
                    }
                    if (++owner == S) { owner = 0; ++idx; }
                }
            }
        }
        asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    }
    if (S > 1) {
        __syncwarp();
        cluster_arrive();
        cluster_wait();  // every partial of this CTA's columns has arrived; nobody writes here any more
    } else if (warp >= 2) {
        asm volatile("bar.sync 1, 128;" ::: "memory");
    }
    if (warp >= 2) {
        // warp w takes the owned rows w, w + 4, ...; a lane owns four consecutive channels
        asm volatile("griddepcontrol.wait;" ::: "memory");  // scales, bias and y belong to the stream order
        const int per = (args.MB + S - 1) / S, ch0 = tile * BM + 4 * lane, left = args.N - ch0;
        float ws[4] = {1.0f, 1.0f, 1.0f, 1.0f}, bs[4] = {0.0f, 0.0f, 0.0f, 0.0f};
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            if (F8 && i < left) ws[i] = __ldg(args.w_scale + ch0 + i);
            if (!F8 && args.bias && i < left) bs[i] = to_f32(static_cast<const T *>(args.bias)[ch0 + i]);
        }
        T *y = static_cast<T *>(args.y) + ch0;
        const bool vec = left >= 4 && (args.ldy & 3) == 0 && (reinterpret_cast<uintptr_t>(args.y) & 7) == 0;
        // the warp's row scales (at most 32), one lane each: asked for together, not row by row between the stores
        const int row_l = (warp - 2 + 4 * lane) * S + rank;
        const float xs_l = F8 && row_l < args.M ? ld_act_f32(args.x_scale + row_l) : 1.0f;
        for (int i = 0, lc = warp - 2, row = lc * S + rank; row < args.M; ++i, lc += 4, row = lc * S + rank) {
            const float xs = F8 ? __shfl_sync(0xffffffffu, xs_l, i) : 1.0f;
            if (left <= 0) continue;
            float4 sum = *reinterpret_cast<const float4 *>(red + (size_t)lc * BM + 4 * lane);
            for (int src = 1; src < S; ++src) {
                const float4 p = *reinterpret_cast<const float4 *>(red + (size_t)(src * per + lc) * BM + 4 * lane);
                sum.x += p.x; sum.y += p.y; sum.z += p.z; sum.w += p.w;
            }
            float val[4] = {sum.x, sum.y, sum.z, sum.w};
            T out[4];
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                out[i] = from_f32<T>(F8 ? ws[i] * (xs * val[i]) : val[i]);
                if (!F8 && args.bias) out[i] = from_f32<T>(to_f32(out[i]) + bs[i]);
            }
            T *dst = y + (size_t)row * args.ldy;
            if (vec) {
                *reinterpret_cast<uint2 *>(dst) = *reinterpret_cast<const uint2 *>(out);
            } else {
                for (int i = 0; i < 4 && i < left; ++i) dst[i] = out[i];
            }
        }
    }

    __syncthreads();
    if (warp == 1) {
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "r"(TMEM_COLS) : "memory");
    }
}

struct SkinnyCall {
    void *y;
    const void *x0, *x1, *w, *bias;
    const float *x_scale, *w_scale;
    size_t m, n, k, ldx, ldw, ldy;
    bool w_static;
};

// CTAs in clusters of S that are on the machine at once, two or one per SM.  A cluster has to fit a GPC: of 148 SMs' 296 / 148
// places the driver's occupancy query gives clusters of two all, of four 284 / 132, of eight 264 / 120.  Past that the last
// clusters are a second round: one per SM, 36 tiles in clusters of four (144 CTAs), e4m3 94 x 4608 x 1408, 16.3 us against 10.3.
inline long long cluster_places(int S, bool two) {
    const long long sms = sm_count();
    if (two) return sms * 7 / 4;
    return S <= 2 ? sms : (S <= 4 ? sms * 8 / 9 : sms * 13 / 16);
}

template <int KIND, bool MN>
int launch(const SkinnyCall &c, cudaStream_t st) {
    constexpr int ELEM = KIND == 0 ? 1 : 2, BK = BKB / ELEM;
    SkinnyArgs a{};
    a.y = c.y; a.x_scale = c.x_scale; a.w_scale = c.w_scale; a.bias = c.bias;
    a.ldy = (int)c.ldy; a.M = (int)c.m; a.N = (int)c.n; a.K = (int)c.k;
    a.MB = (int)((c.m + 15) / 16 * 16);
    a.np = c.x1 ? 2 : 1;
    a.w_static = c.w_static ? 1 : 0;
    if (int rc = wait_ctx(&a.wait)) return rc;
    const int num_kb = (int)((c.k + BK - 1) / BK), sms = sm_count();
    const long long units = (long long)((c.n + BM - 1) / BM);
    const int stage = BM * BKB + a.np * a.MB * BKB;
    // The most ranges of k (a power of two: clusters of 3, 5, ... pack badly) whose CTAs all find a place at once, with two
    // stages each at least.  e4m3, 32 rows, us
    // for S = 1 / 2 / 4 / 8: 4096 x 4096 14.2 / 10.9 / 7.9 / 8.2; 8192 x 4096 14.8 / 12.1 / 10.5 / 16.4; 12288 x 4096
    // 15.5 / 14.6 / 17.9 / 22.9; 22528 x 4096 19.9 / 28.4 / 30.3 / 41.7; 4096 x 11264 30.8 / 21.3 / 13.8 / 12.5.
    // Half an SM's shared memory per CTA when that holds three stages beside the received partials (two, when the units
    // alone outnumber the SMs: W8A16 at 64 rows, 22528 x 4096, 23.4 us against 34.4 us one per SM); otherwise all of it
    // (4096 x 4096 at 64 rows 10.4 -> 9.4 us).
    auto red_bytes = [&](int S) { return S > 1 ? (size_t)S * ((a.MB + S - 1) / S) * BM * sizeof(float) : (size_t)0; };
    const size_t half = 111 * 1024;
    const bool two = (size_t)(units > sms ? 2 : 3) * stage + red_bytes(units > sms ? 1 : 8) + 1024 <= half;
    // Clusters of eight only for up to 16 rows (five stages of weights each, all fetched ahead of the dependency wait) or
    // where four leave most SMs idle: in a decoder layer at 32 streams four are faster (1218 us against 1240 us per four
    // layers), at one stream eight (272 against 288).
    const int most = a.MB <= 16 || units * 6 <= sms ? 8 : 4;
    int S = 1;
    while (S < most && units * S * 2 <= cluster_places(S * 2, two) && num_kb / (S * 2) >= 2) S *= 2;
    const size_t red = red_bytes(S);
    const int nstage = (int)(((two ? half : 2 * half) - 1024 - red) / stage);
    a.nstage = nstage > SK_MAX_STAGES ? SK_MAX_STAGES : nstage;
    a.S = S;
    CUtensorMap mw, mx0, mx1;
    int inner;  // one matrix each: the order (k, rows, 1)
    int rc = MN ? make_map_mn(&mw, c.w, c.n, c.k, c.ldw, 1, 0, &inner) : make_map3(&mw, c.w, ELEM, c.n, c.k, c.ldw, BM, 1, 0, &inner);
    if (rc) return rc;
    if ((rc = make_map3(&mx0, c.x0, ELEM, c.m, c.k, c.ldx, a.MB, 1, 0, &inner))) return rc;
    if ((rc = make_map3(&mx1, c.x1 ? c.x1 : c.x0, ELEM, c.m, c.k, c.ldx, a.MB, 1, 0, &inner))) return rc;
    // never less than what keeps a third CTA off the SM: two of them may hold all of its tensor memory
    size_t smem = (size_t)a.nstage * stage + red + 1024;
    const size_t out = (size_t)a.MB * BM * sizeof(float) + 1024;  // a single CTA's rows, over the drained ring
    if (smem < out) smem = out;
    if (smem < 78 * 1024) smem = 78 * 1024;
    auto kern = gemm_skinny_kernel<KIND, MN>;
    XN_ENSURE_SMEM(kern, smem);
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)(units * S));
    cfg.blockDim = dim3(SK_THREADS);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = st;
    cudaLaunchAttribute attr[2];
    int na = 0;
    if (pdl_enabled()) {
        attr[na].id = cudaLaunchAttributeProgrammaticStreamSerialization;
        attr[na++].val.programmaticStreamSerializationAllowed = 1;
    }
    if (S > 1) {
        attr[na].id = cudaLaunchAttributeClusterDimension;
        attr[na].val.clusterDim.x = (unsigned)S;
        attr[na].val.clusterDim.y = 1;
        attr[na++].val.clusterDim.z = 1;
    }
    cfg.attrs = attr;
    cfg.numAttrs = na;
    XN_CHECK_CUDA(cudaLaunchKernelEx(&cfg, kern, mw, mx0, mx1, a));
    return XN_OK;
}

}  // namespace

// Whether this kernel is the one for m rows against a weight of n channels of k_bytes each (pieces: e4m3 matrices per activation,
// 1 for 16-bit rows).  Up to 64 rows always (the callers know which smaller row counts their weight-streaming kernels still
// win).  From 65 to 128 rows while the channels make at most half as many tiles as there are SMs, so that k can be split, and k is
// long enough to pay for moving MB x 128 partial sums per CTA through the cluster, which the tiled kernel does not do: that cost
// grows with MB^2 (rows, and columns per owner) and is paid back per k stage, twice as fast where two pieces share a weight
// stage.  With fewer than 33 tiles the tiled kernel leaves more of the machine idle and k may be shorter.  us, tiled / this
// kernel: bf16 66 x 4096 x 512 6.2 / 6.5, x 1024 8.8 / 7.2; 128 x 8192 x 2048 14.7 / 15.5, x 4096 23.6 / 21.4; W8A8 128 x 8192 x 1024
// 6.9 / 10.0, 80 x 8192 x 2048 9.7 / 9.8, x 4096 14.3 / 13.1; W8A16 128 x 2048 x 1024 7.2 / 7.8, x 2048 10.3 / 8.5.
bool gemm_skinny_wanted(size_t m, size_t n, size_t k_bytes, int pieces) {
    if (n > 0x7fffff00 || k_bytes > 0x7fffff00 || (n + BM - 1) / BM > 0x7fffffff / 8) return false;
    if (m <= 64) return true;
    const size_t tiles = (n + BM - 1) / BM, mb = (m + 15) / 16 * 16, work = k_bytes * (size_t)pieces;
    if (m > 128 || tiles * 2 > (size_t)sm_count()) return false;
    if (tiles <= 32) {
        const size_t line = mb * mb / 8 > 1024 ? mb * mb / 8 : 1024;
        return pieces == 1 ? work >= line : work > line;
    }
    return work * 25 >= mb * mb * 8 && !(pieces == 1 && mb == 128 && k_bytes > 8192);
}

// y bf16 [m, n] = x_scale[m] * w_scale[n] * (x_hi (+ x_lo)) * wq^T, all operands row-major e4m3.  wq is a static weight.
int launch_skinny_fp8(void *y, const uint8_t *x_hi, const uint8_t *x_lo, const float *x_scale, const uint8_t *wq,
                      const float *w_scale, size_t m, size_t n, size_t k, size_t ldy, cudaStream_t st) {
    const SkinnyCall c{y, x_hi, x_lo, wq, nullptr, x_scale, w_scale, m, n, k, k, k, ldy, true};
    return launch<0, false>(c, st);
}

// 16-bit operands; w_mn: rhs is [k, n] with n contiguous.
int launch_skinny_16bit(xn_dtype dt, void *dst, const void *lhs, const void *rhs, const void *bias, size_t m, size_t n, size_t k,
                        size_t lda, size_t ldb, size_t ldd, bool w_mn, cudaStream_t st) {
    const SkinnyCall c{dst, lhs, nullptr, rhs, bias, nullptr, nullptr, m, n, k, lda, ldb, ldd, rhs_is_static()};
    if (dt == XN_BF16) return w_mn ? launch<1, true>(c, st) : launch<1, false>(c, st);
    return w_mn ? launch<2, true>(c, st) : launch<2, false>(c, st);
}

}  // namespace xn
