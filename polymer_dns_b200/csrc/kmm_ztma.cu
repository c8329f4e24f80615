// kmm_ztma.cu -- the fused step's z transforms (FP64 and the FP32 of the mixed form) with TMA
// tile copies.
//
// Work of the stage (solvers.f90:2578-2803 for the velocity, vorticity and scalar-gradient
// fields): from the y-physical base fields u, v, w, omega_y, du/dy, dw/dy [, c, dc/dy] in column
// layout [f][kx][kz][y], form the nine z-spectral inputs of the x stage (u v w wx wy wz [cx cy
// cz]; wx = dw/dy - i kz v, wz = i kx v - du/dy, cx = i kx c, cz = i kz c), zero-pad kz from nz to
// mz (modes j > nz/2 move to mz - nz + j), inverse c2c along z, and store Q[g][y][z][kx].
//
// Data movement: one CTA per tile of KX consecutive kx and YT consecutive y, one warp per column.
// Its thread 0 issues one tiled TMA load per base field (box: YT y x all nz kz x KX kx), each on its
// own mbarrier.  Each warp's FFT (the warp-private compile-time FFT of kmm_fft.cuh) forms the field's
// z-spectral values from the tiles in its first stage, runs in place in one buffer, and leaves its
// result in a [y][z][kx] staging tile, which a tiled TMA store (box: KX kx x mz z x YT y) writes out
// while the next field is transformed.  52 KB of shared memory per CTA for the inverse and 48 KB for the
// forward transform at mz = 192 in FP64.  Both kinds of tile are swizzled by the length of their rows.
//
// Every wait on an mbarrier is bounded (KMM_OPT_WAIT_LIMIT_MS, default 2 s of %globaltimer); a wait
// that runs out records KMM_ERR_TIMEOUT in the step's status word (the forward transform, which runs
// beside or after the step's report, in the host's late word) and the CTA finishes without the data.
#include <cuda.h>
#include <cudaTypedefs.h>

#include "kmm_internal.cuh"
#include "kmm_async.cuh"
#include "kmm_fft.cuh"
#include "kmm_fused.cuh"

namespace {

__device__ __forceinline__ uint32_t sm_addr(const void *p) { return (uint32_t)__cvta_generic_to_shared(p); }

__device__ __forceinline__ void mbar_init(uint64_t *bar, unsigned count) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(sm_addr(bar)), "r"(count) : "memory");
}

__device__ __forceinline__ void mbar_expect_tx(uint64_t *bar, unsigned bytes) {
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(sm_addr(bar)), "r"(bytes) : "memory");
}

// wait for phase `phase` of a barrier, at most the unit's limit (kasync_wait_ns, default 2 s)
__device__ __forceinline__ bool mbar_wait(uint64_t *bar, unsigned phase) { return kasync::mbar_wait(bar, phase); }

__device__ __forceinline__ void tma_load4(void *dst, const CUtensorMap *tm, int c0, int c1, int c2, int c3,
                                          uint64_t *bar) {
    asm volatile(
        "cp.async.bulk.tensor.4d.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3, %4, %5}], "
        "[%6];" ::"r"(sm_addr(dst)),
        "l"(tm), "r"(c0), "r"(c1), "r"(c2), "r"(c3), "r"(sm_addr(bar))
        : "memory");
}

__device__ __forceinline__ void tma_store4(const CUtensorMap *tm, int c0, int c1, int c2, int c3, const void *src) {
    asm volatile("cp.async.bulk.tensor.4d.global.shared::cta.bulk_group [%0, {%1, %2, %3, %4}], [%5];" ::"l"(tm),
                 "r"(c0), "r"(c1), "r"(c2), "r"(c3), "r"(sm_addr(src))
                 : "memory");
    asm volatile("cp.async.bulk.commit_group;" ::: "memory");
}

// the staging tile may be overwritten once every committed store has read it
__device__ __forceinline__ void tma_store_wait_read() { asm volatile("cp.async.bulk.wait_group.read 0;" ::: "memory"); }

// generic-proxy writes to shared memory -> visible to the TMA (async proxy)
__device__ __forceinline__ void fence_async_smem() { asm volatile("fence.proxy.async.shared::cta;" ::: "memory"); }

}  // namespace

// Element (row, col) of a shared-memory tile whose rows hold COLS values of C and which a tensor
// map moves with the swizzle of its row length (16 bytes: none; 32, 64: the 16-byte chunk index XOR
// address bits 7 (32 bytes) or 7-8 (64 bytes)): a warp's accesses down one column then spread over
// the banks.
template <typename C, int COLS>
__device__ __forceinline__ int tile_idx(int row, int col) {
    constexpr int RB = COLS * (int)sizeof(C), EPC = 16 / (int)sizeof(C);
    static_assert(RB == 16 || RB == 32 || RB == 64, "tile rows of 16, 32 or 64 bytes");
    int ch = col / EPC;
    if (RB == 32) ch ^= (row >> 2) & 1;
    if (RB == 64) ch ^= (row >> 1) & 3;
    return row * COLS + ch * EPC + col % EPC;
}

// the z lengths whose FFT's last stage leaves output z = lane + 32 e in lane `lane` (its stride is
// a multiple of 32), so that the stage can write the lane's registers
template <int MZ>
constexpr bool ZREG = MZ % 32 == 0 && kct::stride(MZ, kct::nfac(MZ) - 1) % 32 == 0;

// One column's transform by a warp: the first stage reads its inputs through ld(z), the stages up
// to the last run in place in the warp's buffer a, out(z, value) receives the result.  before()
// runs once the warp needs nothing but its own buffer or registers any more and before the first
// out(): every thread of the block reaches it.
template <int MZ, typename C, int S, typename LD, typename OUT, typename BEFORE>
__device__ __forceinline__ void z_column(LD ld, OUT out, BEFORE before, C *a, const C *__restrict__ tw) {
    constexpr int L = kct::nfac(MZ);
    const int lane = threadIdx.x & 31;
    const FftBuf<C> buf{a};
    kct::stage_io<C, MZ, 0, S, 1>(ld, buf, tw, lane);
    __syncwarp();
    kct::IpSteps<C, MZ, 1, S, 1, (2 >= L)>::go(a, tw, lane);
    if constexpr (ZREG<MZ>) {
        C rv[MZ / 32];
        auto st = [&](int z, C v) { rv[z >> 5] = v; };
        kct::stage_io<C, MZ, L - 1, S, 1>(buf, st, tw, lane);
        before();
#pragma unroll
        for (int e = 0; e < MZ / 32; ++e) out(lane + 32 * e, rv[e]);
    } else {
        kct::stage_ip<C, MZ, L - 1, S, 1>(a, tw, lane);
        before();
        for (int z = lane; z < MZ; z += 32) out(z, a[fpos<C>(z)]);
    }
}

// blockIdx.z picks one of three groups of q fields that share their base fields -- u, w, omega_y;
// v, wx, wz; dc/dx, dc/dz, dc/dy -- so a CTA holds at most ZB_SLOTS base-field tiles, all loaded at
// its start, and forms (at most) ZB_SLOTS q fields.
#define ZB_SLOTS 3
__device__ __forceinline__ int zb_field(int grp, int k) {
    return grp == 0 ? 2 * k : grp == 1 ? 2 * k + 1 : k == 0 ? 6 : k == 1 ? 8 : 7;
}
// the base field in slot s of a group
__device__ __forceinline__ int zb_base(int grp, int s) {
    return grp == 0 ? (s == 0 ? 0 : s + 1) : grp == 1 ? (s == 0 ? 1 : 6 - s) : 6 + s;
}

template <int MZ, typename C, int KX, int YT, int MINB>
__global__ void __launch_bounds__(KX * YT * 32, MINB)
    k_zb_tma(const __grid_constant__ CUtensorMap tin, const __grid_constant__ CUtensorMap tout,
             const double *__restrict__ wavx, const double *__restrict__ wavz, const C *__restrict__ tw, int nxh,
             int *status) {
    typedef typename kct::Real<C>::T T;
    constexpr int NZ = 2 * MZ / 3, NZH = NZ / 2, TILE = KX * NZ * YT, W = KX * YT;
    extern __shared__ unsigned char zsm_raw[];
    // 1024-byte aligned base: tiles [ZB_SLOTS][KX][NZ][YT], stage [YT][MZ][KX], FFT buffers [W][MZ], barriers
    C *tiles = reinterpret_cast<C *>((reinterpret_cast<uintptr_t>(zsm_raw) + 1023) & ~(uintptr_t)1023);
    C *stage = tiles + (size_t)ZB_SLOTS * TILE;
    C *scr = stage + (size_t)W * MZ;
    uint64_t *bar = reinterpret_cast<uint64_t *>(scr + (size_t)W * flen<C>(MZ));
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int kx0 = blockIdx.x * KX, y0 = blockIdx.y * YT;
    const int kl = warp / YT, y = warp % YT;
    if (threadIdx.x == 0) {
        for (int q = 0; q < ZB_SLOTS; ++q) mbar_init(&bar[q], 1);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    __syncthreads();
    const int grp = blockIdx.z, nslot = grp == 2 ? 2 : ZB_SLOTS;
    if (threadIdx.x == 0) {
        for (int q = 0; q < nslot; ++q) {
            mbar_expect_tx(&bar[q], (unsigned)(TILE * sizeof(C)));
            tma_load4(tiles + (size_t)q * TILE, &tin, 2 * y0, 0, kx0, zb_base(grp, q), &bar[q]);
        }
    }
    const T kxv = kx0 + kl < nxh ? (T)wavx[kx0 + kl] : (T)0;
    const double beta = wavz[1];
    C *a = scr + (size_t)warp * flen<C>(MZ);
    bool ok = true;
    const C zc = kct::mk<C>((T)0, (T)0);
    for (int k = 0; k < ZB_SLOTS; ++k) {
        // q field g (u v w wx wy wz cx cy cz) from the tile in slot s0 and, for wx and wz, v in slot 0
        const int g = zb_field(grp, k), s0 = grp == 2 ? (g == 7 ? 1 : 0) : k;
        ok = mbar_wait(&bar[s0], 0) && ok;
        const C *t0 = tiles + (size_t)s0 * TILE, *t1 = tiles;
        auto ld = [&](int z) {
            C val = zc;
            if (ok && (z < NZH || z >= MZ - NZH)) {
                const int kz = z < NZH ? z : z - (MZ - NZ);
                const int ti = tile_idx<C, YT>(kl * NZ + kz, y);
                const C p = t0[ti];
                switch (g) {
                case 3: {   // wx = dw/dy - i kz v (wavz[kz] = beta (kz or kz - nz), as the context forms it)
                    const T kzv = (T)((double)(kz < NZH ? kz : kz - NZ) * beta);
                    const C vv = t1[ti];
                    val = kct::mk<C>(p.x + kzv * vv.y, p.y - kzv * vv.x);
                } break;
                case 5: {   // wz = i kx v - du/dy
                    const C vv = t1[ti];
                    val = kct::mk<C>(-kxv * vv.y - p.x, kxv * vv.x - p.y);
                } break;
                case 6: val = kct::mk<C>(-kxv * p.y, kxv * p.x); break;   // i kx c
                case 8: {
                    const T kzv = (T)((double)(kz < NZH ? kz : kz - NZ) * beta);
                    val = kct::mk<C>(-kzv * p.y, kzv * p.x);   // i kz c
                } break;
                default: val = p; break;
                }
            }
            return val;
        };
        auto before = [&] {
            if (threadIdx.x == 0) tma_store_wait_read();   // the previous field's store has read the stage
            __syncthreads();
        };
        auto out = [&](int z, C v) { stage[tile_idx<C, KX>(y * MZ + z, kl)] = v; };
        z_column<MZ, C, +1>(ld, out, before, a, tw);
        fence_async_smem();
        __syncthreads();
        if (threadIdx.x == 0) tma_store4(&tout, 2 * kx0, 0, y0, g, stage);
    }
    if (threadIdx.x == 0) {
        tma_store_wait_read();   // shared memory must outlive the last store's read
        // after a timeout, wait (again with the limit) for the tile loads still in flight before the CTA exits
        for (int q = 0; !ok && q < nslot; ++q) mbar_wait(&bar[q], 0);
    }
    if (!ok && lane == 0) atomicMax(status, KMM_ERR_TIMEOUT);
}

// Forward z transform of the x stage's outputs (solvers.f90:3180-3273): R[o][y][z][kx] -> c2c
// along z, truncate to nz (mode j > nz/2 from mz - nz + j), divide by mx mz (FP32: times its
// reciprocal), store in column layout Yo[o][kx][kz][y].  The same CTA tile as the inverse with the
// roles of the two layouts exchanged.  The input tiles pass through two shared-memory slots: fields
// 0 and 1 are loaded at the start, field o + 2 into slot o mod 2 once field o has been read.
#define ZF_SLOTS 2
template <int MZ, typename C, int KX, int YT, int MINB>
__global__ void __launch_bounds__(KX * YT * 32, MINB)
    k_zf_tma(const __grid_constant__ CUtensorMap tin, const __grid_constant__ CUtensorMap tout,
             const C *__restrict__ tw, int nper, double scale, volatile int *status) {
    typedef typename kct::Real<C>::T T;
    constexpr int NZ = 2 * MZ / 3, NZH = NZ / 2, W = KX * YT, TIN = MZ * W, TOUT = NZ * W;
    extern __shared__ unsigned char zsm_raw[];
    // 1024-byte aligned: in tiles [ZF_SLOTS][YT][MZ][KX], out stage [KX][NZ][YT], FFT buffers [W][MZ], barriers
    C *tiles = reinterpret_cast<C *>((reinterpret_cast<uintptr_t>(zsm_raw) + 1023) & ~(uintptr_t)1023);
    C *stage = tiles + (size_t)ZF_SLOTS * TIN;
    C *scr = stage + TOUT;
    uint64_t *bar = reinterpret_cast<uint64_t *>(scr + (size_t)W * flen<C>(MZ));
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int kx0 = blockIdx.x * KX, y0 = blockIdx.y * YT;
    const int kl = warp / YT, y = warp % YT;
    if (threadIdx.x == 0) {
        for (int o = 0; o < nper; ++o) mbar_init(&bar[o], 1);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    __syncthreads();
    unsigned issued = 0;
    bool ok = true;
    const int o0 = blockIdx.z * nper;
    auto load = [&](int o) {
        if (o >= nper || !ok) return;   // nothing is loaded over a tile that did not arrive
        mbar_expect_tx(&bar[o], (unsigned)(TIN * sizeof(C)));
        tma_load4(tiles + (size_t)(o % ZF_SLOTS) * TIN, &tin, 2 * kx0, 0, y0, o0 + o, &bar[o]);
        issued |= 1u << o;
    };
    if (threadIdx.x == 0) {
        load(0);
        load(1);
    }
    const T rs = (T)(1.0 / scale);
    const C zc = kct::mk<C>((T)0, (T)0);
    C *a = scr + (size_t)warp * flen<C>(MZ);
    for (int o = 0; o < nper; ++o) {
        ok = mbar_wait(&bar[o], 0) && ok;
        const C *t = tiles + (size_t)(o % ZF_SLOTS) * TIN;
        auto ld = [&](int z) { return ok ? t[tile_idx<C, KX>(y * MZ + z, kl)] : zc; };
        auto before = [&] {
            if (threadIdx.x == 0) tma_store_wait_read();   // the previous field's store has read the stage
            __syncthreads();
        };
        auto out = [&](int z, C v) {
            if (z < NZH || z >= MZ - NZH) {
                const int kz = z < NZH ? z : z - (MZ - NZ);
                stage[tile_idx<C, YT>(kl * NZ + kz, y)] =
                    sizeof(T) == 8 ? kct::mk<C>((T)(v.x / scale), (T)(v.y / scale)) : kct::mk<C>(v.x * rs, v.y * rs);
            }
        };
        z_column<MZ, C, -1>(ld, out, before, a, tw);
        fence_async_smem();   // also orders this field's tile reads before the TMA load that refills the slot
        __syncthreads();
        if (threadIdx.x == 0) {
            tma_store4(&tout, 2 * y0, 0, kx0, o0 + o, stage);
            load(o + ZF_SLOTS);
        }
    }
    if (threadIdx.x == 0) {
        tma_store_wait_read();
        for (int o = 0; !ok && o < nper; ++o)   // as above
            if ((issued >> o) & 1u) mbar_wait(&bar[o], 0);
    }
    if (!ok && lane == 0) *status = KMM_ERR_TIMEOUT;
}

// ---------------------------------------------------------------------------
// host side: tensor maps (cached per context, re-encoded when a buffer or size changes) and the
// launches
// ---------------------------------------------------------------------------
struct ZtmaPair {
    CUtensorMap in, out;
    const void *src, *dst;
    int nyp, nz, nxh, mz, nsrc, ndst, f32;
};
struct ZtmaMaps {
    ZtmaPair inv, fwd;   // inverse: Y (base fields) -> Q; forward: R -> Yo
};

static PFN_cuTensorMapEncodeTiled_v12000 ztma_encoder() {
    static PFN_cuTensorMapEncodeTiled_v12000 fn = NULL;
    if (!fn) {
        void *p = NULL;
        cudaDriverEntryPointQueryResult q;
        if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &p, cudaEnableDefault, &q) == cudaSuccess &&
            q == cudaDriverEntryPointSuccess)
            fn = (PFN_cuTensorMapEncodeTiled_v12000)p;
    }
    return fn;
}

// this unit's bounded-wait limit on the current device (KMM_OPT_WAIT_LIMIT_MS)
int kmm_ztma_set_wait_limit(unsigned long long ns) { return kasync::kasync_set_wait_limit(ns) == cudaSuccess ? 0 : 1; }

void kmm_ztma_release(kmm_ctx *ctx) {
    free(ctx->ztma);
    ctx->ztma = NULL;
}

bool kmm_ztma_supported(const kmm_ctx *ctx) {
    const int mz = ctx->mz;
    return ctx->use_ztma && (mz == 48 || mz == 96 || mz == 144 || mz == 192);
}

static ZtmaMaps *ztma_maps(kmm_ctx *ctx) {
    if (!ctx->ztma) {
        void *m = NULL;
        if (posix_memalign(&m, 64, sizeof(ZtmaMaps))) return NULL;   // CUtensorMap: 64-byte alignment
        memset(m, 0, sizeof(ZtmaMaps));
        ctx->ztma = m;
    }
    return (ZtmaMaps *)ctx->ztma;
}

static bool pair_current(const ZtmaPair &P, const void *src, const void *dst, const kmm_ctx *ctx, int nsrc, int ndst,
                         int f32) {
    return P.src == src && P.dst == dst && P.nyp == ctx->nyp && P.nz == ctx->nz && P.nxh == ctx->nxh &&
           P.mz == ctx->mz && P.nsrc == nsrc && P.ndst == ndst && P.f32 == f32;
}

static CUtensorMapSwizzle row_swizzle(int bytes) {
    return bytes == 64 ? CU_TENSOR_MAP_SWIZZLE_64B : bytes == 32 ? CU_TENSOR_MAP_SWIZZLE_32B : CU_TENSOR_MAP_SWIZZLE_NONE;
}

// column layout [f][kx][kz][y] as reals (a complex value is 2 reals; FP32 columns padded to an
// even length): (2 nyp, nz, nxh, nf), box (yt values of y, nz, kx columns, 1)
static CUresult map_columns(PFN_cuTensorMapEncodeTiled_v12000 enc, CUtensorMap *m, const void *base,
                            const kmm_ctx *ctx, int nf, CUtensorMapL2promotion l2, bool f32, int kx, int yt) {
    const int nyp = ctx->nyp, nz = ctx->nz, nxh = ctx->nxh;
    const cuuint64_t cb = f32 ? (cuuint64_t)8 * col_ld<float2>(nyp) : (cuuint64_t)16 * nyp;   // column bytes
    cuuint64_t d[4] = {(cuuint64_t)2 * nyp, (cuuint64_t)nz, (cuuint64_t)nxh, (cuuint64_t)nf};
    cuuint64_t st[3] = {cb, (cuuint64_t)nz * cb, (cuuint64_t)nz * nxh * cb};
    cuuint32_t box[4] = {2u * yt, (cuuint32_t)nz, (cuuint32_t)kx, 1};
    cuuint32_t es[4] = {1, 1, 1, 1};
    return enc(m, f32 ? CU_TENSOR_MAP_DATA_TYPE_FLOAT32 : CU_TENSOR_MAP_DATA_TYPE_FLOAT64, 4, (void *)base, d, st, box,
               es, CU_TENSOR_MAP_INTERLEAVE_NONE, row_swizzle(yt * (f32 ? 8 : 16)), l2,
               CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
}

// plane layout [f][y][z][kx] as reals: (2 nxh, mz, nyp, nf), box (kx values, mz, yt, 1)
static CUresult map_planes(PFN_cuTensorMapEncodeTiled_v12000 enc, CUtensorMap *m, const void *base,
                           const kmm_ctx *ctx, int nf, CUtensorMapL2promotion l2, bool f32, int kx, int yt) {
    const int nyp = ctx->nyp, nxh = ctx->nxh, mz = ctx->mz;
    const cuuint64_t eb = f32 ? 8 : 16;   // bytes per complex value
    cuuint64_t d[4] = {(cuuint64_t)2 * nxh, (cuuint64_t)mz, (cuuint64_t)nyp, (cuuint64_t)nf};
    cuuint64_t st[3] = {(cuuint64_t)nxh * eb, (cuuint64_t)mz * nxh * eb, (cuuint64_t)nyp * mz * nxh * eb};
    cuuint32_t box[4] = {2u * kx, (cuuint32_t)mz, (cuuint32_t)yt, 1};
    cuuint32_t es[4] = {1, 1, 1, 1};
    return enc(m, f32 ? CU_TENSOR_MAP_DATA_TYPE_FLOAT32 : CU_TENSOR_MAP_DATA_TYPE_FLOAT64, 4, (void *)base, d, st, box,
               es, CU_TENSOR_MAP_INTERLEAVE_NONE, row_swizzle(kx * (f32 ? 8 : 16)), l2,
               CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
}

static int pair_encode(kmm_ctx *ctx, ZtmaPair &P, bool inverse, const void *src, const void *dst, int nsrc, int ndst,
                       bool f32, int kx, int yt) {
    if (pair_current(P, src, dst, ctx, nsrc, ndst, f32 ? 1 : 0)) return KMM_OK;
    PFN_cuTensorMapEncodeTiled_v12000 enc = ztma_encoder();
    if (!enc) {
        kmm_set_error(ctx, "cuTensorMapEncodeTiled is not available from the driver");
        return KMM_ERR_CUDA;
    }
    CUresult r1, r2;
    if (inverse) {
        r1 = map_columns(enc, &P.in, src, ctx, nsrc, CU_TENSOR_MAP_L2_PROMOTION_L2_128B, f32, kx, yt);
        r2 = map_planes(enc, &P.out, dst, ctx, ndst, CU_TENSOR_MAP_L2_PROMOTION_NONE, f32, kx, yt);
    } else {
        r1 = map_planes(enc, &P.in, src, ctx, nsrc, CU_TENSOR_MAP_L2_PROMOTION_L2_128B, f32, kx, yt);
        r2 = map_columns(enc, &P.out, dst, ctx, ndst, CU_TENSOR_MAP_L2_PROMOTION_NONE, f32, kx, yt);
    }
    if (r1 != CUDA_SUCCESS || r2 != CUDA_SUCCESS) {
        kmm_set_error(ctx, "tensor map encoding failed (%d, %d)", (int)r1, (int)r2);
        P.src = NULL;
        return KMM_ERR_CUDA;
    }
    P.src = src; P.dst = dst; P.nsrc = nsrc; P.ndst = ndst; P.f32 = f32 ? 1 : 0;
    P.nyp = ctx->nyp; P.nz = ctx->nz; P.nxh = ctx->nxh; P.mz = ctx->mz;
    return KMM_OK;
}

// The CTA tile of both transforms: two kx by two y, one warp a column.  A tile's rows in global
// memory are then 32 bytes on either side.  With one kx (16-byte rows on the plane side) the copies'
// row rate bound the kernels at about 100 G rows/s whatever the FFT cost: the FP64 inverse took 188 us
// at 128 x 129 x 128 with a scalar, and 162-191 with the present code and one kx; two kx by two y
// takes 99 (3.7 TB/s), two by four 108, four by two 109, four by four 126, as larger CTAs lose more at
// their barriers.  FP32: 70 us against 85.
#define ZT_KX 2
#define ZT_YT 2
// CTAs per SM: four in FP64 (six: 107 us, the register budget), six in FP32 (four: 73 us)
template <typename C> constexpr int ZT_MINB = sizeof(C) == 16 ? 4 : 6;

template <int MZ, typename C>
static int zb_launch(kmm_ctx *ctx, const C *yp, C *q, int nbase, int nq, const C *tw) {
    constexpr bool f32 = sizeof(C) == 8;
    constexpr int NZ = 2 * MZ / 3, KX = ZT_KX, YT = ZT_YT, W = KX * YT, MINB = ZT_MINB<C>;
    if (f32 && ctx->nxh % 2) return KMM_ERR_UNSUPPORTED;   // a plane row of FP32 values must be a multiple of 16 bytes
    ZtmaMaps *M = ztma_maps(ctx);
    if (!M) return KMM_ERR_NOMEM;
    RET(pair_encode(ctx, M->inv, true, yp, q, nbase, nq, f32, KX, YT));
    const size_t smem = 1024 + sizeof(C) * W * ((size_t)ZB_SLOTS * NZ + MZ + flen<C>(MZ)) + 8 * sizeof(uint64_t);
    const dim3 grid((ctx->nxh + KX - 1) / KX, (ctx->nyp + YT - 1) / YT, nq / ZB_SLOTS);
    RET(kmm_smem_attr(ctx, (const void *)k_zb_tma<MZ, C, KX, YT, MINB>, smem));
    k_zb_tma<MZ, C, KX, YT, MINB><<<grid, W * 32, smem, ctx->stream>>>(M->inv.in, M->inv.out, ctx->d_wavx, ctx->d_wavz,
                                                                       tw, ctx->nxh, ctx->d_status);
    return KMM_OK;   // the caller checks the launch and counts it
}

template <int MZ, typename C>
static int zf_launch(kmm_ctx *ctx, const C *r, C *yo, int nout, const C *tw) {
    constexpr bool f32 = sizeof(C) == 8;
    constexpr int NZ = 2 * MZ / 3, KX = ZT_KX, YT = ZT_YT, W = KX * YT, MINB = ZT_MINB<C>;
    if (f32 && ctx->nxh % 2) return KMM_ERR_UNSUPPORTED;   // a plane row of FP32 values must be a multiple of 16 bytes
    ZtmaMaps *M = ztma_maps(ctx);
    if (!M) return KMM_ERR_NOMEM;
    RET(pair_encode(ctx, M->fwd, false, r, yo, nout, nout, f32, KX, YT));
    const size_t smem = 1024 + sizeof(C) * W * ((size_t)ZF_SLOTS * MZ + NZ + flen<C>(MZ)) + 8 * sizeof(uint64_t);
    // Fields per CTA: all of them in FP64 (58 us at 128 x 129 x 128 against 59 with two and 67 with one,
    // as the ring's loads overlap), two in FP32 (35 against 39 and 44).  A grid of small CTAs' chains
    // that leaves SMs idle is split further: 32 x 33 x 32 (136 tiles) 8.7 us with one field per CTA
    // against 12.7 with four; 64 x 65 x 64 (528) 14.8 with two against 15.6 and 16.9.
    const int tiles = ((ctx->nxh + KX - 1) / KX) * ((ctx->nyp + YT - 1) / YT);
    int nper = nout;
    if (nout % 2 == 0 && (f32 || tiles < 4 * 148)) nper = 2;
    if (tiles <= 148) nper = 1;
    const dim3 grid((ctx->nxh + KX - 1) / KX, (ctx->nyp + YT - 1) / YT, nout / nper);
    RET(kmm_smem_attr(ctx, (const void *)k_zf_tma<MZ, C, KX, YT, MINB>, smem));
    k_zf_tma<MZ, C, KX, YT, MINB><<<grid, W * 32, smem, ctx->stream>>>(M->fwd.in, M->fwd.out, tw, nper,
                                                                       (double)ctx->mx * (double)ctx->mz, &ctx->rep->late);
    return KMM_OK;   // the caller checks the launch and counts it
}

#define ZB_CASE(MM, C) case MM: return zb_launch<MM, C>(ctx, yp, q, nbase, nq, tw);
#define ZF_CASE(MM, C) case MM: return zf_launch<MM, C>(ctx, r, yo, nout, tw);
int kmm_zb_tma(kmm_ctx *ctx, const double2 *yp, double2 *q, int nbase, int nq, const double2 *tw) {
    switch (ctx->mz) {
        ZB_CASE(48, double2) ZB_CASE(96, double2) ZB_CASE(144, double2) ZB_CASE(192, double2)
    default: return KMM_ERR_UNSUPPORTED;
    }
}

int kmm_zf_tma(kmm_ctx *ctx, const double2 *r, double2 *yo, int nout, const double2 *tw) {
    switch (ctx->mz) {
        ZF_CASE(48, double2) ZF_CASE(96, double2) ZF_CASE(144, double2) ZF_CASE(192, double2)
    default: return KMM_ERR_UNSUPPORTED;
    }
}

// FP32 forms (mixed precision)
int kmm_zb_tma32(kmm_ctx *ctx, const float2 *yp, float2 *q, int nbase, int nq, const float2 *tw) {
    switch (ctx->mz) {
        ZB_CASE(48, float2) ZB_CASE(96, float2) ZB_CASE(144, float2) ZB_CASE(192, float2)
    default: return KMM_ERR_UNSUPPORTED;
    }
}

int kmm_zf_tma32(kmm_ctx *ctx, const float2 *r, float2 *yo, int nout, const float2 *tw) {
    switch (ctx->mz) {
        ZF_CASE(48, float2) ZF_CASE(96, float2) ZF_CASE(144, float2) ZF_CASE(192, float2)
    default: return KMM_ERR_UNSUPPORTED;
    }
}
