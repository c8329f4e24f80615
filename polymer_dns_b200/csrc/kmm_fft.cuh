// kmm_fft.cuh -- warp-private Stockham FFTs specialised at compile time for one transform length.
//
// The runtime-plan FFT (fft_warp) spends most of its instructions on integer division, modulo and
// radix dispatch.  Here the length N is a template argument: the radix sequence (8, 4, 2, 3, 5,
// the order of kmm_plan_r8) and every stride are constants, the butterfly loop over j = lane +
// 32 it has a fixed trip count, j % Ns and j / Ns become shifts for the power-of-two strides,
// and the twiddle index r k tstep never reaches N, so it needs no modulo.  The arithmetic per
// butterfly is the same as fft_warp's: twiddle multiply of inputs r >= 1, then the radix-R DFT.
//
// C is double2 or float2; the twiddle table holds exp(-2 pi i m / N), m = 0..N-1, in the same type, and
// after it the packed tables of the stages (tw_off below): stage f's twiddles w^(r k) at (r - 1) NS + k.
// A warp's lanes then read NS consecutive values per r (one to four 128-byte lines), where the strided
// entries r k TSTEP of the natural table lie on up to eight.  x stage at N = 192 (128 x 129 x 128 with scalar) 195 -> 188
// us, at N = 576 (384 x 257 x 384) 4.82 -> 4.51 ms.
#pragma once

#include <type_traits>

#include "kmm_internal.cuh"

namespace kct {

__host__ __device__ constexpr int radix_at(int r) { return r == 0 ? 8 : r == 1 ? 4 : r == 2 ? 2 : r == 3 ? 3 : 5; }

// number of factors of n over radices 8, 4, 2, 3, 5 (-1 when n has another prime factor)
__host__ __device__ constexpr int nfac(int n) {
    int c = 0;
    for (int r = 0; r < 5; ++r)
        while (n % radix_at(r) == 0) {
            n /= radix_at(r);
            ++c;
        }
    return n == 1 ? c : -1;
}

// f-th factor
__host__ __device__ constexpr int fac(int n, int f) {
    int c = 0;
    for (int r = 0; r < 5; ++r)
        while (n % radix_at(r) == 0) {
            if (c == f) return radix_at(r);
            n /= radix_at(r);
            ++c;
        }
    return 1;
}

// product of the first f factors (the Stockham stride Ns of stage f)
__host__ __device__ constexpr int stride(int n, int f) {
    int p = 1;
    for (int i = 0; i < f; ++i) p *= fac(n, i);
    return p;
}

// offset of stage f's twiddles in the packed table of length n (stage 0 has none), and its length tw_off(n, nfac(n))
__host__ __device__ constexpr int tw_off(int n, int f) {
    int o = 0;
    for (int i = 1; i < f; ++i) o += (fac(n, i) - 1) * stride(n, i);
    return o;
}
__host__ __device__ constexpr int tw_packed(int n) { return nfac(n) > 0 ? tw_off(n, nfac(n)) : 0; }
// a table of length n: n natural entries, the packed table of n, (n even) that of n / 2, and (n a multiple of
// 16) the n entries w^(t k) at 16 k + t, t < 16, k < n / 16, of the column kernels' two-pass transform
__host__ __device__ constexpr int tw_lane16(int n) { return n + tw_packed(n) + (n % 2 == 0 ? tw_packed(n / 2) : 0); }
__host__ __device__ constexpr int tw_total(int n) { return tw_lane16(n) + (n % 16 == 0 ? n : 0); }
// where the packed table of length N starts in a table of length TWS N
template <int N, int TWS>
constexpr int tw_base = TWS == 1 ? N : 2 * N + tw_packed(2 * N);

// ---- complex arithmetic on double2 / float2
template <typename C>
struct Real;
template <>
struct Real<double2> {
    typedef double T;
};
template <>
struct Real<float2> {
    typedef float T;
};

template <typename C>
__device__ __forceinline__ C mk(typename Real<C>::T x, typename Real<C>::T y) {
    C c;
    c.x = x;
    c.y = y;
    return c;
}
template <typename C>
__device__ __forceinline__ C add(C a, C b) { return mk<C>(a.x + b.x, a.y + b.y); }
template <typename C>
__device__ __forceinline__ C sub(C a, C b) { return mk<C>(a.x - b.x, a.y - b.y); }
template <typename C>
__device__ __forceinline__ C mul(C a, C b) { return mk<C>(a.x * b.x - a.y * b.y, a.x * b.y + a.y * b.x); }
template <typename C>
__device__ __forceinline__ C scl(C a, typename Real<C>::T s) { return mk<C>(a.x * s, a.y * s); }

}   // namespace kct

// Shared-memory swizzle of the FFT buffers: element x of a 128-byte row r = x / E (E = 8 double2
// or 16 float2 per row) is stored at column (x mod E) xor (r mod E).  Unit-stride runs, the
// stride-R writes of a radix-R stage and the blocked K-per-lane column accesses then spread over
// all banks.  Callers that pass SWZ = true to fft_warp_ct write the input and read the output
// through swz<C>().
template <typename C>
__device__ __forceinline__ int swz(int x) {
    constexpr int RB = sizeof(C) == 16 ? 3 : 4;
    constexpr int RM = (1 << RB) - 1;
    return x ^ ((x >> RB) & RM);
}

// The FFT buffers in FP64 are padded instead, one element after every eight (128 bytes): element x at
// x + x / 8.  The accesses above are as free of conflicts, and where a stage's strides are multiples of
// eight (all but the first stages of 48, 96 and 144) its addresses are one base plus constants, where the
// swizzle takes three or four integer instructions an access: x stage at N = 192 188 -> 173 us, z inverse 97 -> 89.
// FP32 buffers keep the swizzle (their 16-element rows do not match the stages' strides).
template <typename C>
constexpr int FMODE = sizeof(C) == 16 ? 2 : 1;   // 0: plain, 1: swizzled, 2: padded

template <typename C, int MODE = FMODE<C>>
__device__ __forceinline__ int fpos(int x) {
    return MODE == 2 ? x + (x >> 3) : MODE == 1 ? swz<C>(x) : x;
}

// elements of a buffer of n values (n a multiple of 8 where padded)
template <typename C, int MODE = FMODE<C>>
__host__ __device__ constexpr int flen(int n) {
    return MODE == 2 ? n + n / 8 : n;
}

// a transform's buffer as the source or target of a stage
template <typename C, int MODE = FMODE<C>>
struct FftBuf {
    C *p;
};

namespace kct {

// radix-R DFTs, X_q = sum_r v_r exp(S 2 pi i r q / R); the same operation sequence as radix_dft /
// radix8_dft of the runtime FFT
template <typename C, int R, int S>
struct Dft;

template <typename C, int S>
struct Dft<C, 2, S> {
    static __device__ __forceinline__ void run(C *v) {
        const C a0 = v[0], a1 = v[1];
        v[0] = add(a0, a1);
        v[1] = sub(a0, a1);
    }
};

template <typename C, int S>
struct Dft<C, 4, S> {
    static __device__ __forceinline__ void run(C *v) {
        const C a0 = add(v[0], v[2]), a1 = sub(v[0], v[2]);
        const C b0 = add(v[1], v[3]);
        const C d = sub(v[1], v[3]);
        const C b1 = S < 0 ? mk<C>(d.y, -d.x) : mk<C>(-d.y, d.x);   // S i d
        v[0] = add(a0, b0);
        v[1] = add(a1, b1);
        v[2] = sub(a0, b0);
        v[3] = sub(a1, b1);
    }
};

template <typename C, int S>
struct Dft<C, 3, S> {
    static __device__ __forceinline__ void run(C *v) {
        typedef typename Real<C>::T T;
        const T s3 = (T)0.86602540378443864676 * (T)S;
        const C t1 = add(v[1], v[2]);
        const C t2 = sub(v[0], scl(t1, (T)0.5));
        const C d = sub(v[1], v[2]);
        const C t3 = mk<C>(s3 * d.x, s3 * d.y);
        const C o0 = add(v[0], t1);
        v[1] = mk<C>(t2.x - t3.y, t2.y + t3.x);
        v[2] = mk<C>(t2.x + t3.y, t2.y - t3.x);
        v[0] = o0;
    }
};

template <typename C, int S>
struct Dft<C, 5, S> {
    static __device__ __forceinline__ void run(C *v) {
        typedef typename Real<C>::T T;
        const T c5a = (T)0.30901699437494742410, c5b = (T)-0.80901699437494742410;
        const T s5a = (T)0.95105651629515357212 * (T)S, s5b = (T)0.58778525229247312917 * (T)S;
        const C t1 = add(v[1], v[4]), t2 = add(v[2], v[3]);
        const C t3 = sub(v[1], v[4]), t4 = sub(v[2], v[3]);
        const C o0 = add(v[0], add(t1, t2));
        const C r1 = add(v[0], add(scl(t1, c5a), scl(t2, c5b)));
        const C r2 = add(v[0], add(scl(t1, c5b), scl(t2, c5a)));
        const C m1 = add(scl(t3, s5a), scl(t4, s5b));
        const C m2 = sub(scl(t3, s5b), scl(t4, s5a));
        const C i1 = mk<C>(-m1.y, m1.x), i2 = mk<C>(-m2.y, m2.x);
        v[0] = o0;
        v[1] = add(r1, i1);
        v[4] = sub(r1, i1);
        v[2] = add(r2, i2);
        v[3] = sub(r2, i2);
    }
};

template <typename C, int S>
struct Dft<C, 8, S> {
    static __device__ __forceinline__ void run(C *v) {
        typedef typename Real<C>::T T;
        C e[4] = {v[0], v[2], v[4], v[6]}, o[4] = {v[1], v[3], v[5], v[7]};
        Dft<C, 4, S>::run(e);
        Dft<C, 4, S>::run(o);
        const T h = (T)0.70710678118654752440;
        const C t1 = mk<C>(h * (o[1].x - (T)S * o[1].y), h * (o[1].y + (T)S * o[1].x));
        const C t2 = S < 0 ? mk<C>(o[2].y, -o[2].x) : mk<C>(-o[2].y, o[2].x);
        const C t3 = mk<C>(h * (-o[3].x - (T)S * o[3].y), h * (-o[3].y + (T)S * o[3].x));
        v[0] = add(e[0], o[0]);
        v[4] = sub(e[0], o[0]);
        v[1] = add(e[1], t1);
        v[5] = sub(e[1], t1);
        v[2] = add(e[2], t2);
        v[6] = sub(e[2], t2);
        v[3] = add(e[3], t3);
        v[7] = sub(e[3], t3);
    }
};

// element j + r D of a stage's source, r = 0 .. R-1
template <typename C, int D, typename LD>
struct Src {
    LD &ld;
    int j;
    __device__ __forceinline__ Src(LD &l, int jj) : ld(l), j(jj) {}
    __device__ __forceinline__ C operator()(int r) const { return ld(j + r * D); }
};
template <typename C, int D, int MODE>
struct Src<C, D, const FftBuf<C, MODE>> {
    static constexpr bool AFF = MODE == 0 || (MODE == 2 && D % 8 == 0);
    const C *p;
    int j;
    __device__ __forceinline__ Src(const FftBuf<C, MODE> &b, int jj) : p(b.p + (AFF ? fpos<C, MODE>(jj) : 0)), j(jj) {}
    __device__ __forceinline__ C operator()(int r) const {
        return AFF ? p[r * flen<C, MODE>(D)] : p[fpos<C, MODE>(j + r * D)];
    }
};
// element x + q D of its target; x a multiple of R D plus something below D
template <typename C, int R, int D, typename ST>
struct Dst {
    ST &st;
    int x;
    __device__ __forceinline__ Dst(ST &s, int xx) : st(s), x(xx) {}
    __device__ __forceinline__ void operator()(int q, C v) const { st(x + q * D, v); }
};
template <typename C, int R, int D, int MODE>
struct Dst<C, R, D, const FftBuf<C, MODE>> {
    static constexpr bool AFF = MODE == 0 || (MODE == 2 && (D % 8 == 0 || (D == 1 && R == 8)));
    C *p;
    int x;
    __device__ __forceinline__ Dst(const FftBuf<C, MODE> &b, int xx) : p(b.p + (AFF ? fpos<C, MODE>(xx) : 0)), x(xx) {}
    __device__ __forceinline__ void operator()(int q, C v) const {
        p[AFF ? (D == 1 ? q : q * flen<C, MODE>(D)) : fpos<C, MODE>(x + q * D)] = v;
    }
};

// one Stockham stage: butterflies j = 0..N/R-1 of each of the NQ sequences (stored N apart)
// spread over the 32 lanes
template <typename C, int N, int F, int S, int NQ, int MODE, int TWS>
__device__ __forceinline__ void stage(const C *__restrict__ src, C *__restrict__ dst, const C *__restrict__ tw,
                                      int lane) {
    constexpr int R = fac(N, F);
    constexpr int NS = stride(N, F);
    constexpr int NR = N / R;
    constexpr int TW0 = tw_base<N, TWS> + tw_off(N, F);
    constexpr int IT = (NQ * NR + 31) / 32;
#pragma unroll
    for (int it = 0; it < IT; ++it) {
        const int u = lane + 32 * it;
        if ((NQ * NR) % 32 == 0 || u < NQ * NR) {
            const int sq = NQ > 1 ? u / NR : 0;
            const int j = NQ > 1 ? u - sq * NR : u;
            const int base = sq * N;
            const int k = j % NS;
            C v[R];
            const Src<C, NR, const FftBuf<C, MODE>> in(FftBuf<C, MODE>{const_cast<C *>(src)}, base + j);
#pragma unroll
            for (int r = 0; r < R; ++r) {
                C x = in(r);
                if (NS > 1 && r > 0 && k) {
                    C w = __ldg(&tw[TW0 + (r - 1) * NS + k]);
                    if (S > 0) w.y = -w.y;
                    x = mul(x, w);
                }
                v[r] = x;
            }
            Dft<C, R, S>::run(v);
            const Dst<C, R, NS, const FftBuf<C, MODE>> out(FftBuf<C, MODE>{dst}, base + (j - k) * R + k);
#pragma unroll
            for (int q = 0; q < R; ++q) out(q, v[q]);
        }
    }
}

template <typename C, int N, int F, int S, int NQ, int MODE, int TWS, bool END>
struct Step;
template <typename C, int N, int F, int S, int NQ, int MODE, int TWS>
struct Step<C, N, F, S, NQ, MODE, TWS, true> {
    static __device__ __forceinline__ C *go(C *src, C *, const C *, int) { return src; }
};
template <typename C, int N, int F, int S, int NQ, int MODE, int TWS>
struct Step<C, N, F, S, NQ, MODE, TWS, false> {
    static __device__ __forceinline__ C *go(C *src, C *dst, const C *tw, int lane) {
        stage<C, N, F, S, NQ, MODE, TWS>(src, dst, tw, lane);
        __syncwarp();
        return Step<C, N, F + 1, S, NQ, MODE, TWS, (F + 1 >= nfac(N))>::go(dst, src, tw, lane);
    }
};

// stage F of one sequence with its inputs from ld(x) and its outputs to st(x, value): the same
// butterflies, twiddles and operation order as stage()
template <typename C, int N, int F, int S, int TWS, typename LD, typename ST>
__device__ __forceinline__ void stage_io(LD &&ld, ST &&st, const C *__restrict__ tw, int lane) {
    typedef typename std::remove_reference<LD>::type L;
    typedef typename std::remove_reference<ST>::type T;
    constexpr int R = fac(N, F);
    constexpr int NS = stride(N, F);
    constexpr int NR = N / R;
    constexpr int TW0 = tw_base<N, TWS> + tw_off(N, F);
    constexpr int IT = (NR + 31) / 32;
#pragma unroll
    for (int it = 0; it < IT; ++it) {
        const int j = lane + 32 * it;
        if (NR % 32 == 0 || j < NR) {
            const int k = j % NS;
            C v[R];
            const Src<C, NR, L> in(ld, j);
#pragma unroll
            for (int r = 0; r < R; ++r) {
                C x = in(r);
                if (NS > 1 && r > 0 && k) {
                    C w = __ldg(&tw[TW0 + (r - 1) * NS + k]);
                    if (S > 0) w.y = -w.y;
                    x = mul(x, w);
                }
                v[r] = x;
            }
            Dft<C, R, S>::run(v);
            const Dst<C, R, NS, T> out(st, (j - k) * R + k);
#pragma unroll
            for (int q = 0; q < R; ++q) out(q, v[q]);
        }
    }
}

// stage F of one sequence in place in the buffer x (FMODE layout): every lane reads and transforms all
// its butterflies' inputs before the warp writes any output (the same arithmetic as stage())
template <typename C, int N, int F, int S, int TWS>
__device__ __forceinline__ void stage_ip(C *x, const C *__restrict__ tw, int lane) {
    constexpr int R = fac(N, F);
    constexpr int NS = stride(N, F);
    constexpr int NR = N / R;
    constexpr int TW0 = tw_base<N, TWS> + tw_off(N, F);
    constexpr int IT = (NR + 31) / 32;
    C v[IT][R];
#pragma unroll
    for (int it = 0; it < IT; ++it) {
        const int j = lane + 32 * it;
        if (NR % 32 == 0 || j < NR) {
            const int k = j % NS;
            const Src<C, NR, const FftBuf<C>> in(FftBuf<C>{x}, j);
#pragma unroll
            for (int r = 0; r < R; ++r) {
                C u = in(r);
                if (NS > 1 && r > 0 && k) {
                    C w = __ldg(&tw[TW0 + (r - 1) * NS + k]);
                    if (S > 0) w.y = -w.y;
                    u = mul(u, w);
                }
                v[it][r] = u;
            }
            Dft<C, R, S>::run(v[it]);
        }
    }
    __syncwarp();
#pragma unroll
    for (int it = 0; it < IT; ++it) {
        const int j = lane + 32 * it;
        if (NR % 32 == 0 || j < NR) {
            const int k = j % NS;
            const Dst<C, R, NS, const FftBuf<C>> out(FftBuf<C>{x}, (j - k) * R + k);
#pragma unroll
            for (int q = 0; q < R; ++q) out(q, v[it][q]);
        }
    }
    __syncwarp();
}

template <typename C, int N, int F, int S, int TWS, bool END>
struct IpSteps;
template <typename C, int N, int F, int S, int TWS>
struct IpSteps<C, N, F, S, TWS, true> {
    static __device__ __forceinline__ void go(C *, const C *, int) {}
};
template <typename C, int N, int F, int S, int TWS>
struct IpSteps<C, N, F, S, TWS, false> {
    static __device__ __forceinline__ void go(C *x, const C *tw, int lane) {
        stage_ip<C, N, F, S, TWS>(x, tw, lane);
        IpSteps<C, N, F + 1, S, TWS, (F + 2 >= nfac(N))>::go(x, tw, lane);
    }
};

// the stages between the first and the last, ping-ponging between two buffers; returns
// the buffer holding the output of the last of them
template <typename C, int N, int F, int S, int TWS, int MODE, bool END>
struct MidSteps;
template <typename C, int N, int F, int S, int TWS, int MODE>
struct MidSteps<C, N, F, S, TWS, MODE, true> {
    static __device__ __forceinline__ C *go(C *src, C *, const C *, int) { return src; }
};
template <typename C, int N, int F, int S, int TWS, int MODE>
struct MidSteps<C, N, F, S, TWS, MODE, false> {
    static __device__ __forceinline__ C *go(C *src, C *dst, const C *tw, int lane) {
        stage<C, N, F, S, 1, MODE, TWS>(src, dst, tw, lane);
        __syncwarp();
        return MidSteps<C, N, F + 1, S, TWS, MODE, (F + 2 >= nfac(N))>::go(dst, src, tw, lane);
    }
};
}   // namespace kct

// S = -1: exp(-2 pi i jk/N) (FFTW_FORWARD), +1: exp(+...) (FFTW_BACKWARD).  NQ sequences of
// length N lie N apart in a; b is a scratch buffer of the same size (both private to the calling
// warp); the input must be visible to the whole warp (__syncwarp after writing it).  Returns the
// buffer holding the result.  Element x of a buffer is at fpos<C, MODE>(x).  TWS (1 or 2): the
// table is that of length TWS N.
template <typename C, int N, int S, int NQ = 1, int MODE = 0, int TWS = 1>
__device__ __forceinline__ C *fft_warp_ct(C *a, C *b, const C *tw) {
    static_assert(kct::nfac(N) > 0, "transform length must be 2^a 3^b 5^c");
    return kct::Step<C, N, 0, S, NQ, MODE, TWS, false>::go(a, b, tw, threadIdx.x & 31);
}

// fft_warp_ct of one sequence whose first stage reads its input through ld(x) (element x of the
// sequence) and whose last stage writes its output through st(x, value), natural order, so that
// neither needs a copy pass through shared memory; the stages in between use the buffers a and b
// (private to the warp).  pre() runs between the second-last and the last stage
// in every thread of the warp (a block-wide barrier there must be reached by every warp).  Same
// arithmetic as fft_warp_ct.  The last stage reads buffer a when nfac(N) is even, else b; st may
// write the other one.
template <typename C, int N, int S, int TWS = 1, int MODE = FMODE<C>, typename LD, typename ST, typename PRE>
__device__ __forceinline__ void fft_warp_ct_io(const LD ld, const ST st, PRE pre, C *a, C *b, const C *tw) {
    constexpr int L = kct::nfac(N);
    static_assert(L >= 2, "fft_warp_ct_io needs at least two stages");
    const int lane = threadIdx.x & 31;
    const FftBuf<C, MODE> to_a{a};
    kct::stage_io<C, N, 0, S, TWS>(ld, to_a, tw, lane);
    __syncwarp();
    C *src = kct::MidSteps<C, N, 1, S, TWS, MODE, (2 >= L)>::go(a, b, tw, lane);
    pre();
    const FftBuf<C, MODE> from_src{src};
    kct::stage_io<C, N, L - 1, S, TWS>(from_src, st, tw, lane);
}

// fft_warp_ct of one sequence held in one buffer a (FMODE layout) (the input visible to the whole warp):
// every stage but the last runs in place (stage_ip), and the last reads a and writes its output
// through st(x, value), so a warp needs one buffer instead of two.  Same arithmetic
// as fft_warp_ct.
template <typename C, int N, int S, int TWS = 1, typename ST>
__device__ __forceinline__ void fft_warp_ct_ip(C *a, const ST st, const C *tw) {
    constexpr int L = kct::nfac(N);
    static_assert(L >= 1, "transform length must be 2^a 3^b 5^c");
    const int lane = threadIdx.x & 31;
    kct::IpSteps<C, N, 0, S, TWS, (1 >= L)>::go(a, tw, lane);
    const FftBuf<C> from_a{a};
    kct::stage_io<C, N, L - 1, S, TWS>(from_a, st, tw, lane);
}

// the same with every stage in place: the result is left in a (natural order)
template <typename C, int N, int S, int TWS = 1>
__device__ __forceinline__ void fft_warp_ct_inplace(C *a, const C *tw) {
    constexpr int L = kct::nfac(N);
    const int lane = threadIdx.x & 31;
    kct::IpSteps<C, N, 0, S, TWS, (1 >= L)>::go(a, tw, lane);
    kct::stage_ip<C, N, L - 1, S, TWS>(a, tw, lane);
}

// the packed tables behind the n natural entries of a host table t of tw_total(n) values
template <typename C>
inline void tw_pack(C *t, int n) {
    int o = n;
    for (int h = 1; h <= 2; ++h) {   // lengths n and n / 2
        const int N = n / h;
        if (h == 2 && n % 2) break;
        if (kct::nfac(N) <= 0) continue;
        for (int f = 1; f < kct::nfac(N); ++f) {
            const int R = kct::fac(N, f), ns = kct::stride(N, f), step = N / (ns * R);
            for (int r = 1; r < R; ++r)
                for (int k = 0; k < ns; ++k) t[o++] = t[r * k * step * h];
        }
    }
    if (n % 16 == 0)
        for (int k = 0; k < n / 16; ++k)
            for (int l = 0; l < 16; ++l) t[o++] = t[l * k];
}

// the transform lengths with compiled instances (3/2-rule grids of nx, nz = 32, 64, 96, 128, 384
// and the Chebyshev extensions 2 ny = 64, 128, 192, 256, 512)
#define KMM_CT_LEN_LIST(X) X(48) X(64) X(96) X(128) X(144) X(192) X(256) X(512) X(576)

// ---------------------------------------------------------------------------
// In-register DFTs of small lengths (two-pass transforms): X_k = sum_j v_j exp(-2 pi i j k / M),
// natural order in and out.  Lengths that are not a single radix split as M = A B with
// j = B a + b, k = c + A d:  X[c + A d] = sum_b W_M^(bc) W_B^(bd) sum_a v[B a + b] W_A^(ac);
// W_M^j is entry `step` j of the twiddle table tw (a table of length step M).
// ---------------------------------------------------------------------------
template <typename C, int A, int B>
__device__ __forceinline__ void regdft_ab(C *v, const C *__restrict__ tw, int step) {
    constexpr int M = A * B;
    C Q[B][A];
#pragma unroll
    for (int b = 0; b < B; ++b) {
        C u[A];
#pragma unroll
        for (int a = 0; a < A; ++a) u[a] = v[B * a + b];
        kct::Dft<C, A, -1>::run(u);
#pragma unroll
        for (int c = 0; c < A; ++c) Q[b][c] = (b * c) ? kct::mul(u[c], __ldg(tw + step * ((b * c) % M))) : u[c];
    }
#pragma unroll
    for (int c = 0; c < A; ++c) {
        C u[B];
#pragma unroll
        for (int b = 0; b < B; ++b) u[b] = Q[b][c];
        kct::Dft<C, B, -1>::run(u);
#pragma unroll
        for (int d = 0; d < B; ++d) v[c + A * d] = u[d];
    }
}

template <typename C, int M>
struct RegDft;
template <typename C>
struct RegDft<C, 3> {
    static __device__ __forceinline__ void run(C *v, const C *, int) { kct::Dft<C, 3, -1>::run(v); }
};
template <typename C>
struct RegDft<C, 4> {
    static __device__ __forceinline__ void run(C *v, const C *, int) { kct::Dft<C, 4, -1>::run(v); }
};
template <typename C>
struct RegDft<C, 8> {
    static __device__ __forceinline__ void run(C *v, const C *, int) { kct::Dft<C, 8, -1>::run(v); }
};
template <typename C>
struct RegDft<C, 6> {
    static __device__ __forceinline__ void run(C *v, const C *tw, int step) { regdft_ab<C, 2, 3>(v, tw, step); }
};
template <typename C>
struct RegDft<C, 9> {
    static __device__ __forceinline__ void run(C *v, const C *tw, int step) { regdft_ab<C, 3, 3>(v, tw, step); }
};
template <typename C>
struct RegDft<C, 12> {
    static __device__ __forceinline__ void run(C *v, const C *tw, int step) { regdft_ab<C, 4, 3>(v, tw, step); }
};
template <typename C>
struct RegDft<C, 16> {
    static __device__ __forceinline__ void run(C *v, const C *tw, int step) { regdft_ab<C, 4, 4>(v, tw, step); }
};
