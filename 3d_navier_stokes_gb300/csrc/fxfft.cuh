// fxfft.cuh — FP64 line transforms in 64-bit block fixed point.
//
// GB300's FP64 pipe issues 2 lanes per clock and SM (measured: 2.00 DFMA, I2F.F64
// or F2I per clock and SM) against 128 for a 32-bit add and 64 for a 32x32+64-bit
// multiply-add, so an FP64 butterfly costs about 64 issue slots per instruction.
// A transform's own values need no floating exponent: every intermediate value of
// a DFT is a sum of inputs times numbers of modulus <= 1, so it is bounded by the
// line's L1 norm. Each line is therefore scaled by the power of two that puts its
// L1 norm just below 2^61, converted to 64-bit integers, transformed with exact
// 64-bit additions and 64x61-bit twiddle products (both parts of the product that
// reach the result's last bit), and converted back with one rounding. No stage
// needs a shift and nothing can overflow. The absolute error is about one unit of
// 2^-61 of the L1 norm per input and per twiddle product, below the rounding errors
// of the FP64 butterflies it replaces (measured against 64-bit library transforms
// in tests/test_fx_fft.py).
//
// Measured on a GB300 against FP64 butterflies (one RK4 step): 128^3 3.55 -> 0.78 ms, 256^3
// 28.3 -> 5.6 ms, 512^3 250 -> 54 ms; the nonlinear term's error against a 113-bit
// evaluation at 16^3 .. 48^3 falls from 3.1e-16 .. 9.9e-16 to 1.5e-16 .. 2.9e-16.
//
// Lines that hold a NaN or Inf return NaN throughout, as any transform of them
// does; lines whose L1 norm is below 2^-900 (values under about 1e-274) are taken
// as zero.
#pragma once
#include "fft_engine.cuh"

namespace ns3d {

using q64 = long long;

__device__ __forceinline__ q64 madw(int a, int b, q64 c) {
    q64 d;
    asm("mad.wide.s32 %0, %1, %2, %3;" : "=l"(d) : "r"(a), "r"(b), "l"(c));
    return d;
}
__device__ __forceinline__ q64 mulw(int a, int b) {
    q64 d;
    asm("mul.wide.s32 %0, %1, %2;" : "=l"(d) : "r"(a), "r"(b));
    return d;
}

// A twiddle component c in [-1, 1] is c1 2^-31 + c0 2^-62 with |c1| < 2^31 and
// |c0| <= 2^30 (c = +-1: +-(2^31 - 1) for both, off by 2^-62). fx_tw packs
// (cos, sin) as (c1, c0) pairs from the numbers rounded to 2^-62.
__host__ __device__ constexpr int fx_hi(q64 q) {
    const q64 h = (q + (1ll << 30)) >> 31;
    return (int)(h > 2147483647ll ? 2147483647ll : (h < -2147483647ll ? -2147483647ll : h));
}
__host__ __device__ constexpr int fx_lo(q64 q) {
    const q64 l = q - (q64)fx_hi(q) * (1ll << 31);
    return (int)(l > 2147483647ll ? 2147483647ll : (l < -2147483647ll ? -2147483647ll : l));
}

// An integer a as 2^31 ad + a0, 0 <= a0 < 2^31: one funnel shift and one mask
struct FxSplit {
    int ad, a0;
};
__device__ __forceinline__ FxSplit fx_split(q64 a) {
    FxSplit s;
    s.ad = (int)__funnelshift_l((unsigned)a, (unsigned)(a >> 32), 1);
    s.a0 = (int)((unsigned)a & 0x7fffffffu);
    return s;
}
// a * c for a real c = (c1, c0); the product a0 c0 lies below the last bit
__device__ __forceinline__ q64 fx_rmul(q64 a, int c1, int c0) {
    const FxSplit s = fx_split(a);
    const q64 mid = madw(s.a0, c1, mulw(s.ad, c0));
    return madw(s.ad, c1, mid >> 31);
}
// a * (cr + i ci). With |a| <= 2^61 the middle sums stay below 2^63: the low words
// add at most sqrt(2) 2^62, the high ones sqrt(2) 2^60 (|ad| <= 2^30, |c0| <= 2^30).
__device__ __forceinline__ cx<q64> fx_cmul(cx<q64> a, int cr1, int cr0, int ci1, int ci0) {
    const FxSplit r = fx_split(a.x), i = fx_split(a.y);
    const q64 mr = madw(i.a0, -ci1, madw(i.ad, -ci0, madw(r.a0, cr1, mulw(r.ad, cr0))));
    const q64 mi = madw(i.a0, cr1, madw(i.ad, cr0, madw(r.a0, ci1, mulw(r.ad, ci0))));
    return mk<q64>(madw(i.ad, -ci1, madw(r.ad, cr1, mr >> 31)), madw(i.ad, cr1, madw(r.ad, ci1, mi >> 31)));
}
__device__ __forceinline__ cx<q64> cmul(cx<q64> a, int4 w) { return fx_cmul(a, w.x, w.y, w.z, w.w); }
__device__ __forceinline__ void bfly_w(cx<q64> e, cx<q64> o, int4 w, cx<q64>& lo, cx<q64>& hi) {
    const cx<q64> t = cmul(o, w);
    lo = e + t;
    hi = e - t;
}

// cos(2 pi k / 16), cos(2 pi k / 12) times 2^62, the codelets' constants
__device__ constexpr q64 kQ1 = 1ll << 62, kQc16 = 4260642322793532497ll, kQr2 = 3260954456333195553ll,
                         kQs16 = 1764815834521887442ll, kQh3 = 3993837246235628775ll;
__device__ constexpr q64 kQC16[16] = {kQ1, kQc16, kQr2, kQs16, 0, -kQs16, -kQr2, -kQc16,
                                      -kQ1, -kQc16, -kQr2, -kQs16, 0, kQs16, kQr2, kQc16};
__device__ constexpr q64 kQC12[12] = {kQ1, kQh3, kQ1 / 2, 0, -kQ1 / 2, -kQh3, -kQ1, -kQh3, -kQ1 / 2, 0, kQ1 / 2, kQh3};

// lo = e + W_R^K o, hi = e - W_R^K o (see bfly): additions for the trivial angles,
// two real products at odd multiples of 45 degrees, a complex product otherwise
template <int R, int K, bool PK = false>
__device__ __forceinline__ void bfly(cx<q64> e, cx<q64> o, cx<q64>& lo, cx<q64>& hi) {
    constexpr int k = K % R;
    cx<q64> t;
    if constexpr (k == 0) {
        t = o;
    } else if constexpr (4 * k == R) {
        t = mul_mi(o);
    } else if constexpr (2 * k == R) {
        t = mk<q64>(-o.x, -o.y);
    } else if constexpr (4 * k == 3 * R) {
        t = mul_i(o);
    } else if constexpr (R % 3 != 0 && (8 * k) % R == 0) {
        constexpr int e8 = 8 * k / R;   // 1, 3, 5, 7 eighths of a turn
        constexpr int c1 = fx_hi(kQr2), c0 = fx_lo(kQr2);
        const q64 u = fx_rmul(o.x + o.y, c1, c0), v = fx_rmul(o.y - o.x, c1, c0);
        t = e8 == 1 ? mk<q64>(u, v) : e8 == 3 ? mk<q64>(v, -u) : e8 == 5 ? mk<q64>(-u, -v) : mk<q64>(-v, u);
    } else {
        constexpr bool tri = (R % 3 == 0);
        constexpr int n = tri ? 12 : 16, idx = k * n / R;
        static_assert(k * n % R == 0, "no constant for this angle");
        constexpr q64 c = tri ? kQC12[idx % 12] : kQC16[idx % 16];
        constexpr q64 s = tri ? kQC12[(idx + 9) % 12] : kQC16[(idx + 12) % 16];   // sin x = cos(x - 90 degrees)
        t = fx_cmul(o, fx_hi(c), fx_lo(c), fx_hi(-s), fx_lo(-s));                  // W = c - i s
    }
    lo = e + t;
    hi = e - t;
}

template <bool PK> struct Dft<3, cx<q64>, PK> {
    using C = cx<q64>;
    __device__ __forceinline__ static void run(C* a) {
        const C s = a[1] + a[2], d = a[1] - a[2];
        const C m = mk<q64>(a[0].x - (s.x >> 1), a[0].y - (s.y >> 1));
        constexpr int c1 = fx_hi(kQh3), c0 = fx_lo(kQh3);
        const C jd = mk<q64>(fx_rmul(d.y, c1, c0), -fx_rmul(d.x, c1, c0));   // -i sin(60) d
        a[0] = a[0] + s;
        a[1] = m + jd;
        a[2] = m - jd;
    }
    template <bool ONE, typename Wt>
    __device__ __forceinline__ static void run_tw(C* a, const Wt* w) {
        if (!ONE) a[0] = cmul(a[0], w[0]);
        a[1] = cmul(a[1], w[1]);
        a[2] = cmul(a[2], w[2]);
        run(a);
    }
};

// twiddles: the FP64 engines' table holds the packed integers (fx_twiddles) in
// the 16 bytes of each complex entry
template <> struct TwOf<cx<q64>> {
    using tab = int4;
    using type = int4;
    __device__ __forceinline__ static int4 at(const int4* tw, int i) { return __ldg(&tw[i]); }
    __device__ __forceinline__ static int4 one() { return make_int4(2147483647, 2147483647, 0, 0); }
};

// ---------------------------------------------------------------------------
// Scale of a line. Each thread adds the magnitudes of its values as FP32 numbers cut
// from the high words, in units set by its largest exponent (FP64's range does not fit
// FP32's); the threads of a line combine their sums.
// ---------------------------------------------------------------------------
struct FxBound {
    float sum;   // sum of magnitudes / 2^(lo - 896), low by under 2^-19 of itself
    int lo;      // exponent field that the sum's unit belongs to
};
struct FxScale {
    int k;       // values times 2^k are the integers
    bool bad;    // a NaN or Inf in the line
};
constexpr int kFxSpan = 190;   // the largest exponent field is lo + kFxSpan (kept below 254: room for sums)
template <int E>
__device__ __forceinline__ FxBound fx_bound(const cx<double> (&v)[E]) {
    unsigned top = 0u;
#pragma unroll
    for (int s = 0; s < E; ++s)
        top = max(top, max((unsigned)__double2hiint(v[s].x) & 0x7fffffffu, (unsigned)__double2hiint(v[s].y) & 0x7fffffffu));
    FxBound b{0.f, max((int)(top >> 20) - kFxSpan, 0)};
    const unsigned low = (unsigned)b.lo << 20;
    const int base = (int)(0u - ((unsigned)b.lo << 23));
#pragma unroll
    for (int s = 0; s < E; ++s) {
        // the exponent rebased on the multiply pipe; values below the unit's range count as zero
        int x, y;
        asm("mad.lo.s32 %0, %1, 8, %2;" : "=r"(x) : "r"((int)max((unsigned)__double2hiint(v[s].x) & 0x7fffffffu, low)), "r"(base));
        asm("mad.lo.s32 %0, %1, 8, %2;" : "=r"(y) : "r"((int)max((unsigned)__double2hiint(v[s].y) & 0x7fffffffu, low)), "r"(base));
        b.sum += __int_as_float(x);
        b.sum += __int_as_float(y);
    }
    return b;
}
__device__ __forceinline__ FxBound fx_join(FxBound a, FxBound b) {
    const int lo = max(a.lo, b.lo);
    const float fa = __int_as_float(max(127 + a.lo - lo, 0) << 23), fb = __int_as_float(max(127 + b.lo - lo, 0) << 23);
    return FxBound{a.sum * fa + b.sum * fb, lo};
}
// floor(log2(L1 norm)) or above; -4096: nothing to transform; over 1000: NaN, Inf or out of range
__device__ __forceinline__ int fx_exponent(FxBound b) {
    const float f = b.sum * 1.0001f;
    if (b.lo >= 2047 - kFxSpan) return 4096;
    const int e = (int)(__float_as_uint(f) >> 23) - 127 + b.lo - 896;
    return f < 1e-30f || e < -900 ? -4096 : e;
}
__device__ __forceinline__ FxScale fx_scale(int e) {
    return FxScale{e == -4096 ? -4096 : 60 - e, e > 1000};   // |values| 2^k sum to less than 2^61
}
// v 2^k as an integer, cut towards zero
__device__ __forceinline__ q64 fx_from(double v, int k) {
    const int hi = __double2hiint(v), lo = __double2loint(v);
    const int sh = min(1083 - k - (int)(((unsigned)hi << 1) >> 21), 63);   // >= 0: |v| 2^k < 2^61
    const unsigned mh = ((unsigned)hi & 0xfffffu) | 0x100000u;
    const q64 r = (q64)((((unsigned long long)mh << 32 | (unsigned)lo) << 8) >> sh);
    const q64 sgn = hi >> 31;
    return (r ^ sgn) - sgn;
}
// i 2^-k, rounded to nearest: the conversion on the FP64 pipe (idle in a transform), the
// scale as an exponent addition
__device__ __forceinline__ double fx_to(q64 i, int k) {
    const double d = __ll2double_rn(i);
    const int hi = __double2hiint(d);
    return __hiloint2double(hi ? hi - (k << 20) : 0, __double2loint(d));
}

// combine the bounds of the lanes of a warp that differ in the bits of LO..HI-1
template <int LO, int HI>
__device__ __forceinline__ void fx_warp_bound(FxBound& b, unsigned mask) {
#pragma unroll
    for (int o = LO; o < HI; o <<= 1)
        b = fx_join(b, FxBound{__shfl_xor_sync(mask, b.sum, o), __shfl_xor_sync(mask, b.lo, o)});
}

// ---------------------------------------------------------------------------
// A line transform of the passes, v: the thread's E elements (see fft_stages).
// STRIDED passes: the block's NT threads hold TT lines, thread = p TT + t. Line
// passes (TT = 1): P consecutive threads hold a line. `tw` is the engine's table.
// FP32 lines run in floating point. The FP64 result is scaled by 2^-kadd; its slots
// outside the kept band are taken as zero in an inverse transform and left as they
// were by a forward one.
// ---------------------------------------------------------------------------
template <class PL, bool INV, bool PK, int TT, int NT, typename SIdx, typename Sync, int E>
__device__ __forceinline__ void line_fft(cx<float> (&v)[E], cx<float>* sbuf, int p, const cx<float>* __restrict__ tw,
                                         SIdx sidx, Sync sync) {
    if constexpr (INV) PL::template inv<PK>(v, sbuf, p, tw, sidx, sync);
    else PL::template fwd<PK>(v, sbuf, p, tw, sidx, sync);
}
// slot s of every thread lies outside the kept band |k| <= KC = N / 3: a quarter of the
// slots of 16, neither converted nor added (256^3 y passes 0.272 + 0.142 -> 0.255 + 0.132 ms)
template <class PL> constexpr bool fx_outside(int s) {
    return PL::P * s > PL::N / 3 && PL::P * s + PL::P - 1 < PL::N - PL::N / 3;
}
template <class PL, bool INV, bool PK, int TT, int NT, typename SIdx, typename Sync, int E>
__device__ __forceinline__ void line_fft(cx<double> (&v)[E], cx<double>* sbuf, int p,
                                         const cx<double>* __restrict__ tw, SIdx sidx, Sync sync, int kadd = 0) {
    constexpr int P = PL::P;
    FxBound bd = fx_bound(v);
    if constexpr (P > 1) {
        // the lanes of this warp (the last warp of a small block may be short)
        const unsigned mask =
            NT % 32 == 0 || (int)(threadIdx.x | 31) < NT ? 0xffffffffu : (1u << (NT % 32 ? NT % 32 : 31)) - 1u;
        constexpr int span = P * TT < 32 ? P * TT : 32;   // lanes that hold parts of one line's tile
        fx_warp_bound<TT, span>(bd, mask);
        if constexpr (P * TT > 32) {
            // several warps per tile: one entry per warp and line
            constexpr int NW = P * TT / 32;
            __shared__ FxBound part[NT / 32][TT];
            const int w = threadIdx.x / 32, t = threadIdx.x % TT;
            if ((threadIdx.x & 31) < TT) part[w][t] = bd;
            sync();
            const int w0 = w / NW * NW;
            bd = part[w0][t];
#pragma unroll
            for (int q = 1; q < NW; ++q) bd = fx_join(bd, part[w0 + q][t]);
        }
    }
    const FxScale sc = fx_scale(fx_exponent(bd));
    cx<q64> a[E];
#pragma unroll
    for (int s = 0; s < E; ++s) {
        a[s] = mk<q64>(0, 0);
        if (INV && fx_outside<PL>(s)) continue;
        // the inverse transform is the forward one with real and imaginary parts exchanged
        const q64 x = fx_from(v[s].x, sc.k), y = fx_from(v[s].y, sc.k);
        a[s] = INV ? mk<q64>(y, x) : mk<q64>(x, y);
    }
    PL::template fwd<false>(a, reinterpret_cast<cx<q64>*>(sbuf), p, reinterpret_cast<const int4*>(tw), sidx, sync);
    // a line taken as zero keeps its zeros
    const int k = (sc.k == -4096 ? 0 : sc.k) + kadd;
#pragma unroll
    for (int s = 0; s < E; ++s) {
        if (!INV && fx_outside<PL>(s)) continue;
        const double x = fx_to(a[s].x, k), y = fx_to(a[s].y, k);
        v[s] = INV ? mk(y, x) : mk(x, y);
    }
    if (sc.bad) {
        const double nan = __hiloint2double(0x7ff80000, 0);
#pragma unroll
        for (int s = 0; s < E; ++s) v[s] = mk(nan, nan);
    }
}

}  // namespace ns3d
