// fxfft.cuh — FP64 line transforms in 64-bit block fixed point.
//
// GB300's FP64 pipe issues 2 lanes per clock and SM (measured: 2.00 DFMA, I2F.F64
// or F2I per clock and SM) against 128 for a 32-bit add and 64 for a 32x32+64-bit
// multiply-add, so an FP64 butterfly costs about 64 issue slots per instruction.
// A transform's own values need no floating exponent: every intermediate value of
// a DFT is a sum of inputs times numbers of modulus <= 1, so it is bounded by the
// line's L1 norm. Each line is therefore scaled by the power of two that keeps its
// L1 norm below 2^61, held in 64-bit integers and transformed with exact 64-bit
// additions and 64x60-bit twiddle products (both parts of the product that reach the
// result's last bit), so that nothing can overflow. The absolute error is about one unit
// of 2^-61 of the L1 norm per input and per twiddle product. Against the values that
// grows like sqrt(N), an FP64 butterfly's error only like sqrt(log N); long lines
// therefore take their scale in two steps (fx_two).
//
// Between the passes the fields stay integers, each line with its scale k (value =
// integer 2^-k) in a table beside them (FxScales); the next pass brings a line's
// elements to a common scale. Doubles are read and written on the sphere's modes only
// (the x passes), and the integers' range does not end at FP64's exponents.
//
// Measured on a GB300 against FP64 butterflies (one RK4 step): 32^3 0.312 -> 0.073 ms, 128^3
// 3.55 -> 0.63 ms, 256^3 28.3 -> 4.70 ms, 512^3 250 -> 47.1 ms. Relative error of the
// nonlinear term against double-double transforms, butterflies -> these, at 24, 64, 256 and
// 512 points: white fields 7.0, 8.3, 34, 73e-16 -> 2.1, 1.8, 4.1, 4.0e-16 (the packed z lines of
// the butterflies carried u_z beside the larger w_x), k^-5/3 spectra 6.0, 4.7, 6.8, 8.8e-16 ->
// 2.0, 1.6, 2.5, 2.4e-16; white flows in a plane, which have no such pair, at 24, 96, 256 and
// 512 points 5.3, 5.6, 5.7, 6.3e-16 -> 2.2, 2.9, 3.9, 3.7e-16. tests/test_fx_precision.py holds
// plane flows of 24 .. 768 points to a unit of 2^-53 per radix-2 level.
//
// Lines that hold a NaN or Inf carry the scale kFxBad and end as NaN throughout, as any
// transform of them does; lines of zeros the scale kFxZero. The range of inputs and results is
// that of doubles, subnormals among them, and what a line's transform passes through on the
// way has no exponent range to leave.
#pragma once
#include <type_traits>

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

// A twiddle component c in [-1, 1] is c1 2^-30 + c0 2^-60 with |c1| <= 2^30 and
// |c0| <= 2^29, so that quarter turns are exact: equal numbers cancel, as they do in
// FP64. fx_hi and fx_lo give c1 and c0 from c rounded to 2^-60 (a component's error then
// stays below half a unit of a result bounded by 2^61, and is far smaller for lines
// whose values are spread).
constexpr double kQOne = 1152921504606846976.0;   // 2^60
__host__ __device__ constexpr int fx_hi(q64 q) { return (int)((q + (1ll << 29)) >> 30); }
__host__ __device__ constexpr int fx_lo(q64 q) { return (int)(q - (q64)fx_hi(q) * (1ll << 30)); }

// An integer a, |a| < 2^61, as 2^30 ad + a0, 0 <= a0 < 2^30: one funnel shift and one mask
struct FxSplit {
    int ad, a0;
};
__device__ __forceinline__ FxSplit fx_split(q64 a) {
    FxSplit s;
    s.ad = (int)__funnelshift_l((unsigned)a, (unsigned)(a >> 32), 2);
    s.a0 = (int)((unsigned)a & 0x3fffffffu);
    return s;
}
// a * c, |a| < 2^62 (the sum of an element's parts may reach sqrt(2) 2^61), for a constant
// c in (0, 1) given as 2^62 c, from 31-bit halves; the product a0 c0 lies below half the last bit
template <q64 Q, bool ROUND> __device__ __forceinline__ q64 fx_rmul(q64 a) {
    constexpr int c1 = (int)((Q + (1ll << 30)) >> 31), c0 = (int)(Q - (q64)c1 * (1ll << 31));
    const int ad = (int)__funnelshift_l((unsigned)a, (unsigned)(a >> 32), 1);
    const int a0 = (int)((unsigned)a & 0x7fffffffu);
    const q64 mid = madw(a0, c1, ROUND ? madw(ad, c0, 1ll << 30) : mulw(ad, c0));
    return madw(ad, c1, mid >> 31);
}
// a * (cr + i ci), cut or with ROUND to nearest. The middle sums stay below 2^62: |ad| <= 2^31
// times |c0| <= 2^29 and a0 < 2^30 times |c1| <= 2^30, at most sqrt(2) 2^60 from each pair.
template <bool ROUND = false>
__device__ __forceinline__ cx<q64> fx_cmul(cx<q64> a, int cr1, int cr0, int ci1, int ci0) {
    const FxSplit r = fx_split(a.x), i = fx_split(a.y);
    const q64 tr = ROUND ? madw(r.ad, cr0, 1ll << 29) : mulw(r.ad, cr0);
    const q64 ti = ROUND ? madw(r.ad, ci0, 1ll << 29) : mulw(r.ad, ci0);
    const q64 mr = madw(i.a0, -ci1, madw(i.ad, -ci0, madw(r.a0, cr1, tr)));
    const q64 mi = madw(i.a0, cr1, madw(i.ad, cr0, madw(r.a0, ci1, ti)));
    return mk<q64>(madw(i.ad, -ci1, madw(r.ad, cr1, mr >> 30)), madw(i.ad, cr1, madw(r.ad, ci1, mi >> 30)));
}
__device__ __forceinline__ cx<q64> cmul(cx<q64> a, int4 w) { return fx_cmul(a, w.x, w.y, w.z, w.w); }
__device__ __forceinline__ void bfly_w(cx<q64> e, cx<q64> o, int4 w, cx<q64>& lo, cx<q64>& hi) {
    const cx<q64> t = cmul(o, w);
    lo = e + t;
    hi = e - t;
}
// a stage twiddle whose products round to nearest
struct FxRounded : int4 {
    FxRounded() = default;
    __device__ __forceinline__ FxRounded(int4 w) : int4(w) {}
};
__device__ __forceinline__ cx<q64> cmul(cx<q64> a, FxRounded w) { return fx_cmul<true>(a, w.x, w.y, w.z, w.w); }
__device__ __forceinline__ void bfly_w(cx<q64> e, cx<q64> o, FxRounded w, cx<q64>& lo, cx<q64>& hi) {
    const cx<q64> t = cmul(o, w);
    lo = e + t;
    hi = e - t;
}

// cos(2 pi k / 16), cos(2 pi k / 12) times 2^60, the codelets' constants, and sqrt(1/2) and
// sqrt(3/4) times 2^62 (fx_rmul)
__device__ constexpr q64 kQ1 = 1ll << 60, kQc16 = 1065160580698383124ll, kQr2 = 815238614083298888ll,
                         kQs16 = 441203958630471860ll, kQh3 = 998459311558907194ll;
constexpr q64 kQr2x4 = 3260954456333195553ll, kQh3x4 = 3993837246235628775ll;
__device__ constexpr q64 kQC16[16] = {kQ1, kQc16, kQr2, kQs16, 0, -kQs16, -kQr2, -kQc16,
                                      -kQ1, -kQc16, -kQr2, -kQs16, 0, kQs16, kQr2, kQc16};
__device__ constexpr q64 kQC12[12] = {kQ1, kQh3, kQ1 / 2, 0, -kQ1 / 2, -kQh3, -kQ1, -kQh3, -kQ1 / 2, 0, kQ1 / 2, kQh3};

// lo = e + W_R^K o, hi = e - W_R^K o (see bfly): additions for the trivial angles,
// two real products at odd multiples of 45 degrees, a complex product otherwise; PK
// rounds the products to nearest
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
        const q64 u = fx_rmul<kQr2x4, PK>(o.x + o.y), v = fx_rmul<kQr2x4, PK>(o.y - o.x);
        t = e8 == 1 ? mk<q64>(u, v) : e8 == 3 ? mk<q64>(v, -u) : e8 == 5 ? mk<q64>(-u, -v) : mk<q64>(-v, u);
    } else {
        constexpr bool tri = (R % 3 == 0);
        constexpr int n = tri ? 12 : 16, idx = k * n / R;
        static_assert(k * n % R == 0, "no constant for this angle");
        constexpr q64 c = tri ? kQC12[idx % 12] : kQC16[idx % 16];
        constexpr q64 s = tri ? kQC12[(idx + 9) % 12] : kQC16[(idx + 12) % 16];   // sin x = cos(x - 90 degrees)
        t = fx_cmul<PK>(o, fx_hi(c), fx_lo(c), fx_hi(-s), fx_lo(-s));                  // W = c - i s
    }
    lo = e + t;
    hi = e - t;
}

template <bool PK> struct Dft<3, cx<q64>, PK> {
    using C = cx<q64>;
    __device__ __forceinline__ static void run(C* a) {
        const C s = a[1] + a[2], d = a[1] - a[2];
        const C m = mk<q64>(a[0].x - (s.x >> 1), a[0].y - (s.y >> 1));
        const C jd = mk<q64>(fx_rmul<kQh3x4, PK>(d.y), -fx_rmul<kQh3x4, PK>(d.x));   // -i sin(60) d
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
    __device__ __forceinline__ static int4 one() { return make_int4(1 << 30, 0, 0, 0); }
};

// ---------------------------------------------------------------------------
// Scale of a line. Each thread bounds the sum of its magnitudes in units set by its
// largest value; the threads of a line combine their sums.
// ---------------------------------------------------------------------------
constexpr int kFxZero = 30000, kFxBad = -30000;
struct FxBound {
    float sum;   // the magnitudes sum to sum 2^e, low by under 2^-19 of itself
    int e;
};
// Doubles: FP32 numbers cut from the high words with the exponent rebased on the multiply
// pipe (largest field base + kFxSpan: room for sums); smaller values count as zero, and a
// thread with nothing in its high words (below 2^-1042) as one unit of them.
constexpr int kFxSpan = 190;
template <int E>
__device__ __forceinline__ FxBound fx_bound(const cx<double> (&v)[E]) {
    unsigned top = 0u, low_words = 0u;
#pragma unroll
    for (int s = 0; s < E; ++s) {
        top = max(top, max((unsigned)__double2hiint(v[s].x) & 0x7fffffffu, (unsigned)__double2hiint(v[s].y) & 0x7fffffffu));
        low_words |= (unsigned)__double2loint(v[s].x) | (unsigned)__double2loint(v[s].y);
    }
    const int lo = max((int)(top >> 20) - kFxSpan, 0);
    const unsigned low = (unsigned)lo << 20;
    const int base = (int)(0u - ((unsigned)lo << 23));
    FxBound b{0.f, top >= 0x7ff00000u ? -kFxBad : lo - 896};
#pragma unroll
    for (int s = 0; s < E; ++s) {
        int x, y;
        asm("mad.lo.s32 %0, %1, 8, %2;" : "=r"(x) : "r"((int)max((unsigned)__double2hiint(v[s].x) & 0x7fffffffu, low)), "r"(base));
        asm("mad.lo.s32 %0, %1, 8, %2;" : "=r"(y) : "r"((int)max((unsigned)__double2hiint(v[s].y) & 0x7fffffffu, low)), "r"(base));
        b.sum += __int_as_float(x);
        b.sum += __int_as_float(y);
    }
    if (top == 0u && low_words != 0u) b.sum = __int_as_float(8);
    return b;
}
// Integers (|a| <= 2^61) with their scales: sums of the high words' upper bits, aligned to
// the thread's smallest scale, in units of 2^38; at most 2^28 for 16 elements.
template <int E>
__device__ __forceinline__ FxBound fx_bound(const cx<q64> (&a)[E], const int (&k)[E]) {
    int km = kFxZero;
#pragma unroll
    for (int s = 0; s < E; ++s) km = min(km, k[s]);
    unsigned sum = 2 * E;   // cut parts
#pragma unroll
    for (int s = 0; s < E; ++s) {
        const int sh = min(6 + k[s] - km, 31);
        sum += ((unsigned)abs((int)(a[s].x >> 32)) >> sh) + ((unsigned)abs((int)(a[s].y >> 32)) >> sh);
    }
    return FxBound{(float)sum, 38 - km};
}
__device__ __forceinline__ FxBound fx_join(FxBound a, FxBound b) {
    const int e = max(a.e, b.e);
    const float fa = __int_as_float(max(127 + a.e - e, 0) << 23), fb = __int_as_float(max(127 + b.e - e, 0) << 23);
    return FxBound{a.sum * fa + b.sum * fb, e};
}
// combine the bounds of the lanes of a warp that differ in the bits of LO..HI-1
template <int LO, int HI>
__device__ __forceinline__ void fx_warp_bound(FxBound& b) {
#pragma unroll
    for (int o = LO; o < HI; o <<= 1)
        b = fx_join(b, FxBound{__shfl_xor_sync(0xffffffffu, b.sum, o), __shfl_xor_sync(0xffffffffu, b.e, o)});
}
template <int LO, int HI>
__device__ __forceinline__ int fx_warp_min(int k) {
#pragma unroll
    for (int o = LO; o < HI; o <<= 1) k = min(k, __shfl_xor_sync(0xffffffffu, k, o));
    return k;
}
// Lines of 512 points and more take their scale in two steps. Scaled by the whole line's L1 norm,
// 2 N / sqrt(N) times its L2 norm where it is spread, the inputs lose log2 N bits, which from 512
// points on is more than FP64 butterflies lose. The first stage works inside a thread, so that the
// threads' own norms bound it: the inputs are scaled by the largest of those, and the stage's
// outputs, sqrt(16) times as large by then, shifted to the line's scale (FxLater). From 768 points
// on the products round to nearest as well: cut, each loses half a unit on average, which adds up
// over the lines (at 768 points two thirds of the error lay in modes of kx = 0). White flow in a
// plane, relative error of the right-hand side at 512, 768 and 1024 points with one step 7.0, 11
// and 20e-16, butterflies 6.3, 5.6 and 6.1e-16, now 3.7, 4.4 and 4.4e-16. The two steps cost 4 % of
// a 512^3 step, rounding as much again (so not below 768 points).
template <int N> constexpr bool fx_two() { return N >= 512; }
template <int N> constexpr bool fx_round() { return N > 512; }
template <bool ROUND> struct FxLater {
    template <typename W> using Tw = typename std::conditional<ROUND, FxRounded, W>::type;
    int s;
    __device__ __forceinline__ cx<q64> operator()(cx<q64> a) const {
        const q64 half = (1ll << s) >> 1;
        return mk<q64>((a.x + half) >> s, (a.y + half) >> s);
    }
};
template <int N> __device__ __forceinline__ auto fx_mid(int s) {
    if constexpr (fx_two<N>()) return FxLater<fx_round<N>()>{s};
    else return AsIs();
}
// bits between the scale `first` of the first stage and a line's
template <bool TWO> __device__ __forceinline__ int fx_later(int first, int k) {
    return TWO && k != kFxZero && k != kFxBad ? min(max(first - k, 0), 31) : 0;
}
// The bound of a line of a strided tile: NT threads of the block hold tiles of TT lines, P
// threads each, thread = (tile P + p) TT + t; with TWO the smallest `first` of its threads
template <bool TWO, int P, int TT, int NT, typename Sync>
__device__ __forceinline__ FxBound fx_line_bound(FxBound b, int& first, Sync sync) {
    static_assert(NT % 32 == 0, "whole warps");
    if constexpr (P > 1) {
        constexpr int span = P * TT < 32 ? P * TT : 32;   // lanes that hold parts of one tile
        fx_warp_bound<TT, span>(b);
        if constexpr (TWO) first = fx_warp_min<TT, span>(first);
        if constexpr (P * TT > 32) {
            // several warps per tile: one entry per warp and line
            constexpr int NW = P * TT / 32;
            __shared__ FxBound part[NT / 32][TT];
            __shared__ int firsts[TWO ? NT / 32 : 1][TT];
            const int w = threadIdx.x / 32, t = threadIdx.x % TT;
            if ((threadIdx.x & 31) < TT) {
                part[w][t] = b;
                if constexpr (TWO) firsts[w][t] = first;
            }
            sync();
            const int w0 = w / NW * NW;
            b = part[w0][t];
#pragma unroll
            for (int q = 1; q < NW; ++q) b = fx_join(b, part[w0 + q][t]);
            if constexpr (TWO) {
#pragma unroll
                for (int q = 0; q < NW; ++q) first = min(first, firsts[w0 + q][t]);
            }
        }
    }
    return b;
}
// The largest scale at which a line of this bound sums to less than 2^(61 - spare), kFxZero
// or kFxBad
__device__ __forceinline__ int fx_scale(FxBound b, int spare) {
    if (b.e >= -kFxBad - 1000) return kFxBad;
    const float f = b.sum * 1.0001f;
    const int e = (int)(__float_as_uint(f) >> 23) - 127 + b.e;
    return f == 0.f || e < -20000 ? kFxZero : 60 - spare - e;
}
// of doubles: no finer than the smallest normal number needs (fx_from)
__device__ __forceinline__ int fx_scale_in(FxBound b, int spare) {
    const int k = fx_scale(b, spare);
    return k == kFxZero ? k : min(k, 1082);
}
// and of integers: no finer than the finest common scale of the elements
__device__ __forceinline__ int fx_scale_of(FxBound b, int spare) {
    const int k = fx_scale(b, spare);
    return k == kFxBad || k == kFxZero ? k : min(k, 38 - b.e);
}
// v 2^k as an integer, cut towards zero (|v| 2^k < 2^61, k <= 1082 unless v is zero)
__device__ __forceinline__ q64 fx_from(double v, int k) {
    const int hi = __double2hiint(v), lo = __double2loint(v);
    const unsigned mag = (unsigned)hi & 0x7fffffffu;
    const unsigned mh = min(mag, ((unsigned)hi & 0xfffffu) | 0x100000u);   // subnormals: no leading bit,
    const int sh = min(1083 - k - (int)(mag >> 20), 1082 - k);             // the smallest normal's exponent
    unsigned long long r;
    asm("shr.u64 %0, %1, %2;" : "=l"(r) : "l"(((unsigned long long)mh << 32 | (unsigned)lo) << 8), "r"(sh));   // 0 past 63
    const q64 sgn = hi >> 31;
    return ((q64)r ^ sgn) - sgn;
}
// an integer at scale k0 to the line's scale k <= k0, rounded to nearest
__device__ __forceinline__ cx<q64> fx_align(cx<q64> a, int k0, int k) {
    const int sh = min(max(k0 - k, 0), 63);
    const q64 half = (q64)((1ull << sh) >> 1);
    return mk<q64>((a.x + half) >> sh, (a.y + half) >> sh);
}
// i 2^-k, rounded to nearest: the conversion on the FP64 pipe, the scale as an exponent
// addition (-1020 <= -k, |i| < 2^62)
__device__ __forceinline__ double fx_to(q64 i, int k) {
    const double d = __ll2double_rn(i);
    const int hi = __double2hiint(d);
    return __hiloint2double(hi ? hi - (k << 20) : 0, __double2loint(d));
}
// Scales beyond the ones fx_to takes: convert at fx_near(k), then multiply by fx_far(k), a power
// of two whose product rounds to a subnormal, zero or infinity; NaN for bad lines
__device__ __forceinline__ int fx_near(int k) { return min(max(k, -900), 1020); }
__device__ __forceinline__ double fx_far(int k) {
    return __hiloint2double(k == kFxBad ? 0x7ff80000 : (1023 + min(max(fx_near(k) - k, -1022), 1023)) << 20, 0);
}
__device__ __forceinline__ double fx_to_any(q64 a, int k) {
    const double d = fx_to(a, fx_near(k));
    return fx_near(k) == k ? d : d * fx_far(k);
}
// slot s of every thread lies outside the kept band |k| <= KC = N / 3: a quarter of the
// slots of 16, neither loaded nor added by an inverse transform, nor stored by a forward
// one (256^3 y passes, when they took 0.272 + 0.142 ms: to 0.255 + 0.132; now 0.201 + 0.108)
template <class PL> constexpr bool fx_outside(int s) {
    return PL::P * s > PL::N / 3 && PL::P * s + PL::P - 1 < PL::N - PL::N / 3;
}

}  // namespace ns3d
