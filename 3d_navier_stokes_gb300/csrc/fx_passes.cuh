// fx_passes.cuh — the passes of the FP64 engines, on the 64-bit integer line transforms
// of fxfft.cuh. Layouts and launch grids are those of the FP32 passes in
// ns3d_kernels.cuh; the work array W holds integers.
#pragma once
#include "ns3d_kernels.cuh"

namespace ns3d {

// Scales of the lines of W after each pass, member after member (fx_scales_ints ints each):
// one per line of the pass that wrote it.
struct FxScales {
    int* x;   // after P1: [6 fields][N ky][NZP]
    int* y;   // after P2: [6][N x][NZP]
    int* z;   // after P3: [3][N x][N y]
    int* w;   // after P4: [3][N x][NZP]
};
template <int N> constexpr long long fx_scales_ints() { return 15LL * N * Geo<N>::NZP + 3LL * N * N; }
template <int N> __device__ __forceinline__ FxScales fx_scales(int* base, long long member) {
    int* b = base + member * fx_scales_ints<N>();
    constexpr long long c = (long long)N * Geo<N>::NZP;
    return FxScales{b, b + 6 * c, b + 15 * c, b + 12 * c};
}

// ---------------------------------------------------------------------------
// x passes, on FxPlan<N>::X, fx_tile pencils per CTA. `aux` holds 1/k2 for k2 <= KC^2 (0 at 0) and
// then the N wavenumbers of the x rows, so that no mode pays an FP64 division or
// conversion.
// ---------------------------------------------------------------------------
template <int N> constexpr int fxinv_threads() { return fx_tile<N>() * FxPlan<N>::X::P; }
template <int N> constexpr int fxfwd_threads() { return 3 * fx_tile<N, true>() * FxPlan<N>::X::P; }
constexpr int fx_log2(int n) { return n <= 1 ? 0 : 1 + fx_log2(n / 2); }
constexpr int fx_ctas(int per_sm, int threads) { return per_sm / threads < 1 ? 1 : per_sm / threads; }
// CTAs per SM the passes are compiled for. Inverse: 640 threads (96 registers) from 16
// threads per line, 512 below (256^3 0.164 -> 0.160 ms, 128^3 0.0253 against 0.0258).
// Forward: two CTAs of 384 threads or one of 768 (80 registers, a few spills, but one
// CTA's transforms under the other's FP64 work: 256^3 0.208 -> 0.166 ms, 512^3 1.96 ->
// 1.51 ms, now 0.163 and 1.47 ms), 576 threads with smaller CTAs (128^3 0.0395 -> 0.0343 ms,
// 0.0411 with 768).
template <int N> constexpr int fxinv_ctas() { return fx_ctas(FxPlan<N>::X::P >= 16 ? 640 : 512, fxinv_threads<N>()); }
template <int N> constexpr int fxfwd_ctas() { return fx_ctas(fxfwd_threads<N>() >= 384 ? 768 : 576, fxfwd_threads<N>()); }
template <int N> constexpr int fxinv_smem() { return N * fx_tile<N>() * 16; }
template <int N> constexpr int fxfwd_smem() { return 3 * N * fx_tile<N, true>() * 16; }

// P1: one field of u, w = i k x u of one tile per CTA (blockIdx.z = 6 member + field).
// The curl is formed on the modes of the sphere (a third of a column's rows), where the
// FP64 pipe has to do less than for the transformed columns, and the six fields are
// independent CTAs, which fills the chip at small N (32^3: 11 us per launch, 27 us with
// the six transforms in one CTA, now 8.4 us; 256^3: 0.19 against 0.25 ms, now 0.157). The
// inputs' second and third reads hit L2.
template <int N>
__global__ void __launch_bounds__(fxinv_threads<N>(), fxinv_ctas<N>())
k_xinv_fx(const cx<double>* __restrict__ U, cx<q64>* __restrict__ W, int* __restrict__ scales,
          const int4* __restrict__ tw, const double* __restrict__ aux) {
    const long long dep = pdl_begin();
    U += dep;
    W += dep;
    scales += dep;
    using G = Geo<N>;
    using PL = typename FxPlan<N>::X;
    constexpr int TT = fx_tile<N>(), E = PL::E, P = PL::P, NT = TT * P;
    constexpr bool kPow2 = (N & (N - 1)) == 0;
    extern __shared__ __align__(16) unsigned char smem_raw[];
    cx<q64>* sbuf = reinterpret_cast<cx<q64>*>(smem_raw);
    const int t = threadIdx.x % TT, p = threadIdx.x / TT;
    const int kz0 = blockIdx.x * TT, kz = kz0 + t;
    const int ky = (int)blockIdx.y - G::KC;
    const int j = ky < 0 ? ky + N : ky;
    if (ky * ky + kz0 * kz0 > G::KC2) return;
    const int f = blockIdx.z % 6;
    U += (long long)(blockIdx.z / 6) * 3 * G::FS;
    W += (long long)blockIdx.z * G::FS;
    const int rem = kz <= G::KC ? G::KC2 - ky * ky - kz * kz : -1;
    const long long off = (long long)j * G::NZP + kz, xs = (long long)N * G::NZP;
    const double* kxs = aux + G::KC2 + 1;
    const double fky = ky, fkz = kz;
    StridedIdx<TT, PL::R1> sidx{t};
    SyncBlock sync;
    // f < 3: u_f; else i (ca u_a - cb u_b) with kx as ca of w_z and cb of w_y
    const int c = f - 3, ia = c == 0 ? 2 : c == 1 ? 0 : 1, ib = c == 0 ? 1 : c == 1 ? 2 : 0;
    const cx<double>* A = U + (f < 3 ? f : ia) * G::FS + off;
    const cx<double>* B = U + ib * G::FS + off;
    cx<double> v[E];
    if (f < 3) {
#pragma unroll
        for (int s = 0; s < E; ++s) {
            const int i = p + P * s, kx = kof<N>(i);
            v[s] = czero<double>();
            if (P * s > G::KC && P * s + P - 1 < N - G::KC) continue;   // |kx| > KC in every thread
            if (kx * kx <= rem) v[s] = A[(long long)i * xs];
        }
    } else {
#pragma unroll
        for (int s = 0; s < E; ++s) {
            const int i = p + P * s, kx = kof<N>(i);
            v[s] = czero<double>();
            if (P * s > G::KC && P * s + P - 1 < N - G::KC) continue;
            if (kx * kx <= rem) {
                const cx<double> a = A[(long long)i * xs], b = B[(long long)i * xs];
                const double fkx = __ldg(&kxs[i]);
                const double ca = c == 0 ? fky : c == 1 ? fkz : fkx, cb = c == 0 ? fkz : c == 1 ? fkx : fky;
                v[s] = mk(cb * b.y - ca * a.y, ca * a.x - cb * b.x);
            }
        }
    }
    if (!kPow2) {
#pragma unroll
        for (int s = 0; s < E; ++s)
            if (!(P * s > G::KC && P * s + P - 1 < N - G::KC)) v[s] = v[s] * (1.0 / ((double)N * N * N));
    }
    constexpr bool TWO = fx_two<N>();
    FxBound b = fx_bound(v);
    int first = TWO ? fx_scale_in(b, 0) : 0;
    b = fx_line_bound<TWO, P, TT, NT>(b, first, sync);
    const int k = fx_scale_in(b, 0), later = fx_later<TWO>(first, k);
    cx<q64> a[E];
#pragma unroll
    for (int s = 0; s < E; ++s)
        // an inverse transform is the forward one with real and imaginary parts exchanged
        a[s] = fx_outside<PL>(s) ? mk<q64>(0, 0) : mk<q64>(fx_from(v[s].y, k + later), fx_from(v[s].x, k + later));
    PL::template fwd<fx_round<N>()>(a, sbuf, p, tw, sidx, sync, fx_mid<N>(later));
    if (rem >= 0) {
#pragma unroll
        for (int s = 0; s < E; ++s) W[off + (long long)(p + P * s) * xs] = mk<q64>(a[s].y, a[s].x);
        // 1/N^3 of a power of two goes into the scale
        if (p == 0)
            fx_scales<N>(scales, blockIdx.z / 6).x[((long long)f * N + j) * G::NZP + kz] =
                k + (kPow2 && k != kFxZero && k != kFxBad ? 3 * fx_log2(N) : 0);
    }
}

// P2 / P4: FFT along y in place, grid and masks of k_ypass; the elements of a line come
// with scales of their own (per ky after P1, per y after P3).
template <int N> constexpr int fxy_tile() { return FxPlan<N>::A::P * 8 <= 512 ? 8 : 4; }
template <int N> constexpr int fxy_threads() { return fxy_tile<N>() * FxPlan<N>::A::P; }
// 512 threads per SM (128 registers); 640 with at most 12 elements per thread (192^3 0.118 ->
// 0.114 ms; 256^3, 16 elements: 0.201 against 0.207 ms)
template <int N> constexpr int fxy_ctas() { return fx_ctas(FxPlan<N>::A::E <= 12 ? 640 : 512, fxy_threads<N>()); }
template <int N, bool INV>
__global__ void __launch_bounds__(fxy_threads<N>(), fxy_ctas<N>())
k_ypass_fx(cx<q64>* __restrict__ W, int* __restrict__ scales, const int4* __restrict__ tw) {
    const long long dep = pdl_begin();
    W += dep;
    scales += dep;
    using G = Geo<N>;
    using PL = typename FxPlan<N>::A;
    constexpr int TT = fxy_tile<N>(), E = PL::E, P = PL::P, NT = TT * P;
    constexpr int NF = INV ? 6 : 3;
    extern __shared__ __align__(16) unsigned char smem_raw[];
    cx<q64>* sbuf = reinterpret_cast<cx<q64>*>(smem_raw);
    const int t = threadIdx.x % TT, p = threadIdx.x / TT;
    const int kz = blockIdx.x * TT + t, i = blockIdx.y;
    const bool colok = kz <= G::KC;
    const int rem = G::KC2 - kz * kz;
    const int mem = blockIdx.z / NF, f = blockIdx.z % NF;
    cx<q64>* base = W + ((long long)mem * 6 + f) * G::FS + (long long)i * N * G::NZP + kz;
    const FxScales sc = fx_scales<N>(scales, mem);
    const int* kin = INV ? sc.x + (long long)f * N * G::NZP + kz : sc.z + ((long long)f * N + i) * N;
    StridedIdx<TT, PL::R1> sidx{t};
    SyncBlock sync;
    cx<q64> a[E];
    int ke[E];
#pragma unroll
    for (int s = 0; s < E; ++s) {
        const int jj = p + P * s, ky = kof<N>(jj);
        a[s] = mk<q64>(0, 0);
        ke[s] = kFxZero;
        if (INV && fx_outside<PL>(s)) continue;
        if (colok && (!INV || ky * ky <= rem)) {
            a[s] = base[(long long)jj * G::NZP];
            ke[s] = kin[INV ? (long long)jj * G::NZP : jj];
        }
    }
    constexpr bool TWO = fx_two<N>();
    FxBound b = fx_bound(a, ke);
    int first = TWO ? fx_scale_of(b, 0) : 0;
    b = fx_line_bound<TWO, P, TT, NT>(b, first, sync);
    const int k = fx_scale_of(b, 0), later = fx_later<TWO>(first, k);
#pragma unroll
    for (int s = 0; s < E; ++s) {
        if (INV && fx_outside<PL>(s)) continue;
        const cx<q64> v = fx_align(a[s], ke[s], k + later);
        a[s] = INV ? mk<q64>(v.y, v.x) : v;
    }
    PL::template fwd<fx_round<N>()>(a, sbuf, p, tw, sidx, sync, fx_mid<N>(later));
    if (!colok) return;
#pragma unroll
    for (int s = 0; s < E; ++s) {
        const int jj = p + P * s, ky = kof<N>(jj);
        if (!INV && fx_outside<PL>(s)) continue;
        if (INV) base[(long long)jj * G::NZP] = mk<q64>(a[s].y, a[s].x);
        else if (ky * ky <= rem) base[(long long)jj * G::NZP] = a[s];
    }
    if (p == 0) (INV ? sc.y : sc.w)[((long long)f * N + i) * G::NZP + kz] = k;
}

// h / 3 to the nearest: the product with 1/3, corrected by its exact residual (the final step of
// division by Markstein, IBM J. Res. Dev. 34, 1990). A division costs a 32^3 step 2 us; the product
// alone is off by up to a unit, the same in every stage and step.
__device__ __forceinline__ double third(double h) {
    const double q = h * (1.0 / 3.0);
    return fma(fma(-3.0, q, h), 1.0 / 3.0, q);
}
// P5: three groups of threads transform one component each, leave the rows of the band in
// their exchange buffers, and all threads share the modes of the tile for the stage
// algebra. The mode loop's FP64 work is a large part (FP64 pipe 44 % busy at 256^3 with the
// division and conversions it had), so 1/k2 comes from `aux` and the per-step factors are
// formed once per thread. Three groups instead of one after the other: 24 -> 14 us per
// launch at 32^3, 0.226 -> 0.212 ms at 256^3 (now 10 us and 0.163 ms).
template <int N, int INTEG, int MODE>
__global__ void __launch_bounds__(fxfwd_threads<N>(), fxfwd_ctas<N>())
k_xfwd_fx(const cx<q64>* __restrict__ W, int* __restrict__ scales, cx<double>* __restrict__ U,
          cx<double>* __restrict__ UT, cx<double>* __restrict__ ACC, const int4* __restrict__ tw,
          const StepDev* __restrict__ sd,
          const cx<double>* __restrict__ tab, const double* __restrict__ aux, cx<double>* __restrict__ K,
          double* __restrict__ dpart, const RkStage rs) {
    const long long dep = pdl_begin();
    W += dep;
    scales += dep;
    U += dep;
    UT += dep;
    ACC += dep;
    sd += dep;
    tab += dep;
    K += dep;
    dpart += dep;
    using G = Geo<N>;
    using PL = typename FxPlan<N>::X;
    using C = cx<double>;
    constexpr int TT = fx_tile<N, true>(), E = PL::E, P = PL::P, NG = TT * P, NT = 3 * NG;
    extern __shared__ __align__(16) unsigned char smem_raw[];
    C* buf = reinterpret_cast<C*>(smem_raw);   // [3 components][N rows][TT]
    const int g = threadIdx.x / NG;
    const int t = threadIdx.x % TT, p = threadIdx.x % NG / TT;
    const int kz0 = blockIdx.x * TT;
    const int ky = (int)blockIdx.y - G::KC;
    const int j = ky < 0 ? ky + N : ky;
    {
        const long long mem = blockIdx.z;   // ensemble member
        W += mem * 6 * G::FS;
        U += mem * 3 * G::FS;
        UT += mem * 3 * G::FS;
        ACC += mem * 3 * G::FS;
        sd += mem;
        tab += mem * (G::KC2 + 1);
        if (INTEG == INT_TAB) {
            K += mem * 18 * G::FS;
            dpart += (mem * gridDim.y * gridDim.x + (long long)blockIdx.y * gridDim.x + blockIdx.x) * 3;
        }
    }
    if (ky * ky + kz0 * kz0 > G::KC2) {
        if (INTEG == INT_TAB && rs.kind == 2 && threadIdx.x < 3) dpart[threadIdx.x] = 0.0;
        return;
    }
    const long long xs = (long long)N * G::NZP;
    C* sbuf = buf + (size_t)g * N * TT;
    __shared__ int line_scale[3][TT];
    // the stage algebra's modes of this thread: rows r0 + it RPI, it < NIT, of the band's 2 KC + 1;
    // their state is loaded CH rows at a time, before the transform where that is all of them
    constexpr int RPI = NT / TT, NIT = (2 * G::KC + RPI) / RPI, CH = NIT < 2 ? 1 : 2;
    constexpr bool needU = MODE <= X_STAGE4 && !(INTEG == INT_IFRK4 && MODE == X_STAGE4);
    constexpr bool needA = MODE <= X_STAGE4 && MODE != X_STAGE1 && INTEG != INT_TAB;
    const int r0 = threadIdx.x / TT, kz = kz0 + t, kp2 = ky * ky + kz * kz;
    const double fkz = kz;
    C us[CH][3], as[CH][3];
    auto load_state = [&](int it, C (&u)[3], C (&a)[3]) {
        const int r = r0 + it * RPI, kx = r - G::KC;
        if (r > 2 * G::KC || kz > G::KC || kx * kx + kp2 > G::KC2) return;
        const long long q = (long long)(kx < 0 ? kx + N : kx) * xs + (long long)j * G::NZP + kz;
#pragma unroll
        for (int c = 0; c < 3; ++c) {
            if (needU) u[c] = U[c * G::FS + q];
            if (needA) a[c] = ACC[c * G::FS + q];
        }
    };
    if (NIT <= CH)
#pragma unroll
        for (int q = 0; q < CH; ++q) load_state(q, us[q], as[q]);
    {
        const bool colok = kz <= G::KC && ky * ky + kz * kz <= G::KC2;
        const cx<q64>* src = W + g * G::FS + (long long)j * G::NZP + kz;
        const int* kin = fx_scales<N>(scales, blockIdx.z).w + (long long)g * N * G::NZP + kz;
        cx<q64> a[E];
        int ke[E];
#pragma unroll
        for (int s = 0; s < E; ++s) {
            a[s] = colok ? src[(long long)(p + P * s) * xs] : mk<q64>(0, 0);
            ke[s] = colok ? kin[(p + P * s) * G::NZP] : kFxZero;
        }
        // the state rows of this tile into L2 (the groups share the rows)
        if (g == 0) xfwd_prefetch_state<double, N, INTEG, MODE, E, P, TT>(U, ACC, K, rs, p, t, ky, kz0, j);
        StridedIdx<TT, PL::R1> sidx{t};
        static_assert(NG % 32 == 0, "a group has whole warps");
        SyncGroup sync{1 + g, NG};
        constexpr bool TWO = fx_two<N>();
        FxBound b = fx_bound(a, ke);
        int first = TWO ? fx_scale_of(b, 0) : 0;
        b = fx_line_bound<TWO, P, TT, NT>(b, first, sync);
        const int k = fx_scale_of(b, 0), later = fx_later<TWO>(first, k);
#pragma unroll
        for (int s = 0; s < E; ++s) a[s] = fx_align(a[s], ke[s], k + later);
        PL::template fwd<fx_round<N>()>(a, reinterpret_cast<cx<q64>*>(sbuf), p, tw, sidx, sync, fx_mid<N>(later));
        const int kn = fx_near(k);
#pragma unroll
        for (int s = 0; s < E; ++s)
            if (!fx_outside<PL>(s)) sbuf[(p + P * s) * TT + t] = mk(fx_to(a[s].x, kn), fx_to(a[s].y, kn));
        if (p == 0) line_scale[g][t] = k;
    }
    __syncthreads();
    // rare scales: the mode loop multiplies by what the conversions left out (a branch beside those
    // parts them from the last stage's additions, which cover them: 96^3 21.7 -> 23.4 us with a loop
    // of its own behind them, 28 us with their code in it)
    const bool far = line_scale[0][t] != fx_near(line_scale[0][t]) || line_scale[1][t] != fx_near(line_scale[1][t]) ||
                     line_scale[2][t] != fx_near(line_scale[2][t]);

    const double* kxs = aux + G::KC2 + 1;
    const double fky = ky;
    const double h = MODE <= X_STAGE4 ? sd->dt : 0.0;
    const double h2 = 0.5 * h, h3 = third(h), h6 = 0.5 * h3;
    double es[3] = {0.0, 0.0, 0.0};   // DP5CN error partial sums
#pragma unroll 1
    for (int it0 = 0; it0 < NIT; it0 += CH) {
      if (NIT > CH)
#pragma unroll
        for (int q = 0; q < CH; ++q) load_state(it0 + q, us[q], as[q]);
#pragma unroll
      for (int ch = 0; ch < CH; ++ch) {
        const int r = r0 + (it0 + ch) * RPI;
        const int kx = r - G::KC, i = kx < 0 ? kx + N : kx;
        const int k2 = kx * kx + kp2;
        if (r > 2 * G::KC || kz > G::KC || k2 > G::KC2) continue;
        const long long idx = (long long)i * xs + (long long)j * G::NZP + kz;
        C n[3];
#pragma unroll
        for (int c = 0; c < 3; ++c) n[c] = buf[(c * N + i) * TT + t];
        if (far) {
#pragma unroll
            for (int c = 0; c < 3; ++c) {
                const int k = line_scale[c][t];
                if (k != fx_near(k)) n[c] = n[c] * fx_far(k);
            }
        }
        if (MODE != X_PLAIN) {
            // Leray projection; the mean is removed
            const double fkx = __ldg(&kxs[i]), kinv = __ldg(&aux[k2]);
            const C d = mk((n[0].x * fkx + n[1].x * fky + n[2].x * fkz) * kinv,
                           (n[0].y * fkx + n[1].y * fky + n[2].y * fkz) * kinv);
            n[0] = n[0] - d * fkx;
            n[1] = n[1] - d * fky;
            n[2] = n[2] - d * fkz;
            if (k2 == 0) n[0] = n[1] = n[2] = czero<double>();
        }
        if constexpr (MODE == X_RHS || MODE == X_PLAIN) {
#pragma unroll
            for (int c = 0; c < 3; ++c) ACC[c * G::FS + idx] = n[c];
        } else if constexpr (INTEG == INT_TAB) {
            const C ab = ldg(&tab[k2]);
#pragma unroll
            for (int c = 0; c < 3; ++c) {
                const long long q = c * G::FS + idx;
                C acc = n[c] * rs.c_cur, ea = n[c] * rs.e_cur;
#pragma unroll
                for (int jj = 0; jj < 6; ++jj) {
                    if (jj < rs.nk && (rs.c[jj] != 0.0 || rs.e[jj] != 0.0)) {
                        const C kj = K[(long long)jj * 3 * G::FS + q];
                        acc = acc + kj * rs.c[jj];
                        if (rs.kind == 2) ea = ea + kj * rs.e[jj];
                    }
                }
                if (rs.store >= 0) K[(long long)rs.store * 3 * G::FS + q] = n[c];
                const C u = us[ch][c];
                if (rs.kind == 0) {
                    UT[q] = u + acc * h;
                } else if (rs.kind == 1) {
                    U[q] = u * ab.x + acc * ab.y;
                } else {
                    const C un = u * ab.x + acc * ab.y;
                    ACC[q] = un;
                    const C df = ea * ab.y;
                    const double m0 = sqrt(u.x * u.x + u.y * u.y), m1 = sqrt(un.x * un.x + un.y * un.y);
                    const double den = sd->dp_atol + (m0 > m1 ? m0 : m1) * sd->dp_rtol;
                    es[c] += (df.x * df.x + df.y * df.y) / (den * den);
                }
            }
        } else if constexpr (INTEG == INT_IFRK4) {
            const C ef = ldg(&tab[k2]);
            const double Eh = ef.x, Ef = ef.y;
            const double cu = MODE == X_STAGE3 ? h * Eh : h2, ca = h3 * Eh;
#pragma unroll
            for (int c = 0; c < 3; ++c) {
                const long long q = c * G::FS + idx;
                if (MODE == X_STAGE1) {
                    const C u = us[ch][c];
                    UT[q] = (u + n[c] * h2) * Eh;
                    ACC[q] = (u + n[c] * h6) * Ef;
                } else if (MODE == X_STAGE4) {
                    U[q] = as[ch][c] + n[c] * h6;
                } else {
                    UT[q] = us[ch][c] * (MODE == X_STAGE2 ? Eh : Ef) + n[c] * cu;
                    ACC[q] = as[ch][c] + n[c] * ca;
                }
            }
        } else {
#pragma unroll
            for (int c = 0; c < 3; ++c) {
                const long long q = c * G::FS + idx;
                if (MODE == X_STAGE4) {
                    const C ab = ldg(&tab[k2]);
                    U[q] = us[ch][c] * ab.x + (as[ch][c] + n[c] * (1.0 / 6.0)) * ab.y;
                } else {
                    UT[q] = us[ch][c] + n[c] * (MODE == X_STAGE3 ? h : h2);
                    ACC[q] = MODE == X_STAGE1 ? n[c] * (1.0 / 6.0) : as[ch][c] + n[c] * (1.0 / 3.0);
                }
            }
        }
      }
    }
    if constexpr (INTEG == INT_TAB) {
        if (rs.kind == 2) dp_block_sum<NT>(es, dpart);
    }
}

// ---------------------------------------------------------------------------
// P3, MODE as in k_zpass (0: c2r, u x w, r2c; 1: c2r to real_out [6][N][N][N]; 2: r2c of
// real_out [3][N][N][N]). A CTA takes ZP pairs of adjacent lines; three groups of P
// threads own one complex transform each. Each of a line's fields gets a scale of its own
// (2^60 bounds its L1 norm), group g turns fields 2g, 2g+1 into real space, the threads
// form the products >> 60 of u x w from the 30-bit halves and bring the two of a
// component to one scale, and the groups transform (Nx, Ny) of both lines and (Nz_a, Nz_b) back,
// every real line with a shift of its own that bounds its L1 norm by 2^60. The
// transforms exchange through the group's own third of the line's buffer, which
// then holds its real-space output, so 96 bytes of shared memory per grid point of
// a pair are enough for four 96-thread CTAs per SM; where a group lies inside a
// warp it synchronises with its warp only. 1.24 -> 0.60 ms per launch at 256^3 against
// the CTA-synchronous pass with transforms that convert at both ends and FP64 products (CTAs
// of 192 and 384 threads, whose warps run in step, measured 0.64 and 0.73 ms then); with the
// work array in integers 0.556, with the scales per field and the peaks below 0.567 ms.
// Issue bound.
// ---------------------------------------------------------------------------
// Exchange slots of a line, 16-byte elements, 8 lanes (one wavefront) at a time: m + (m >> A),
// lines XS slots apart. One pad slot per 16 counts 2.0 - 2.1 wavefronts per access at 8, 24 and
// 48 points and 1.33 at 64, these 1.2 and 1.0; at 96 and 192 points (1.4 to 1.2) nothing was
// gained.
// From 256 points on a line's own peaks, not the bound by its modes, set the scales of the products'
// operands: operands of 2^60 / sqrt(N) each lose log2 N bits between them. White flow in a plane,
// relative error of the right-hand side at 128, 192, 256, 384 and 512 points without the peaks 2.6,
// 4.1, 5.9, 6.8 and 8.8e-16 (FP64 butterflies 5.0, 6.1, 5.7, 5.9 and 6.3e-16), with them at 256,
// 384 and 512 3.9, 5.5 and 7.0e-16; they cost 3.5 % of this pass (0.547 -> 0.567 ms at 256^3).
template <int N> constexpr bool zfx_peaks() { return N >= 256; }
template <int N> struct FxLay { static constexpr int A = 4, XS = zpad<N>(); };
template <> struct FxLay<8> { static constexpr int A = 2, XS = 12; };
template <> struct FxLay<24> { static constexpr int A = 4, XS = 28; };
template <> struct FxLay<48> { static constexpr int A = 2, XS = 60; };
template <> struct FxLay<64> { static constexpr int A = 3, XS = 72; };
// line pairs per CTA (>= 96 threads)
template <int N> constexpr int zfx_pairs() { return (95 + 3 * FxPlan<N>::A::P) / (3 * FxPlan<N>::A::P); }
template <int N> constexpr int zfx_smem() { return zfx_pairs<N>() * 6 * FxLay<N>::XS * 16; }
template <int N> constexpr int zfx_threads() { return 3 * FxPlan<N>::A::P * zfx_pairs<N>(); }
constexpr int zfx_fit(int by_regs, int by_smem) { return by_regs < by_smem ? (by_regs < 1 ? 1 : by_regs) : by_smem; }
// CTAs per SM: 384 threads (168 registers each) or what the buffers allow
template <int N> constexpr int zfx_minb() { return zfx_fit(384 / zfx_threads<N>(), 227 * 1024 / (zfx_smem<N>() + 2048)); }
template <int P> struct SyncLine {   // the P threads of a line transform
    __device__ __forceinline__ void operator()() const {
        if constexpr (P <= 32) __syncwarp();
        else __syncthreads();
    }
};
// The halves of a 2^h, 0 <= h <= 28
__device__ __forceinline__ FxSplit fx_split(q64 a, int h) {
    FxSplit s;
    s.ad = (int)__funnelshift_l((unsigned)a, (unsigned)(a >> 32), h + 2);
    s.a0 = (int)((unsigned)a << h & 0x3fffffffu);
    return s;
}
// a b 2^-60 for |a|, |b| <= 2^60, from 30-bit halves (the product of the low halves would
// add less than one unit)
__device__ __forceinline__ q64 fx_product(FxSplit a, FxSplit b) {
    return madw(a.ad, b.ad, madw(a.ad, b.a0, mulw(a.a0, b.ad)) >> 30);
}
// a b - c d with shifts that bring both to one scale
__device__ __forceinline__ q64 fx_cross(FxSplit a, FxSplit b, FxSplit c, FxSplit d, int2 sh) {
    return (fx_product(a, b) >> sh.x) - (fx_product(c, d) >> sh.y);
}
// scale k of a difference of products a and b of scales ka, kb, and the shifts that bring them to it
struct FxCross {
    int k;
    int2 sh;
};
__device__ __forceinline__ FxCross fx_cross_scale(int ka, int kb) {
    const int k = min(ka, kb);
    return FxCross{k, make_int2(min(ka - k, 63), min(kb - k, 63))};
}
// scale of a spectrum (twice itself) from the scale of the products (sums of two lines' scales,
// so that a bad or zero line shows) and the real line's shift
__device__ __forceinline__ int fx_product_scale(int k, int sh) {
    return k < kFxBad / 2 ? kFxBad : k > kFxZero / 2 ? kFxZero : k - 60 - sh + 1;
}

template <int N, int MODE>
__global__ void __launch_bounds__(zfx_threads<N>(), zfx_minb<N>())
k_zfx(cx<q64>* __restrict__ W, int* __restrict__ scales, const int4* __restrict__ tw, double* __restrict__ real,
      StepDev* __restrict__ sd, int want_umax) {
    const long long dep = pdl_begin();
    W += dep;
    scales += dep;
    real += dep;
    sd += dep;
    using G = Geo<N>;
    using PL = typename FxPlan<N>::A;
    constexpr int E = PL::E, P = PL::P, ZP = zfx_pairs<N>(), XS = FxLay<N>::XS;
    constexpr int NW = P > 32 ? P / 32 : 1;    // warps per line
    constexpr int NLOW = (G::KC + P) / P;      // slots s that can hold a mode p + P s <= KC
    W += (long long)blockIdx.y * 6 * G::FS;    // ensemble member
    extern __shared__ __align__(16) unsigned char smem_raw[];
    cx<q64>* buf = reinterpret_cast<cx<q64>*>(smem_raw);   // [ZP][2 lines][3 groups][XS]
    __shared__ FxBound bound[ZP][6][NW];                    // a line's L1 norm per field
    __shared__ uint2 count[ZP][3][NW], most[ZP][3][NW];     // a real line's sums and its threads' largest (P > 32)
    __shared__ int firsts[ZP][6][NW];                       // scales of a line's first stage
    __shared__ int scale[2 * ZP][6];                        // per line: its fields' scales
    __shared__ unsigned peak[2 * ZP][3][NW];                // and a group's two peaks (leading zeros)
    __shared__ int product[2 * ZP][3];                      // and those of its products
    const int p = threadIdx.x % P;
    const int g = (threadIdx.x / P) % 3;
    const int lp = threadIdx.x / (3 * P);
    const long long la = 2 * ((long long)blockIdx.x * ZP + lp);
    const FxScales sc = fx_scales<N>(scales, blockIdx.y);
    PadIdx<FxLay<N>::A, 1> sidx;
    SyncLine<P> sync;

    constexpr bool TWO = fx_two<N>();
    int kA = 0, kB = 0;   // scales of what a group writes
    // lines a and b to real space, then the products back: one copy of the transform's code
    // (instruction fetch is a cost of these long unrolled bodies)
#pragma unroll 1
    for (int L = MODE == 2 ? 2 : 0; L < (MODE == 1 ? 2 : 3); ++L) {
        cx<q64>* sb;
        cx<q64> a[E];
        int later = 0;   // bits of the scale that come after the first stage
        if (L < 2) {
            sb = buf + ((lp * 2 + L) * 3 + g) * XS;
            const cx<q64>* A = W + (long long)(2 * g) * G::FS + (la + L) * G::NZP;
            const int* kin = sc.y + ((long long)2 * g * N + (la + L) / N) * G::NZP;
            constexpr long long kf = (long long)N * G::NZP;   // to the next field's scales
            cx<q64> ra[NLOW], rb[NLOW];
            int kea[NLOW], keb[NLOW];
#pragma unroll
            for (int s = 0; s < NLOW; ++s) {
                const int m = p + P * s;
                ra[s] = rb[s] = mk<q64>(0, 0);
                kea[s] = keb[s] = kFxZero;
                if (m <= G::KC) {
                    ra[s] = A[m];
                    rb[s] = A[G::FS + m];
                    kea[s] = kin[m];
                    keb[s] = kin[kf + m];
                    if (m == 0) ra[s].y = rb[s].y = 0;   // c2r takes the real part of the mean
                }
            }
            FxBound ba = fx_bound(ra, kea), bb = fx_bound(rb, keb);
            if constexpr (TWO) {
                // a thread's modes come once as they are and once as the conjugates in another thread's slots:
                // half of 2^60 for each of the two fields keeps its inputs' sum below 2^61
                const int fa = fx_warp_min<1, (P < 32 ? P : 32)>(fx_scale_of(ba, 2));
                const int fb = fx_warp_min<1, (P < 32 ? P : 32)>(fx_scale_of(bb, 2));
                if (p % 32 == 0) {
                    firsts[lp][2 * g][p / 32] = fa;
                    firsts[lp][2 * g + 1][p / 32] = fb;
                }
            }
            fx_warp_bound<1, (P < 32 ? P : 32)>(ba);
            fx_warp_bound<1, (P < 32 ? P : 32)>(bb);
            if (p % 32 == 0) {
                bound[lp][2 * g][p / 32] = ba;
                bound[lp][2 * g + 1][p / 32] = bb;
            }
            __syncthreads();
            // a scale for each field, so that a component far below the others keeps its bits: every
            // mode but the mean counts twice (its conjugate), so its modes sum to half of 2^60
            int kfield[2];
#pragma unroll
            for (int h = 0; h < 2; ++h) {
                FxBound b = bound[lp][2 * g + h][0];
#pragma unroll
                for (int w = 1; w < NW; ++w) b = fx_join(b, bound[lp][2 * g + h][w]);
                kfield[h] = fx_scale_of(b, 2);
                if (p == 0) scale[2 * lp + L][2 * g + h] = kfield[h];
            }
            if constexpr (TWO) {
                // the two fields share the transform, so the shift as well
                later = 31;
#pragma unroll
                for (int h = 0; h < 2; ++h) {
                    int f = firsts[lp][2 * g + h][0];
#pragma unroll
                    for (int w = 1; w < NW; ++w) f = min(f, firsts[lp][2 * g + h][w]);
                    if (kfield[h] != kFxZero) later = min(later, fx_later<TWO>(f, kfield[h]));
                }
            }
            const int ka = kfield[0] + later, kb = kfield[1] + later;
            if (MODE == 1) {
                kA = kfield[0];
                kB = kfield[1];
            }
#pragma unroll
            for (int s = 0; s < E; ++s) a[s] = mk<q64>(0, 0);
#pragma unroll
            for (int s = 0; s < NLOW; ++s) {
                const int m = p + P * s;
                const cx<q64> va = fx_align(ra[s], kea[s], ka), vb = fx_align(rb[s], keb[s], kb);
                // a + i b at m, conj(a) + i conj(b) at N - m, real and imaginary parts exchanged (inverse)
                a[s] = mk<q64>(va.y + vb.x, va.x - vb.y);
                if (m > 0 && m <= G::KC) sb[sidx(N - m)] = mk<q64>(vb.x - va.y, va.x + vb.y);
            }
            sync();
#pragma unroll
            for (int s = 0; s < E; ++s)
                if (P * s + P - 1 >= N - G::KC && p + P * s >= N - G::KC) a[s] = sb[sidx(p + P * s)];
            sync();
        } else {
            // forward: group 0 -> line a (Nx + i Ny), 1 -> line b, 2 -> Nz_a + i Nz_b
            cx<q64>* ba = buf + lp * 6 * XS;   // line a's buffers; line b's 3 XS further
            sb = g == 0 ? ba : g == 1 ? ba + 3 * XS : ba + XS;
            if constexpr (MODE == 0) {
                // u x w: (ux, uy), (uz, wx), (wy, wz) -> (Nx, Ny), (Nz, -); 3 P / 2 threads per line
                constexpr int NL = 3 * P / 2;
                static_assert(P % 2 == 0 && (E % 2 == 0 || !zfx_peaks<N>()), "whole threads per line, elements in pairs");
                const int line = threadIdx.x / NL;   // of the CTA's 2 ZP
                int h[6], k[6];   // bits to a field's peak, and its scale with them
#pragma unroll
                for (int f = 0; f < 6; ++f) {
                    h[f] = 0;
                    if constexpr (zfx_peaks<N>()) {
                        unsigned t = peak[line][f / 2][0];
#pragma unroll
                        for (int w = 1; w < NW; ++w) t = __vimin3_u16x2(t, t, peak[line][f / 2][w]);
                        h[f] = max((int)(f % 2 ? t >> 16 : t & 0xffffu) - 4, 0);   // values below 2^60
                    }
                    k[f] = scale[line][f] + h[f];
                }
                const FxCross cn = fx_cross_scale(k[1] + k[5], k[2] + k[4]), cy = fx_cross_scale(k[2] + k[3], k[0] + k[5]),
                              cz = fx_cross_scale(k[0] + k[4], k[1] + k[3]);
                if (threadIdx.x % NL == 0) {
                    product[line][0] = cn.k;
                    product[line][1] = cy.k;
                    product[line][2] = cz.k;
                }
                const int kx = scale[line][0], ky = scale[line][1], kz = scale[line][2], ku = min(kx, min(ky, kz));
                const int sx = min(kx - ku, 63), sy = min(ky - ku, 63), sz = min(kz - ku, 63);
                q64 top = 0;   // the largest |ux| + |uy| + |uz|
                for (int n = threadIdx.x % NL; n < N; n += NL) {
                    cx<q64>* r = buf + line * 3 * XS + sidx(n);
                    const cx<q64> v1 = r[0], v2 = r[XS], v3 = r[2 * XS];
                    const FxSplit ux = fx_split(v1.x, h[0]), uy = fx_split(v1.y, h[1]), uz = fx_split(v2.x, h[2]);
                    const FxSplit wx = fx_split(v2.y, h[3]), wy = fx_split(v3.x, h[4]), wz = fx_split(v3.y, h[5]);
                    r[0] = mk<q64>(fx_cross(uy, wz, uz, wy, cn.sh), fx_cross(uz, wx, ux, wz, cy.sh));
                    r[XS].x = fx_cross(ux, wy, uy, wx, cz.sh);
                    if (want_umax) {
                        const q64 sp = (llabs(v1.x) >> sx) + (llabs(v1.y) >> sy) + (llabs(v2.x) >> sz);
                        top = sp > top ? sp : top;
                    }
                }
                if (want_umax) {
                    double um = fx_to_any(top, ku);
#pragma unroll
                    for (int o = 16; o > 0; o >>= 1) um = fmax(um, __shfl_xor_sync(0xffffffffu, um, o));
                    if ((threadIdx.x & 31) == 0) Bits<double>::amax(&sd[blockIdx.y].umax_bits, um);
                }
                __syncthreads();

                unsigned hx = 0u, hy = 0u;
#pragma unroll
                for (int s = 0; s < E; ++s) {
                    a[s] = sb[sidx(p + P * s)];
                    if (g == 2) a[s].y = sb[3 * XS + sidx(p + P * s)].x;
                    hx += ((unsigned)abs((int)(a[s].x >> 32)) >> 10) + 1u;
                    hy += ((unsigned)abs((int)(a[s].y >> 32)) >> 10) + 1u;
                }
                unsigned mx = hx, my = hy;
                // |x| < 2^42 per count: a shift of the bit length over 18 bounds the line's sum by 2^60
#pragma unroll
                for (int o = 1; o < (P < 32 ? P : 32); o <<= 1) {
                    hx += __shfl_xor_sync(0xffffffffu, hx, o);
                    hy += __shfl_xor_sync(0xffffffffu, hy, o);
                    if constexpr (TWO) {
                        mx = max(mx, __shfl_xor_sync(0xffffffffu, mx, o));
                        my = max(my, __shfl_xor_sync(0xffffffffu, my, o));
                    }
                }
                if constexpr (NW > 1) {
                    if (p % 32 == 0) {
                        count[lp][g][p / 32] = make_uint2(hx, hy);
                        most[lp][g][p / 32] = make_uint2(mx, my);
                    }
                    __syncthreads();
                    hx = hy = 0u;
#pragma unroll
                    for (int w = 0; w < NW; ++w) {
                        hx += count[lp][g][w].x;
                        hy += count[lp][g][w].y;
                        mx = max(mx, most[lp][g][w].x);
                        my = max(my, most[lp][g][w].y);
                    }
                }
                const int shx = max(0, 14 - __clz(hx)), shy = max(0, 14 - __clz(hy));
                if constexpr (TWO) later = min(shx - max(0, 14 - __clz(mx)), shy - max(0, 14 - __clz(my)));
                const int s0x = shx - later, s0y = shy - later;
                const q64 rx = (1ll << s0x) >> 1, ry = (1ll << s0y) >> 1;
#pragma unroll
                for (int s = 0; s < E; ++s) a[s] = mk<q64>((a[s].x + rx) >> s0x, (a[s].y + ry) >> s0y);
                // the spectra's scales (one more for the halves)
                kA = fx_product_scale(product[2 * lp + (g == 1 ? 1 : 0)][g == 2 ? 2 : 0], shx);
                kB = fx_product_scale(product[2 * lp + (g == 0 ? 0 : 1)][g == 2 ? 2 : 1], shy);
            } else {
                constexpr long long kReal = (long long)N * N * N;
                const double* r0 = real + (g == 2 ? 2 * kReal : 0) + (g == 1 ? la + 1 : la) * N;
                const double* r1 = real + (g == 2 ? 2 * kReal : kReal) + (g == 0 ? la : la + 1) * N;
                cx<double> v[E];
#pragma unroll
                for (int s = 0; s < E; ++s) v[s] = mk(r0[p + P * s], r1[p + P * s]);
                FxBound b = fx_bound(v);
                int first = TWO ? fx_warp_min<1, (P < 32 ? P : 32)>(fx_scale_in(b, 1)) : 0;
                fx_warp_bound<1, (P < 32 ? P : 32)>(b);
                if constexpr (NW > 1) {
                    if (p % 32 == 0) {
                        bound[lp][g][p / 32] = b;
                        firsts[lp][g][p / 32] = first;
                    }
                    __syncthreads();
                    b = bound[lp][g][0];
                    first = min(firsts[lp][g][0], firsts[lp][g][1]);
#pragma unroll
                    for (int w = 1; w < NW; ++w) b = fx_join(b, bound[lp][g][w]);
                }
                static_assert(NW <= 2, "two warps' firsts");
                const int k = fx_scale_in(b, 1);
                later = fx_later<TWO>(first, k);
#pragma unroll
                for (int s = 0; s < E; ++s) a[s] = mk<q64>(fx_from(v[s].x, k + later), fx_from(v[s].y, k + later));
                kA = kB = k == kFxZero || k == kFxBad ? k : k + 1;
            }
            sync();
        }
        PL::template fwd<fx_round<N>()>(a, sb, p, tw, sidx, sync, fx_mid<N>(later));
        if (L < 2 && MODE == 0) {
#pragma unroll
            for (int s = 0; s < E; ++s) sb[sidx(p + P * s)] = mk<q64>(a[s].y, a[s].x);
            if constexpr (zfx_peaks<N>()) {
                int hia = 0, hib = 0, loa = -1, lob = -1;
#pragma unroll
                for (int s = 0; s < E; s += 2) {
                    const int ha = (int)(a[s].y >> 32), hb = (int)(a[s].x >> 32);
                    const int ga = (int)(a[s + 1].y >> 32), gb = (int)(a[s + 1].x >> 32);
                    hia = __vimax3_s32(hia, ha, ga);
                    loa = __vimin3_s32(loa, ha, ga);
                    hib = __vimax3_s32(hib, hb, gb);
                    lob = __vimin3_s32(lob, hb, gb);
                }
                unsigned zeros = __clz(max(hia, ~loa)) | __clz(max(hib, ~lob)) << 16;
#pragma unroll
                for (int o = 1; o < (P < 32 ? P : 32); o <<= 1)
                    zeros = __vimin3_u16x2(zeros, zeros, __shfl_xor_sync(0xffffffffu, zeros, o));
                if (p % 32 == 0) peak[2 * lp + L][g][p / 32] = zeros;
            }
            // the line's real space is complete, and its bounds are read
            __syncthreads();
        } else if (L < 2) {
            double* r = real + (long long)2 * g * N * N * N + (la + L) * N;
#pragma unroll
            for (int s = 0; s < E; ++s) {
                r[p + P * s] = fx_to_any(a[s].y, kA);
                r[(long long)N * N * N + p + P * s] = fx_to_any(a[s].x, kB);
            }
            __syncthreads();
        } else {
#pragma unroll
            for (int s = 0; s < E; ++s)   // only the slots read below: N - m
                if (P * s + P - 1 >= N - G::KC || s == 0) sb[sidx(p + P * s)] = a[s];
            sync();
            const int fA = g == 2 ? 2 : 0, fB = g == 2 ? 2 : 1;
            const long long lA = g == 1 ? la + 1 : la, lB = g == 0 ? la : la + 1;
            cx<q64>* outA = W + fA * G::FS + lA * G::NZP;
            cx<q64>* outB = W + fB * G::FS + lB * G::NZP;
            if (p == 0) {
                sc.z[(long long)fA * N * N + lA] = kA;
                sc.z[(long long)fB * N * N + lB] = kB;
            }
#pragma unroll
            for (int s = 0; s < NLOW; ++s) {
                const int m = p + P * s;
                if (m <= G::KC) {
                    const cx<q64> zm = a[s], zc = sb[sidx(m == 0 ? 0 : N - m)];
                    outA[m] = mk<q64>(zm.x + zc.x, zm.y - zc.y);
                    outB[m] = mk<q64>(zm.y + zc.y, zc.x - zm.x);
                }
            }
        }
    }
}

}  // namespace ns3d
