// fx_passes.cuh — the x and z passes of the FP64 engines, on the 64-bit integer
// line transforms of fxfft.cuh (the y passes are k_ypass with line_fft). Layouts and
// launch grids are those of the FP32 passes in ns3d_kernels.cuh.
#pragma once
#include "ns3d_kernels.cuh"

namespace ns3d {

// ---------------------------------------------------------------------------
// x passes: the z lines' plan (16 elements per thread where N allows, one or two
// exchanges), fx_tile pencils per CTA. `aux` holds 1/k2 for k2 <= KC^2 (0 at 0) and
// then the N wavenumbers of the x rows, so that no mode pays an FP64 division or
// conversion.
// ---------------------------------------------------------------------------
template <int N> constexpr int fxinv_threads() { return fx_tile<N>() * Plans<N>::A::P; }
template <int N> constexpr int fxfwd_threads() { return 3 * fx_tile<N, true>() * Plans<N>::A::P; }
constexpr int fx_log2(int n) { return n <= 1 ? 0 : 1 + fx_log2(n / 2); }
constexpr int fx_ctas(int per_sm, int threads) { return per_sm / threads < 1 ? 1 : per_sm / threads; }
template <int N> constexpr int fxinv_smem() { return N * fx_tile<N>() * 16; }
template <int N> constexpr int fxfwd_smem() { return 3 * N * fx_tile<N, true>() * 16; }

// P1: one field of u, w = i k x u of one tile per CTA (blockIdx.z = 6 member + field).
// The curl is formed on the modes of the sphere (a third of a column's rows), where the
// FP64 pipe has to do less than for the transformed columns, and the six fields are
// independent CTAs, which fills the chip at small N (32^3: 11 us per launch, 27 us with
// the six transforms in one CTA; 256^3: 0.19 against 0.25 ms). The inputs' second and
// third reads hit L2.
template <int N>
__global__ void __launch_bounds__(fxinv_threads<N>(), fx_ctas(512, fxinv_threads<N>()))
k_xinv_fx(const cx<double>* __restrict__ U, cx<double>* __restrict__ W, const cx<double>* __restrict__ tw,
          const double* __restrict__ aux) {
    const long long dep = pdl_begin();
    U += dep;
    W += dep;
    using G = Geo<N>;
    using PL = typename Plans<N>::A;
    constexpr int TT = fx_tile<N>(), E = PL::E, P = PL::P, NT = TT * P;
    constexpr bool kPow2 = (N & (N - 1)) == 0;
    extern __shared__ __align__(16) unsigned char smem_raw[];
    cx<double>* sbuf = reinterpret_cast<cx<double>*>(smem_raw);
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
    // 1/N^3 of a power of two goes into the exponent
    line_fft<PL, true, false, TT, NT>(v, sbuf, p, tw, sidx, sync, kPow2 ? 3 * fx_log2(N) : 0);
    if (rem >= 0) {
#pragma unroll
        for (int s = 0; s < E; ++s) W[off + (long long)(p + P * s) * xs] = v[s];
    }
}

// P5: three groups of threads transform one component each, leave the rows of the band in
// their exchange buffers, and all threads share the modes of the tile for the stage
// algebra. The mode loop's FP64 work is a large part (FP64 pipe 44 % busy at 256^3 with the
// division and conversions it had), so 1/k2 comes from `aux` and the per-step factors are
// formed once per thread. Three groups instead of one after the other: 24 -> 14 us per
// launch at 32^3, 0.226 -> 0.212 ms at 256^3.
template <int N, int INTEG, int MODE>
__global__ void __launch_bounds__(fxfwd_threads<N>(), fx_ctas(384, fxfwd_threads<N>()))
k_xfwd_fx(const cx<double>* __restrict__ W, cx<double>* __restrict__ U, cx<double>* __restrict__ UT,
          cx<double>* __restrict__ ACC, const cx<double>* __restrict__ tw, const StepDev* __restrict__ sd,
          const cx<double>* __restrict__ tab, const double* __restrict__ aux, cx<double>* __restrict__ K,
          double* __restrict__ dpart, const RkStage rs) {
    const long long dep = pdl_begin();
    W += dep;
    U += dep;
    UT += dep;
    ACC += dep;
    sd += dep;
    tab += dep;
    K += dep;
    dpart += dep;
    using G = Geo<N>;
    using PL = typename Plans<N>::A;
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
    {
        const int kz = kz0 + t;
        const bool colok = kz <= G::KC && ky * ky + kz * kz <= G::KC2;
        const C* src = W + g * G::FS + (long long)j * G::NZP + kz;
        C v[E];
#pragma unroll
        for (int s = 0; s < E; ++s) v[s] = colok ? src[(long long)(p + P * s) * xs] : czero<double>();
        // the state rows of this tile into L2 (the groups share the rows)
        if (g == 0) xfwd_prefetch_state<double, N, INTEG, MODE, E, P, TT>(U, ACC, K, rs, p, t, ky, kz0, j);
        StridedIdx<TT, PL::R1> sidx{t};
        if constexpr (NG % 32 == 0) {
            const SyncGroup sync{1 + g, NG};
            line_fft<PL, false, false, TT, NT>(v, sbuf, p, tw, sidx, sync);
        } else {
            line_fft<PL, false, false, TT, NT>(v, sbuf, p, tw, sidx, SyncBlock());
        }
#pragma unroll
        for (int s = 0; s < E; ++s)
            if (!(P * s > G::KC && P * s + P - 1 < N - G::KC)) sbuf[(p + P * s) * TT + t] = v[s];
    }
    __syncthreads();

    const double* kxs = aux + G::KC2 + 1;
    const double fky = ky;
    const double h = MODE <= X_STAGE4 ? sd->dt : 0.0;
    const double h2 = 0.5 * h, h3 = h * (1.0 / 3.0), h6 = h * (1.0 / 6.0);
    double es[3] = {0.0, 0.0, 0.0};   // DP5CN error partial sums
    // rows |kx| <= KC of the tile, NT / TT rows at a time (NT is a multiple of TT)
    const int kz = kz0 + t, kp2 = ky * ky + kz * kz;
    const double fkz = kz;
#pragma unroll 2
    for (int r = threadIdx.x / TT; r < 2 * G::KC + 1; r += NT / TT) {
        const int kx = r - G::KC, i = kx < 0 ? kx + N : kx;
        const int k2 = kx * kx + kp2;
        if (kz > G::KC || k2 > G::KC2) continue;
        const long long idx = (long long)i * xs + (long long)j * G::NZP + kz;
        C n[3];
#pragma unroll
        for (int c = 0; c < 3; ++c) n[c] = buf[(c * N + i) * TT + t];
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
                const C u = U[q];
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
                    const C u = U[q];
                    UT[q] = (u + n[c] * h2) * Eh;
                    ACC[q] = (u + n[c] * h6) * Ef;
                } else if (MODE == X_STAGE4) {
                    U[q] = ACC[q] + n[c] * h6;
                } else {
                    UT[q] = U[q] * (MODE == X_STAGE2 ? Eh : Ef) + n[c] * cu;
                    ACC[q] = ACC[q] + n[c] * ca;
                }
            }
        } else {
#pragma unroll
            for (int c = 0; c < 3; ++c) {
                const long long q = c * G::FS + idx;
                if (MODE == X_STAGE4) {
                    const C ab = ldg(&tab[k2]);
                    U[q] = U[q] * ab.x + (ACC[q] + n[c] * (1.0 / 6.0)) * ab.y;
                } else {
                    UT[q] = U[q] + n[c] * (MODE == X_STAGE3 ? h : h2);
                    ACC[q] = MODE == X_STAGE1 ? n[c] * (1.0 / 6.0) : ACC[q] + n[c] * (1.0 / 3.0);
                }
            }
        }
    }
    if constexpr (INTEG == INT_TAB) {
        if (rs.kind == 2) dp_block_sum<NT>(es, dpart);
    }
}

// ---------------------------------------------------------------------------
// P3 for FP64 (fxfft.cuh): the whole line stays in 64-bit integers between the
// load and the store. A CTA takes ZP pairs of adjacent lines; three groups of P
// threads own one complex transform each. Per line the velocity and the vorticity
// get one scale each (2^60 bounds the L1 norm of every component), group g turns
// fields 2g, 2g+1 into real space, the threads form u x w >> 60 from the 32-bit
// halves, and the groups transform (Nx, Ny) of both lines and (Nz_a, Nz_b) back,
// every real line with a shift of its own that bounds its L1 norm by 2^60. The
// transforms exchange through the group's own third of the line's buffer, which
// then holds its real-space output, so 96 bytes of shared memory per grid point of
// a pair are enough for four 96-thread CTAs per SM; where a group lies inside a
// warp it synchronises with its warp only. 1.24 -> 0.60 ms per launch at 256^3 against
// the CTA-synchronous pass with transforms that convert at both ends and FP64 products;
// issue bound (49 % of slots, instruction fetch the largest stall: CTAs of 192 and 384
// threads, whose warps run in step, measured 0.64 and 0.73 ms).
// ---------------------------------------------------------------------------
// line pairs per CTA (>= 96 threads)
template <int N> constexpr int zfx_pairs() { return (95 + 3 * Plans<N>::A::P) / (3 * Plans<N>::A::P); }
template <int N> constexpr int zfx_smem() { return zfx_pairs<N>() * 6 * zpad<N>() * 16; }
template <int N> constexpr int zfx_threads() { return 3 * Plans<N>::A::P * zfx_pairs<N>(); }
constexpr int zfx_fit(int by_regs, int by_smem) { return by_regs < by_smem ? (by_regs < 1 ? 1 : by_regs) : by_smem; }
// CTAs per SM: 384 threads (168 registers each) or what the buffers allow
template <int N> constexpr int zfx_minb() { return zfx_fit(384 / zfx_threads<N>(), 227 * 1024 / (zfx_smem<N>() + 2048)); }
template <int P> struct SyncLine {   // the P threads of a line transform
    __device__ __forceinline__ void operator()() const {
        if constexpr (P <= 32) __syncwarp();
        else __syncthreads();
    }
};
// (a b - c d) >> 60 for |a|, |b|, |c|, |d| < 2^60, from 31-bit halves (the products of
// the low halves are below the last bits kept); a4 = 4 a.ad, c4 = 4 c.ad
__device__ __forceinline__ q64 fx_cross(FxSplit a, int a4, FxSplit b, FxSplit c, int c4, FxSplit d) {
    const q64 mid = madw(a.ad, b.a0, mulw(a.a0, b.ad)) - madw(c.ad, d.a0, mulw(c.a0, d.ad));
    return madw(a4, b.ad, mid >> 29) - mulw(c4, d.ad);
}

template <int N>
__global__ void __launch_bounds__(zfx_threads<N>(), zfx_minb<N>())
k_zfx(cx<double>* __restrict__ W, const cx<double>* __restrict__ tw, StepDev* __restrict__ sd, int want_umax) {
    const long long dep = pdl_begin();
    W += dep;
    sd += dep;
    using G = Geo<N>;
    using PL = typename Plans<N>::A;
    constexpr int E = PL::E, P = PL::P, ZP = zfx_pairs<N>(), XS = zpad<N>();
    constexpr int NW = P > 32 ? P / 32 : 1;    // warps per line
    constexpr int NLOW = (G::KC + P) / P;      // slots s that can hold a mode p + P s <= KC
    W += (long long)blockIdx.y * 6 * G::FS;    // ensemble member
    extern __shared__ __align__(16) unsigned char smem_raw[];
    cx<q64>* buf = reinterpret_cast<cx<q64>*>(smem_raw);   // [ZP][2 lines][3 groups][XS]
    __shared__ FxBound bound[ZP][6][NW];                    // a line's L1 norm per field
    __shared__ uint2 count[ZP][3][NW];                      // a real line's sums (P > 32)
    __shared__ int2 scale[ZP][2];                           // per line: ku, kw (bad lines: ku = kBad)
    constexpr int kBad = 1 << 20;
    const int p = threadIdx.x % P;
    const int g = (threadIdx.x / P) % 3;
    const int lp = threadIdx.x / (3 * P);
    const long long la = 2 * ((long long)blockIdx.x * ZP + lp);
    const int4* twq = reinterpret_cast<const int4*>(tw);
    PaddedIdx sidx;
    SyncLine<P> sync;

    int shx = 0, shy = 0;
    // lines a and b to real space, then the products back: one copy of the transform's code
    // (instruction fetch is a cost of these long unrolled bodies)
#pragma unroll 1
    for (int L = 0; L < 3; ++L) {
        cx<q64>* sb;
        cx<q64> a[E];
        if (L < 2) {
            sb = buf + ((lp * 2 + L) * 3 + g) * XS;
            const cx<double>* A = W + (long long)(2 * g) * G::FS + (la + L) * G::NZP;
            const cx<double>* B = A + G::FS;
            cx<double> ra[NLOW], rb[NLOW];
#pragma unroll
            for (int s = 0; s < NLOW; ++s) {
                const int m = p + P * s;
                ra[s] = rb[s] = czero<double>();
                if (m <= G::KC) {
                    ra[s] = A[m];
                    rb[s] = B[m];
                    if (m == 0) ra[s].y = rb[s].y = 0.0;   // c2r takes the real part of the mean
                }
            }
            FxBound ba = fx_bound(ra), bb = fx_bound(rb);
            fx_warp_bound<1, (P < 32 ? P : 32)>(ba, 0xffffffffu);
            fx_warp_bound<1, (P < 32 ? P : 32)>(bb, 0xffffffffu);
            if (p % 32 == 0) {
                bound[lp][2 * g][p / 32] = ba;
                bound[lp][2 * g + 1][p / 32] = bb;
            }
            __syncthreads();
            // the scales: every mode but the mean counts twice (its conjugate), so half of 2^60 per component
            int kk[2];
            bool bad = false;
#pragma unroll
            for (int h = 0; h < 2; ++h) {
                int e = -4096;
#pragma unroll
                for (int c = 0; c < 3; ++c) {
                    FxBound b = bound[lp][3 * h + c][0];
#pragma unroll
                    for (int w = 1; w < NW; ++w) b = fx_join(b, bound[lp][3 * h + c][w]);
                    e = max(e, fx_exponent(b));
                }
                const FxScale sc = fx_scale(e);
                kk[h] = sc.k;
                bad = bad || sc.bad;
            }
            const int ku = kk[0] - 2, kw = kk[1] - 2;
            if (p == 0 && g == 0) scale[lp][L] = make_int2(bad ? kBad : ku, kw);
            const int ka = g < 2 ? ku : kw, kb = g < 1 ? ku : kw;
#pragma unroll
            for (int s = 0; s < E; ++s) a[s] = mk<q64>(0, 0);
#pragma unroll
            for (int s = 0; s < NLOW; ++s) {
                const int m = p + P * s;
                const q64 ax = fx_from(ra[s].x, ka), ay = fx_from(ra[s].y, ka);
                const q64 bx = fx_from(rb[s].x, kb), by = fx_from(rb[s].y, kb);
                // a + i b at m, conj(a) + i conj(b) at N - m, real and imaginary parts exchanged (inverse)
                a[s] = mk<q64>(ay + bx, ax - by);
                if (m > 0 && m <= G::KC) sb[sidx(N - m)] = mk<q64>(bx - ay, ax + by);
            }
            sync();
#pragma unroll
            for (int s = 0; s < E; ++s)
                if (P * s + P - 1 >= N - G::KC && p + P * s >= N - G::KC) a[s] = sb[sidx(p + P * s)];
            sync();
        } else {
            // u x w: (ux, uy), (uz, wx), (wy, wz) -> (Nx, Ny), (Nz, -)
            double um = 0.0;
            for (int idx = threadIdx.x; idx < ZP * 2 * N; idx += 3 * P * ZP) {
                const int line = idx / N, n = idx % N;   // line = pair 2 + L
                cx<q64>* r = buf + line * 3 * XS + sidx(n);
                const cx<q64> v1 = r[0], v2 = r[XS], v3 = r[2 * XS];
                const FxSplit ux = fx_split(v1.x), uy = fx_split(v1.y), uz = fx_split(v2.x);
                const FxSplit wx = fx_split(v2.y), wy = fx_split(v3.x), wz = fx_split(v3.y);
                const int ux4 = 4 * ux.ad, uy4 = 4 * uy.ad, uz4 = 4 * uz.ad;
                r[0] = mk<q64>(fx_cross(uy, uy4, wz, uz, uz4, wy), fx_cross(uz, uz4, wx, ux, ux4, wz));
                r[XS].x = fx_cross(ux, ux4, wy, uy, uy4, wx);
                if (want_umax) {
                    const int ku = scale[line / 2][line % 2].x;
                    const q64 sp = llabs(v1.x) + llabs(v1.y) + llabs(v2.x);
                    // lines of tiny values were taken as zero (ku far below the exponent range)
                    if (ku > -2000 && ku < kBad) um = fmax(um, fx_to(sp, ku));
                }
            }
            if (want_umax) {
#pragma unroll
                for (int o = 16; o > 0; o >>= 1) um = fmax(um, __shfl_xor_sync(0xffffffffu, um, o));
                if ((threadIdx.x & 31) == 0) Bits<double>::amax(&sd[blockIdx.y].umax_bits, um);
            }
            __syncthreads();

            // forward: group 0 -> line a (Nx + i Ny), 1 -> line b, 2 -> Nz_a + i Nz_b
            cx<q64>* ba = buf + lp * 6 * XS;   // line a's buffers; line b's 3 XS further
            sb = g == 0 ? ba : g == 1 ? ba + 3 * XS : ba + XS;
            unsigned hx = 0u, hy = 0u;
#pragma unroll
            for (int s = 0; s < E; ++s) {
                a[s] = sb[sidx(p + P * s)];
                if (g == 2) a[s].y = sb[3 * XS + sidx(p + P * s)].x;
                hx += ((unsigned)abs((int)(a[s].x >> 32)) >> 10) + 1u;
                hy += ((unsigned)abs((int)(a[s].y >> 32)) >> 10) + 1u;
            }
            // |x| < 2^42 per count: a shift of the bit length over 18 bounds the line's sum by 2^60
#pragma unroll
            for (int o = 1; o < (P < 32 ? P : 32); o <<= 1) {
                hx += __shfl_xor_sync(0xffffffffu, hx, o);
                hy += __shfl_xor_sync(0xffffffffu, hy, o);
            }
            if constexpr (NW > 1) {
                if (p % 32 == 0) count[lp][g][p / 32] = make_uint2(hx, hy);
                __syncthreads();
                hx = hy = 0u;
#pragma unroll
                for (int w = 0; w < NW; ++w) {
                    hx += count[lp][g][w].x;
                    hy += count[lp][g][w].y;
                }
            }
            shx = max(0, 14 - __clz(hx));
            shy = max(0, 14 - __clz(hy));
            const q64 rx = (1ll << shx) >> 1, ry = (1ll << shy) >> 1;
#pragma unroll
            for (int s = 0; s < E; ++s) a[s] = mk<q64>((a[s].x + rx) >> shx, (a[s].y + ry) >> shy);
            sync();
        }
        PL::template fwd<false>(a, sb, p, twq, sidx, sync);
        if (L < 2) {
#pragma unroll
            for (int s = 0; s < E; ++s) sb[sidx(p + P * s)] = mk<q64>(a[s].y, a[s].x);
            // the line's real space is complete, and its bounds are read
            __syncthreads();
        } else {
#pragma unroll
            for (int s = 0; s < E; ++s)   // only the slots read below: N - m
                if (P * s + P - 1 >= N - G::KC || s == 0) sb[sidx(p + P * s)] = a[s];
            sync();
            const int2 s0 = scale[lp][g == 1 ? 1 : 0], s1 = scale[lp][g == 0 ? 0 : 1];   // of the two outputs' lines
            cx<double>* outA = W + (g == 2 ? 2 * G::FS : 0) + (g == 1 ? la + 1 : la) * G::NZP;
            cx<double>* outB = W + (g == 2 ? 2 * G::FS : G::FS) + (g == 0 ? la : la + 1) * G::NZP;
            // the spectra's scales (one more for the halves); out of the exponent range: zero below
            // (and for lines taken as zero), NaN above
            const int kA = s0.x + s0.y - 60 - shx + 1, kB = s1.x + s1.y - 60 - shy + 1;
            const bool tinyA = kA > 1020 || min(s0.x, s0.y) < -2000, tinyB = kB > 1020 || min(s1.x, s1.y) < -2000;
            const bool bad = s0.x == kBad || s1.x == kBad || (!tinyA && kA < -900) || (!tinyB && kB < -900);
#pragma unroll
            for (int s = 0; s < NLOW; ++s) {
                const int m = p + P * s;
                if (m <= G::KC) {
                    const cx<q64> zm = a[s], zc = sb[sidx(m == 0 ? 0 : N - m)];
                    cx<double> oa = mk(fx_to(zm.x + zc.x, kA), fx_to(zm.y - zc.y, kA));
                    cx<double> ob = mk(fx_to(zm.y + zc.y, kB), fx_to(zc.x - zm.x, kB));
                    if (tinyA) oa = czero<double>();
                    if (tinyB) ob = czero<double>();
                    if (bad) oa = ob = mk(__hiloint2double(0x7ff80000, 0), __hiloint2double(0x7ff80000, 0));
                    outA[m] = oa;
                    outB[m] = ob;
                }
            }
        }
    }
}

}  // namespace ns3d
