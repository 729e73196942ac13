// fftb_line.cuh -- the single-axis line kernel: one launch transforms the lines of one axis.
//
// Bound: memory.  A pass reads every line once and writes it once, so the kernel keeps a line in
// registers from its load to its store: the first butterfly's points come straight from global
// memory into the registers that transform them, the last butterfly's results are stored
// straight from registers, and shared memory carries only the exchanges between the stages
// (S - 1 of them; up to 4096 points S is at most five, and two or three for most lengths).  Every thread issues all of its line's loads before it
// waits for the first, which is what keeps enough bytes in flight.  Per launch, bytes read and
// written over the time on a B200, this kernel and the pass kernel it replaced (fftb_pass.cuh: all
// points through shared memory before and after the transform): 512^3 f32 R2C 172 us = 6.2 TB/s
// (406 us), x or y C2C 215 us = 5.0 TB/s (533 us), x sandwich 305 us (1118 us); 256^3 f64 C2C
// 51-53 us = 5.1-5.3 TB/s (74-82 us); 192^3 f32 C2C 16.4 us (30.7 us).
//
// Lines are n = r_0 r_1 ... points (Stockham order: Govindaraju et al., "High performance
// discrete Fourier transforms on graphics processors", SC 2008); the plan takes the fewest
// stages of radices up to 16 (float lines above 256 points: two of up to 32, line_plan) and, of those,
// the most even ones, so a stage's n / r_i butterflies
// fill the line's T threads.
//
// Two thread mappings: ROW (the points of a line are neighbours in memory: consecutive threads
// take consecutive points) and COL (the lines are: consecutive threads take the same point of
// consecutive lines, and a line group's rows are contiguous segments).  A pass whose input or
// output side has the other order stages that side through shared memory (in_t / out_t).
//
// The inverse transform is the forward one with its results stored in reverse order (X_inv[p] =
// X_fwd[-p mod n]), so one copy of the butterflies serves both directions.  The sandwich runs the
// second transform with the radices reversed: its first stage then takes its points where the
// last stage of the forward one left them, in the registers of the same thread.
#pragma once

#include "fftb_device.cuh"
#include "fftb_internal.h"

namespace fftb {

// ---------------------------------------------------------------- plan
struct LinePlan {
    int S = 1;                 // stages
    int r[5] = {1, 1, 1, 1, 1};  // radices, descending
    int T = 1;                 // threads per line
    int E = 1;                 // complex values a thread holds
};

__host__ __device__ constexpr bool line_radix_ok(int r)
{
    return (r >= 2 && r <= 16) || r == 18 || r == 20 || r == 24 || r == 25 || r == 30 || r == 32;
}

// The most even factorisation of n into S radices (descending): minimal largest radix, then
// maximal smallest, none above top.  false if there is none.
__host__ __device__ constexpr bool line_factor(int n, int S, int top, int *out)
{
    if (S == 1) {
        if (!line_radix_ok(n) || n > top) return false;
        out[0] = n;
        return true;
    }
    int best[5] = {};
    bool have = false;
    for (int r = top; r >= 2; --r) {
        if (n % r || !line_radix_ok(r)) continue;
        int rest[5] = {};
        if (!line_factor(n / r, S - 1, r, rest)) continue;
        // largest radix r falls with the loop, so the last hit has the smallest largest radix;
        // the recursion has already made the rest as even as it can be
        best[0] = r;
        for (int i = 0; i + 1 < S; ++i) best[i + 1] = rest[i];
        have = true;
    }
    for (int i = 0; i < S; ++i) out[i] = best[i];
    return have;
}

// (The chirp-z pass, two transforms of at least 2 n points, took 5 to 16 times as long on lengths
// such as 150, 180 and 1000, which now have a plan.)
//
// ROW lines split every composite length (a thread per line would read its points one line
// apart) and take the larger of equally good thread counts; COL lines the smaller.
// emax bounds the values a thread holds.  top: the largest radix of a two-stage plan above 256 points.
// In float up to 32 (64 registers of values, 16 warps per SM): a third stage costs another
// exchange and set of twiddles, and these kernels are bound by issue and shared-memory
// wavefronts: 512-point columns of 512^3 241 -> 218 us and their sandwich 369 -> 316 (16 x 32 for
// 8 x 8 x 8), 400-point columns 311 -> 247 (20 x 20), 480-point sandwich 303 -> 246, 320-point rows
// 168 -> 138.  In double 32 values would take 128 registers: three stages.
__host__ __device__ constexpr LinePlan line_plan(int n, bool row, int emax, int top)
{
    LinePlan p;
    if (n <= 1) return p;
    bool have = false;
    for (int S = 1; S <= 5 && !have; ++S) {
        if (S == 1 && row && n > 3) {
            bool prime = true;
            for (int d = 2; d * d <= n; ++d)
                if (n % d == 0) prime = false;
            if (!prime) continue;
        }
        int r[5] = {};
        if (line_factor(n, S, S == 2 && n > 256 ? top : 16, r)) {
            have = true;
            p.S = S;
            for (int i = 0; i < S; ++i) p.r[i] = r[i];
        }
    }
    if (!have) {
        p.S = 0;
        return p;
    }
    int best = 0;
    for (int t = 1; t <= n / p.r[p.S - 1]; ++t) {
        int e = 0, cost = 0;
        for (int i = 0; i < p.S; ++i) {
            const int nb = n / p.r[i], per = (nb + t - 1) / t;
            if (per * p.r[i] > e) e = per * p.r[i];
            cost += per * p.r[i] * t;
        }
        const int lim = emax > p.r[0] ? emax : p.r[0];
        if (e > lim) continue;
        if (best == 0 || cost < best || (row && cost == best)) {
            best = cost;
            p.T = t;
            p.E = e;
        }
    }
    return p;
}

// entries of the stage tables of a plan: stage i > 0 holds w_{Ns r_i}^(r j), r = 1 .. r_i - 1,
// j < Ns = r_0 ... r_{i-1}, at [off + (r - 1) Ns + j]
__host__ __device__ constexpr int line_table_size(const LinePlan &p)
{
    int n = 0, ns = 1;
    for (int i = 0; i < p.S; ++i) {
        if (i > 0) n += (p.r[i] - 1) * ns;
        ns *= p.r[i];
    }
    return n;
}

// the plan of the sandwich's second transform: the same radices in reverse
__host__ __device__ constexpr LinePlan line_reverse(const LinePlan &p)
{
    LinePlan q = p;
    for (int i = 0; i < p.S; ++i) q.r[i] = p.r[p.S - 1 - i];
    return q;
}

// The exchange of a line after stage i: writes (b / Ns)(BS + pad) + b % Ns + q Ns, reads
// b + (b / BS) pad + q (NB + NB / BS pad), BS = Ns r_i, NB = n / r_{i+1} (a multiple of BS).
__host__ __device__ constexpr int line_conflicts_at(const LinePlan &p, int n, int T, int lp, int lanes, int i, int pad)
{
    int ns = 1;
    for (int k = 0; k < i; ++k) ns *= p.r[k];
    const int bs = ns * p.r[i];
    int total = 0;
    for (int rd = 0; rd < 2; ++rd) {
        int hit[32] = {}, worst = 0;
        for (int l = 0; l < lanes; ++l) {
            const int g = l / T, b = l % T;
            if (b >= n / p.r[rd ? i + 1 : i]) continue;
            const int a = g * lp + (rd ? b + (b / bs) * pad : (b / ns) * (bs + pad) + b % ns);
            if (++hit[a % lanes] > worst) worst = hit[a % lanes];
        }
        total += worst;
    }
    return total;
}
__host__ __device__ constexpr int line_pad(const LinePlan &p, int n, int T, int lanes, int i)
{
    int best = 0, bc = 1 << 30;
    for (int pad = 0; pad < lanes; ++pad) {
        const int c = line_conflicts_at(p, n, T < lanes ? T : lanes, 0, T < lanes ? T : lanes, i, pad);
        if (c < bc) {
            bc = c;
            best = pad;
        }
    }
    return best;
}
__host__ __device__ constexpr int line_pitch(const LinePlan &p, int n, int T, int lanes)
{
    int m = n, ns = 1;
    for (int i = 0; i + 1 < p.S; ++i) {
        ns *= p.r[i];
        const int sz = n + (n / ns) * line_pad(p, n, T, lanes, i);
        if (sz > m) m = sz;
    }
    return m;
}
__host__ __device__ constexpr int line_conflicts(const LinePlan &p, int n, int T, int lp, int lanes)
{
    int c = 0;
    for (int i = 0; i + 1 < p.S; ++i) c += line_conflicts_at(p, n, T, lp, lanes, i, line_pad(p, n, T, lanes, i));
    return c;
}

constexpr int kBatchThreads = 256;  // threads of a batch kernel's block, whatever its tiles need

constexpr int kLineEmax = 16;  // 16 complex values: 32 (float) or 64 (double) registers (radices above take more)

template <typename R, int N, bool ROW> struct LineShape {
    static constexpr LinePlan P = line_plan(N, ROW, kLineEmax, sizeof(R) == 4 ? 32 : 16);
    static constexpr LinePlan Q = line_reverse(P);
    static constexpr int T = P.T, E = P.E;
    // lines per CTA.  ROW: as near to 256 threads as fills its warps best.  COL: 256 threads, and
    // segments of 64 bytes (8 float, 4 double lines) where 1024 threads and 160 KB of exchange area
    // allow them (float columns of 1500, 2000 and 4096 points get 32 bytes, 2401 and 3000 points 16) (512^3 f32 Poisson back to back: 1113 us with 64-byte segments, 1137 with 128).
    // Double lines of one thread: past 32 lines while the tile is below 6 KB, because a CTA of one warp
    // with a few values a thread is bound by CTA starts (2^22 points as C2C columns of 1, 2 and 4
    // points 136 -> 36, 69 -> 25 and 35 -> 22 us, R2C of 4, 8 and 16 points 35 -> 13, 18 -> 11 and
    // 11 -> 10; longer lines gain nothing, and lose 4% with a staged side).
    static constexpr int row_lines()
    {
        int best = 1, bw = 1 << 30;
        for (int g = 1; g * T <= 384 || g == 1; ++g) {
            const int th = g * T, warps = (th + 31) / 32;
            if (warps > 12 && g > 1) break;
            // idle lanes per 1024 and the distance from eight warps
            const int waste = (warps * 32 - th) * 1024 / (warps * 32) + 12 * (warps > 8 ? warps - 8 : 8 - warps);
            const bool whole = 32 % T != 0 || th % 32 == 0;  // warp-local exchanges need whole warps
            if (whole && waste < bw) {
                bw = waste;
                best = g;
            }
        }
        return best;
    }
    static constexpr int col_lines()
    {
        const int lo = sizeof(R) == 4 ? 8 : 4, hi = sizeof(R) == 4 ? 128 : 32;
        int g = 1;
        while (g * 2 * T <= 256 && (g < hi || (g < 128 && g * N < 384))) g *= 2;
        while (g < lo && g * 2 * T <= 1024) g *= 2;
        while (g > 1 && (size_t)g * N * 2 * sizeof(R) > 160 * 1024) g /= 2;
        return g;
    }
    static constexpr int G = ROW ? row_lines() : col_lines();
    static constexpr int NT = G * T;
    // Exchanges: after stage i, point p sits at p + (p / BS) pad, BS = Ns r_i, the pad and the line
    // pitch chosen for the fewest bank conflicts; the offsets stay linear in a butterfly's points.
    // LANES: points of one line among the lanes that share a shared-memory wavefront
    static constexpr int WAVE = sizeof(R) == 4 ? 16 : 8;
    static constexpr int LANES = ROW ? WAVE : (WAVE > G ? WAVE / G : 1);
    static constexpr int PITCH0 = line_pitch(P, N, T, LANES) > line_pitch(Q, N, T, LANES)
                                      ? line_pitch(P, N, T, LANES)
                                      : line_pitch(Q, N, T, LANES);
    static constexpr int pitch()
    {
        int best = PITCH0, bc = 1 << 30;
        for (int lp = PITCH0; lp < PITCH0 + LANES; ++lp) {
            const int c = ROW && T < LANES ? line_conflicts(P, N, T, lp, LANES) + line_conflicts(Q, N, T, lp, LANES) : 0;
            if (c < bc) {
                bc = c;
                best = lp;
            }
        }
        return best;
    }
    static constexpr int LP = pitch();
    static constexpr int STEP = ROW ? 1 : G;          // between points of a line in natural order
    static constexpr bool WARP = ROW && 32 % T == 0;  // a line's threads share a warp
    static constexpr size_t EX = (size_t)G * LP;      // exchange area, entries
    static constexpr int SP = (N + 1) | 1;                              // staged line pitch (in_t / out_t)
    static constexpr size_t ST = (size_t)G * SP;
    // CTAs per SM the registers are budgeted for: 64 registers a thread (float; 80 and 128 with
    // more than 16 and 20 values), 128 (double)
    static constexpr int MINB = (65536 / (sizeof(R) == 4 ? (E > 20 ? 128 : E > 16 ? 80 : 64) : 128)) / (NT < 32 ? 32 : NT) > 0
                                    ? (65536 / (sizeof(R) == 4 ? (E > 20 ? 128 : E > 16 ? 80 : 64) : 128)) / (NT < 32 ? 32 : NT)
                                    : 1;
};

// ---------------------------------------------------------------- butterflies
// sine and cosine by their power series (|x| <= pi; the terms fall below 1e-40 by the 30th)
__host__ __device__ constexpr double ct_sin(double x)
{
    double t = x, r = x;
    for (int i = 1; i < 30; ++i) { t *= -x * x / ((2 * i) * (2 * i + 1)); r += t; }
    return r;
}
__host__ __device__ constexpr double ct_cos(double x)
{
    double t = 1, r = 1;
    for (int i = 1; i < 30; ++i) { t *= -x * x / ((2 * i - 1) * (2 * i)); r += t; }
    return r;
}
// exp(2 pi i m / M), m < M
template <int M> struct CtTable {
    double c[M] = {}, s[M] = {};
    constexpr CtTable()
    {
        for (int m = 0; m < M; ++m) {
            const double x = 6.283185307179586476925286766559 * (2 * m > M ? m - M : m) / M;
            c[m] = ct_cos(x);
            s[m] = ct_sin(x);
        }
    }
};
// n = A B with coprime A and B (Good 1958, Thomas 1963: the prime factor algorithm): input
// index B n1 + A n2, output index k with k = k1 mod A and k = k2 mod B, and no twiddles between.
__host__ __device__ constexpr int pfa_out(int A, int B, int k1, int k2)
{
    for (int k = 0; k < A * B; ++k)
        if (k % A == k1 && k % B == k2) return k;
    return 0;
}

template <typename R, int RAD, typename C> __device__ __forceinline__ void line_dft(C *v);

template <typename R, int A, int B, typename C> __device__ __forceinline__ void dft_pfa(C *v)
{
    C u[A * B];
#pragma unroll
    for (int n2 = 0; n2 < B; ++n2) {
        C c[A];
#pragma unroll
        for (int n1 = 0; n1 < A; ++n1) c[n1] = v[(B * n1 + A * n2) % (A * B)];
        line_dft<R, A>(c);
#pragma unroll
        for (int k1 = 0; k1 < A; ++k1) u[k1 * B + n2] = c[k1];
    }
#pragma unroll
    for (int k1 = 0; k1 < A; ++k1) {
        line_dft<R, B>(u + k1 * B);
#pragma unroll
        for (int k2 = 0; k2 < B; ++k2) v[pfa_out(A, B, k1, k2)] = u[k1 * B + k2];
    }
}

// cos (want = 0) and sin (want = 1) of 2 pi m / P, m = 0 .. (P - 1) / 2, for the prime radices
// 11 and 13
template <int P> __host__ __device__ constexpr double prime_cs(int want, int m)
{
    static_assert(P == 11 || P == 13, "prime radix");
    constexpr double c11[] = {1.00000000000000000000, 0.84125353283118120551, 0.41541501300188643508,
                              -0.14231483827328514358, -0.65486073394528510061, -0.95949297361449736865};
    constexpr double s11[] = {0.00000000000000000000, 0.54064081745559755543, 0.90963199535451833011,
                              0.98982144188093268422, 0.75574957435425826890, 0.28173255684142967104};
    constexpr double c13[] = {1.00000000000000000000, 0.88545602565320991051, 0.56806474673115581187,
                              0.12053668025532304764, -0.35460488704253562142, -0.74851074817110108128,
                              -0.97094181742605201180};
    constexpr double s13[] = {0.00000000000000000000, 0.46472317204376856203, 0.82298386589365635224,
                              0.99270887409805397272, 0.93501624268541483342, 0.66312265824079519305,
                              0.23931566428755776665};
    if (P == 11) return want ? s11[m] : c11[m];
    return want ? s13[m] : c13[m];
}

// odd prime radix from its even and odd parts: X[k], X[p - k] = v0 + sum_m c(mk) a_m -+ i s(mk) b_m
template <typename R, int P, typename C> __device__ __forceinline__ void dft_prime(C *v)
{
    constexpr int H = (P - 1) / 2;
    C a[H], b[H], o[P];
    o[0] = v[0];
#pragma unroll
    for (int m = 0; m < H; ++m) {
        a[m] = cadd(v[m + 1], v[P - 1 - m]);
        b[m] = csub(v[m + 1], v[P - 1 - m]);
        o[0] = cadd(o[0], a[m]);
    }
#pragma unroll
    for (int k = 1; k <= H; ++k) {
        C x = v[0], y = mk<R>(R(0), R(0));
#pragma unroll
        for (int m = 1; m <= H; ++m) {
            const int e = (m * k) % P, q = e <= H ? e : P - e;
            const R c = R(prime_cs<P>(0, q)), s = R(e <= H ? prime_cs<P>(1, q) : -prime_cs<P>(1, q));
            x.x += c * a[m - 1].x;
            x.y += c * a[m - 1].y;
            y.x += s * b[m - 1].x;
            y.y += s * b[m - 1].y;
        }
        const C iy = mul_si<-1>(y);  // -i y: the forward transform
        o[k] = cadd(x, iy);
        o[P - k] = csub(x, iy);
    }
#pragma unroll
    for (int k = 0; k < P; ++k) v[k] = o[k];
}

// 9 = 3 x 3 with the twiddles w_9^(n k), forward
template <typename R, typename C> __device__ __forceinline__ void dft9(C *v)
{
    constexpr R c1 = R(0.76604444311897801345), s1 = R(0.64278760968653936292);  // 2 pi / 9
    constexpr R c2 = R(0.17364817766693035894), s2 = R(0.98480775301220802032);  // 4 pi / 9
    constexpr R c4 = R(-0.93969262078590842791), s4 = R(0.34202014332566871291);  // 8 pi / 9
    C u[3][3];
#pragma unroll
    for (int n = 0; n < 3; ++n) {
        C c[3] = {v[n], v[n + 3], v[n + 6]};
        dft3<-1, C, R>(c);
#pragma unroll
        for (int k = 0; k < 3; ++k) u[k][n] = c[k];
    }
    u[1][1] = cmulc(u[1][1], mk<R>(c1, s1));
    u[1][2] = cmulc(u[1][2], mk<R>(c2, s2));
    u[2][1] = cmulc(u[2][1], mk<R>(c2, s2));
    u[2][2] = cmulc(u[2][2], mk<R>(c4, s4));
#pragma unroll
    for (int k = 0; k < 3; ++k) {
        dft3<-1, C, R>(u[k]);
#pragma unroll
        for (int m = 0; m < 3; ++m) v[k + 3 * m] = u[k][m];
    }
}

// A x B with the twiddles w_AB^(n k) between
template <typename R, int A, int B, typename C> __device__ __forceinline__ void dft_ct(C *v)
{
    C u[A][B];
#pragma unroll
    for (int n = 0; n < B; ++n) {
        C c[A];
#pragma unroll
        for (int m = 0; m < A; ++m) c[m] = v[n + B * m];
        line_dft<R, A>(c);
#pragma unroll
        for (int k = 0; k < A; ++k) {
            constexpr CtTable<A * B> w{};
            u[k][n] = n * k == 0 ? c[k] : cmulc(c[k], mk<R>(R(w.c[n * k]), R(w.s[n * k])));
        }
    }
#pragma unroll
    for (int k = 0; k < A; ++k) {
        line_dft<R, B>(u[k]);
#pragma unroll
        for (int m = 0; m < B; ++m) v[k + A * m] = u[k][m];
    }
}

// forward DFT of RAD values in registers
template <typename R, int RAD, typename C> __device__ __forceinline__ void line_dft(C *v)
{
    if constexpr (RAD == 18) dft_pfa<R, 2, 9>(v);
    else if constexpr (RAD == 20) dft_pfa<R, 4, 5>(v);
    else if constexpr (RAD == 24) dft_pfa<R, 3, 8>(v);
    else if constexpr (RAD == 30) dft_pfa<R, 2, 15>(v);
    else if constexpr (RAD == 25) dft_ct<R, 5, 5>(v);
    else if constexpr (RAD == 32) dft_ct<R, 4, 8>(v);
    else if constexpr (RAD == 6) dft_pfa<R, 2, 3>(v);
    else if constexpr (RAD == 9) dft9<R>(v);
    else if constexpr (RAD == 10) dft_pfa<R, 2, 5>(v);
    else if constexpr (RAD == 11 || RAD == 13) dft_prime<R, RAD>(v);
    else if constexpr (RAD == 12) dft_pfa<R, 3, 4>(v);
    else if constexpr (RAD == 14) dft_pfa<R, 2, 7>(v);
    else if constexpr (RAD == 15) dft_pfa<R, 3, 5>(v);
    else dft_radix<-1, RAD, C, R>(v, nullptr, 1);
}

// ---------------------------------------------------------------- staged core
__host__ __device__ constexpr int line_ns(const LinePlan &p, int stage)
{
    int ns = 1;
    for (int i = 0; i < stage; ++i) ns *= p.r[i];
    return ns;
}
__host__ __device__ constexpr int line_tab_off(const LinePlan &p, int stage)
{
    int n = 0, ns = 1;
    for (int i = 0; i < stage; ++i) {
        if (i > 0) n += (p.r[i] - 1) * ns;
        ns *= p.r[i];
    }
    return n;
}

template <typename R, int N, bool ROW> __device__ __forceinline__ void line_sync()
{
    if constexpr (LineShape<R, N, ROW>::WARP) __syncwarp();
    else __syncthreads();
}

// Stages STAGE .. S-1 of the forward transform.  v holds the PER butterflies of this stage:
// v[k r + q] = point b + q n / r of butterfly b = t + k T.  ln: this line in the exchange area.
template <typename R, int N, bool ROW, bool REV, int STAGE>
__device__ __forceinline__ void line_stages(cpx<R> *v, cpx<R> *ln, const cpx<R> *__restrict__ tab, int t)
{
    using C = cpx<R>;
    using S = LineShape<R, N, ROW>;
    constexpr LinePlan P = REV ? S::Q : S::P;
    constexpr int RAD = P.r[STAGE], NB = N / RAD, T = S::T, PER = (NB + T - 1) / T, NS = line_ns(P, STAGE);
    constexpr bool FULL = PER * T == NB;
    if constexpr (STAGE > 0) {
        const C *tw = tab + line_tab_off(P, STAGE);
#pragma unroll
        for (int k = 0; k < PER; ++k) {
            const int b = t + k * T;
            if (FULL || b < NB) {
                const int j = STAGE == P.S - 1 ? b : b % NS;
#pragma unroll
                for (int q = 1; q < RAD; ++q) v[k * RAD + q] = cmul(v[k * RAD + q], __ldg(&tw[(q - 1) * NS + j]));
            }
        }
    }
#pragma unroll
    for (int k = 0; k < PER; ++k) line_dft<R, RAD>(v + k * RAD);
    if constexpr (STAGE + 1 < P.S) {
        constexpr int RN = P.r[STAGE + 1], NBN = N / RN, PERN = (NBN + T - 1) / T;
        constexpr bool FULLN = PERN * T == NBN;
        constexpr int BS = NS * RAD, PAD = line_pad(P, N, T, S::LANES, STAGE), ST = S::STEP;
        line_sync<R, N, ROW>();  // earlier reads of the exchange area are done
#pragma unroll
        for (int k = 0; k < PER; ++k) {
            const int b = t + k * T;
            if (FULL || b < NB) {
                C *w = ln + ((b / NS) * (BS + PAD) + b % NS) * ST;
#pragma unroll
                for (int q = 0; q < RAD; ++q) w[q * NS * ST] = v[k * RAD + q];
            }
        }
        line_sync<R, N, ROW>();
#pragma unroll
        for (int k = 0; k < PERN; ++k) {
            const int b = FULLN || t + k * T < NBN ? t + k * T : 0;  // (a thread without one repeats the first)
            const C *r = ln + (b + (b / BS) * PAD) * ST;
#pragma unroll
            for (int q = 0; q < RN; ++q) v[k * RN + q] = r[q * (NBN + NBN / BS * PAD) * ST];
        }
        line_stages<R, N, ROW, REV, STAGE + 1>(v, ln, tab, t);
    }
}

// Spectral factor of the sandwich: scale, sign / |k|^2 and the Gaussian; the part of |k|^2 that does
// not depend on the point is formed once per line
template <typename R> struct LineFactor {
    R base = R(0);
    int pn = 0, phalf = 0;  // the points' own axis (0: none)
    __device__ __forceinline__ void init(const PassArgs &a, int b0, int b1, int b2)
    {
#pragma unroll
        for (int ax = 0; ax < 4; ++ax) {
            if (ax >= a.ep_naxes) break;
            const int src = a.ep_src[ax], n = a.ep_n[ax];
            if (src == 0) {
                pn = n;
                phalf = a.ep_half[ax];
                continue;
            }
            const int i = src == 1 ? b0 : (src == 2 ? b1 : b2);
            const R k = R(a.ep_half[ax] || i <= n / 2 ? i : i - n);
            base += k * k;
        }
    }
    __device__ __forceinline__ R k2(int p) const
    {
        const R k = R(phalf || p <= pn / 2 ? p : p - pn);
        return pn ? base + k * k : base;
    }
};

// a line's EP_SCALE / EP_HALFW factor (the half axis is a batch axis of a C2C pass)
template <typename R> __device__ __forceinline__ R line_scale(const PassArgs &a, int b0, int b1, int b2)
{
    R f = R(a.ep_scale);
    if (a.ep_mode & EP_HALFW) {
#pragma unroll
        for (int ax = 0; ax < 4; ++ax) {
            if (ax >= a.ep_naxes) break;
            const int src = a.ep_src[ax], n = a.ep_n[ax];
            const int i = src == 1 ? b0 : (src == 2 ? b1 : b2);
            if (src != 0 && a.ep_half[ax] && i != 0 && 2 * i != n) f *= R(a.ep_hw);
        }
    }
    return f;
}

// direction of a store: known at compile time (unit), and then whether backwards
template <bool U, bool B> struct LineDir {
    static constexpr bool unit = U, back = B;
};

// One CTA's lines: tile `tile` of the pass.  BATCH: called from the batch kernels, whose blocks may
// have more threads than the tile (the extra ones repeat the first and store nothing) and whose
// passes have no staged side, no long-line twiddle and no programmatic launch.
template <typename R, int N, bool ROW, bool SAND, bool BATCH>
__device__ __forceinline__ void line_body(const PassArgs &__restrict__ a, const void *in_ptr, void *out_ptr,
                                          long long tile, unsigned char *smem_raw, long long *soff)
{
    using C = cpx<R>;
    using S = LineShape<R, N, ROW>;
    constexpr LinePlan P = S::P;
    constexpr int T = S::T, G = S::G, NT = S::NT, ST = S::STEP;
    constexpr int R0 = P.r[0], NB0 = N / R0, PER0 = (NB0 + T - 1) / T;
    // the last stage's radix (the sandwich ends with the reversed plan's last, r_0)
    constexpr int RL = SAND ? P.r[0] : P.r[P.S - 1], NBL = N / RL, PERL = (NBL + T - 1) / T;
    constexpr int PH = (N / 2 + T) / T;  // pairs (k, N - k), k = t + T i <= N/2, of a thread
    // an extra thread takes the place of thread tid - NT, which has to be one of the tile; it repeats that
    // thread's exchange writes, which only block-wide barriers order
    static_assert(!BATCH || (NT <= kBatchThreads && 2 * NT >= kBatchThreads), "extra threads stay in the tile");
    static_assert(!BATCH || !S::WARP || NT == kBatchThreads, "whole tiles where a warp orders its own exchanges");
    C *s = reinterpret_cast<C *>(smem_raw);
    const int tid = BATCH && threadIdx.x >= NT ? threadIdx.x - NT : threadIdx.x;
    const int g = ROW ? tid / T : tid % G, t = ROW ? tid - g * T : tid / G;
    C *ln = ROW ? s + g * S::LP : s + g;
    C *st = s + g * S::SP;  // this line in a staged side
    // threads past the last line repeat it and store nothing
    const bool has = tile * G + g < a.nlines;
    const bool act = has && (!BATCH || threadIdx.x < NT);
    const long long l = has ? tile * G + g : a.nlines - 1;
    int b0, b1, b2;
    if (a.c_shift >= 0) {  // l < 2^31: the divisions as multiplications (PassArgs)
        const unsigned q = (unsigned)(((unsigned long long)(unsigned)l * a.c0_mul) >> (a.c_shift & 63));
        b0 = (int)((unsigned)l - q * (unsigned)a.c0);
        b2 = (int)(((unsigned long long)q * a.c1_mul) >> (a.c_shift >> 6));
        b1 = (int)(q - (unsigned)b2 * (unsigned)a.c1);
    } else {
        const long long q = l / a.c0;
        b0 = (int)(l - q * a.c0);
        b2 = (int)(q / a.c1);
        b1 = (int)(q - (long long)b2 * a.c1);
    }
    const long long io = b0 * a.ib0 + b1 * a.ib1 + b2 * a.ib2;
    // Programmatic launch: the next pass may start its CTAs (they wait here) while this one's last
    // run, and this one waits for the whole of the pass before it, so the launch gap and the index
    // arithmetic above overlap.  Nothing before this line reads a buffer; every load of one after
    // it is an ordinary load (the tables alone are read as constants).  Back to back: 192^3 f32
    // Poisson 76.9 -> 66.4 us, 32^3 f64 25.4 -> 18.2, 2048^2 forward 26.7 -> 21.8, 256^3 f64 round
    // trip 306 -> 302.
    if constexpr (!BATCH) asm volatile("griddepcontrol.launch_dependents;\n\tgriddepcontrol.wait;\n" ::: "memory");
    const int kind = SAND ? (int)K_SANDWICH : a.kind;
    const bool half = !SAND && a.half;
    // the direct side of a ROW pass has unit stride
    const long long is = ROW ? 1 : a.is, os = ROW ? 1 : a.os;
    const bool in_t = !BATCH && !a.line_in, out_t = !BATCH && !a.line_out;
    const long long left = a.nlines - tile * G;
    const int rows = left < G ? (int)left : G;  // lines of this CTA

    C v[S::E];
    // v <- points of this thread's first-stage butterflies: x(p, offset p st) of each
    auto load = [&](long long st, auto x) {
#pragma unroll
        for (int k = 0; k < PER0; ++k) {
            const int b = PER0 * T == NB0 || t + k * T < NB0 ? t + k * T : 0;
            long long off = b * st;
#pragma unroll
            for (int q = 0; q < R0; ++q, off += NB0 * st) v[k * R0 + q] = x(b + q * NB0, off);
        }
    };
    // copies of a staged side: f(line of the CTA, point), the points or the lines fastest
    auto staged = [&](int n, bool pts_fast, auto f) {
        if (pts_fast) {
#pragma unroll 4
            for (int e = tid; e < rows * n; e += NT) f(e / n, e % n);
        } else {
#pragma unroll 4
            for (int e = tid; e < G * n; e += NT)
                if (e % G < rows) f(e % G, e / G);
        }
    };
    // packed half-length line of a half spectrum (x: its bin 0, st: between bins): Z[k] = E + i O and
    // Z[N-k] = conj(E - i O) with E = X[k] + conj X[N-k], O = (X[k] - conj X[N-k]) conj(w_2N^k), DC and
    // Nyquist counted with their real parts.  Each pair is read once and goes through the
    // exchange area to the threads that start the transform.
    // EP_DERIV multiplies bin b by i b first (the derivative along a half axis).
    const bool drv = !SAND && (a.ep_mode & EP_DERIV);
    auto times_ik = [](int k, C x) -> C { return mk<R>(-R(k) * x.y, R(k) * x.x); };
    auto load_packed = [&](bool stage, const C *x, long long st) {
        C xa[PH], xb[PH];
        const C *pa = x + t * st, *pb = x + (N - t) * st;
#pragma unroll
        for (int i = 0; i < PH; ++i, pa += T * st, pb -= T * st) {
            const bool ok = i + 1 < PH || t + T * i <= N / 2;
            xa[i] = ok ? *pa : mk<R>(R(0), R(0));
            xb[i] = ok ? *pb : mk<R>(R(0), R(0));
        }
        if (drv) {
#pragma unroll
            for (int i = 0; i < PH; ++i) {
                xa[i] = times_ik(t + T * i, xa[i]);
                xb[i] = times_ik(N - t - T * i, xb[i]);
            }
        }
        if (stage) __syncthreads();  // every line is read before the packed ones overwrite them
        const C *tw = reinterpret_cast<const C *>(a.tw) + t;
#pragma unroll
        for (int i = 0; i < PH; ++i) {
            const int k = t + T * i;
            if (i + 1 < PH || k <= N / 2) {
                C xk = xa[i], xm = cconj(xb[i]);
                if (i == 0 && t == 0) {
                    xk.y = R(0);
                    xm.y = R(0);
                }
                const C e = cadd(xk, xm);
                const C io = mul_si<1>(cmulc(csub(xk, xm), __ldg(tw + T * i)));
                ln[k * ST] = cadd(e, io);
                if (i > 0 || t > 0) ln[(N - k) * ST] = cconj(csub(e, io));
            }
        }
        line_sync<R, N, ROW>();
        load(ST, [&](int p, long long) { return ln[p * ST]; });
    };
    // full line of a half spectrum: bin p from x, which holds bin p or (p > N/2) bin N - p
    auto extend = [&](int p, C x) -> C {
        if (drv) x = times_ik(p <= N / 2 ? p : N - p, x);
        if (p > N / 2) x = cconj(x);
        if (p == 0 || 2 * p == N) x.y = R(0);
        return x;
    };

    // ------------------------------------------------------------ load
    if (in_t) {
        // the input's other order: its lines go through shared memory, [line][SP]
        if (t == 0) soff[g] = io;
        __syncthreads();
        staged(kind == K_C2R ? (half ? N + 1 : N / 2 + 1) : N, a.in_pts_fast, [&](int gg, int p) {
            C *d = &s[gg * S::SP + p];
            if (kind == K_R2C) {
                const R *src = reinterpret_cast<const R *>(in_ptr) + soff[gg];
                if (half) {
                    cp_async<sizeof(R)>(&d->x, src + (2 * p) * a.is, true);
                    cp_async<sizeof(R)>(&d->y, src + (2 * p + 1) * a.is, true);
                } else {
                    cp_async<sizeof(R)>(&d->x, src + p * a.is, true);
                    d->y = R(0);
                }
            } else {
                const long long pi =
                    a.in_blk ? (long long)(p / a.in_blk) * a.in_hi + (long long)(p % a.in_blk) * a.is : p * a.is;
                cp_async<sizeof(C)>(d, reinterpret_cast<const C *>(in_ptr) + soff[gg] + pi, true);
            }
        });
        cp_async_wait_all();
        __syncthreads();
        if (kind == K_C2R && half) {
            load_packed(true, st, 1);
        } else {
            if (kind == K_C2R) load(1, [&](int p, long long) { return extend(p, st[p <= N / 2 ? p : N - p]); });
            else load(1, [&](int p, long long) { return st[p]; });
            __syncthreads();  // the staged lines are read before the exchanges overwrite them
        }
    } else if (!SAND && kind == K_R2C) {
        const R *in = reinterpret_cast<const R *>(in_ptr) + io;
        if (half && a.pair_io) load(2, [&](int, long long o) { return *reinterpret_cast<const C *>(in + o); });
        else if (half) load(2 * is, [&](int, long long o) { return mk<R>(in[o], in[o + is]); });
        else load(is, [&](int, long long o) { return mk<R>(in[o], R(0)); });
    } else {
        const C *in = reinterpret_cast<const C *>(in_ptr) + io;
        if (SAND || kind != K_C2R) load(is, [&](int, long long o) { return in[o]; });
        else if (half) load_packed(false, in, is);
        else load(is, [&](int p, long long) { return extend(p, in[(p <= N / 2 ? p : N - p) * is]); });
    }

    // ------------------------------------------------------------ transform
    const C *tab = reinterpret_cast<const C *>(a.ltw);
    line_stages<R, N, ROW, false, 0>(v, ln, tab, t);
    if constexpr (SAND) {
        // the forward transform's results sit where the reversed plan's first stage takes them
        constexpr int RF = P.r[P.S - 1], NBF = N / RF, PERF = (NBF + T - 1) / T;
        LineFactor<R> fac;
        fac.init(a, b0, b1, b2);
        const R sc = R(a.ep_scale), ss = sc * R(a.ep_sign), gs = R(a.ep_gauss);
        auto multiply = [&](auto f) {
#pragma unroll
            for (int k = 0; k < PERF; ++k)
#pragma unroll
                for (int q = 0; q < RF; ++q) v[k * RF + q] = f(t + k * T + q * NBF, v[k * RF + q]);
        };
        if (a.ep_mode & EP_GAUSS)
            multiply([&](int p, C z) {
                const R k2 = fac.k2(p);
                R f = sc;
                if (a.ep_mode & EP_POISSON) f = k2 == R(0) ? R(0) : ss / k2;
                return cscale(z, f * exp(-k2 * gs));
            });
        else if (a.ep_mode & EP_POISSON)
            multiply([&](int p, C z) {
                const R k2 = fac.k2(p);
                return cscale(z, k2 == R(0) ? R(0) : ss / k2);
            });
        else if (a.ep_mode & EP_DERIV)  // i k along the lines' own full axis, the Nyquist bin at +n/2
            multiply([&](int p, C z) { return cscale(times_ik(p <= N / 2 ? p : p - N, z), sc); });
        else
            multiply([&](int, C z) { return cscale(z, sc); });
        line_stages<R, N, ROW, true, 0>(v, ln, tab + line_table_size(P), t);
    }

    // ------------------------------------------------------------ epilogue
    const bool inv = SAND || kind == K_C2C_INV || kind == K_C2R;  // result i is point -i mod N
    if (!SAND && a.ep_mode) {
        if (!BATCH && (a.ep_mode & EP_TWIDDLE)) {
            // the four-step twiddle of a long line: p < L1 and j < L2, so p j < L needs no reduction
            const C *eptw = reinterpret_cast<const C *>(a.ep_tw);
            const int j = a.ep_src[0] == 1 ? b0 : (a.ep_src[0] == 2 ? b1 : b2);
#pragma unroll
            for (int k = 0; k < PERL; ++k) {
                const int b = PERL * T == NBL || t + k * T < NBL ? t + k * T : 0;
#pragma unroll
                for (int q = 0; q < RL; ++q) {
                    const int i = b + q * NBL, p = inv && i ? N - i : i;
                    const C w = eptw[(long long)p * j];
                    v[k * RL + q] = inv ? cmulc(v[k * RL + q], w) : cmul(v[k * RL + q], w);
                }
            }
        }
        if (a.ep_mode & (EP_SCALE | EP_HALFW)) {
            const R f = line_scale<R>(a, b0, b1, b2);
#pragma unroll
            for (int i = 0; i < S::E; ++i) v[i] = cscale(v[i], f);
        }
    }

    // ------------------------------------------------------------ store
    const long long oo = b0 * a.ob0 + b1 * a.ob1 + b2 * a.ob2;
    // f(point p, offset p st, value) for the results of this thread's last-stage butterflies
    auto walk = [&](long long st, auto rev, auto f) {
        constexpr bool UNIT = decltype(rev)::unit;  // the direction is known at compile time
        const bool back = UNIT ? decltype(rev)::back : inv;
#pragma unroll
        for (int k = 0; k < PERL; ++k) {
            const int b = t + k * T;
            if (PERL * T == NBL || b < NBL) {
                const int p0 = back ? N - b : b;
                long long off = p0 * st;
                const long long step = (back ? -NBL : NBL) * st;
#pragma unroll
                for (int q = 0; q < RL; ++q, off += step) {
                    const bool zero = back && k == 0 && q == 0 && t == 0;
                    f(zero ? 0 : (back ? p0 - q * NBL : p0 + q * NBL), zero ? 0 : off, v[k * RL + q]);
                }
            }
        }
    };
    auto store = [&](long long st, auto f) {
        if constexpr (ROW) {
            if (inv) walk(st, LineDir<true, true>{}, f);
            else walk(st, LineDir<true, false>{}, f);
        } else {
            walk(st, LineDir<false, false>{}, f);
        }
    };
    if (!SAND && kind == K_R2C && half) {
        // X[k] = E + w^k O, X[N-k] = conj(E - w^k O), E = (Z[k] + conj Z[N-k]) / 2,
        // O = -i (Z[k] - conj Z[N-k]) / 2, w = w_2N: the line goes through the exchange area once
        // more, to pair k with N - k
        line_sync<R, N, ROW>();
        walk(1, LineDir<true, false>{}, [&](int p, long long, C z) { ln[p * ST] = z; });
        line_sync<R, N, ROW>();
        C xa[PH], xb[PH];
        const C *tw = reinterpret_cast<const C *>(a.tw) + t;
#pragma unroll
        for (int i = 0; i < PH; ++i) {
            const int k = i + 1 < PH || t + T * i <= N / 2 ? t + T * i : 0;
            const int m = (i > 0 && i + 1 < PH) || k > 0 ? N - k : 0;
            const C zk = ln[k * ST], zm = cconj(ln[m * ST]);
            const C e = cscale(cadd(zk, zm), R(0.5)), o = cscale(mul_si<-1>(csub(zk, zm)), R(0.5));
            const C w = cmul(o, __ldg(tw + (i + 1 < PH || t + T * i <= N / 2 ? T * i : 0)));
            xa[i] = cadd(e, w);
            xb[i] = cconj(csub(e, w));
        }
        if (out_t) {
            __syncthreads();  // every line is read before the staged ones overwrite them
#pragma unroll
            for (int i = 0; i < PH; ++i) {
                const int k = t + T * i;
                if (i + 1 < PH || k <= N / 2) {
                    st[k] = xa[i];
                    st[N - k] = xb[i];
                }
            }
        } else if (act) {
            C *pa = reinterpret_cast<C *>(out_ptr) + oo + t * os, *pb = reinterpret_cast<C *>(out_ptr) + oo + (N - t) * os;
#pragma unroll
            for (int i = 0; i < PH; ++i, pa += T * os, pb -= T * os) {
                if (i + 1 < PH || t + T * i <= N / 2) {
                    *pa = xa[i];
                    *pb = xb[i];
                }
            }
        }
    } else if (out_t) {
        __syncthreads();
        store(1, [&](int p, long long, C z) { st[p] = z; });
    } else if (act) {
        if (!SAND && kind == K_C2R) {
            R *o = reinterpret_cast<R *>(out_ptr) + oo;
            if (!half) store(os, [&](int, long long f, C z) { o[f] = z.x; });
            else if (a.pair_io) store(2, [&](int, long long f, C z) { *reinterpret_cast<C *>(o + f) = z; });
            else
                store(2 * os, [&](int, long long f, C z) {
                    o[f] = z.x;
                    o[f + os] = z.y;
                });
        } else {
            C *o = reinterpret_cast<C *>(out_ptr) + oo;
            if (!SAND && kind == K_R2C) store(os, [&](int p, long long f, C z) { if (p <= N / 2) o[f] = z; });
            else store(os, [&](int, long long f, C z) { o[f] = z; });
        }
    }
    if (out_t) {
        // the output's other order, from the staged lines
        if (t == 0) soff[g] = oo;
        __syncthreads();
        staged(kind == K_R2C ? (half ? N + 1 : N / 2 + 1) : N, a.out_pts_fast, [&](int gg, int p) {
            const C z = s[gg * S::SP + p];
            if (kind == K_C2R) {
                R *o = reinterpret_cast<R *>(out_ptr) + soff[gg];
                if (half) {
                    o[(2 * p) * a.os] = z.x;
                    o[(2 * p + 1) * a.os] = z.y;
                } else {
                    o[p * a.os] = z.x;
                }
            } else {
                C *o = reinterpret_cast<C *>(out_ptr) + soff[gg];
                if (a.out_blk) {  // a slab exchange's pack: block q of the points, or a peer's buffer
                    const int q = p / a.out_blk;
                    C *base = a.out_peer[q] ? reinterpret_cast<C *>(a.out_peer[q]) + soff[gg] : o + (long long)q * a.out_hi;
                    base[(long long)(p - q * a.out_blk) * a.os] = z;
                } else {
                    o[p * a.os] = z;
                }
            }
        });
    }
}

template <typename R, int N, bool ROW, bool SAND>
__global__ void __launch_bounds__(LineShape<R, N, ROW>::NT, LineShape<R, N, ROW>::MINB)
    fftb_line_kernel(const __grid_constant__ PassArgs a)
{
    extern __shared__ __align__(16) unsigned char smem_raw[];
    __shared__ long long soff[LineShape<R, N, ROW>::G];  // line offsets of a staged side
    line_body<R, N, ROW, SAND, false>(a, a.in, a.out, blockIdx.x, smem_raw, soff);
}

// what the host needs of one line length and mapping
struct LineKernelInfo {
    int nf = 0, row = 0;
    int G = 0, NT = 0;
    size_t smem = 0, smem_t = 0;  // exchange area alone; with a staged side
    LinePlan plan;
    const void *fn = nullptr, *fn_sand = nullptr;
};

template <typename R, int N, bool ROW> inline LineKernelInfo line_kernel_info()
{
    using S = LineShape<R, N, ROW>;
    LineKernelInfo k;
    k.nf = N;
    k.row = ROW;
    k.G = S::G;
    k.NT = S::NT;
    k.smem = sizeof(cpx<R>) * S::EX;
    constexpr size_t staged = sizeof(cpx<R>) * (S::EX > S::ST ? S::EX : S::ST);
    static_assert(staged + S::G * sizeof(long long) + 1024 <= 228 * 1024, "a CTA's shared memory, its line offsets and 1 KB of the system's");
    k.smem_t = staged;
    k.plan = S::P;
    k.fn = (const void *)&fftb_line_kernel<R, N, ROW, false>;
    k.fn_sand = (const void *)&fftb_line_kernel<R, N, ROW, true>;
    return k;
}

} // namespace fftb
