// kernels_demon.cu -- the per-link demon microcanonical sweep
// (demon_microcanonical, field-demon.h:25-126).
//
// The reference updates the links one after another in site-index order
// (x0 fastest, mu = 0..3 inner), each update seeing every earlier one, and four
// global demons decide every hit: the sweep is sequential by definition.  One
// CTA walks the links of one chain in that order (independent chains of an
// ensemble run side by side, one CTA each).  What bounds it is the latency of
// one link's work: the staple paths, their sums and the two hits.  The work of
// neighbouring links overlaps as far as the order allows:
//
//  * in stage l (one block barrier each) the path warps multiply out the 168
//    staple paths of link l while one warp runs the hits of link l - 1, one
//    prepares link l + 1's proposals and three stage links;
//  * link l - 1 changes during stage l.  It enters the paths of link l only as
//    the first step, U_(mu-1)(x) forward, of 27 paths (mu > 0) or the second
//    step of one rectangle (mu = 0): those paths are multiplied out with the
//    unit matrix in its place (and in place of the steps before it), and the
//    hits of link l complete their sums with the link itself.  This holds when
//    the offsets -2..2 are distinct sites, every extent >= 5; below that the
//    same kernel runs the hits of l - 1 before the paths of l (8^3 x 4: 2.46 us
//    per link, 6^4: 1.87);
//  * a hit's action change is linear in the staple sum, ReTr(Y S) with
//    Y = v - m v for the proposal m: the path warps contract each path with the
//    three Y (first hit, second after a rejected or an accepted first) where
//    they multiply it out, so that no staple sum is ever formed;
//  * window: the 353 distinct links of the four links' paths, one window per
//    site, staged for site s + 1 during the four stages of site s by 16-byte
//    cp.async copies.  The links of sites s + 1, s and s - 1, which change after
//    a window was staged, are read from small site buffers that the hits
//    keep current;
//  * paths: 24 threads in each of seven warps, a warp holding paths of one
//    staple kind, so that a kind's sums end in its warps.  A thread multiplies
//    two rows of four products and reconstructs the third; the three-link
//    plaquette paths are padded with a unit slot and adjoints are formed by the
//    loads' addresses, so every thread runs the same instructions.  The window's slots
//    are numbered so that the eight threads that load together find their links
//    in different bank groups.
//
// Measured, us per link: 3.21 with paths, sums and hits one after another behind
// three barriers (6^4 and 8^3 x 4), now 1.87 and 2.46.  Of a stage's 3500 cycles
// the products of a path take 2400 (two path warps share an SM quarter's FP64
// pipe, 2.1 cycles per instruction), its contraction 600, the sum over eight
// lanes 280; the hits take 2700 of them beside.  At most 12 warps: a thirteenth
// would leave a thread 128 registers (2.1 us).
#include <stdint.h>

#include <algorithm>
#include <cstring>
#include <initializer_list>
#include <utility>
#include <vector>

#include "kernels.h"
#include "rng.cuh"

namespace magb {

namespace {

// one warp each for the proposals and the hits (the latter on the SM quarter with the
// fewest path warps), kPathWarps of 24 threads with a path each, the rest stage links
constexpr int kPrepareWarp = 0, kHitWarp = 1, kPathWarp0 = 2, kPathWarps = 7, kPathsPerWarp = 24;
constexpr int kStageWarp0 = kPathWarp0 + kPathWarps, kStageWarps = 3;
constexpr int kDemonThreads = 32 * (kStageWarp0 + kStageWarps);
constexpr int kPaths = kDemonPaths;  // 6 + 18 + 72 + 72
static_assert(kPaths == kPathWarps * kPathsPerWarp, "one thread per path");
constexpr int kSteps = 5;
constexpr size_t kLinkBytes = 144;  // 9 complex doubles
constexpr int kSiteLinks = 2 * kDemonWindow;  // the site buffers follow the two windows
constexpr size_t kDemonDynSmem = (kSiteLinks + 16) * kLinkBytes;
enum { RNG_DEMON_SU2 = 4, RNG_DEMON_SUBGROUP = 5 };

__device__ __forceinline__ int wrap(int v, int L) { return v < 0 ? v + L : (v >= L ? v - L : v); }

__device__ __forceinline__ void cp16(void* sdst, const void* gsrc) {
    const unsigned sa = (unsigned)__cvta_generic_to_shared(sdst);
    asm volatile("cp.async.ca.shared.global [%0], [%1], 16;\n" ::"r"(sa), "l"(gsrc) : "memory");
}
__device__ __forceinline__ void cp_wait_all() { asm volatile("cp.async.wait_all;\n" ::: "memory"); }

// the draws of random_su3_from_su2(0.9, rng) (field-matrix.h:36-65) from Philox counters
// (link, sweep, hit): a0 uniform in [0.9, 1), a1..a3 in [-1, 1) scaled to |a| = sqrt(1 - a0^2),
// and the SU(2) subgroup (1,2), (0,2) or (0,1) by a draw % 3
__device__ void su2_draw(unsigned long long seed, uint32_t link, uint32_t sweep, uint32_t hit, double a[4], int& sub) {
    uint32_t c1[4] = {link, sweep, hit, (uint32_t)RNG_DEMON_SU2};
    uint32_t c2[4] = {link, sweep, hit, (uint32_t)RNG_DEMON_SUBGROUP};
    philox4x32_10(c1, (uint32_t)seed, (uint32_t)(seed >> 32));
    philox4x32_10(c2, (uint32_t)seed, (uint32_t)(seed >> 32));
    const double small = 0.9;
    auto u = [](uint32_t v) { return ((double)v + 0.5) * 2.3283064365386963e-10; };
    const double a0 = small + (1.0 - small) * u(c1[0]);
    const double a1 = -1.0 + 2.0 * u(c1[1]), a2 = -1.0 + 2.0 * u(c1[2]), a3 = -1.0 + 2.0 * u(c1[3]);
    const double norm = sqrt((1. - a0 * a0) / (a1 * a1 + a2 * a2 + a3 * a3));
    a[0] = a0;
    a[1] = a1 * norm;
    a[2] = a2 * norm;
    a[3] = a3 * norm;
    sub = (int)(c2[0] % 3u);
}

// the proposal is the unit matrix but for rows / columns i, j:
//   m_ii = a0 + i a3, m_ij = a2 + i a1, m_ji = -a2 + i a1, m_jj = a0 - i a3
struct Su2 {
    int i, j;
    cplx<double> ii, ij, ji, jj;
};
__device__ __forceinline__ Su2 su2_of(double a0, double a1, double a2, double a3, int sub) {
    Su2 m;
    m.i = sub == 0 ? 1 : 0;
    m.j = sub == 2 ? 1 : 2;
    m.ii = mk(a0, a3);
    m.ij = mk(a2, a1);
    m.ji = mk(-a2, a1);
    m.jj = mk(a0, -a3);
    return m;
}
__device__ __forceinline__ cplx<double> pick(const cplx<double>& a, const cplx<double>& b, const cplx<double>& c, int r) {
    return r == 0 ? a : (r == 1 ? b : c);
}
// one column of v <- m v: rows i, j change
__device__ __forceinline__ void apply_su2_col(cplx<double> col[3], const Su2& m) {
    const cplx<double> vi = pick(col[0], col[1], col[2], m.i);
    const cplx<double> vj = pick(col[0], col[1], col[2], m.j);
    cplx<double> ni = cmul<false, false>(m.ii, vi);
    cmac<false, false, false>(ni, m.ij, vj);
    cplx<double> nj = cmul<false, false>(m.ji, vi);
    cmac<false, false, false>(nj, m.jj, vj);
#pragma unroll
    for (int r = 0; r < 3; r++) {
        if (r == m.i) col[r] = ni;
        if (r == m.j) col[r] = nj;
    }
}
// a staged link, or its adjoint (by the addresses and signs: every lane runs the same product code)
__device__ __forceinline__ mat3<double> load_oriented(const double2* q, bool fwd) {
    const int sr = fwd ? 3 : 1, sc = fwd ? 1 : 3;
    const long long flip = fwd ? 0 : (long long)0x8000000000000000ull;
    mat3<double> o;
#pragma unroll
    for (int r = 0; r < 3; r++)
#pragma unroll
        for (int c = 0; c < 3; c++) {
            const double2 v = q[r == c ? 4 * r : r * sr + c * sc];
            o.e[r][c] = mk(v.x, __longlong_as_double(__double_as_longlong(v.y) ^ flip));
        }
    return o;
}

// element (r, c) of a staged link or of its adjoint
__device__ __forceinline__ cplx<double> oriented(const double2* q, bool fwd, int r, int c) {
    const double2 v = q[fwd ? 3 * r + c : 3 * c + r];
    return mk(v.x, fwd ? v.y : -v.y);
}

__global__ void __launch_bounds__(kDemonThreads, 1) k_demon_sweep(const DemonJob* jobs, double2* aos,
                                                                  const DemonTables* tabs, int sweep, double e_max,
                                                                  DemonState* states) {
    const ChainInfo ci = jobs[blockIdx.x].ci;
    double2* U = aos + jobs[blockIdx.x].aos_off;
    const unsigned long long seed = jobs[blockIdx.x].seed;
    DemonState* st = states + blockIdx.x;
    // [2][kDemonWindow] windows of sites s and s + 1, [4][4] links of sites s - 2 .. s + 1 (site % 4)
    extern __shared__ __align__(16) double2 links[];
    auto site_link = [&](int s, int d) { return links + (kSiteLinks + 4 * (s & 3) + d) * 9; };
    // by link % 3: the candidates v, m0 v, m1 v, m1 m0 v and the Y of the three action changes
    __shared__ __align__(16) double2 cand[3][4][9];
    __shared__ __align__(16) double2 ymat[3][3][9];
    // by link % 2: the paths that wait for a link, the other paths' action changes by eight lanes
    __shared__ __align__(16) double2 tail[2][kDemonLate][9];
    __shared__ double psum[2][kPathWarps][4][3];
    // hits: sums of the waiting paths by kind, Y times the link they wait for
    __shared__ __align__(16) double2 late[4][9], lu[9], yu[2][3][9];
    __shared__ double draw_a[2][4];
    __shared__ int draw_sub[2];
    __shared__ uint16_t loc[2][kDemonWindow];  // where a window slot's link is: index into `links`
    // slots of the five steps, five bits of orientation, 1 + index into `tail`
    __shared__ __align__(16) uint4 path[4][kPaths];
    __shared__ int8_t sfirst[4][5];
    __shared__ int spk[kDemonWindow];
    for (int i = threadIdx.x; i < 4 * kPaths; i += blockDim.x) {
        const uint16_t* sl = &tabs->slot[0][0][0] + kSteps * i;
        const uint8_t* fw = &tabs->fwd[0][0][0] + kSteps * i;
        uint32_t f = 0;
        for (int k = 0; k < kSteps; k++) f |= (uint32_t)(fw[k] != 0) << k;
        (&path[0][0])[i] = make_uint4(sl[0] | (uint32_t)sl[1] << 16, sl[2] | (uint32_t)sl[3] << 16, sl[4] | f << 16,
                                      (uint32_t)(1 + (&tabs->late[0][0])[i]));
    }
    if (threadIdx.x < 20) (&sfirst[0][0])[threadIdx.x] = (&tabs->first[0][0])[threadIdx.x];
    for (int i = threadIdx.x; i < kDemonWindow; i += blockDim.x) spk[i] = tabs->packed[i];
    const int ns = tabs->nslot, lslot = tabs->lslot, uslot = tabs->uslot;
    const bool lfwd = tabs->lfwd, ufwd = tabs->ufwd;
    const int t = threadIdx.x, lane = t & 31, warp = t >> 5;
    double E = st->E[lane & 3];  // hits: demon lane % 4
    long long acc = 0, rej = 0;
    __syncthreads();
    const int nsite = ci.V;
    // the offsets -2..2 are distinct sites: the paths of a link may run ahead of its predecessor's hits
    const bool ahead = ci.L[0] >= 5 && ci.L[1] >= 5 && ci.L[2] >= 5 && ci.L[3] >= 5;

    // Stage part `part` (0..3; -1: all) of site s's window into buffer s % 2 with the nw warps from
    // w0 on: lane k of a round forms the source of slot base + k, the round's 32 slots are then
    // copied as 288 consecutive 16-byte pieces.  Part 0 also stages the site's own four links.
    // Links of site s or of the two sites before it are read from the site buffers.  Each part
    // first waits for the copies of the part before it, the last one for its own as well.
    auto stage_site = [&](int s, int part, int w0, int nw) {
        cp_wait_all();
        const int wb = s & 1;
        int x[4];
        int r = s;
        x[0] = r % ci.L[0]; r /= ci.L[0];
        x[1] = r % ci.L[1]; r /= ci.L[1];
        x[2] = r % ci.L[2]; r /= ci.L[2];
        x[3] = r;
        const int n0 = part < 0 ? 0 : (ns * part) / 4, n1 = part < 0 ? ns : (ns * (part + 1)) / 4;
        const int w = warp - w0;
        if (part <= 0 && w == 0) {
            cp16(site_link(s, 0) + lane, U + (size_t)s * 36 + lane);
            if (lane < 4) cp16(site_link(s, 0) + 32 + lane, U + (size_t)s * 36 + 32 + lane);
        }
        for (int base = n0 + 32 * w; base < n1; base += 32 * nw) {
            const int n = base + lane;
            int src = -1;  // link index; -1: nothing to copy
            if (n < n1) {
                const int pk = spk[n];
                const int d = pk >> 16;
                int at = wb * kDemonWindow + n;
                if (d >= 4) {
                    double2* dst = links + (size_t)at * 9;
#pragma unroll
                    for (int j = 0; j < 9; j++) dst[j] = make_double2(j == 0 || j == 4 || j == 8 ? 1.0 : 0.0, 0.0);
                } else {
                    const int g = wrap(x[0] + (pk & 15) - 4, ci.L[0]) +
                                  wrap(x[1] + ((pk >> 4) & 15) - 4, ci.L[1]) * ci.stride[1] +
                                  wrap(x[2] + ((pk >> 8) & 15) - 4, ci.L[2]) * ci.stride[2] +
                                  wrap(x[3] + ((pk >> 12) & 15) - 4, ci.L[3]) * ci.stride[3];
                    const int back = s - g;
                    if (back >= 0 && back <= 2)
                        at = kSiteLinks + 4 * (g & 3) + d;
                    else
                        src = g * 4 + d;
                }
                loc[wb][n] = (uint16_t)at;
            }
            double2* dst0 = links + ((size_t)wb * kDemonWindow + base) * 9;
#pragma unroll
            for (int rr = 0; rr < 9; rr++) {
                const int f = rr * 32 + lane;
                const int q = f / 9, j = f - 9 * q;
                const int a = __shfl_sync(0xffffffffu, src, q);
                if (a >= 0) cp16(dst0 + f, U + (size_t)a * 9 + j);
            }
        }
        if (part < 0 || part == 3) cp_wait_all();
    };
    // proposals of link l (one warp): the two draws, the candidate links and Y = v - m0 v,
    // v - m1 v, m0 v - m1 m0 v; v does not change before its own hits
    auto prepare = [&](int l) {
        if (lane < 2) {
            double a[4];
            int sub;
            su2_draw(seed, (uint32_t)l, (uint32_t)sweep, (uint32_t)lane, a, sub);
#pragma unroll
            for (int k = 0; k < 4; k++) draw_a[lane][k] = a[k];
            draw_sub[lane] = sub;
        }
        __syncwarp();
        if (lane < 9) {
            const int r = lane / 3, c = lane % 3, b = l % 3;
            const double(*a)[4] = draw_a;
            const Su2 m0 = su2_of(a[0][0], a[0][1], a[0][2], a[0][3], draw_sub[0]);
            const Su2 m1 = su2_of(a[1][0], a[1][1], a[1][2], a[1][3], draw_sub[1]);
            cplx<double> v[3], v0[3], v1[3], v01[3];
            const double2* vp = site_link(l >> 2, l & 3);
#pragma unroll
            for (int k = 0; k < 3; k++) {
                const double2 q = vp[3 * k + c];
                v[k] = v0[k] = v1[k] = mk(q.x, q.y);
            }
            apply_su2_col(v0, m0);
            apply_su2_col(v1, m1);
#pragma unroll
            for (int k = 0; k < 3; k++) v01[k] = v0[k];
            apply_su2_col(v01, m1);
            const cplx<double> e = pick(v[0], v[1], v[2], r), e0 = pick(v0[0], v0[1], v0[2], r);
            const cplx<double> e1 = pick(v1[0], v1[1], v1[2], r), e01 = pick(v01[0], v01[1], v01[2], r);
            cand[b][0][lane] = make_double2(e.re, e.im);
            cand[b][1][lane] = make_double2(e0.re, e0.im);
            cand[b][2][lane] = make_double2(e1.re, e1.im);
            cand[b][3][lane] = make_double2(e01.re, e01.im);
            ymat[b][0][lane] = make_double2(e.re - e0.re, e.im - e0.im);
            ymat[b][1][lane] = make_double2(e.re - e1.re, e.im - e1.im);
            ymat[b][2][lane] = make_double2(e0.re - e01.re, e0.im - e01.im);
        }
        __syncwarp();
    };
    // the paths of link l (kPathWarps warps): ReTr(Y P) summed over the kind's paths, P daggered
    // for plaquettes and rectangles (get_staple_dagger / get_rectangular_dagger) and not for
    // chairs and twists; a path that waits for link l - 1 goes to `tail`
    auto paths = [&](int l) {
        const int mu = l & 3, w = warp - kPathWarp0;
        // rectangles on lanes 0..17 and plaquettes on lanes 24..29 of the first warp, 24 chairs or
        // twists in each of the others: eight lanes never hold two kinds
        const int p = w > 0 ? w * kPathsPerWarp + lane : lane < 18 ? 6 + lane : lane - 24;
        double a[3] = {0.0, 0.0, 0.0};
        if (w > 0 ? lane < kPathsPerWarp : lane < 18 || (lane >= 24 && lane < 30)) {
            const uint4 d = path[mu][p];
            const uint16_t* at = loc[(l >> 2) & 1];
            const double2* q[kSteps] = {links + at[d.x & 0xffff] * 9, links + at[d.x >> 16] * 9,
                                        links + at[d.y & 0xffff] * 9, links + at[d.y >> 16] * 9,
                                        links + at[d.z & 0xffff] * 9};
            mat3<double> m = load_oriented(q[0], d.z & 0x10000u);
#pragma unroll
            for (int i = 1; i < kSteps; i++) m = mul_2r(m, load_oriented(q[i], d.z & (0x10000u << i)));
            reconstruct_row2(m);
            if (d.w) {
                double2* o = tail[l & 1][d.w - 1];
#pragma unroll
                for (int k = 0; k < 9; k++) o[k] = make_double2(m.e[k / 3][k % 3].re, m.e[k / 3][k % 3].im);
            } else {
                double acc[3][3] = {};
#pragma unroll
                for (int k = 0; k < 9; k++) {
                    cplx<double> e;
                    e.re = w == 0 ? m.e[k / 3][k % 3].re : m.e[k % 3][k / 3].re;
                    e.im = w == 0 ? m.e[k / 3][k % 3].im : -m.e[k % 3][k / 3].im;
#pragma unroll
                    for (int G = 0; G < 3; G++) {
                        const double2 y = ymat[l % 3][G][k];
                        acc[G][k % 3] = fma(y.y, e.im, fma(y.x, e.re, acc[G][k % 3]));
                    }
                }
#pragma unroll
                for (int G = 0; G < 3; G++) a[G] = (acc[G][0] + acc[G][1]) + acc[G][2];
            }
        }
#pragma unroll
        for (int o = 4; o; o >>= 1)
#pragma unroll
            for (int G = 0; G < 3; G++) a[G] += __shfl_xor_sync(0xffffffffu, a[G], o);
        if ((lane & 7) == 0)
#pragma unroll
            for (int G = 0; G < 3; G++) psum[l & 1][w][lane >> 3][G] = a[G];
    };
    // the two hits of link l (one warp)
    auto hits = [&](int l) {
        const int s = l >> 2, mu = l & 3, b = l % 3;
        // sums R of the waiting paths by kind: lanes 0..26 an element of rectangles, chairs or
        // twists each, then lanes 0..8 of the one plaquette
        {
            const int k = 1 + lane / 9, e = lane % 9;
            cplx<double> R[3];
#pragma unroll
            for (int x = 0; x < 3; x++) R[x] = mk(0.0, 0.0);
            if (lane < 27) {
                const int f0 = sfirst[mu][k], f1 = sfirst[mu][k + 1];
#pragma unroll
                for (int i = 0; i < 12; i++)
                    if (f0 + i < f1) {
                        const double2 v = tail[l & 1][f0 + i][e];
                        R[i % 3].re += v.x;
                        R[i % 3].im += v.y;
                    }
                late[k][e] = make_double2((R[0].re + R[1].re) + R[2].re, (R[0].im + R[1].im) + R[2].im);
            }
            if (lane < 9) late[0][lane] = sfirst[mu][1] > 0 ? tail[l & 1][0][lane] : make_double2(0.0, 0.0);
        }
        // the link they wait for, u: U_(mu-1)(x), or the rectangle's first two links when mu = 0
        const double2* u = site_link(s, (mu + 3) & 3);
        if (mu == 0) {
            const double2* lp = links + loc[s & 1][lslot] * 9;
            const double2* up = links + loc[s & 1][uslot] * 9;
            if (lane < 9) {
                cplx<double> o = mk(0.0, 0.0);
#pragma unroll
                for (int x = 0; x < 3; x++)
                    cmac<false, false, false>(o, oriented(lp, lfwd, lane / 3, x), oriented(up, ufwd, x, lane % 3));
                lu[lane] = make_double2(o.re, o.im);
            }
            u = lu;
            __syncwarp();
        }
        // u^+ Y for the daggered kinds, Y u for the others
#pragma unroll
        for (int round = 0; round < 2; round++) {
            const int j = lane + 32 * round;
            if (j < 54) {
                const int h = j / 27, G = (j % 27) / 9, r = (j % 9) / 3, c = j % 3;
                const double2* y = ymat[b][G];
                const double2* pa = h ? y + 3 * r : u + r;
                const double2* pb = h ? u + c : y + c;
                cplx<double> o = mk(0.0, 0.0);
#pragma unroll
                for (int x = 0; x < 3; x++) {
                    const double2 va = pa[h ? x : 3 * x], vb = pb[3 * x];
                    cmac<false, false, false>(o, mk(va.x, h ? va.y : -va.y), mk(vb.x, vb.y));
                }
                yu[h][G][3 * r + c] = make_double2(o.re, o.im);
            }
        }
        __syncwarp();
        // lane 4 G + k: demon k; G = 0 the first hit, G = 1 the second after a rejected first,
        // G = 2 the second after an accepted first (ReTr(v S) - ReTr(m v S), field-demon.h:75-78)
        const int G = lane < 12 ? lane >> 2 : 0, k = lane & 3;
        double d[3] = {0.0, 0.0, 0.0}, rest[3] = {0.0, 0.0, 0.0};
#pragma unroll
        for (int e = 0; e < 9; e++) {
            const double2 y = yu[k >> 1][G][e];
            const double2 v = late[k][k < 2 ? e : 3 * (e % 3) + e / 3];
            d[e % 3] = fma(y.x, v.x, d[e % 3]);
            d[e % 3] = fma(k < 2 ? y.y : -y.y, v.y, d[e % 3]);
        }
        // eight-lane sums: 3 of the first warp are rectangles, its fourth the plaquettes; chairs
        // and twists have three warps each
        const double(*ps)[4][3] = psum[l & 1] + (k < 2 ? 0 : 3 * k - 5);
#pragma unroll
        for (int i = 0; i < 9; i++)
            if (k >= 2 || (k == 1 && i < 3)) rest[i % 3] += ps[i / 3][i % 3][G];
        if (k == 0) rest[0] = ps[0][3][G];
        const double dS = ((rest[0] + rest[1]) + rest[2]) + ((d[0] + d[1]) + d[2]);
        const double first = E - __shfl_sync(0xffffffffu, dS, k);  // the demon after an accepted first hit
        const double after = (G == 2 ? first : E) - dS;
        const unsigned in = __ballot_sync(0xffffffffu, after > -e_max && after < e_max);
        const bool ok0 = (in & 0xfu) == 0xfu;
        const bool ok1 = ((in >> (ok0 ? 8 : 4)) & 0xfu) == 0xfu;
        const double moved = __shfl_sync(0xffffffffu, after, k + (ok1 ? (ok0 ? 8 : 4) : 0));
        if (ok0 || ok1) {
            E = moved;
            if (lane < 9) {
                const double2 o = cand[b][(ok0 ? 1 : 0) + (ok1 ? 2 : 0)][lane];
                site_link(s, mu)[lane] = o;
                U[((size_t)s * 4 + mu) * 9 + lane] = o;
            }
        }
        acc += (ok0 ? 1 : 0) + (ok1 ? 1 : 0);
        rej += (ok0 ? 0 : 1) + (ok1 ? 0 : 1);
        __syncwarp();
    };

    stage_site(0, -1, 0, kDemonThreads / 32);
    __syncthreads();
    const int nlink = 4 * nsite;
    if (warp == kPrepareWarp) prepare(0);
    __syncthreads();
    for (int l = 0; l <= nlink; l++) {
        if (warp == kHitWarp) {
            if (l > 0) hits(l - 1);
        } else if (warp == kPrepareWarp) {
            if (l + 1 < nlink) prepare(l + 1);
        } else if (warp >= kStageWarp0) {
            const int s = (l >> 2) + 1;
            if (s < nsite) stage_site(s, l & 3, kStageWarp0, kStageWarps);
        }
        if (!ahead) __syncthreads();
        if (warp >= kPathWarp0 && warp < kStageWarp0 && l < nlink) paths(l);
        __syncthreads();
    }
    if (warp == kHitWarp && lane < 4) {
        st->E[lane] = E;
        if (lane == 0) {
            st->accept += acc;
            st->reject += rej;
        }
    }
}

// the staple paths of a link in direction mu in the reference's order: plaquette staples
// (field-hmc.h:228-239), rectangles (:142-198), chairs and twists (field-staple.h:27-120);
// 0-3 forward, 4-7 backward, -1 pads the three-link paths
void demon_paths(int8_t out[4][kPaths][kSteps]) {
    for (int mu = 0; mu < 4; mu++) {
        int p = 0;
        auto put = [&](std::initializer_list<int> d) {
            int i = 0;
            for (int v : d) out[mu][p][i++] = (int8_t)v;
            for (; i < kSteps; i++) out[mu][p][i] = -1;
            p++;
        };
        for (int nu = 0; nu < 4; nu++) {
            if (nu == mu) continue;
            put({nu, mu, nu + 4});
            put({nu + 4, mu, nu});
        }
        for (int nu = 0; nu < 4; nu++) {
            if (nu == mu) continue;
            put({nu, mu, mu, nu + 4, mu + 4});
            put({nu + 4, mu, mu, nu, mu + 4});
            put({nu, nu, mu, nu + 4, nu + 4});
            put({nu + 4, nu + 4, mu, nu, nu});
            put({mu + 4, nu, mu, mu, nu + 4});
            put({mu + 4, nu + 4, mu, mu, nu});
        }
        for (int twist = 0; twist < 2; twist++)
            for (int nu = 0; nu < 4; nu++) {
                if (nu == mu) continue;
                for (int la = 0; la < 4; la++) {
                    if (la == nu || la == mu) continue;
                    const int chair[4][4] = {{nu, la, la + 4, nu + 4}, {nu, la + 4, la + 4, nu},
                                             {nu + 4, la, la, nu + 4}, {nu + 4, la + 4, la, nu}};
                    const int tw[4][4] = {{nu, la, nu + 4, la + 4}, {nu, la + 4, nu + 4, la},
                                          {nu + 4, la, nu, la + 4}, {nu + 4, la + 4, nu, la}};
                    for (int b = 0; b < 4; b++)
                        for (int ins = 1; ins < 4; ins++) {
                            const int* base = twist ? tw[b] : chair[b];
                            int d[5], k = 0;
                            for (int i = 0; i < 4; i++) {
                                if (i == ins) d[k++] = mu;
                                d[k++] = base[i];
                            }
                            put({d[0], d[1], d[2], d[3], d[4]});
                        }
                }
            }
    }
}

}  // namespace

bool build_demon_tables(DemonTables* T) {
    std::memset(T, 0, sizeof(*T));
    int8_t paths[4][kPaths][kSteps];
    demon_paths(paths);
    // the distinct (site offset, direction) pairs over the four directions, and the unit matrix
    // (direction 4) that pads the three-link paths
    std::vector<int> keys;
    auto key_of = [&](const int y[4], int d) {
        const int key = ((y[0] + 4) & 15) | (((y[1] + 4) & 15) << 4) | (((y[2] + 4) & 15) << 8) |
                        (((y[3] + 4) & 15) << 12) | (d << 16);
        for (size_t k = 0; k < keys.size(); k++)
            if (keys[k] == key) return (int)k;
        keys.push_back(key);
        return (int)keys.size() - 1;
    };
    const int zero[4] = {0, 0, 0, 0}, before[4] = {-1, 0, 0, 0};
    const int unit = key_of(zero, 4);
    int lkey = -1, ukey = -1;
    for (int mu = 0; mu < 4; mu++) {
        // the link updated before this one, and the step at which paths meet it
        const int prev = mu > 0 ? key_of(zero, mu - 1) : key_of(before, 3), meets = mu > 0 ? 0 : 1;
        int n = 0;
        for (int p = 0; p < kPaths; p++) {
            if (p == 0 || p == 6 || p == 24 || p == 96) T->first[mu][p == 0 ? 0 : p == 6 ? 1 : p == 24 ? 2 : 3] = (int8_t)n;
            int y[4] = {0, 0, 0, 0}, key[kSteps];
            T->late[mu][p] = -1;
            for (int i = 0; i < kSteps; i++) {
                const int d = paths[mu][p][i];
                T->fwd[mu][p][i] = d < 4;
                key[i] = unit;
                if (d < 0) continue;
                const int a = d & 3;
                if (d >= 4) y[a]--;
                if (y[a] < -2 || y[a] > 2) return false;
                key[i] = key_of(y, a);
                if (d < 4) y[a]++;
                if (key[i] == prev) {
                    if (i != meets || T->late[mu][p] >= 0 || n >= kDemonLate) return false;
                    T->late[mu][p] = (int8_t)n++;
                }
            }
            if (T->late[mu][p] >= 0) {
                if (mu == 0) {
                    if (n > 1 || p < 6 || p >= 24) return false;
                    lkey = key[0];
                    T->lfwd = T->fwd[mu][p][0];
                    ukey = key[1];
                    T->ufwd = T->fwd[mu][p][1];
                } else if (!T->fwd[mu][p][0]) {
                    return false;
                }
                for (int i = 0; i <= meets; i++) {
                    key[i] = unit;
                    T->fwd[mu][p][i] = 1;
                }
            }
            for (int i = 0; i < kSteps; i++) T->slot[mu][p][i] = (uint16_t)key[i];
        }
        T->first[mu][4] = (int8_t)n;
    }
    // Slots: 16-byte loads are served for eight threads at a time, and the bank group of element e
    // of a link is (slot + e) % 8; two links that a group reads the same way meet in all nine
    // elements when their slots agree modulo 8, a link and an adjoint (element 3 c + r against
    // 3 r + c) in three of them, and in two when the slots differ by 2, 4 or 6.  Greedy choice of
    // slot % 8, most used link first, then passes that move a link to where it meets fewer
    const int nkey = (int)keys.size();
    using Read = std::pair<int, int>;  // link, orientation
    std::vector<std::vector<Read>> groups;
    std::vector<std::vector<std::pair<int, int>>> member(nkey);  // group, orientation
    for (int mu = 0; mu < 4; mu++)
        for (int i = 0; i < kSteps; i++)
            for (int p0 = 0, p1; p0 < kPaths; p0 = p1) {
                // the eight-lane groups: plaquettes, 8 + 8 + 2 rectangles, eights of the others
                p1 = p0 == 0 ? 6 : p0 == 22 ? 24 : p0 + 8;
                std::vector<Read> g;
                for (int p = p0; p < p1; p++) {
                    const Read k{T->slot[mu][p][i], T->fwd[mu][p][i]};
                    if (std::find(g.begin(), g.end(), k) == g.end()) g.push_back(k);
                }
                for (const Read& k : g) member[k.first].push_back({(int)groups.size(), k.second});
                groups.push_back(g);
            }
    std::vector<int> order(nkey), res(nkey, -1);
    int used[8] = {0};
    for (int k = 0; k < nkey; k++) order[k] = k;
    std::stable_sort(order.begin(), order.end(), [&](int a, int b) { return member[a].size() > member[b].size(); });
    for (int pass = 0; pass < 8; pass++)
        for (int k : order) {
            if (res[k] >= 0) used[res[k]]--;
            int cost[8] = {0};
            for (const auto& g : member[k])
                for (const Read& o : groups[g.first])
                    if (o.first != k && res[o.first] >= 0) {
                        const int at = res[o.first];
                        if (o.second == g.second) {
                            cost[at] += 9;
                        } else {
                            cost[at] += 3;
                            for (int d = 2; d < 8; d += 2) cost[(at + d) & 7] += 2;
                        }
                    }
            int best = -1;
            for (int r = 0; r < 8; r++)
                if (used[r] < kDemonWindow / 8 && (best < 0 || cost[r] < cost[best])) best = r;
            if (best < 0) return false;
            res[k] = best;
            used[best]++;
        }
    std::vector<int> slot(nkey);
    int count[8] = {0};
    for (int n = 0; n < kDemonWindow; n++) T->packed[n] = keys[unit];  // slots without a link
    for (int k = 0; k < nkey; k++) {
        slot[k] = res[k] + 8 * count[res[k]]++;
        T->packed[slot[k]] = keys[k];
        T->nslot = std::max(T->nslot, slot[k] + 1);
    }
    for (int mu = 0; mu < 4; mu++)
        for (int p = 0; p < kPaths; p++)
            for (int i = 0; i < kSteps; i++) T->slot[mu][p][i] = (uint16_t)slot[T->slot[mu][p][i]];
    if (lkey < 0) return false;
    T->lslot = slot[lkey];
    T->uslot = slot[ukey];
    return true;
}

void launch_demon_sweeps(const DemonJob* jobs, int njobs, double* aos, const DemonTables* tabs, int sweep,
                         double e_max, DemonState* states, cudaStream_t s) {
    cudaFuncSetAttribute(k_demon_sweep, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kDemonDynSmem);
    k_demon_sweep<<<(unsigned)njobs, kDemonThreads, kDemonDynSmem, s>>>(jobs, reinterpret_cast<double2*>(aos), tabs,
                                                                        sweep, e_max, states);
}

}  // namespace magb
