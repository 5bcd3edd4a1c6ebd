// kernels_smear.cu -- stout smearing and its derivative on plaquettes (plaq_ops.cuh).
//
// A level is two launches, forward and backward alike: one over plaquettes (a block
// of six warps holds the six planes of a 32-site tile), whose results go to memory
// as algebra elements, and one over links, which adds up the terms of its six
// plaquettes (three at the site, three at x - nu) and does the rest of the level.
//
// Backward, per link and level: about 1450 multiply-adds instead of 3456 in the
// one-thread-per-link chain rule and 156 instead of 450 loaded reals, because a
// plaquette is formed once for its four links; the price is 1.8 KB per site (FP64)
// of intermediate results.  Measured at 32^4 (ms per launch): chain rule + Lambda
// 1.65 + 0.57 FP64, 0.69 + 0.24 FP32 before; k_plaq_chain + k_chain_gather 0.72 +
// 0.31 FP64, 0.36 + 0.16 FP32 at the power cap of a run (k_plaq_chain 0.59 by itself at
// full clock).  k_chain_gather moves 1.7 KB per site at 0.9 of the HBM rate (5.8 TB/s in
// FP64); k_plaq_chain keeps the FP64 pipe 61% busy at 12 warps per SM.
#include "kernels.h"
#include "plaq_ops.cuh"

namespace magb {

namespace {

constexpr int kPlaqBlock = 6 * MAG_TILE;
constexpr int kLinkBlock = 4 * MAG_TILE;

// plane of warp w: (0,1) (0,2) (0,3) (1,2) (1,3) (2,3)
__device__ __forceinline__ void plane_of(int w, int& p, int& q) {
    p = w < 3 ? 0 : w < 5 ? 1 : 2;
    q = w < 3 ? w + 1 : w < 5 ? w - 1 : 3;
}
// index of the plane of directions i != j
__device__ __forceinline__ int plane_index(int i, int j) {
    const int p = i < j ? i : j, q = i < j ? j : i;
    return p == 0 ? q - 1 : p + q;
}

__device__ __forceinline__ bool locate_tile(const DevGeom& g, ChainInfo& ci, Site& st) {
    const int gs = blockIdx.x * MAG_TILE + (threadIdx.x & 31);
    ci = g.nchain == 1 ? g.one : g.chains[g.c2c[gs / MAG_CHUNK]];
    const int s = gs - ci.off;
    if (s >= ci.V) return false;
    decode(ci, s, st);
    return true;
}

// The twelve (link, plane) terms of the tile's links that start at its own sites:
// slot 3 mu + i for the link in direction mu and its i-th other direction.  A thread
// writes the two slots of its plane; the block adds the three slots of each link.
template <typename T>
struct site_terms {
    static constexpr int kPieces = AlgPlanes<T>::kPieces, kPer = AlgPlanes<T>::kPer;
    alg_piece<T> v[12][kPieces][MAG_TILE];
    __device__ __forceinline__ void put(int i, int lane, const herm8<T>& h) {
#pragma unroll
        for (int j = 0; j < kPieces; j++)
#pragma unroll
            for (int k = 0; k < kPer; k++) v[i][j][lane].v[k] = h.h[j * kPer + k];
    }
    __device__ __forceinline__ herm8<T> get(int i, int lane) const {
        herm8<T> h;
#pragma unroll
        for (int j = 0; j < kPieces; j++)
#pragma unroll
            for (int k = 0; k < kPer; k++) h.h[j * kPer + k] = v[i][j][lane].v[k];
        return h;
    }
    // after a barrier: the sums of the four links, shared out over the six warps
    __device__ __forceinline__ void sum_links(const AlgPlanes<T>& Loc, int g, int w, int lane) const {
        for (int r = w; r < 4 * kPieces; r += 6) {
            const int mu = r / kPieces, j = r - mu * kPieces;
            alg_piece<T> a = v[3 * mu][j][lane];
            const alg_piece<T> b = v[3 * mu + 1][j][lane], c = v[3 * mu + 2][j][lane];
#pragma unroll
            for (int k = 0; k < kPer; k++) a.v[k] = (a.v[k] + b.v[k]) + c.v[k];
            const_cast<alg_piece<T>*>(Loc.at(mu, g))[j * MAG_TILE] = a;
        }
    }
};

// S = (P - P^dag) / 2i of every plaquette (plane fields 0..5 of S)
template <typename T>
__global__ void __launch_bounds__(kPlaqBlock, sizeof(T) == 8 ? 4 : 3) k_plaq_sin(DevGeom g, LinkPlanes<T> U, AlgPlanes<T> S) {
    after_previous();
    ChainInfo ci;
    Site st;
    if (!locate_tile(g, ci, st)) return;
    const int w = threadIdx.x >> 5;
    int p, q;
    plane_of(w, p, q);
    const int gp = nb_sel(ci, st, p, 1), gq = nb_sel(ci, st, q, 1);
    S.store(w, st.g, herm_convert<T>(plaq_sin(plaquette_wide(U, st.g, gp, gq, p, q), 1.0)));
}

// -i TA(stp U^dag) of link (x, mu), stp its six staples, from the plaquettes at x and x - nu
template <typename T>
__device__ __forceinline__ herm8<T> staple_angle(const LinkPlanes<T>& U, const AlgPlanes<T>& S, const ChainInfo& ci,
                                                 const Site& st, int mu) {
    herm8<T> sum = herm_zero<T>();
#pragma unroll
    for (int i = 0; i < 3; i++) {
        const int nu = i + (i >= mu ? 1 : 0), w = plane_index(mu, nu), gm = nb_sel(ci, st, nu, -1);
        const T sign = mu < nu ? T(-1) : T(1);
        const herm8<T> y = transport_dn(U.load(nu, gm), S.load(w, gm));
        const herm8<T> up = S.load(w, st.g);
#pragma unroll
        for (int k = 0; k < 8; k++) sum.h[k] = fmaT(sign, up.h[k] - y.h[k], sum.h[k]);
    }
    return sum;
}

// Q = -i rho TA(stp U^dag) (field-multi.h:32-39), U' = e^{iQ} U.  Q is kept for the derivative
// where the caller gives a place for it; without, 256 of 1792 B per site and level less go to
// memory, which bounds it (Hamiltonian of 24^3 x 48 with three levels 1.80 -> 1.72 ms)
__global__ void __launch_bounds__(kLinkBlock, 5) k_stout_apply(DevGeom g, LinkPlanes<double> U, AlgPlanes<double> S,
                                                            LinkPlanes<double> Uout, AlgPlanes<double> Q) {
    after_previous();
    ChainInfo ci;
    Site st;
    if (!locate_tile(g, ci, st)) return;
    const int mu = threadIdx.x >> 5;
    const herm8<double> q = scaled(staple_angle(U, S, ci, st, mu), ci.rho);
    if (Q.p) Q.store(mu, st.g, q);
    Uout.store(mu, st.g, exp_times(q, U.load(mu, st.g)));
}

// Wilson force F = i beta/3 TA(U A^dag), A the plaquette staples (field-hmc.h:394-421)
template <typename T>
__global__ void __launch_bounds__(kLinkBlock) k_wilson_force(DevGeom g, LinkPlanes<T> U, AlgPlanes<T> S,
                                                             AlgPlanes<T> F) {
    after_previous();
    ChainInfo ci;
    Site st;
    if (!locate_tile(g, ci, st)) return;
    const int mu = threadIdx.x >> 5;
    F.store(mu, st.g, scaled(staple_angle(U, S, ci, st, mu), (T)(ci.beta / 3.0)));
}

// rows 0, 1 of every plaquette (plane fields 0..5 of Pl)
template <typename T>
__global__ void __launch_bounds__(kPlaqBlock, sizeof(T) == 8 ? 2 : 4) k_plaq(DevGeom g, LinkPlanes<T> U, RowPlanes<T> Pl) {
    after_previous();
    ChainInfo ci;
    Site st;
    if (!locate_tile(g, ci, st)) return;
    const int w = threadIdx.x >> 5;
    int p, q;
    plane_of(w, p, q);
    Pl.store(w, st.g, convert<T>(plaquette_wide(U, st.g, nb_sel(ci, st, p, 1), nb_sel(ci, st, q, 1), p, q)));
}

// Iwasaki force i TA(U A^dag) without its beta/3, A = c0 staples + c1 rectangles
// (field-hmc.h:142-198, 226-269), as the loops through each plaquette P: the 1x2
// rectangles that contain P are its products with the plaquette across each of its
// four sides,
//   A P,  A = a P(x+p) a^dag           (b is not on it)
//   P B,  B = a-^dag P(x-p) a-,  a- = U_p(x-p)  (d is not on it)
//   P D,  D = d P(x+q) d^dag           (c is not on it)
//   E P,  E = d-^dag P(x-q) d-,  d- = U_q(x-q)  (a is not on it).
// A link's term is the (L - L^dag) / 2i of its loops, moved to the link's start along
// the loop: b's start along a (E P, which does not hold a, is P E there) and c's along
// d (P B is B P), P E = P (E P) P^dag and B P = P^dag (P B) P.  With R the weighted
// (L - L^dag) / 2i of the four products and R0 that of P
//   a: -(R0 + RA + RB + RD),                  d: R0 + RA + RD + RE,
//   b: -a^dag (R0 + RB + RD + P RE P^dag) a,  c: d^dag (R0 + RA + RE + P^dag RB P) d.
// Every rectangle is formed twice (from each of its plaquettes) instead of six times,
// from nine matrices read instead of 24 per direction.  Loc and Rem as in k_plaq_chain.
template <typename T, int MINB>
__global__ void __launch_bounds__(kPlaqBlock, MINB) k_plaq_rect(DevGeom g, LinkPlanes<T> U, RowPlanes<T> Pl,
                                                                AlgPlanes<T> Loc, AlgPlanes<T> Rem) {
    after_previous();
    __shared__ site_terms<T> sm;
    ChainInfo ci;
    Site st;
    const bool ok = locate_tile(g, ci, st);
    const int w = threadIdx.x >> 5, lane = threadIdx.x & 31;
    if (ok) {
        int p, q;
        plane_of(w, p, q);
        const int ip = 3 * p + q - 1, iq = 3 * q + p;
        const T k0 = (T)ci.c0, k1 = (T)ci.c1;
        // operands are loaded again for each use (L1) instead of staying in registers, unless
        // the block has an SM's registers to itself
        auto fresh = []() {
            if (MINB > 1) asm volatile("" ::: "memory");
        };
        // the rectangles' terms are added up before R0, which is ten times their size
        herm8<T> lb, lc, t, u;
        {
            const int gm = nb_sel(ci, st, q, -1);
            mat3<T> x = mul_dn_2r(U.load_cols01(q, gm), Pl.load(w, gm));
            x = mul_2r(x, U.load(q, gm));
            const mat3<T> P = Pl.load(w, st.g);
            lc = plaq_sin(mul_su3(x, P), k1);  // RE
            sm.put(iq, lane, lc);
            lb = transport_nd(P, lc);
            t = plaq_sin(P, k0);  // R0
        }
        fresh();
        {
            const int gm = nb_sel(ci, st, p, -1);
            mat3<T> x = mul_nd_2r(Pl.load_rows01(w, st.g), U.load(p, gm));
            x = mul_2r(x, Pl.load(w, gm));
            const herm8<T> r = plaq_sin(mul_su3(x, U.load(p, gm)), k1);  // RB
            sm.put(ip, lane, r);
            herm_add(lb, r);
            herm_add(lc, transport_dn(Pl.load(w, st.g), r));
        }
        fresh();
        {
            mat3<T> x = mul_2r(U.load_rows01(p, st.g), Pl.load(w, nb_sel(ci, st, p, 1)));
            x = mul_nd_2r(x, U.load(p, st.g));
            u = plaq_sin(mul_su3(x, Pl.load(w, st.g)), k1);  // RA
            herm_add(lc, u);
        }
        herm_add(lc, t);
        fresh();
        Rem.store(ip, st.g, transport_dn(U.load(q, st.g), lc));
        {
            mat3<T> x = mul_2r(Pl.load_rows01(w, st.g), U.load(q, st.g));
            x = mul_2r(x, Pl.load(w, nb_sel(ci, st, q, 1)));
            const herm8<T> r = plaq_sin(mul_nd_su3(x, U.load(q, st.g)), k1);  // RD
            herm_add(lb, r);
            herm_add(u, r);
        }
        herm_add(lb, t);
        fresh();
#pragma unroll
        for (int k = 0; k < 8; k++) lb.h[k] = -lb.h[k];
        Rem.store(iq, st.g, transport_dn(U.load(p, st.g), lb));
        herm8<T> y = sm.get(ip, lane);
#pragma unroll
        for (int k = 0; k < 8; k++) y.h[k] = -t.h[k] - (u.h[k] + y.h[k]);
        sm.put(ip, lane, y);
        herm_add(u, sm.get(iq, lane));
        herm_add(t, u);
        sm.put(iq, lane, t);
    }
    __syncthreads();
    if (ok) sm.sum_links(Loc, st.g, w, lane);
}

// The Wilson action's derivative with respect to the smeared top links and Lambda and Dir of the
// top level.  With the derivative written and read between two kernels a force took (us) 29.1
// instead of 27.1 at 8^4 FP64 with one level, 62.2 instead of 59 at 6 x 10 x 14 x 9 with two,
// 2130 instead of 2035 at 32^4 with one, 36.6 instead of 33.8 at 12^4 mixed.
template <typename T>
__global__ void __launch_bounds__(kLinkBlock) k_wilson_lambda(DevGeom g, LinkPlanes<T> U, AlgPlanes<T> S,
                                                              AlgPlanes<T> Q, AlgPlanes<T> Lam, AlgPlanes<T> Dir) {
    after_previous();
    ChainInfo ci;
    Site st;
    if (!locate_tile(g, ci, st)) return;
    const int mu = threadIdx.x >> 5;
    const herm8<T> x = scaled(staple_angle(U, S, ci, st, mu), (T)(ci.beta / 3.0));
    herm8<T> lam, dir;
    lambda_adjoint(Q.load(mu, st.g), x, lam, dir);
    Lam.store(mu, st.g, lam);
    Dir.store(mu, st.g, dir);
}

// Chain rule over the plaquettes.  The variation of rho Tr(M S), M = Lambda_d -
// Lambda_a + D - A with A = a Lambda_b a^dag, D = d Lambda_c d^dag (the plaquette's
// part of sum Tr(Lambda dQ): Q_a = -rho S, Q_d = rho S, Q_b = -rho a^dag S a,
// Q_c = rho d^dag S d), with respect to the four links is
//   y_a = G+ + i [S, A],  y_d = G- - i [S, D],  y_b = a^dag G+ a,  y_c = d^dag G- d,
//   G+- = +-{C, M} / 2 + i [S, M] / 2,  C = (P + P^dag) / 2.
// y_a and y_d, summed over the planes through shared memory, go to Loc; y_b and y_c
// belong to the links (x+p, q) and (x+q, p) and go to the plane fields Rem[3 link + i]
// at x, i = the plane's other direction counted without the link's own.
template <typename T, int MINB>
__global__ void __launch_bounds__(kPlaqBlock, MINB) k_plaq_chain(DevGeom g, LinkPlanes<T> U, AlgPlanes<T> Lam,
                                                                 AlgPlanes<T> Loc, AlgPlanes<T> Rem) {
    after_previous();
    __shared__ site_terms<T> sm;
    ChainInfo ci;
    Site st;
    const bool ok = locate_tile(g, ci, st);
    const int w = threadIdx.x >> 5, lane = threadIdx.x & 31;
    if (ok) {
        int p, q;
        plane_of(w, p, q);
        const int gp = nb_sel(ci, st, p, 1), gq = nb_sel(ci, st, q, 1);
        const int ip = 3 * p + q - 1, iq = 3 * q + p;
        // the thread's two slots hold A and D until y_a and y_d replace them
        // a and d are loaded again (L1) for each use instead of staying in registers, unless
        // the block has an SM's registers to itself
        auto link = [&](int d) {
            if (MINB > 1) asm volatile("" ::: "memory");
            return U.load(d, st.g);
        };
        const mat3<T> P =
            plaquette(U.load_rows01(p, st.g), U.load(q, gp), U.load(p, gq), U.load_rows01(q, st.g));
        const herm8<T> S = plaq_sin(P, (T)ci.rho);
        const herm9<T> C = plaq_cos(P, (T)ci.rho);
        herm8<T> M = transport_nd(link(q), Lam.load(p, gq));
        sm.put(iq, lane, M);
        {
            const herm8<T> A = transport_nd(link(p), Lam.load(q, gp));
            sm.put(ip, lane, A);
            herm_sub(M, A);
        }
        herm_add(M, Lam.load(q, st.g));
        herm_sub(M, Lam.load(p, st.g));
        const herm8<T> anti = anticomm_half(C, M);
        herm8<T> gm = comm_i(S, M);
#pragma unroll
        for (int k = 0; k < 8; k++) gm.h[k] *= T(0.5);
        herm8<T> gpl = gm;
        herm_add(gpl, anti);
        herm_sub(gm, anti);
        asm volatile("" ::: "memory");
        herm8<T> y = comm_i(S, sm.get(ip, lane));
        herm_add(y, gpl);
        sm.put(ip, lane, y);
        y = gm;
        herm_sub(y, comm_i(S, sm.get(iq, lane)));
        sm.put(iq, lane, y);
        Rem.store(iq, st.g, transport_dn(link(p), gpl));
        Rem.store(ip, st.g, transport_dn(link(q), gm));
    }
    __syncthreads();
    if (ok) sm.sum_links(Loc, st.g, w, lane);
}

// Loc(x) + sum_nu Rem(x - nu) (+ Dir unless TOP, times beta/3 if TOP): the derivative
// with respect to a level's link (TOP: the gauge force of the top links)
template <typename T, bool TOP>
__device__ __forceinline__ herm8<T> gathered(const AlgPlanes<T>& Loc, const AlgPlanes<T>& Rem, const AlgPlanes<T>& Dir,
                                             const ChainInfo& ci, const Site& st, int mu) {
    herm8<T> x = Loc.load(mu, st.g);
    herm8<T> d = herm_zero<T>();
    if (!TOP) d = Dir.load(mu, st.g);
    herm8<T> r[3];
#pragma unroll
    for (int i = 0; i < 3; i++) {
        const int nu = i + (i >= mu ? 1 : 0);
        r[i] = Rem.load(3 * mu + i, nb_sel(ci, st, nu, -1));
    }
    // in double: the terms are of one size and an FP32 addition's rounding is as large as theirs;
    // bound by memory, the kernels take no longer
#pragma unroll
    for (int k = 0; k < 8; k++) {
        double a = (double)x.h[k];
        if (!TOP) a += (double)d.h[k];
        a = ((a + (double)r[0].h[k]) + (double)r[1].h[k]) + (double)r[2].h[k];
        if (TOP) a *= ci.beta / 3.0;
        x.h[k] = (T)a;
    }
    return x;
}

// Lambda and Dir of the level below from the gathered derivative
template <typename T, bool TOP>
__global__ void __launch_bounds__(kLinkBlock) k_chain_gather(DevGeom g, AlgPlanes<T> Loc, AlgPlanes<T> Rem,
                                                             AlgPlanes<T> Dir, AlgPlanes<T> Q, AlgPlanes<T> Lam) {
    after_previous();
    ChainInfo ci;
    Site st;
    if (!locate_tile(g, ci, st)) return;
    const int mu = threadIdx.x >> 5;
    const herm8<T> x = gathered<T, TOP>(Loc, Rem, Dir, ci, st, mu);
    herm8<T> lam, dir;
    lambda_adjoint(Q.load(mu, st.g), x, lam, dir);
    Lam.store(mu, st.g, lam);
    Dir.store(mu, st.g, dir);
}

// the site one step along d (k = 1 or -1)
__device__ __forceinline__ Site step_site(const ChainInfo& ci, const Site& st, int d, int k) {
    Site n = st;
    n.g = nb_sel(ci, st, d, k);
#pragma unroll
    for (int e = 0; e < 4; e++) {
        if (e != d) continue;
        const int w = st.x[e] + k;
        n.x[e] = w < 0 ? w + ci.L[e] : w >= ci.L[e] ? w - ci.L[e] : w;
    }
    return n;
}

// The force of a thin link from its free-link force x.  Constrained segments
// (field-hmc.h:399-407): the last link's force is zero, every other link's is
// F(x + mu) - U^dag F(x) U of the free-link forces (the next link's is gathered again).
template <typename T, bool TOP>
__device__ __forceinline__ herm8<T> constrained(herm8<T> x, int cc, const LinkPlanes<T>& U, const AlgPlanes<T>& Loc,
                                                const AlgPlanes<T>& Rem, const AlgPlanes<T>& Dir, const ChainInfo& ci,
                                                const Site& st, int mu) {
    if (cc == 100) return herm_zero<T>();
    if (cc == 0) return x;
    herm8<T> y = gathered<T, TOP>(Loc, Rem, Dir, ci, step_site(ci, st, mu, 1), mu);
    herm_sub(y, transport_dn(U.load(mu, st.g), x));
    return y;
}

// The force of the thin links; KICK: P += eps F (field-hmc.h:427-440) without storing F
template <typename T, bool TOP, bool KICK>
__global__ void __launch_bounds__(kLinkBlock) k_force_gather(DevGeom g, LinkPlanes<T> U, AlgPlanes<T> Loc,
                                                             AlgPlanes<T> Rem, AlgPlanes<T> Dir, AlgPlanes<T> F,
                                                             AlgPlanes<double> P, double eps) {
    after_previous();
    ChainInfo ci;
    Site st;
    if (!locate_tile(g, ci, st)) return;
    const int mu = threadIdx.x >> 5;
    const herm8<T> x = constrained<T, TOP>(gathered<T, TOP>(Loc, Rem, Dir, ci, st, mu), constraint_case(ci, st, mu), U,
                                           Loc, Rem, Dir, ci, st, mu);
    if (KICK) {
        herm8<double> p = P.load(mu, st.g);
#pragma unroll
        for (int k = 0; k < 8; k++) p.h[k] += (double)x.h[k] * eps;
        P.store(mu, st.g, p);
    } else {
        F.store(mu, st.g, x);
    }
}

// The force-gradient step's links U' = e^{i eps F} U with the constraint rules
// (field-hmc.h:497-503), F as in k_force_gather but not stored: a segment's link that
// moves with the one before it forms that link's force too.  Apart (force, then link
// update) an 8^4 trajectory takes 0.63 instead of 0.57 ms; at 128 registers FP64 spills.
template <typename T, bool TOP>
__global__ void __launch_bounds__(kLinkBlock, sizeof(T) == 8 ? 2 : 4) k_force_evolve(DevGeom g, LinkPlanes<T> U, AlgPlanes<T> Loc,
                                                             AlgPlanes<T> Rem, AlgPlanes<T> Dir, double eps,
                                                             LinkPlanes<T> Uout) {
    after_previous();
    ChainInfo ci;
    Site st;
    if (!locate_tile(g, ci, st)) return;
    const int mu = threadIdx.x >> 5;
    const int cc = constraint_case(ci, st, mu);
    const herm8<T> x = gathered<T, TOP>(Loc, Rem, Dir, ci, st, mu);
    Uout.store(mu, st.g, evolve_link<T>(U.load(mu, st.g), eps, cc, [&](bool previous) {
                   if (!previous) return constrained<T, TOP>(x, cc, U, Loc, Rem, Dir, ci, st, mu);
                   // the link before: F = (free force here) - U^dag (its free force) U
                   const Site b = step_site(ci, st, mu, -1);
                   herm8<T> y = x;
                   herm_sub(y, transport_dn(U.load(mu, b.g), gathered<T, TOP>(Loc, Rem, Dir, ci, b, mu)));
                   return y;
               }));
}

// Up to one block per SM the FP64 plaquette kernels take the registers of two (the same
// arithmetic; no reloads, no spills): 8^4 force with one level 0.042 -> 0.035 ms; with
// more tiles than SMs two blocks per SM are faster (10 x 8^3: 0.0151 against 0.0158 ms).
constexpr unsigned kSoloTiles = 148;
unsigned tiles(const DevGeom& g) { return (unsigned)(g.vpad / MAG_TILE); }

}  // namespace

void launch_stout_level(const DevGeom& g, LinkPlanes<double> U, LinkPlanes<double> Uout, AlgPlanes<double> Q,
                        AlgPlanes<double> S, cudaStream_t s) {
    launch_after(k_plaq_sin<double>, tiles(g), kPlaqBlock, 0, s, g, U, S);
    launch_after(k_stout_apply, tiles(g), kLinkBlock, 0, s, g, U, S, Uout, Q);
}
template <typename T>
void launch_plaq_chain(const DevGeom& g, LinkPlanes<T> U, AlgPlanes<T> Lam, AlgPlanes<T> Loc, AlgPlanes<T> Rem,
                       cudaStream_t s) {
    // blocks of six warps per SM: two of FP64 (168 registers, no spills; three would spill 1 KB
    // and take 1.8 times as long), three of FP32 (96 registers; two 0.431 against 0.369 ms at 32^4)
    if constexpr (sizeof(T) == 8) {
        if (tiles(g) <= kSoloTiles) return launch_after(k_plaq_chain<T, 1>, tiles(g), kPlaqBlock, 0, s, g, U, Lam, Loc, Rem);
    }
    launch_after(k_plaq_chain<T, sizeof(T) == 8 ? 2 : 3>, tiles(g), kPlaqBlock, 0, s, g, U, Lam, Loc, Rem);
}
template <typename T>
void launch_chain_gather(const DevGeom& g, AlgPlanes<T> Loc, AlgPlanes<T> Rem, AlgPlanes<T> Dir, bool top,
                         AlgPlanes<T> Q, AlgPlanes<T> Lam, cudaStream_t s) {
    if (top) launch_after(k_chain_gather<T, true>, tiles(g), kLinkBlock, 0, s, g, Loc, Rem, Dir, Q, Lam);
    else launch_after(k_chain_gather<T, false>, tiles(g), kLinkBlock, 0, s, g, Loc, Rem, Dir, Q, Lam);
}
template <typename T>
void launch_force_gather(const DevGeom& g, LinkPlanes<T> U, AlgPlanes<T> Loc, AlgPlanes<T> Rem, AlgPlanes<T> Dir,
                         bool top, const ForceUse<T>& use, cudaStream_t s) {
#define L_(TOP, KICK)                                                                                              \
    launch_after(k_force_gather<T, TOP, KICK>, tiles(g), kLinkBlock, 0, s, g, U, Loc, Rem, Dir, use.F, use.P, use.eps)
    if (use.kind == ForceUse<T>::kEvolve) {
        if (top) launch_after(k_force_evolve<T, true>, tiles(g), kLinkBlock, 0, s, g, U, Loc, Rem, Dir, use.eps, use.Uout);
        else launch_after(k_force_evolve<T, false>, tiles(g), kLinkBlock, 0, s, g, U, Loc, Rem, Dir, use.eps, use.Uout);
    } else if (use.kind == ForceUse<T>::kKick) {
        if (top) L_(true, true);
        else L_(false, true);
    } else {
        if (top) L_(true, false);
        else L_(false, false);
    }
#undef L_
}
template <typename T>
void launch_plaq_rect(const DevGeom& g, LinkPlanes<T> U, RowPlanes<T> Pl, AlgPlanes<T> Loc, AlgPlanes<T> Rem,
                      cudaStream_t s) {
    launch_after(k_plaq<T>, tiles(g), kPlaqBlock, 0, s, g, U, Pl);
    // two blocks of six warps per SM in both precisions (three: 0.81 against 0.75 ms FP32 at 32^4,
    // twice as slow in FP64, from spills; with two FP64 spills 136 bytes at 168 registers)
    if constexpr (sizeof(T) == 8) {
        if (tiles(g) <= kSoloTiles) return launch_after(k_plaq_rect<T, 1>, tiles(g), kPlaqBlock, 0, s, g, U, Pl, Loc, Rem);
    }
    launch_after(k_plaq_rect<T, 2>, tiles(g), kPlaqBlock, 0, s, g, U, Pl, Loc, Rem);
}
template <typename T>
void launch_wilson_force(const DevGeom& g, LinkPlanes<T> U, AlgPlanes<T> S, AlgPlanes<T> F, cudaStream_t s) {
    launch_after(k_plaq_sin<T>, tiles(g), kPlaqBlock, 0, s, g, U, S);
    launch_after(k_wilson_force<T>, tiles(g), kLinkBlock, 0, s, g, U, S, F);
}
template <typename T>
void launch_wilson_lambda(const DevGeom& g, LinkPlanes<T> U, AlgPlanes<T> S, AlgPlanes<T> Q, AlgPlanes<T> Lam,
                          AlgPlanes<T> Dir, cudaStream_t s) {
    launch_after(k_plaq_sin<T>, tiles(g), kPlaqBlock, 0, s, g, U, S);
    launch_after(k_wilson_lambda<T>, tiles(g), kLinkBlock, 0, s, g, U, S, Q, Lam, Dir);
}

#define MAG_INSTANTIATE(T)                                                                                          \
    template void launch_wilson_lambda<T>(const DevGeom&, LinkPlanes<T>, AlgPlanes<T>, AlgPlanes<T>, AlgPlanes<T>,  \
                                          AlgPlanes<T>, cudaStream_t);                                              \
    template void launch_plaq_chain<T>(const DevGeom&, LinkPlanes<T>, AlgPlanes<T>, AlgPlanes<T>, AlgPlanes<T>,     \
                                       cudaStream_t);                                                               \
    template void launch_chain_gather<T>(const DevGeom&, AlgPlanes<T>, AlgPlanes<T>, AlgPlanes<T>, bool,            \
                                         AlgPlanes<T>, AlgPlanes<T>, cudaStream_t);                                 \
    template void launch_force_gather<T>(const DevGeom&, LinkPlanes<T>, AlgPlanes<T>, AlgPlanes<T>, AlgPlanes<T>,   \
                                         bool, const ForceUse<T>&, cudaStream_t);                                   \
    template void launch_plaq_rect<T>(const DevGeom&, LinkPlanes<T>, RowPlanes<T>, AlgPlanes<T>, AlgPlanes<T>,      \
                                      cudaStream_t);                                                                \
    template void launch_wilson_force<T>(const DevGeom&, LinkPlanes<T>, AlgPlanes<T>, AlgPlanes<T>, cudaStream_t);
MAG_INSTANTIATE(float)
MAG_INSTANTIATE(double)
#undef MAG_INSTANTIATE

}  // namespace magb
