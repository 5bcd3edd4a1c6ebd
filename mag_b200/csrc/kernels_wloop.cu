// kernels_wloop.cu -- Wilson loops (field-wloop.h:26-99) and the constrained
// plaquette (field-matrix.h:407-443), FP64 with double-double sums.
//
// Planar R x T loops reuse line products: for one spatial direction i the
// lines S_R(x) = U_i(x) ... U_i(x+(R-1)i) are built once for R = 1..Rmax; the
// temporal line T_T(x) grows by one link per T; then
//   W_i(R,T)(x) = ReTr( S_R(x) T_T(x+R i) S_R(x+T t)^dag T_T(x)^dag )
// costs two products and one trace per (x, R, T) instead of 2(R+T)-1 products.
//
// Unitary links of one chain go further (launch_wilson_gauged): with the temporal lines
// G(x, t) = U_t(x, 0) ... U_t(x, t-1), T_T(x, t) = G(x, t)^-1 G(x, t + T) and a loop is
// the trace of two lines,
//   W_i(R, T)(x, t) = ReTr(A_R(x, t) B_R(x, t + T)^dag),
//   B_R(x) = G(x) S_R(x) G(x + R i)^dag,  A_R(x) = G(x)^-dag S_R(x) G(x + R i)^-1:
// no product at all, 18 multiply-adds.  B_R continues over the boundary as
// B_R(x, t + Lt) = P(x) B_R(x, t) P(x + R i)^dag (P the Polyakov line).  With exactly
// unitary links A would be B; links are unitary to rounding (or to what an integration
// left), and G is their product with nothing added.  With H = G G^dag = 1 + h,
//   A_R(x) = H(x)^-1 B_R(x) H(x + R i)^-1,  H^-1 = 1 - h
// up to h^2 (1e-20 for links 1e-12 off).  So the loops are those of the links as they
// are, of any determinant: 1e-16 from 64-bit loops as the line products are, where G made
// special unitary and A = B are 5e-15 off (and wrong for a determinant that is not one).
// The lines of a few spatial sites over all t stay on the SM while R grows; nothing but
// the gauged links and h is read.  24^3 x 48, R, T <= 8, on the device: 10.7 ms by line
// products, 1.29 ms so (0.98 ms with A = B).
#include "kernels.h"
#include "plaq_ops.cuh"

namespace magb {

namespace {

constexpr int kBlock = 256;

__device__ __forceinline__ bool locate(const DevGeom& g, int gs, ChainInfo& ci, Site& st) {
    if (gs >= g.vpad) return false;
    ci = g.chains[g.c2c[gs / MAG_CHUNK]];
    const int s = gs - ci.off;
    if (s >= ci.V) return false;
    decode(ci, s, st);
    return true;
}

__device__ __forceinline__ int wrap_shift(const ChainInfo& ci, int xd, int d, int k) {
    int w = (xd + k) % ci.L[d];
    if (w < 0) w += ci.L[d];
    return (w - xd) * ci.stride[d];
}

__device__ __forceinline__ dd2 two_sum(double a, double b) {
    const double s = a + b, bp = s - a;
    return dd2{s, (a - (s - bp)) + (b - bp)};
}
__device__ __forceinline__ dd2 dd_add(dd2 a, dd2 b) {
    dd2 s = two_sum(a.hi, b.hi);
    s.lo += a.lo + b.lo;
    return two_sum(s.hi, s.lo);
}
__device__ dd2 block_reduce(dd2 v) {
    __shared__ dd2 sm[kBlock / 32];
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        dd2 w{__shfl_down_sync(0xffffffffu, v.hi, o), __shfl_down_sync(0xffffffffu, v.lo, o)};
        v = dd_add(v, w);
    }
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    __syncthreads();
    if (lane == 0) sm[wid] = v;
    __syncthreads();
    if (wid == 0) {
        v = lane < (int)(blockDim.x >> 5) ? sm[lane] : dd2{0.0, 0.0};
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) {
            dd2 w{__shfl_down_sync(0xffffffffu, v.hi, o), __shfl_down_sync(0xffffffffu, v.lo, o)};
            v = dd_add(v, w);
        }
    }
    return v;
}

// line(x) <- prev(x) U_d(x + k d)   (prev = nullptr: line(x) = U_d(x))
__global__ void k_line_extend(DevGeom g, LinkPlanes<double> U, int d, LinkPlanes<double> prev, int k,
                              LinkPlanes<double> out) {
    ChainInfo ci;
    Site st;
    if (!locate(g, blockIdx.x * blockDim.x + threadIdx.x, ci, st)) return;
    const mat3<double> u = U.load(d, st.g + wrap_shift(ci, st.x[d], d, k));
    out.store(0, st.g, prev.p ? mul(prev.load(0, st.g), u) : u);
}

// partial[block * Rmax + R-1] = sum_x ReTr W_i(R, T)(x).  The R values are
// taken four at a time: a thread forms its site's four loops (their loads
// issued together) and the block reduces the four sums at once, instead of one
// block reduction (two barriers) per R.  ReTr(S_R(x) T(x+Ri) S_R(x+Tt)^dag
// T(x)^dag) = ReTr(a c^dag) with a = S_R(x) T(x+Ri), c = T(x) S_R(x+Tt): two
// products and one trace of a product per loop.
constexpr int kRChunk = 4;
__global__ void __launch_bounds__(kBlock, 2) k_wloop_accum(DevGeom g, LinkPlanes<double> lines, int Rmax,
                                                           LinkPlanes<double> tl, int i, int T, dd2* partial) {
    __shared__ dd2 sm[kBlock / 32][kRChunk];
    ChainInfo ci;
    Site st;
    const bool ok = locate(g, blockIdx.x * blockDim.x + threadIdx.x, ci, st);
    int gT = 0, gR = 0;
    if (ok) {
        gT = st.g + wrap_shift(ci, st.x[3], 3, T);
        gR = st.x[i];
    }
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    for (int R0 = 1; R0 <= Rmax; R0 += kRChunk) {
        double v[kRChunk];
#pragma unroll
        for (int r = 0; r < kRChunk; r++) {
            const int R = R0 + r;
            v[r] = 0.0;
            if (ok && R <= Rmax) {
                const LinkPlanes<double> S{lines.p + (size_t)(R - 1) * 9 * lines.vpad, lines.vpad};
                const mat3<double> a = mul(S.load(0, st.g), tl.load(0, st.g + wrap_shift(ci, gR, i, R)));
                const mat3<double> c = mul(tl.load(0, st.g), S.load(0, gT));
                v[r] = retr_mul_nd(a, c);
            }
        }
#pragma unroll
        for (int r = 0; r < kRChunk; r++)
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) v[r] += __shfl_down_sync(0xffffffffu, v[r], o);
        __syncthreads();  // the previous chunk's sums have been read
        if (lane == 0)
#pragma unroll
            for (int r = 0; r < kRChunk; r++) sm[wid][r] = dd2{v[r], 0.0};
        __syncthreads();
        if (threadIdx.x < kRChunk && R0 + (int)threadIdx.x <= Rmax) {
            dd2 s = sm[0][threadIdx.x];
            for (int w = 1; w < kBlock / 32; w++) s = dd_add(s, sm[w][threadIdx.x]);
            partial[(size_t)blockIdx.x * Rmax + R0 - 1 + threadIdx.x] = s;
        }
    }
}

// generic closed paths from every site (or from coarse sites when mag > 0):
// sum over paths of ReTr of the path-ordered product (get_path_ordered_product,
// field-matrix.h:102-131); dirs: 0..3 forward, 4..7 backward
__global__ void k_paths(DevGeom g, LinkPlanes<double> U, const int* dirs, int npath, int plen, int coarse_mag,
                        dd2* partial) {
    ChainInfo ci;
    Site st;
    dd2 v{0.0, 0.0};
    if (locate(g, blockIdx.x * blockDim.x + threadIdx.x, ci, st)) {
        bool active = true;
        if (coarse_mag > 0)
            for (int d = 0; d < 4; d++) active = active && (st.x[d] % coarse_mag == 0);
        if (active) {
            double acc = 0.0;
            for (int p = 0; p < npath; p++) {
                int y[4] = {st.x[0], st.x[1], st.x[2], st.x[3]};
                int gy = st.g;
                mat3<double> m = unit_mat<double>();
                for (int k = 0; k < plen; k++) {
                    const int d = dirs[p * plen + k];
                    if (d < 0) break;
                    if (d < 4) {
                        m = mul(m, U.load(d, gy));
                        const int sh = wrap_shift(ci, y[d], d, 1);
                        gy += sh;
                        y[d] = y[d] + 1 < ci.L[d] ? y[d] + 1 : 0;
                    } else {
                        const int e = d - 4;
                        const int sh = wrap_shift(ci, y[e], e, -1);
                        gy += sh;
                        y[e] = y[e] > 0 ? y[e] - 1 : ci.L[e] - 1;
                        m = mul_nd(m, U.load(e, gy));
                    }
                }
                acc += retr(m);
            }
            v.hi = acc;
        }
    }
    v = block_reduce(v);
    if (threadIdx.x == 0) partial[blockIdx.x] = v;
}

// per chain: out[c * nq + q] = sum of partial[b * nq + q] over the chain's blocks
__global__ void k_finalize_multi(DevGeom g, const dd2* partial, int nq, dd2* out) {
    const int c = blockIdx.x;
    const ChainInfo ci = g.chains[c];
    const int b0 = ci.off / kBlock, b1 = (ci.off + ci.V + kBlock - 1) / kBlock;
    for (int q = 0; q < nq; q++) {
        dd2 v{0.0, 0.0};
        for (int b = b0 + threadIdx.x; b < b1; b += blockDim.x) v = dd_add(v, partial[(size_t)b * nq + q]);
        v = block_reduce(v);
        if (threadIdx.x == 0) out[c * nq + q] = v;
        __syncthreads();
    }
}

// ---------------------------------------------------------- temporal gauge
// h = m m^dag - 1 of a nearly unitary m
__device__ __forceinline__ herm9<double> gram_off_one(const mat3<double>& m) {
    herm9<double> h;
#pragma unroll
    for (int i = 0; i < 3; i++)
#pragma unroll
        for (int j = i; j < 3; j++) {
            cplx<double> s = cmul<false, true>(m.e[i][0], m.e[j][0]);
            cmac<false, true, false>(s, m.e[i][1], m.e[j][1]);
            cmac<false, true, false>(s, m.e[i][2], m.e[j][2]);
            if (i == j) {
                h.d[i] = s.re - 1.0;
            } else {
                h.z[2 * (i + j - 1)] = s.re;
                h.z[2 * (i + j - 1) + 1] = s.im;
            }
        }
    return h;
}
// The gauge form takes links within 1e-12 of unitary ones (1e-15 after a reunitarisation,
// 1e-13 after a long integration), NaN not among them
__device__ __forceinline__ bool is_unitary(const mat3<double>& m) {
    const herm9<double> h = gram_off_one(m);
    bool ok = true;
#pragma unroll
    for (int k = 0; k < 3; k++) ok = ok && fabs(h.d[k]) <= 1e-12;
#pragma unroll
    for (int k = 0; k < 6; k++) ok = ok && fabs(h.z[k]) <= 1e-12;
    return ok;
}
// h of every site: its nine reals in five 16-byte pieces, one site after another (the four sites of a
// block on a long chain 320 bytes together; in nine rows 32 bytes each: 48^3 x 96 34 against 23 ms)
struct HermSites {
    double2* p;
    __device__ __forceinline__ herm9<double> load(int s) const {
        const double2* q = p + 5 * (long)s;
        const double2 a = q[0], b = q[1], c = q[2], d = q[3], e = q[4];
        return herm9<double>{{a.x, a.y, b.x}, {b.y, c.x, c.y, d.x, d.y, e.x}};
    }
    __device__ __forceinline__ void store(int s, const herm9<double>& h) const {
        double2* q = p + 5 * (long)s;
        q[0] = make_double2(h.d[0], h.d[1]);
        q[1] = make_double2(h.d[2], h.z[0]);
        q[2] = make_double2(h.z[1], h.z[2]);
        q[3] = make_double2(h.z[3], h.z[4]);
        q[4] = make_double2(h.z[5], 0.0);
    }
};
// (x, y, z) += sign (x, y, z) h, a row; with CONJ h's transpose, so that a column (x, y, z)^T
// gets sign h (x, y, z)^T
template <bool CONJ>
__device__ __forceinline__ void add_row_times(cplx<double>& x, cplx<double>& y, cplx<double>& z, const herm9<double>& h,
                                              double sign) {
    const cplx<double> h01 = mk(sign * h.z[0], sign * (CONJ ? -h.z[1] : h.z[1]));
    const cplx<double> h02 = mk(sign * h.z[2], sign * (CONJ ? -h.z[3] : h.z[3]));
    const cplx<double> h12 = mk(sign * h.z[4], sign * (CONJ ? -h.z[5] : h.z[5]));
    const cplx<double> a = x, b = y, c = z;
    x = mk(fma(sign * h.d[0], a.re, a.re), fma(sign * h.d[0], a.im, a.im));
    cmac<false, true, false>(x, b, h01);
    cmac<false, true, false>(x, c, h02);
    y = mk(fma(sign * h.d[1], b.re, b.re), fma(sign * h.d[1], b.im, b.im));
    cmac<false, false, false>(y, a, h01);
    cmac<false, true, false>(y, c, h12);
    z = mk(fma(sign * h.d[2], c.re, c.re), fma(sign * h.d[2], c.im, c.im));
    cmac<false, false, false>(z, a, h02);
    cmac<false, false, false>(z, b, h12);
}
// m (1 + sign h) and (1 + sign h) m
__device__ __forceinline__ void scale_right(mat3<double>& m, const herm9<double>& h, double sign) {
#pragma unroll
    for (int r = 0; r < 3; r++) add_row_times<false>(m.e[r][0], m.e[r][1], m.e[r][2], h, sign);
}
__device__ __forceinline__ void scale_left(mat3<double>& m, const herm9<double>& h, double sign) {
#pragma unroll
    for (int c = 0; c < 3; c++) add_row_times<true>(m.e[0][c], m.e[1][c], m.e[2][c], h, sign);
}

constexpr int kGaugeBlock = 64;
// G(x, t) = U_t(x, 0) ... U_t(x, t-1), h of it, and the Polyakov line P(x) = G(x, Lt); one
// thread per spatial site, the next link loaded while the current one is multiplied
__global__ void __launch_bounds__(kGaugeBlock) k_temporal_gauge(ChainInfo ci, LinkPlanes<double> U,
                                                                LinkPlanes<double> G, HermSites H,
                                                                LinkPlanes<double> P, int* bad) {
    after_previous();
    const int vs = ci.L[0] * ci.L[1] * ci.L[2];
    const int x = blockIdx.x * kGaugeBlock + threadIdx.x;
    if (x >= vs) return;
    mat3<double> g = unit_mat<double>(), u = U.load(3, ci.off + x);
    bool ok = true;
    for (int t = 0; t < ci.L[3]; t++) {
        const mat3<double> next = U.load(3, ci.off + x + vs * (t + 1 < ci.L[3] ? t + 1 : 0));
        G.store(0, x + vs * t, g);
        H.store(x + vs * t, gram_off_one(g));
        ok = ok && is_unitary(u);
        g = mul(g, u);
        u = next;
    }
    P.store(0, x, g);
    if (!ok) *bad = 1;
}

// V_i(x) = G(x) U_i(x) G(x + i)^dag, the three spatial directions
__global__ void __launch_bounds__(kBlock) k_gauge_links(ChainInfo ci, LinkPlanes<double> U, LinkPlanes<double> G,
                                                        LinkPlanes<double> V, int* bad) {
    after_previous();
    const int s = blockIdx.x * kBlock + threadIdx.x, i = blockIdx.y;
    if (s >= ci.V) return;
    Site st;
    decode(ci, s, st);
    const mat3<double> u = U.load(i, st.g);
    if (!is_unitary(u)) *bad = 1;
    const int sn = s + nb_sel(ci, st, i, 1) - st.g;
    V.store(i, s, mul_nd(mul(G.load(0, s), u), G.load(0, sn)));
}

// One block: NX spatial sites (blockDim = NX times the groups of SL time slices, in
// whole warps), direction i = blockIdx.y.  Shared memory holds B_R of the sites for
// t in [0, Lt + Tmax), a thread A_R of its SL slices.  It extends these lines, then takes
// the traces of its slices with the slices up to T + SL - 1 later, each read once for SL
// loops, TC values of T at a time (4 where Tmax is no more).  Bound by the FP64 pipe and
// shared-memory reads in turn, at the twelve warps per SM that the registers allow: two
// slices at 168 registers 1.29 ms at 24^3 x 48 (R, T <= 8) and 0.152 at 16^4, at 144 or
// 128 (spills) 1.50 and 1.59; three slices spill (1.63, 0.25), with A read back from
// shared memory and corrected there 1.28 and 0.172.  Blocks of 64 contiguous bytes per
// element instead of 128 (four sites): 1.58 ms.  A block walks the groups of NX sites
// with stride gridDim.x and adds up its
// part[((i Rmax + R-1) Tmax + T-1) gridDim.x + block].
constexpr int kGaugedBlocks = 592;  // per direction at most: four per SM
// the block's slots for n slices, sl per thread
__host__ __device__ __forceinline__ int gauged_slots(int n, int sl) { return (n + sl - 1) / sl * sl; }
template <int NX, int SL, int TC>
__global__ void __maxnreg__(168) k_wloop_gauged(ChainInfo ci, LinkPlanes<double> V, HermSites H,
                                                      LinkPlanes<double> P, int Rmax, int Tmax, dd2* part) {
    after_previous();
    extern __shared__ __align__(16) unsigned char wsm[];
    cplx<double>* S = reinterpret_cast<cplx<double>*>(wsm);  // [gauged_slots][9][NX]
    __shared__ double red[8][TC];
    const int Lt = ci.L[3], vs = ci.L[0] * ci.L[1] * ci.L[2], i = blockIdx.y;
    const int nx = threadIdx.x % NX, t0 = (threadIdx.x / NX) * SL;
    const int Li = i == 0 ? ci.L[0] : i == 1 ? ci.L[1] : ci.L[2];
    const int si = i == 0 ? 1 : i == 1 ? ci.L[0] : ci.L[0] * ci.L[1];
    // slice t is in slot t / SL of the t % SL-th part: the threads of a warp, SL slices apart, read
    // neighbouring slots.  With the slices one after another, two per thread and fewer than eight
    // sites meet in the same banks (48^3 x 96, four sites, R, T <= 8: 44 against 34 ms)
    const int part_slots = gauged_slots(Lt + Tmax, SL) / SL;
    auto line = [&](int t) { return S + ((t % SL) * part_slots + t / SL) * 9 * NX + nx; };
    auto put = [&](int t, const mat3<double>& m) {
        cplx<double>* b = line(t);
#pragma unroll
        for (int k = 0; k < 9; k++) b[k * NX] = m.e[k / 3][k % 3];
    };
    auto get = [&](int t) {
        mat3<double> m;
        const cplx<double>* b = line(t);
#pragma unroll
        for (int k = 0; k < 9; k++) m.e[k / 3][k % 3] = b[k * NX];
        return m;
    };
    const int last = Lt + Tmax - 1;
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5, nw = blockDim.x >> 5;
    for (int x0 = blockIdx.x * NX; x0 < vs; x0 += gridDim.x * NX) {
        mat3<double> a[SL];
        for (int R = 1; R <= Rmax; R++) {
            const int x = x0 + nx;
            const bool site = x < vs;
            // coordinate along i and the index of x + k i
            const int xi = i == 0 ? x % ci.L[0] : i == 1 ? x / ci.L[0] % ci.L[1] : x / (ci.L[0] * ci.L[1]);
            auto along = [&](int k) { return x + ((xi + k) % Li - xi) * si; };
            const int xr = site ? along(R - 1) : 0, xe = site ? along(R) : 0, xs = site ? x : 0;
            // 1. this thread's slices: E_R = A_{R-1} V_i(x + (R-1) i), E_1 = H^-1 V_i; B_R = H E_R goes to
            // shared memory, A_R = E_R H(x + R i)^-1 stays
#pragma unroll
            for (int j = 0; j < SL; j++) {
                const int t = t0 + j;
                if (t >= Lt) {
                    set_zero(a[j]);
                    continue;
                }
                const mat3<double> v = V.load(i, xr + vs * t);
                const herm9<double> h = H.load(xs + vs * t);
                if (R == 1) {
                    if (site) a[j] = v;
                    else set_zero(a[j]);
                    scale_left(a[j], h, -1.0);
                } else {
                    a[j] = mul(a[j], v);
                }
                mat3<double> b = a[j];
                scale_left(b, h, 1.0);
                put(t, b);
                scale_right(a[j], H.load(xe + vs * t), -1.0);
            }
            // 2. the slices past the boundary, from this thread's own slices, a row at a time
#pragma unroll 1
            for (int t = t0; t < t0 + SL && t < Lt && t < Tmax; t++) {
                const cplx<double>* from = line(t);
                cplx<double>* to = line(Lt + t);
#pragma unroll 1
                for (int r = 0; r < 3; r++) {
                    cplx<double> y[3] = {};
#pragma unroll
                    for (int k = 0; k < 3; k++) {
                        const cplx<double> p = P.at(0, xs)[(3 * r + k) * MAG_TILE];
#pragma unroll
                        for (int c = 0; c < 3; c++) cmac<false, false, false>(y[c], p, from[(3 * k + c) * NX]);
                    }
#pragma unroll
                    for (int c = 0; c < 3; c++) {
                        cplx<double> z = mk(0.0, 0.0);
#pragma unroll
                        for (int k = 0; k < 3; k++)
                            cmac<false, true, false>(z, y[k], P.at(0, xe)[(3 * c + k) * MAG_TILE]);
                        to[(3 * r + c) * NX] = z;
                    }
                }
            }
            __syncthreads();
            // 3. traces, TC values of T at a time
            for (int Tb = 0; Tb < Tmax; Tb += TC) {
                double acc[TC];
#pragma unroll
                for (int k = 0; k < TC; k++) acc[k] = 0.0;
#pragma unroll
                for (int u = 1; u < TC + SL; u++) {
                    const int t = t0 + Tb + u;
                    const mat3<double> b = get(t < last ? t : last);  // beyond the last slice: only a[j] = 0 or T > Tmax
#pragma unroll
                    for (int j = 0; j < SL; j++)
                        if (u - j >= 1 && u - j <= TC) acc[u - j - 1] += retr_mul_nd(a[j], b);
                }
                // the warp's sums: TC values over 32 lanes, half of them kept at each step
#pragma unroll
                for (int h = TC / 2, o = 16; h >= 1; h /= 2, o /= 2) {
                    const bool up = lane & o;
#pragma unroll
                    for (int k = 0; k < h; k++) {
                        const double give = up ? acc[k] : acc[k + h], keep = up ? acc[k + h] : acc[k];
                        acc[k] = keep + __shfl_xor_sync(0xffffffffu, give, o);
                    }
                }
#pragma unroll
                for (int o = 16 / TC; o >= 1; o /= 2) acc[0] += __shfl_xor_sync(0xffffffffu, acc[0], o);
                // the lane's upper bits select the value
                if (lane % (32 / TC) == 0) red[wid][lane / (32 / TC)] = acc[0];
                __syncthreads();
                if (threadIdx.x < TC && Tb + (int)threadIdx.x < Tmax) {
                    dd2 v{red[0][threadIdx.x], 0.0};
                    for (int w = 1; w < nw; w++) v = dd_add(v, dd2{red[w][threadIdx.x], 0.0});
                    dd2* p = part + ((size_t)(i * Rmax + R - 1) * Tmax + Tb + threadIdx.x) * gridDim.x + blockIdx.x;
                    *p = x0 == (int)blockIdx.x * NX ? v : dd_add(*p, v);
                }
                __syncthreads();
            }
        }
    }
}

// out[(R-1) Tmax + T-1] = the sum over directions and blocks
__global__ void k_wloop_gauged_sum(int nblk, int RT, const dd2* part, dd2* out) {
    after_previous();
    dd2 v{0.0, 0.0};
    for (int i = 0; i < 3; i++)
        for (int b = threadIdx.x; b < nblk; b += blockDim.x)
            v = dd_add(v, part[((size_t)i * RT + blockIdx.x) * nblk + b]);
    v = block_reduce(v);
    if (threadIdx.x == 0) out[blockIdx.x] = v;
}

unsigned blocks(const DevGeom& g) { return (unsigned)((g.vpad + kBlock - 1) / kBlock); }

}  // namespace

// Shape of k_wloop_gauged: slices per thread and the most spatial sites per block (32 down
// to 1) whose lines take at most 72 KB (three blocks per SM) and whose slice groups fit 256
// threads; 0 sites: none, the chain is too long in time.
struct GaugedShape {
    int nx, sl;
};
static int gauged_fit(const ChainInfo& ci, int Tmax, int sl) {
    const int groups = (ci.L[3] + sl - 1) / sl;
    for (int nx = 32; nx >= 1; nx /= 2)
        if ((size_t)nx * gauged_slots(ci.L[3] + Tmax, sl) * 144 <= 72 * 1024 && nx * groups <= 256) return nx;
    return 0;
}
static GaugedShape gauged_shape(const ChainInfo& ci, int Tmax) {
    if (Tmax > ci.L[3]) return {0, 2};
    const int vs = ci.L[0] * ci.L[1] * ci.L[2];
    // Two slices per thread read each line for two traces.  Chains that leave an SM fewer than
    // about five warps of such threads are bound by a thread's own work: one slice each, in
    // blocks that spread over the SMs.  One measurement, one slice against two: 8^4 to R, T = 4
    // 30 against 39 us, 8^3 x 16 to 8 63 against 86 (12,000 threads of two), 10^3 x 20 to 6 74
    // against 72 (30,000), 12^4 to 4 54 against 51, 16^4 to 4 115 against 84.
    if (3L * vs * ((ci.L[3] + 1) / 2) < 25000) {
        int nx = gauged_fit(ci, Tmax, 1);
        while (nx > 4 && 3 * ((vs + nx - 1) / nx) < 148) nx /= 2;
        if (nx) return {nx, 1};
    }
    return {gauged_fit(ci, Tmax, 2), 2};
}
int wilson_gauged_sites(const ChainInfo& ci, int Tmax) { return gauged_shape(ci, Tmax).nx; }
static int gauged_blocks(const ChainInfo& ci, int nx) {
    const int groups = (ci.L[0] * ci.L[1] * ci.L[2] + nx - 1) / nx;
    return groups < kGaugedBlocks ? groups : kGaugedBlocks;
}
size_t wilson_gauged_partials(const ChainInfo& ci, int Rmax, int Tmax) {
    const int nx = wilson_gauged_sites(ci, Tmax);
    return nx ? (size_t)3 * Rmax * Tmax * gauged_blocks(ci, nx) : 0;
}

template <int NX, int SL, int TC>
static cudaError_t wloop_gauged(const ChainInfo& ci, LinkPlanes<double> V, HermSites H, LinkPlanes<double> P, int Rmax,
                                int Tmax, dd2* part, cudaStream_t s) {
    const int groups = (ci.L[3] + SL - 1) / SL;
    const int threads = (NX * groups + 31) / 32 * 32;
    const size_t smem = (size_t)NX * gauged_slots(ci.L[3] + Tmax, SL) * 144;
    const cudaError_t e =
        cudaFuncSetAttribute(k_wloop_gauged<NX, SL, TC>, cudaFuncAttributeMaxDynamicSharedMemorySize, 72 * 1024);
    if (e != cudaSuccess) return e;
    launch_after(k_wloop_gauged<NX, SL, TC>, dim3(gauged_blocks(ci, NX), 3), threads, smem, s, ci, V, H, P, Rmax,
                 Tmax, part);
    return cudaGetLastError();
}
template <int NX>
static cudaError_t wloop_gauged(const ChainInfo& ci, int sl, LinkPlanes<double> V, HermSites H, LinkPlanes<double> P,
                                int Rmax, int Tmax, dd2* part, cudaStream_t s) {
    if (Tmax <= 4)
        return sl == 1 ? wloop_gauged<NX, 1, 4>(ci, V, H, P, Rmax, Tmax, part, s)
                       : wloop_gauged<NX, 2, 4>(ci, V, H, P, Rmax, Tmax, part, s);
    return sl == 1 ? wloop_gauged<NX, 1, 8>(ci, V, H, P, Rmax, Tmax, part, s)
                   : wloop_gauged<NX, 2, 8>(ci, V, H, P, Rmax, Tmax, part, s);
}

// One chain's planar loops in the temporal gauge: G and V, P scratch planes of the
// chain's V (1 and 3 directions) and L0 L1 L2 sites, H nine reals per site, local site indices;
// out[(R-1) Tmax + T-1] = sum over the directions and sites; *bad is set when a link
// is not unitary (the sums are then not the loops).
cudaError_t launch_wilson_gauged(const ChainInfo& ci, LinkPlanes<double> U, int Rmax, int Tmax, LinkPlanes<double> G,
                                 LinkPlanes<double> V, LinkPlanes<double> P, double* h, dd2* part, dd2* out, int* bad,
                                 cudaStream_t s) {
    const HermSites H{reinterpret_cast<double2*>(h)};
    const GaugedShape shape = gauged_shape(ci, Tmax);
    const int nx = shape.nx, vs = ci.L[0] * ci.L[1] * ci.L[2];
    launch_after(k_temporal_gauge, (vs + kGaugeBlock - 1) / kGaugeBlock, kGaugeBlock, 0, s, ci, U, G, H, P,
                 bad);
    launch_after(k_gauge_links, dim3((ci.V + kBlock - 1) / kBlock, 3), kBlock, 0, s, ci, U, G, V, bad);
    cudaError_t e = cudaErrorInvalidValue;
    switch (nx) {
        case 32: e = wloop_gauged<32>(ci, shape.sl, V, H, P, Rmax, Tmax, part, s); break;
        case 16: e = wloop_gauged<16>(ci, shape.sl, V, H, P, Rmax, Tmax, part, s); break;
        case 8: e = wloop_gauged<8>(ci, shape.sl, V, H, P, Rmax, Tmax, part, s); break;
        case 4: e = wloop_gauged<4>(ci, shape.sl, V, H, P, Rmax, Tmax, part, s); break;
        case 2: e = wloop_gauged<2>(ci, shape.sl, V, H, P, Rmax, Tmax, part, s); break;
        case 1: e = wloop_gauged<1>(ci, shape.sl, V, H, P, Rmax, Tmax, part, s); break;
        default: return e;
    }
    if (e != cudaSuccess) return e;
    launch_after(k_wloop_gauged_sum, Rmax * Tmax, kBlock, 0, s, gauged_blocks(ci, nx), Rmax * Tmax, part, out);
    return cudaGetLastError();
}

// lines: Rmax consecutive single-direction planes (9 * vpad complex each);
// tl, tl2: two single-direction planes for the temporal line (ping-pong).
// out[((i * Tmax + T-1) * nchain + c) * Rmax + R-1] = sum over the chain's sites
// of ReTr W_i(R, T) for spatial direction i; partial holds blocks * Rmax entries.
void launch_wilson_planar(const DevGeom& g, LinkPlanes<double> U, int Rmax, int Tmax, LinkPlanes<double> lines,
                          LinkPlanes<double> tl, LinkPlanes<double> tl2, dd2* partial, dd2* out, cudaStream_t s) {
    const unsigned nb = blocks(g);
    for (int i = 0; i < 3; i++) {
        for (int R = 1; R <= Rmax; R++) {
            LinkPlanes<double> cur{lines.p + (size_t)(R - 1) * 9 * lines.vpad, lines.vpad};
            LinkPlanes<double> prev{R > 1 ? lines.p + (size_t)(R - 2) * 9 * lines.vpad : nullptr, lines.vpad};
            k_line_extend<<<nb, kBlock, 0, s>>>(g, U, i, prev, R - 1, cur);
        }
        LinkPlanes<double> a = tl, b = tl2;
        for (int T = 1; T <= Tmax; T++) {
            k_line_extend<<<nb, kBlock, 0, s>>>(g, U, 3, T > 1 ? a : LinkPlanes<double>{nullptr, 0}, T - 1, b);
            k_wloop_accum<<<nb, kBlock, 0, s>>>(g, lines, Rmax, b, i, T, partial);
            k_finalize_multi<<<g.nchain, kBlock, 0, s>>>(g, partial, Rmax,
                                                         out + (size_t)(i * Tmax + (T - 1)) * g.nchain * Rmax);
            LinkPlanes<double> t = a;
            a = b;
            b = t;
        }
    }
}

void launch_wilson_general(const DevGeom& g, LinkPlanes<double> U, const int* dirs, int npath, int plen,
                           int coarse_mag, dd2* partial, dd2* out, cudaStream_t s) {
    k_paths<<<blocks(g), kBlock, 0, s>>>(g, U, dirs, npath, plen, coarse_mag, partial);
    k_finalize_multi<<<g.nchain, kBlock, 0, s>>>(g, partial, 1, out);
}

}  // namespace magb
