// fnec_plain.cu -- plain FP64 Hallen kernels with bit-exact operation order.
//
// Every arithmetic operation below is one separately rounded IEEE
// operation (explicit _rn intrinsics; the file is also built with
// -fmad=false), issued in the order the reference issues it, and sin, cos
// and hypot return the platform libm's values (fnec_libm.cuh restates
// glibc's algorithms; the self term's ln comes from the host libm, see
// DevSeg::self_log).  Given the
// same inputs the Gram matrix, the elimination and the back substitution
// therefore reproduce the reference CPU path bit for bit; pivot order is
// chosen with the reference's "last maximum by hypot" rule.
//
// Kernels (one launch each, all units of a batch at once):
//   k_expand_segments  geometry.rs:710-754     one CTA per GW wire
//   k_hallen_rhs       excitation.rs:119-244   one CTA per unit
//   k_fill_exact       matrix.rs:186-331       16x16 tiles of Z, tile list
//   k_gram_zz          linear.rs:765-780       32x32 tiles of Z^H [Z | y], upper triangle
//   k_gram_ccols       linear.rs:765-780       the -cos(k s) columns (sparse)
//   k_gram_finish      linear.rs:757-785       constraint rows, then +1e-8 I
//   k_panel_cluster    linear.rs:1343-1370     NB columns, a thread per row, up to 8 CTAs per unit
//   k_panel            linear.rs:1343-1370     the same from global memory, one CTA per unit
//   k_panel_grid       linear.rs:1343-1370     NB columns of a panel above 3,072 rows, many CTAs
//   k_swap_u12         linear.rs:1358-1369     deferred swaps + U block row
//   k_trailing         linear.rs:1362-1369     A22 -= L21 U12, 32x32 or 64x64 tiles
//   k_backsub          linear.rs:1372-1381     one CTA per unit: a chain warp, two product warps
//   k_feedpoints       solve_session.rs:846-947
#include <algorithm>
#include <cstdio>
#include <climits>
#include <map>
#include <mutex>
#include <unordered_map>
#include <utility>

#include "fnec_grid.cuh"
#include "fnec_kernels.h"
#include "fnec_libm.cuh"
#include "fnec_math.cuh"

namespace fnec {

// Gauss-Legendre tables as written in matrix.rs:39-72 (15 decimal digits).
__constant__ double c_gl_n4[4] = {-0.861136311594953, -0.339981043584856, 0.339981043584856,
                                  0.861136311594953};
__constant__ double c_gl_w4[4] = {0.347854845137454, 0.652145154862626, 0.652145154862626,
                                  0.347854845137454};
__constant__ double c_gl_n8[8] = {-0.960289856497536, -0.796666477413627, -0.525532409916329,
                                  -0.183434642495650, 0.183434642495650,  0.525532409916329,
                                  0.796666477413627,  0.960289856497536};
__constant__ double c_gl_w8[8] = {0.101228536290376, 0.222381034453374, 0.313706645877887,
                                  0.362683783378362, 0.362683783378362, 0.313706645877887,
                                  0.222381034453374, 0.101228536290376};

// ---------------------------------------------------------------------------
// geometry
// ---------------------------------------------------------------------------
__global__ void k_expand_segments(const DevWire *__restrict__ wires, int nw, DevSeg *segs) {
    int w = blockIdx.x;
    if (w >= nw) return;
    DevWire gw = wires[w];
    double dx = D_SUB(gw.end[0], gw.start[0]);
    double dy = D_SUB(gw.end[1], gw.start[1]);
    double dz = D_SUB(gw.end[2], gw.start[2]);
    double wl = D_SQRT(D_ADD(D_ADD(D_MUL(dx, dx), D_MUL(dy, dy)), D_MUL(dz, dz)));
    double dir0 = D_DIV(dx, wl), dir1 = D_DIV(dy, wl), dir2 = D_DIV(dz, wl);
    double nn = (double)gw.nseg;
    double seg_len = D_DIV(wl, nn);
    for (uint32_t i = threadIdx.x; i < gw.nseg; i += blockDim.x) {
        double t0 = D_DIV((double)i, nn);
        double t1 = D_DIV(D_ADD((double)i, 1.0), nn);
        double tm = D_MUL(D_ADD(t0, t1), 0.5);
        DevSeg s;
        s.start[0] = D_ADD(gw.start[0], D_MUL(dx, t0));
        s.start[1] = D_ADD(gw.start[1], D_MUL(dy, t0));
        s.start[2] = D_ADD(gw.start[2], D_MUL(dz, t0));
        s.end[0] = D_ADD(gw.start[0], D_MUL(dx, t1));
        s.end[1] = D_ADD(gw.start[1], D_MUL(dy, t1));
        s.end[2] = D_ADD(gw.start[2], D_MUL(dz, t1));
        s.mid[0] = D_ADD(gw.start[0], D_MUL(dx, tm));
        s.mid[1] = D_ADD(gw.start[1], D_MUL(dy, tm));
        s.mid[2] = D_ADD(gw.start[2], D_MUL(dz, tm));
        s.dir[0] = dir0;
        s.dir[1] = dir1;
        s.dir[2] = dir2;
        s.len = seg_len;
        s.rad = gw.radius;
        s.tag = gw.tag;
        s.tag_index = i + 1;
        s.self_log = gw.self_log;
        segs[gw.seg_off + i] = s;
    }
}

// ---------------------------------------------------------------------------
// Hallen RHS: cos(k s_local) per merged conductor and the delta-gap term
// -j (2 pi / eta0) V sin(k |s - s_src|) on the source's conductor.
// ---------------------------------------------------------------------------
__global__ void k_hallen_rhs(const UnitDesc *__restrict__ solves, const AntDesc *__restrict__ ants,
                             const DevSeg *__restrict__ segs, const int32_t *__restrict__ ibuf,
                             const DevSource *__restrict__ srcs, const double *__restrict__ dtab,
                             cx *rhs_buf, double *cos_buf, double scale) {
    UnitDesc u = solves[blockIdx.x];  // one right-hand side
    AntDesc a = ants[u.ant];
    if (a.hom2) return;  // a receiving antenna: k_planewave_field / k_planewave_rhs
    const DevSeg *sg = segs + a.seg_off;
    const int32_t *comp = ibuf + a.comp_off;
    const int32_t *sptr = ibuf + a.sptr_off;
    const DevSource *src = srcs + a.src_off + sptr[u.rhs];
    int n_src = sptr[u.rhs + 1] - sptr[u.rhs];
    double k = u.k_fill;
    if (a.paths) {
        // build_hallen_rhs_paths (excitation.rs:264-341): cos(k s) and the
        // source terms along each path's signed arc length s, times the
        // traversal signs; every EX card drives its whole path
        const double *s_mid = dtab + a.arc_off, *sgn = s_mid + a.n;
        const int32_t *col = ibuf + a.rowwire_off;
        for (int m = threadIdx.x; m < a.n; m += blockDim.x) {
            if (u.rhs == 0) {
                double sn, cs;
                fnec_libm::libm_sincos(D_MUL(k, s_mid[m]), &sn, &cs);
                cos_buf[u.cos_off + m] = D_MUL(sgn[m], cs);
            }
            cx r = cx_make(0.0, 0.0);
            for (int q = 0; q < n_src; ++q) {
                DevSource s = src[q];
                if (col[m] != col[s.feed]) continue;
                double ds = fabs(D_SUB(s_mid[m], s_mid[s.feed]));
                double ss, sc;
                fnec_libm::libm_sincos(D_MUL(k, ds), &ss, &sc);
                cx t = cx_mul(cx_make(0.0, D_MUL(-scale, ss)), cx_make(s.v_re, s.v_im));
                double f = D_MUL(sgn[m], sgn[s.feed]);
                r = cx_add(r, cx_make(D_MUL(t.re, f), D_MUL(t.im, f)));
            }
            rhs_buf[u.rhs_off + m] = r;
        }
        return;
    }
    for (int m = threadIdx.x; m < a.n; m += blockDim.x) {
        int first = comp[2 * m], last = comp[2 * m + 1];
        const double *wd = sg[first].dir;
        double wm0 = D_DIV(D_ADD(sg[first].mid[0], sg[last].mid[0]), 2.0);
        double wm1 = D_DIV(D_ADD(sg[first].mid[1], sg[last].mid[1]), 2.0);
        double wm2 = D_DIV(D_ADD(sg[first].mid[2], sg[last].mid[2]), 2.0);
        double dl0 = D_SUB(sg[m].mid[0], wm0);
        double dl1 = D_SUB(sg[m].mid[1], wm1);
        double dl2 = D_SUB(sg[m].mid[2], wm2);
        double s_local = D_ADD(D_ADD(D_MUL(dl0, wd[0]), D_MUL(dl1, wd[1])), D_MUL(dl2, wd[2]));
        if (u.rhs == 0) {  // cos(k s) belongs to the system: written once
            double sn, cs;
            fnec_libm::libm_sincos(D_MUL(k, s_local), &sn, &cs);
            cos_buf[u.cos_off + m] = cs;
        }
        cx r = cx_make(0.0, 0.0);
        for (int q = 0; q < n_src; ++q) {
            DevSource s = src[q];
            if (m < s.comp_first || m > s.comp_last) continue;
            const DevSeg &f = sg[s.feed];
            double d0 = D_SUB(sg[m].mid[0], f.mid[0]);
            double d1 = D_SUB(sg[m].mid[1], f.mid[1]);
            double d2 = D_SUB(sg[m].mid[2], f.mid[2]);
            double sd = D_ADD(D_ADD(D_MUL(d0, f.dir[0]), D_MUL(d1, f.dir[1])), D_MUL(d2, f.dir[2]));
            double ss, sc;
            fnec_libm::libm_sincos(D_MUL(k, fabs(sd)), &ss, &sc);
            cx t = cx_mul(cx_make(0.0, D_MUL(-scale, ss)), cx_make(s.v_re, s.v_im));
            r = cx_add(r, t);
        }
        rhs_buf[u.rhs_off + m] = r;
    }
}

// ---------------------------------------------------------------------------
// Plane-wave forcing (planewave.rs:162-254 per wire, :278-348 per path).
// k_planewave_field: the tangential incident field of every segment for
// every incidence direction, E_p = sign_p (e . d_p) exp(+j k r_hat . r_p)
// with d_p the direction of the wire's first segment (per-wire form) or of
// the segment itself (path form); the solve's x vector holds it until the
// solve overwrites x.  Solve 0 of each system also writes cos(k s) and
// sin(k s), times the sign, as the two homogeneous columns.
// It also tabulates sin(k |s_m - s_p|) for the rows p of m's wire or path
// (ascending), which no incidence direction changes, after the two columns.
// k_planewave_rhs: rhs_m = sign_m (-j 2 pi / eta0) sum_p E_p sin(k |s_m -
// s_p|) dl_p over those rows in ascending order, reading the table.
// Every operation is the reference's, in its order; sign = 1 in the
// per-wire form, where multiplying by it is exact.
// ---------------------------------------------------------------------------
__global__ void k_planewave_field(const UnitDesc *__restrict__ solves, int ns, const AntDesc *__restrict__ ants,
                                  const DevSeg *__restrict__ segs, const int32_t *__restrict__ ibuf,
                                  const double *__restrict__ dtab, cx *xbuf, double *cos_buf) {
    const int p = blockIdx.x * blockDim.x + threadIdx.x;
    for (int si = blockIdx.y; si < ns; si += gridDim.y) {  // solves beyond the grid's y limit
        UnitDesc u = solves[si];
        AntDesc a = ants[u.ant];
        if (!a.hom2 || p >= a.n) continue;
        const DevSeg *sg = segs + a.seg_off;
        const double *wv = dtab + a.wave_off + 10 * (int64_t)u.rhs;  // r_hat[3], pol re[3], pol im[3]
        const double *dir = a.paths ? sg[p].dir : sg[ibuf[a.comp_off + 2 * p]].dir;
        const double s = dtab[a.arc_off + p], sgn = dtab[a.arc_off + a.n + p];
        const double k = u.k_fill;
        cx coup = cx_make(0.0, 0.0);
        for (int c = 0; c < 3; ++c) coup = cx_add(coup, cx_make(D_MUL(wv[3 + c], dir[c]), D_MUL(wv[6 + c], dir[c])));
        const double phase = D_MUL(
            k, D_ADD(D_ADD(D_MUL(wv[0], sg[p].mid[0]), D_MUL(wv[1], sg[p].mid[1])), D_MUL(wv[2], sg[p].mid[2])));
        double sn, cs;
        fnec_libm::libm_sincos(phase, &sn, &cs);
        const cx e = cx_mul(coup, cx_make(D_MUL(1.0, cs), D_MUL(1.0, sn)));  // from_polar(1, phase)
        xbuf[u.x_off + p] = cx_make(D_MUL(e.re, sgn), D_MUL(e.im, sgn));
        if (u.rhs == 0) {
            double ss, sc;
            fnec_libm::libm_sincos(D_MUL(k, s), &ss, &sc);
            cos_buf[u.cos_off + p] = D_MUL(sgn, sc);
            cos_buf[u.cos_off + a.n + p] = D_MUL(sgn, ss);
            const int32_t col = ibuf[a.rowwire_off + p];
            const int32_t *wptr = ibuf + a.wptr_off, *wrow = ibuf + a.wrow_off;
            double *kt = cos_buf + u.cos_off + 2 * (int64_t)a.n + ibuf[a.koff_off + p];
            for (int q = wptr[col]; q < wptr[col + 1]; ++q) {
                double ks, kc;
                fnec_libm::libm_sincos(D_MUL(k, fabs(D_SUB(s, dtab[a.arc_off + wrow[q]]))), &ks, &kc);
                kt[q - wptr[col]] = ks;
            }
        }
    }
}

__global__ void k_planewave_rhs(const UnitDesc *__restrict__ solves, int ns, const AntDesc *__restrict__ ants,
                                const DevSeg *__restrict__ segs, const int32_t *__restrict__ ibuf,
                                const double *__restrict__ dtab, const double *__restrict__ cos_buf,
                                const cx *__restrict__ xbuf, cx *rhs_buf, double scale) {
    const int m = blockIdx.x * blockDim.x + threadIdx.x;
    for (int si = blockIdx.y; si < ns; si += gridDim.y) {
        UnitDesc u = solves[si];
        AntDesc a = ants[u.ant];
        if (!a.hom2 || m >= a.n) continue;
        const DevSeg *sg = segs + a.seg_off;
        const double *s_mid = dtab + a.arc_off, *sgn = s_mid + a.n;
        const int32_t col = ibuf[a.rowwire_off + m];  // the wire's cos column
        const int32_t *wptr = ibuf + a.wptr_off, *wrow = ibuf + a.wrow_off;
        const cx *e = xbuf + u.x_off;
        const double *kt = cos_buf + u.cos_off + 2 * (int64_t)a.n + ibuf[a.koff_off + m];
        cx acc = cx_make(0.0, 0.0);
        for (int q = wptr[col]; q < wptr[col + 1]; ++q) {
            const int p = wrow[q];
            const double ks = kt[q - wptr[col]];
            const cx ep = e[p];
            const double len = sg[p].len;
            acc = cx_add(acc, cx_make(D_MUL(D_MUL(ep.re, ks), len), D_MUL(D_MUL(ep.im, ks), len)));
        }
        const cx r = cx_mul(cx_make(0.0, -scale), acc);
        rhs_buf[u.rhs_off + m] = cx_make(D_MUL(r.re, sgn[m]), D_MUL(r.im, sgn[m]));
    }
}

// Peak |I| of each plane-wave solve (solve_session.rs:354): the largest
// hypot over the segment currents, NaN when the solve failed.
__global__ void k_receive_peaks(const UnitDesc *__restrict__ solves, const AntDesc *__restrict__ ants,
                                const cx *__restrict__ xbuf, const int32_t *__restrict__ status, double *peak) {
    UnitDesc u = solves[blockIdx.x];
    if (!ants[u.ant].hom2) return;
    double v = 0.0;
    for (int m = threadIdx.x; m < u.n; m += 32) v = fmax(v, cx_norm(xbuf[u.x_off + m]));
    for (int o = 16; o > 0; o >>= 1) v = fmax(v, __shfl_xor_sync(0xffffffffu, v, o));
    if (threadIdx.x == 0) peak[blockIdx.x] = status[u.sys] != 0 ? __longlong_as_double(0x7ff8000000000000ll) : v;
}

// ---------------------------------------------------------------------------
// Z fill
// ---------------------------------------------------------------------------
// G(R) = exp(-jkR)/R with exp(0 + jt) = (cos t, sin t) (num-complex exp)
__device__ __forceinline__ cx green_k_exact(double r, double k) {
    double sn, cs;
    fnec_libm::libm_sincos(D_MUL(-k, r), &sn, &cs);
    return cx_make(D_DIV(cs, r), D_DIV(sn, r));
}

// The fill of a 16 x 16 tile by 256 threads.  What bounds it is the FP64
// pipe (about 85 operations a sample) once the rest keeps out of its way:
// - the sin/cos table sits in shared memory as four arrays (the lanes look
//   up different points; from global memory those scattered reads took
//   three quarters of the kernel's time, 30 % FP64 pipe);
// - a sample's source point mid + node * half * dir depends on (source,
//   node) alone and is formed once per tile.  The PEC image's points are the
//   direct ones of the mirrored node with z negated: the nodes are symmetric
//   and a rounded sum with both signs turned is the same sum turned;
// - the square root and the two divisions of G(R) share one reciprocal
//   square root (sqrt_recip).
// Two nodes in flight per thread at 4 CTAs per SM (one: 4.50 ms, 2 CTAs with
// 128 registers: 5.2 ms).  Measured, 512 random antennas: 9.26 -> 4.36 ms,
// FP64 pipe 30 -> 57 %; the rest is issue slots of the branches and selects.
struct FillTile {
    double tab[4][112];     // the sin/cos table by part
    double rs[8][3][16];    // source points (node, axis, source)
    double om[3][16], od[3][16], sd[3][16];
    double half[16], a2[16], self_log[16];
};

struct LmSharedTable {
    const double (*t)[112];
    __device__ __forceinline__ fnec_libm::LmEntry operator()(int i) const {
        return {t[0][i], t[1][i], t[2][i], t[3][i]};
    }
};

// w G(R) at R^2 = x added to the sums
__device__ __forceinline__ void add_green(double x, double k, double w, const LmSharedTable &tab, double &sre,
                                          double &sim) {
    double gr, gi, sn, cs;
    SqrtRecip sr = sqrt_recip(x);
    double t = D_MUL(-k, sr.r);
    const uint32_t kt = (uint32_t)(fnec_libm::lm_bits(t) >> 32) & 0x7fffffffu;
    if (sqrt_recip_domain(x) && kt >= 0x39b00000u) {  // kR at least 2^-100: its sine's quotient stays normal
        fnec_libm::libm_sincos(t, &sn, &cs, tab);
        gr = div_by(cs, sr);
        gi = div_by(sn, sr);
    } else {
        const cx g = green_k_exact(D_SQRT(x), k);
        gr = g.re;
        gi = g.im;
    }
    sre = D_ADD(sre, D_MUL(w, gr));
    sim = D_ADD(sim, D_MUL(w, gi));
}

// matrix.rs:186-218: Z[i][j] for rows row0.. and columns col0.. of one system
__device__ __forceinline__ void fill_exact_tile(FillTile &sh, const DevSeg *__restrict__ sg, int n, double k,
                                                int ground, int row0, int col0, cx *__restrict__ z) {
    const int tid = threadIdx.x;
    for (int e = tid; e < 440; e += 256) sh.tab[e & 3][e >> 2] = __ldg(&fnec_libm::libm_sincos_tab_dev[e]);
    if (tid < 128) {  // (source, node)
        const int j = min(col0 + (tid & 15), n - 1), m = tid >> 4;
        const DevSeg &s = sg[j];
        const double half = D_MUL(s.len, 0.5), sc = D_MUL(c_gl_n8[m], half);
#pragma unroll
        for (int c = 0; c < 3; ++c) sh.rs[m][c][tid & 15] = D_ADD(s.mid[c], D_MUL(sc, s.dir[c]));
        if (m == 0) {
#pragma unroll
            for (int c = 0; c < 3; ++c) sh.sd[c][tid] = s.dir[c];
            sh.half[tid] = half;
            sh.a2[tid] = D_MUL(s.rad, s.rad);
            sh.self_log[tid] = s.self_log;
        }
    } else if (tid < 144) {
        const int i = min(row0 + tid - 128, n - 1);
#pragma unroll
        for (int c = 0; c < 3; ++c) {
            sh.om[c][tid - 128] = sg[i].mid[c];
            sh.od[c][tid - 128] = sg[i].dir[c];
        }
    }
    __syncthreads();
    const int ii = tid >> 4, jj = tid & 15;
    const int i = row0 + ii, j = col0 + jj;
    if (i >= n || j >= n) return;
    const LmSharedTable tab{sh.tab};
    const double o0 = sh.om[0][ii], o1 = sh.om[1][ii], o2 = sh.om[2][ii];
    const double half = sh.half[jj], a2 = sh.a2[jj];
    cx direct = cx_make(0.0, 0.0), img = cx_make(0.0, 0.0);
#pragma unroll 1
    for (int image = 0; image <= (ground == 1 ? 1 : 0); ++image) {
        // matrix.rs:297-331 elem; image (:265-279): position (x, y, -z), current (-Jx, -Jy, +Jz)
        double sre = 0.0, sim = 0.0;
        if (i == j && !image) {
#pragma unroll 1
            for (int m = 0; m < 4; ++m) {
                double l = D_MUL(c_gl_n4[m], half);
                double r_eff = D_SQRT(D_ADD(D_MUL(l, l), a2));
                cx g = green_k_exact(r_eff, k);
                sre = D_ADD(sre, D_MUL(c_gl_w4[m], D_SUB(g.re, D_DIV(1.0, r_eff))));
                sim = D_ADD(sim, D_MUL(c_gl_w4[m], g.im));
            }
            sre = D_ADD(D_MUL(sre, half), sh.self_log[jj]);
            sim = D_MUL(sim, half);
        } else {
            const int flip = image ? 7 : 0;
            const uint32_t turn = image ? 0x80000000u : 0u;
#pragma unroll 2
            for (int m = 0; m < 8; ++m) {
                const double(*p)[16] = sh.rs[m ^ flip];
                const double r0 = D_SUB(o0, p[0][jj]), r1 = D_SUB(o1, p[1][jj]);
                const double r2 = D_SUB(o2, fnec_libm::lm_turn(p[2][jj], turn));
                const double r_sq = D_ADD(D_ADD(D_MUL(r0, r0), D_MUL(r1, r1)), D_MUL(r2, r2));
                add_green(D_ADD(r_sq, a2), k, c_gl_w8[m], tab, sre, sim);
            }
            sre = D_MUL(sre, half);
            sim = D_MUL(sim, half);
        }
        const double d0 = sh.sd[0][jj], d1 = sh.sd[1][jj];
        const double cos_alpha = D_ADD(D_ADD(D_MUL(sh.od[0][ii], image ? -d0 : d0),
                                             D_MUL(sh.od[1][ii], image ? -d1 : d1)),
                                       D_MUL(sh.od[2][ii], sh.sd[2][jj]));
        const cx v = cx_make(D_MUL(sre, cos_alpha), D_MUL(sim, cos_alpha));
        if (image) img = v;
        else direct = v;
    }
    z[(int64_t)i * n + j] = cx_add(direct, img);
}

// One CTA of 256 threads fills a 16x16 tile of one unit's Z.
__global__ void __launch_bounds__(256, 4) k_fill_exact(const UnitDesc *__restrict__ units,
                                                       const AntDesc *__restrict__ ants,
                                                       const DevSeg *__restrict__ segs,
                                                       const int4 *__restrict__ tiles, cx *zbuf) {
    __shared__ FillTile sh;
    const int4 t = tiles[blockIdx.x];  // (unit, row0, col0, -)
    const UnitDesc &u = units[t.x];
    const AntDesc &a = ants[u.ant];
    fill_exact_tile(sh, segs + a.seg_off, a.n, u.k_fill, a.ground, t.y, t.z, zbuf + u.z_off);
}

// Fill for caller-provided segments (ZSegmentInput): same arithmetic.
__global__ void __launch_bounds__(256, 4) k_fill_exact_flat(const DevSeg *__restrict__ sg, int n,
                                                            double k, int ground, cx *z) {
    __shared__ FillTile sh;
    fill_exact_tile(sh, sg, n, k, ground, blockIdx.y * 16, blockIdx.x * 16, z);
}

// ---------------------------------------------------------------------------
// Gram:  A[i][j] = sum_r conj(M[r][i]) M[r][j]  (r ascending, no FMA)
// ---------------------------------------------------------------------------
// Part 1: i < N, j <= N over the Z rows r < N, where column j == N is the
// RHS y (aty).  A CTA owns one 32 x 32 output tile on or above the diagonal
// with a 2 x 2 block per thread, k-chunks of 16.  The entry below the
// diagonal is its mirror's conjugate bit for bit: the products of the two
// are the same numbers with the imaginary part's subtraction turned round,
// rounding is symmetric, and a sum that starts at +0 never becomes -0 (so
// the mirrored imaginary part is 0 - im, not -im).
// The FP64 pipe bounds it.  Measured, Gram phase: 512 random antennas 10.1 ms
// with all 64 x 64 tiles, 6.1 with those of the triangle, 5.7 with 32 x 32
// ones (less of a tile past N and past the diagonal); one N = 255 system
// 0.142 -> 0.077 ms (36 CTAs for 10); N = 1680 the same at either width.
__global__ void __launch_bounds__(256) k_gram_zz(const UnitDesc *__restrict__ units,
                                                 const int4 *__restrict__ tiles,
                                                 const cx *__restrict__ zbuf,
                                                 const cx *__restrict__ rhs_buf, cx *abuf) {
    constexpr int T = GRAM_TILE, P = T / 16;
    __shared__ cx s_l[16][T];      // conj side: Z[r][i0 + ii]
    __shared__ cx s_r[16][T + 1];  // right side: B[r][j0 + jj], B = [Z | y]
    int4 t = tiles[blockIdx.x];
    UnitDesc u = units[t.x];
    int n = u.n;
    int i0 = t.y, j0 = t.z;
    const cx *z = zbuf + u.z_off;
    const cx *y = rhs_buf + u.rhs_off;
    int tid = threadIdx.x;
    int ty = tid / 16, tx = tid % 16;
    cx acc[P][P];
#pragma unroll
    for (int a = 0; a < P; ++a)
#pragma unroll
        for (int b = 0; b < P; ++b) acc[a][b] = cx_make(0.0, 0.0);
    for (int r0 = 0; r0 < n; r0 += 16) {
        // load 16 x T of each side
        for (int e = tid; e < 16 * T; e += 256) {
            int rr = e / T, cc = e % T;
            int r = r0 + rr;
            int ci = i0 + cc, cj = j0 + cc;
            cx lv = cx_make(0.0, 0.0), rv = cx_make(0.0, 0.0);
            if (r < n) {
                if (ci < n) lv = z[(int64_t)r * n + ci];
                if (cj < n) rv = z[(int64_t)r * n + cj];
                else if (cj == n) rv = y[r];
            }
            s_l[rr][cc] = lv;
            s_r[rr][cc] = rv;
        }
        __syncthreads();
        int kmax = min(16, n - r0);
        for (int kk = 0; kk < kmax; ++kk) {
            cx lv[P], rv[P];
#pragma unroll
            for (int a = 0; a < P; ++a) lv[a] = s_l[kk][ty + 16 * a];
#pragma unroll
            for (int b = 0; b < P; ++b) rv[b] = s_r[kk][tx + 16 * b];
#pragma unroll
            for (int a = 0; a < P; ++a)
#pragma unroll
                for (int b = 0; b < P; ++b) acc[a][b] = cx_add(acc[a][b], cx_conj_mul(lv[a], rv[b]));
        }
        __syncthreads();
    }
    int w1 = u.s + 1;
    cx *A = abuf + u.a_off;
#pragma unroll
    for (int a = 0; a < P; ++a) {
        int i = i0 + ty + 16 * a;
        if (i >= n) continue;
#pragma unroll
        for (int b = 0; b < P; ++b) {
            int j = j0 + tx + 16 * b;
            if (j < n) {
                A[(int64_t)i * w1 + j] = acc[a][b];
                if (j0 > i0) A[(int64_t)j * w1 + i] = cx_make(acc[a][b].re, D_SUB(0.0, acc[a][b].im));
            } else if (j == n) {
                A[(int64_t)i * w1 + u.s] = acc[a][b];
            }
        }
    }
}

// Part 2: the homogeneous columns N+w (M[r][N+w] = -cos_r for rows of wire
// w, zero elsewhere; zero products change neither value nor sign of a sum
// that starts at +0, so only the wire's rows are visited, in ascending r).
// grid.x = wire column w, grid.y = unit; threads stride over i in [0, N]
// (i == N is the y column).
__global__ void k_gram_ccols(const UnitDesc *__restrict__ units, const AntDesc *__restrict__ ants,
                             const int32_t *__restrict__ ibuf, const cx *__restrict__ zbuf,
                             const cx *__restrict__ rhs_buf, const double *__restrict__ cos_buf,
                             cx *abuf) {
    UnitDesc u = units[blockIdx.y];
    AntDesc a = ants[u.ant];
    int w = blockIdx.x;
    if (w >= a.w) return;
    int n = u.n, s = u.s, w1 = s + 1;
    const cx *z = zbuf + u.z_off;
    const cx *y = rhs_buf + u.rhs_off;
    // the plane-wave form's odd columns hold -sin(k s): the second half
    const double *cv = cos_buf + u.cos_off + ((a.hom2 && (w & 1)) ? n : 0);
    const int32_t *wptr = ibuf + a.wptr_off;
    const int32_t *wrow = ibuf + a.wrow_off;
    cx *A = abuf + u.a_off;
    int b = wptr[w], e = wptr[w + 1];
    for (int i = threadIdx.x; i <= n; i += blockDim.x) {
        cx col = cx_make(0.0, 0.0);  // A[i][N+w]  (i < N)
        cx row = cx_make(0.0, 0.0);  // A[N+w][i]  (i < N), or A[N+w][S] for i == N
        for (int q = b; q < e; ++q) {
            int r = wrow[q];
            cx c = cx_make(-cv[r], 0.0);
            cx zi = (i < n) ? z[(int64_t)r * n + i] : y[r];
            if (i < n) col = cx_add(col, cx_conj_mul(zi, c));
            row = cx_add(row, cx_conj_mul(c, zi));
        }
        if (i < n) {
            A[(int64_t)i * w1 + n + w] = col;
            A[(int64_t)(n + w) * w1 + i] = row;
        } else {
            A[(int64_t)(n + w) * w1 + s] = row;
        }
    }
    // the W x W block row of this column: the sum of squares on the
    // diagonal, and in the plane-wave form the cos-sin cross sum of the same
    // wire (its rows ascending, as the reference's sum over all rows); exact
    // zeros elsewhere
    for (int v = threadIdx.x; v < a.w; v += blockDim.x) {
        cx d = cx_make(0.0, 0.0);
        if (v == w || (a.hom2 && v == (w ^ 1))) {
            const double *cw = cos_buf + u.cos_off + ((a.hom2 && (v & 1)) ? n : 0);
            for (int q = b; q < e; ++q) {
                const int r = wrow[q];
                d = cx_add(d, cx_conj_mul(cx_make(-cv[r], 0.0), cx_make(-cw[r], 0.0)));
            }
        }
        A[(int64_t)(n + w) * w1 + n + v] = d;
    }
}

// Part 3: constraint rows (free-end I = 0 rows, then junction rows, in
// row order), then the Tikhonov term +1e-8 on the diagonal.
__global__ void k_gram_finish(const UnitDesc *__restrict__ units, const AntDesc *__restrict__ ants,
                              const DevConstraint *__restrict__ cons,
                              const int32_t *__restrict__ codes, cx *abuf) {
    UnitDesc u = units[blockIdx.x];
    AntDesc a = ants[u.ant];
    int w1 = u.s + 1;
    cx *A = abuf + u.a_off;
    const DevConstraint *cg = cons + a.con_off;
    const int32_t *cc = codes + a.conv_off;
    for (int g = threadIdx.x; g < a.n_con; g += blockDim.x) {
        DevConstraint c = cg[g];
        cx e = A[(int64_t)c.i * w1 + c.j];
        for (int t = 0; t < c.count; ++t) {
            int code = cc[c.begin + t];
            cx uv = cx_make((code & 2) ? -1.0 : 1.0, 0.0);
            cx vv = cx_make((code & 1) ? -1.0 : 1.0, 0.0);
            e = cx_add(e, cx_conj_mul(uv, vv));
        }
        A[(int64_t)c.i * w1 + c.j] = e;
    }
    __syncthreads();
    for (int i = threadIdx.x; i < u.s; i += blockDim.x) {
        cx d = A[(int64_t)i * w1 + i];
        A[(int64_t)i * w1 + i] = cx_add(d, cx_make(1e-8, 0.0));
    }
}

// ---------------------------------------------------------------------------
// Blocked GEPP with the reference's per-element operation order.
// Panel columns c0 .. c0+NB-1 are factored right-looking inside the panel;
// the row swaps are applied to the trailing columns afterwards, and every
// trailing element then receives its updates in the same column order as
// the unblocked loop, so the result is identical to linear.rs:1343-1370.
// The multipliers f = a[r][c] / a[c][c] are stored in place of a[r][c]
// (the reference leaves a[r][c] - f*a[c][c] there, which it never reads).
// ---------------------------------------------------------------------------
constexpr int NB = 32;

// Pivot reduction: largest hypot, ties resolved to the larger row index
// (Iterator::max_by keeps the last maximum).
__device__ __forceinline__ void piv_better(double &bv, int &bi, double v, int i) {
    if (v > bv || (v == bv && i > bi)) {
        bv = v;
        bi = i;
    }
}

__global__ void __launch_bounds__(256) k_panel(const UnitDesc *__restrict__ units, int c0,
                                               cx *abuf, int32_t *piv_buf, int32_t *status,
                                               const int32_t *__restrict__ order, int base) {
    __shared__ double s_v[8];
    __shared__ int s_i[8];
    __shared__ int s_p;
    __shared__ cx s_prow[NB];
    int ui = order[base + blockIdx.x];
    UnitDesc u = units[ui];
    int s = u.s;
    if (c0 >= s || status[ui] != 0) return;
    int w1 = s + 1;
    cx *A = abuf + u.a_off;
    int32_t *piv = piv_buf + u.piv_off;
    int nb = min(NB, s - c0);
    int tid = threadIdx.x, lane = tid & 31, wid = tid >> 5;
    for (int c = c0; c < c0 + nb; ++c) {
        // --- pivot search over rows c..s-1 of column c
        double bv = -1.0;
        int bi = -1;
        for (int r = c + tid; r < s; r += blockDim.x) piv_better(bv, bi, cx_norm(A[(int64_t)r * w1 + c]), r);
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) {
            double ov = __shfl_down_sync(0xffffffffu, bv, o);
            int oi = __shfl_down_sync(0xffffffffu, bi, o);
            piv_better(bv, bi, ov, oi);
        }
        if (lane == 0) {
            s_v[wid] = bv;
            s_i[wid] = bi;
        }
        __syncthreads();
        if (tid == 0) {
            double v = s_v[0];
            int p = s_i[0];
            for (int q = 1; q < (int)(blockDim.x >> 5); ++q) piv_better(v, p, s_v[q], s_i[q]);
            // linear.rs:1354 singular test on the chosen pivot (NaN never passes <)
            if (p < 0 || v < 1e-30) {
                status[ui] = -(c + 1);
                p = -1;
            }
            s_p = p;
            piv[c] = p;
        }
        __syncthreads();
        int p = s_p;
        if (p < 0) return;
        // --- swap rows c and p inside the panel columns
        if (p != c && tid < nb) {
            int k = c0 + tid;
            cx t0 = A[(int64_t)c * w1 + k];
            A[(int64_t)c * w1 + k] = A[(int64_t)p * w1 + k];
            A[(int64_t)p * w1 + k] = t0;
        }
        __syncthreads();
        if (tid < nb) s_prow[tid] = A[(int64_t)c * w1 + c0 + tid];
        __syncthreads();
        cx diag = s_prow[c - c0];
        // --- eliminate below the pivot inside the panel
        for (int r = c + 1 + tid; r < s; r += blockDim.x) {
            cx *row = A + (int64_t)r * w1;
            cx f = cx_div(row[c], diag);
            row[c] = f;
            for (int k = c + 1; k < c0 + nb; ++k) row[k] = cx_sub(row[k], cx_mul(f, s_prow[k - c0]));
        }
        __syncthreads();
    }
}

__device__ __forceinline__ void cp_async_cx(cx *dst, const cx *src) {
    const uint32_t d = (uint32_t)__cvta_generic_to_shared(dst);
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(d), "l"(src) : "memory");
}

// The panel factorisation of systems up to CP_MAX_CTAS * CP_MAX_ROWS rows: a
// thread per row, the panel in shared memory, the 16 columns being factored
// in registers, and a cluster of CTAs where one CTA's rows do not suffice.
// A column's latency is what bounds it (one system) or the FP64 work of the
// rows (many), so a column takes two barriers and no square root:
// - Rows never move.  Each thread carries the position its row has reached
//   (pos); the pivot's becomes c, and the row that stood at c takes the
//   pivot's.  Rows are written to their positions at the end.
// - The pivot is the largest hypot, the last of equals (piv_better).  Rows
//   are first compared by the high word of re^2 + im^2: a row whose word is
//   two or more below the largest is smaller by 2^-21, relative, and its
//   hypot (within an ulp of exact) is smaller too.  With one row left it is
//   the pivot; otherwise, and where the squares leave the safe range, the
//   hypots are compared as the reference does.
// - The quotients f = a / diag share the reciprocal of |diag|^2 (Markstein's
//   correction, as div_by), correctly rounded inside its exponent range.
// Every element receives f = a_rc / a_cc and a_rk -= f a_ck in column order,
// as in k_panel; the second 16 columns take the first 16 columns' updates in
// the same order before they are factored.
// Measured, factor phase, against one CTA of 256 threads per panel with a
// warp per row and the panel, hypots and divisions from shared memory:
// one N = 255 system 2.04 -> 0.70 ms, 512 random antennas 25.4 -> 10.6 ms,
// 20 x 20 mesh (S = 2520) 19.0 -> 11.8 ms.  About 2,500 cycles a column;
// spreading a short panel over more CTAs costs more in cluster barriers than
// its shorter columns give (N = 255: 0.71 at 256 rows a CTA, 0.84 at 64).
constexpr int CP_MAX_ROWS = 384;  // rows (threads) per CTA: 512 B of panel each
constexpr int CP_MAX_CTAS = 8;    // the portable cluster size
constexpr int CP_W = 16;          // columns held in registers

struct alignas(16) CpRow {  // a candidate pivot row and what the choice needs
    uint32_t hi;            // high word of |a[0]|^2, plus one (0: no row)
    int cnt;                // 1: no other row within the margin
    int pos;                // the row's position
    int pad;
    double z;               // 1 / |a[0]|^2 (recip_rn)
    double v;               // slow path: hypot of a[0]
    cx a[CP_W];             // its entries from the current column on
};
constexpr int CP_WARPS = CP_MAX_ROWS / 32;
struct alignas(16) CpShared {
    CpRow warp[2][CP_WARPS];    // each warp's candidate, by column parity
    CpRow cta[2][CP_MAX_CTAS];  // each CTA's, written by the CTAs of the cluster
    double w_v[CP_WARPS];
    int w_pos[CP_WARPS];
    int pos_of[CP_MAX_ROWS];
};
static size_t cp_smem(int rows) { return sizeof(CpShared) + sizeof(cx) * NB * (size_t)(rows + 1); }

__device__ __forceinline__ uint32_t cluster_rank() {
    uint32_t r;
    asm("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
    return r;
}
__device__ __forceinline__ void cluster_barrier() {
    asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}
// 16-byte store to the same shared-memory address of CTA `rank` of the cluster
__device__ __forceinline__ void st_cluster(void *p, uint32_t rank, uint4 v) {
    const uint32_t a = (uint32_t)__cvta_generic_to_shared(p);
    uint32_t ra;
    asm("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(ra) : "r"(a), "r"(rank));
    asm volatile("st.shared::cluster.v4.u32 [%0], {%1, %2, %3, %4};" ::"r"(ra), "r"(v.x), "r"(v.y), "r"(v.z), "r"(v.w)
                 : "memory");
}

// 1/x rounded to nearest for 2^-400 <= x < 2^400 whose mantissa is not all
// ones: a first guess (2^-20), two Newton steps and Markstein's last one,
// without the branch of a general division, so that it overlaps the column
// updates beside it.
__device__ __forceinline__ double recip_rn(double x) {
    double y;
    asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(x));
#pragma unroll
    for (int q = 0; q < 3; ++q) y = D_FMA(D_FMA(-x, y, 1.0), y, y);
    return y;
}

// num-complex's a / b for the quotients of one pivot b: ns = |b|^2 and
// z = recip_rn(ns).  Each quotient is corrected from z (div_by) where the
// residuals stay normal, else divided as it stands.
__device__ __forceinline__ cx cp_div(cx a, cx b, double ns, double z) {
    const double re = D_ADD(D_MUL(a.re, b.re), D_MUL(a.im, b.im));
    const double im = D_SUB(D_MUL(a.im, b.re), D_MUL(a.re, b.im));
    auto ok = [](double v) {  // 2^-400 <= |v| < 2^400
        const uint32_t k = fnec_libm::lm_hi(v) & 0x7fffffffu;
        return k - 0x26f00000u < 0x58f00000u - 0x26f00000u;
    };
    if (ok(ns) && (uint32_t)fnec_libm::lm_bits(ns) != 0xffffffffu && (ok(re) || re == 0.0) && (ok(im) || im == 0.0))
        return cx_make(div_by(re, {ns, z}), div_by(im, {ns, z}));
    return cx_make(D_DIV(re, ns), D_DIV(im, ns));
}

// The exact choice among a CTA's rows (piv_better over hypots): out of line,
// the column loop seldom needs it.  The warps' winners go through sh.w_*;
// `clustered` waits for the whole cluster, whose CTAs have then all read the
// column's first candidates.
__device__ __noinline__ int exact_pivot(CpShared &sh, cx a0, int pos, bool act, int nw, bool clustered, double *v_out) {
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    double v = -1.0;
    int p = -1;
    if (act) piv_better(v, p, cx_norm(a0), pos);
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        const double ov = __shfl_xor_sync(0xffffffffu, v, o);
        const int oi = __shfl_xor_sync(0xffffffffu, p, o);
        piv_better(v, p, ov, oi);
    }
    if (lane == 0) {
        sh.w_v[wid] = v;
        sh.w_pos[wid] = p;
    }
    if (clustered) cluster_barrier();
    else __syncthreads();
    v = -1.0;
    p = -1;
    for (int q = 0; q < nw; ++q) piv_better(v, p, sh.w_v[q], sh.w_pos[q]);
    *v_out = v;
    return p;
}

// One system per cluster of nc CTAs (CL: nc > 1).
template <bool CL>
__global__ void __launch_bounds__(CP_MAX_ROWS, 1) k_panel_cluster(const UnitDesc *__restrict__ units, int c0, cx *abuf,
                                                               int32_t *piv_buf, int32_t *status,
                                                               const int32_t *__restrict__ order, int base, int nc) {
    extern __shared__ __align__(16) unsigned char s_raw[];
    CpShared &sh = *reinterpret_cast<CpShared *>(s_raw);
    cx *s_f = reinterpret_cast<cx *>(s_raw + sizeof(CpShared));  // [NB][T + 1], by data row
    const int T = blockDim.x, ld = T + 1, nw = T >> 5;
    const int rank = CL ? (int)cluster_rank() : 0;
    const int ui = order[base + blockIdx.x / nc];
    const UnitDesc u = units[ui];
    const int s = u.s;
    if (c0 >= s || status[ui] != 0) return;  // the same in every CTA of the cluster
    const int w1 = s + 1, nb = min(NB, s - c0), m = s - c0;
    cx *A = abuf + u.a_off;
    const int tid = threadIdx.x, lane = tid & 31, wid = tid >> 5;
    const int row0 = rank * T, nl = max(0, min(T, m - row0));  // this CTA's rows
    for (int e = tid; e < nl * nb; e += T) {
        const int rr = e / nb, q = e % nb;
        cp_async_cx(&s_f[q * ld + rr], &A[(int64_t)(c0 + row0 + rr) * w1 + c0 + q]);
    }
    asm volatile("cp.async.commit_group;\n\tcp.async.wait_group 0;" ::: "memory");
    if (CL) cluster_barrier();  // every CTA runs before its shared memory is written
    else __syncthreads();
    const bool mine = tid < nl;
    int pos = c0 + row0 + tid;  // the row's current position
    int ord = mine ? NB : -1;   // the panel column it became the pivot of; NB: none yet, -1: no row
    // a row of this CTA to the same place in every CTA of the cluster, by
    // `n` threads of index `t` (the row is visible to them)
    auto spread = [&](const CpRow *from, CpRow *to, int t, int n) {
        constexpr int Q = sizeof(CpRow) / 16;
        for (int e = t; e < Q * nc; e += n) st_cluster((uint4 *)to + e % Q, e / Q, ((const uint4 *)from)[e % Q]);
    };
    int par = 0;
    for (int h = 0; h * CP_W < nb; ++h) {
        const int hb = h * CP_W, ncol = min(CP_W, nb - hb);
        cx a[CP_W];
#pragma unroll
        for (int k = 0; k < CP_W; ++k) a[k] = mine && k < ncol ? s_f[(hb + k) * ld + tid] : cx_make(0.0, 0.0);
        // the earlier half's updates, pivot by pivot
        for (int c = 0; c < hb; ++c, par ^= 1) {
            if (ord == c) {
#pragma unroll
                for (int k = 0; k < CP_W; ++k) sh.warp[par][0].a[k] = a[k];
            }
            const CpRow *src = &sh.warp[par][0];
            if (CL) {
                src = &sh.cta[par][0];
                const bool owner = __any_sync(0xffffffffu, ord == c);
                __syncwarp();
                if (owner) spread(&sh.warp[par][0], &sh.cta[par][0], lane, 32);
                cluster_barrier();
            } else {
                __syncthreads();
            }
            if (ord > c) {
                const cx f = s_f[c * ld + tid];
#pragma unroll
                for (int k = 0; k < CP_W; ++k) a[k] = cx_sub(a[k], cx_mul(f, src->a[k]));
            }
        }
        if (mine && ord < hb) {
#pragma unroll
            for (int k = 0; k < CP_W; ++k)
                if (k < ncol) s_f[(hb + k) * ld + tid] = a[k];
        }
        // |a[0]|^2, its reciprocal, and the warp's candidate among its rows
        // without a pivot; the reciprocal and the reductions overlap the
        // updates of the other columns when these follow in the same pass
        double n2 = 0.0, z = 0.0;
        unsigned near = 0, top = 0;
        uint32_t wm = 0;
        auto choose = [&](bool act) {
            n2 = D_ADD(D_MUL(a[0].re, a[0].re), D_MUL(a[0].im, a[0].im));
            z = recip_rn(n2);
            const uint32_t key = act ? min(fnec_libm::lm_hi(n2) & 0x7fffffffu, 0x7ff00000u) : 0u;
            wm = __reduce_max_sync(0xffffffffu, key);
            near = __ballot_sync(0xffffffffu, act && key + 1 >= wm);
            top = __ballot_sync(0xffffffffu, act && key == wm);
        };
        auto announce = [&](int pr) {
            CpRow &w = sh.warp[pr][wid];
            if (lane == (top ? __ffs(top) - 1 : 0)) {
#pragma unroll
                for (int k = 0; k < CP_W; ++k) w.a[k] = a[k];
                w.z = z;
                w.hi = top ? wm + 1 : 0;
                w.cnt = __popc(near);
                w.pos = pos;
            }
        };
        choose(ord > hb);
        announce(par);
        for (int lc = 0; lc < ncol; ++lc, par ^= 1) {
            const int col = hb + lc;
            const bool act = ord > col;
            __syncthreads();
            // the largest of n candidates: one is set if no other comes near it
            uint32_t gm;
            int best, p;
            bool one;
            auto largest = [&](const CpRow *cand, int n) {
                const uint4 in = lane < n ? *reinterpret_cast<const uint4 *>(cand + lane) : make_uint4(0, 0, 0, 0);
                gm = __reduce_max_sync(0xffffffffu, in.x);
                best = __ffs(__ballot_sync(0xffffffffu, in.x == gm)) - 1;
                const unsigned cn = __ballot_sync(0xffffffffu, in.x + 1 >= gm && (lane == best || in.x > 0));
                one = __popc(cn) == 1 && __shfl_sync(0xffffffffu, (int)in.y, best) == 1;
                p = __shfl_sync(0xffffffffu, (int)in.z, best);
            };
            largest(sh.warp[par], nw);
            const CpRow *piv = &sh.warp[par][best];
            if (CL) {  // the same among the CTAs
                if (tid == 0 && !one) sh.warp[par][best].cnt = 2;
                if (wid == 0) {
                    __syncwarp();
                    spread(piv, &sh.cta[par][rank], lane, 32);
                }
                cluster_barrier();
                largest(sh.cta[par], nc);
                piv = &sh.cta[par][best];
            }
            // near ties, squares out of range, a column near the singular bound
            if (!one || gm - 1 >= 0x7ff00000u || gm - 1 < 0x34100000u) {
                double v;
                p = exact_pivot(sh, a[0], pos, act, nw, CL, &v);
                if (p < 0 ? tid == 0 : act && pos == p) {  // the CTA's candidate, in warp slot 0
                    CpRow &w = sh.warp[par][0];
#pragma unroll
                    for (int k = 0; k < CP_W; ++k) w.a[k] = a[k];
                    w.z = z;
                    w.v = v;
                    w.pos = p;
                }
                __syncthreads();
                piv = &sh.warp[par][0];
                if (CL) {
                    if (wid == 0) spread(piv, &sh.cta[par][rank], lane, 32);
                    cluster_barrier();
                    v = -1.0;
                    p = -1;
                    best = 0;
                    for (int q = 0; q < nc; ++q) {
                        const int before = p;
                        piv_better(v, p, sh.cta[par][q].v, sh.cta[par][q].pos);
                        if (p != before) best = q;
                    }
                    piv = &sh.cta[par][best];
                }
                // linear.rs:1354 singular test on the chosen pivot (NaN never passes <)
                if (p < 0 || v < 1e-30) p = -1;
            }
            if (rank == 0 && tid == 0) {
                piv_buf[u.piv_off + c0 + col] = p;
                if (p < 0) status[ui] = -(c0 + col + 1);
            }
            if (p < 0) return;  // the same in every CTA of the cluster
            const cx *prow = piv->a;
            const int left = ncol - lc;  // columns left, this one included
            cx f = cx_make(0.0, 0.0);
            const bool row = act && pos != p;  // a row below the pivot
            if (act && !row) {                 // the pivot row: its entries are final
                ord = col;
                pos = c0 + col;
#pragma unroll
                for (int k = 0; k < CP_W; ++k)
                    if (k < left) s_f[(col + k) * ld + tid] = a[k];
            } else if (row) {
                if (pos == c0 + col) pos = p;
                const cx diag = prow[0];
                const double ns = D_ADD(D_MUL(diag.re, diag.re), D_MUL(diag.im, diag.im));
                f = cp_div(a[0], diag, ns, piv->z);
                s_f[col * ld + tid] = f;
                // the columns shift down by one as they are updated
                a[0] = cx_sub(a[1], cx_mul(f, prow[1]));
            }
            if (left > 1) choose(row);
            if (row) {
#pragma unroll
                for (int k0 = 2; k0 < CP_W; k0 += 2) {
                    if (k0 < left) {
#pragma unroll
                        for (int k = k0; k < k0 + 2; ++k) a[k - 1] = cx_sub(a[k], cx_mul(f, prow[k]));
                    }
                }
            }
            if (left > 1) announce(par ^ 1);
        }
    }
    if (mine) sh.pos_of[tid] = pos;
    __syncthreads();
    for (int e = tid; e < nl * nb; e += T) {
        const int rr = e / nb, q = e % nb;
        A[(int64_t)sh.pos_of[rr] * w1 + c0 + q] = s_f[q * ld + rr];
    }
    if (CL) cluster_barrier();
}

// Panels taller than the largest cluster holds: the grid-wide panel of
// fnec_grid.cuh over gridDim.x CTAs per unit (gridDim.y units, the tallest
// first), launched cooperatively.  Bit-identical to k_panel.
struct ExactPanelOps {
    using E = cx;
    using V = double;
    static constexpr double V_NONE = -1.0;
    __device__ static double key(cx a) { return cx_norm(a); }
    __device__ static void better(double &bv, int &bi, double v, int i) { piv_better(bv, bi, v, i); }
    __device__ static cx div(cx a, cx b) { return cx_div(a, b); }
    __device__ static cx sub_mul(cx acc, cx f, cx p) { return cx_sub(acc, cx_mul(f, p)); }
    __device__ static bool singular(double v) { return v < 1e-30; }  // linear.rs:1354
    __device__ static cx load_cg(const cx *p) {
        double2 d = __ldcg(reinterpret_cast<const double2 *>(p));
        return cx_make(d.x, d.y);
    }
};

__global__ void __launch_bounds__(256) k_panel_grid(const UnitDesc *__restrict__ units,
                                                    const int32_t *__restrict__ order, int c0, cx *abuf,
                                                    int32_t *piv_buf, int32_t *status, PanelXchg<cx> *xg,
                                                    GridSync *gs) {
    extern __shared__ cx s_gpan[];
    int ui = order[blockIdx.y];
    UnitDesc u = units[ui];
    if (status[ui] != 0) return;
    panel_grid_body<ExactPanelOps, NB, 256>(abuf + u.a_off, (int64_t)u.s + 1, u.s, c0, piv_buf + u.piv_off,
                                            &status[ui], xg + blockIdx.y, gs + blockIdx.y, (int)gridDim.x,
                                            (int)blockIdx.x, s_gpan);
}

// Deferred swaps and the U12 block row.  A CTA of 128 threads owns SU_COLS
// columns outside the panel.  The panel's swaps are first followed on row
// numbers alone, so the rows they touch (the panel's NB and up to NB below)
// are all loaded at once and each row takes its final one's values: one
// memory latency where following them on the values took up to NB in turn.
// Right of the panel, row c0 + q then receives the updates of panel columns
// c0 .. c0 + q - 1 in order, four lanes per column, each with every fourth
// row, the pivot column's entry by shuffle.
// Measured, per step of one N = 255 system: 24 -> 15 us (its factor 0.70 ->
// 0.65 ms); 512 random antennas' steps together 1.95 -> 1.58 ms.
constexpr int SU_COLS = 32;
constexpr int SU_LD = SU_COLS + 2;

__global__ void __launch_bounds__(4 * SU_COLS) k_swap_u12(const UnitDesc *__restrict__ units, int c0, cx *abuf,
                                                         const int32_t *__restrict__ piv_buf,
                                                         const int32_t *__restrict__ status,
                                                         const int32_t *__restrict__ order, int base) {
    extern __shared__ cx s_su[];
    cx(*s_v)[SU_LD] = reinterpret_cast<cx(*)[SU_LD]>(s_su);                     // [2 NB] rows before the swaps
    cx(*s_L)[NB + 1] = reinterpret_cast<cx(*)[NB + 1]>(s_su + 2 * NB * SU_LD);  // the panel's block
    __shared__ int s_row[2 * NB], s_idx[2 * NB], s_slot[NB];
    int ui = order[base + blockIdx.y];
    UnitDesc u = units[ui];
    int s = u.s;
    if (c0 >= s || status[ui] != 0) return;
    const int nb = min(NB, s - c0);
    const int w1 = s + 1;
    cx *A = abuf + u.a_off;
    const int t = threadIdx.x;
    // columns left of the panel (earlier panels' multipliers) come last:
    // swaps only, so that every row of L ends up with the row it belongs to
    const int n_left = (c0 + SU_COLS - 1) / SU_COLS, x = (int)blockIdx.x - ((int)gridDim.x - n_left);
    const bool left = x >= 0;
    const int K0 = left ? x * SU_COLS : c0 + nb + (int)blockIdx.x * SU_COLS;  // column s is the right-hand side
    const int K1 = left ? c0 : s + 1;
    if (K0 >= K1) return;
    if (t < NB) {
        // slot t: panel row c0 + t; slot NB + q: the row below the panel that
        // pivot q names first (-1: none)
        const int p = t < nb ? piv_buf[u.piv_off + c0 + t] : -1;
        int slot = p < c0 + nb ? p - c0 : -1;  // p >= c0 always
        for (int q = NB - 1; q >= 0; --q) {
            const int pq = __shfl_sync(0xffffffffu, p, q);
            if (p >= c0 + nb && pq == p) slot = NB + q;  // ends at the first
        }
        s_slot[t] = slot;
        s_row[t] = t < nb ? c0 + t : -1;
        s_row[NB + t] = slot == NB + t ? p : -1;
        s_idx[t] = t;
        s_idx[NB + t] = NB + t;
        __syncwarp();
        if (t == 0)
            for (int q = 0; q < nb; ++q) {
                const int o = s_slot[q], i0 = s_idx[q];
                s_idx[q] = s_idx[o];
                s_idx[o] = i0;
            }
    }
    __syncthreads();
    for (int e = t; e < 2 * NB * SU_COLS; e += 4 * SU_COLS) {
        const int r = s_row[e / SU_COLS], K = K0 + e % SU_COLS;
        if (r >= 0 && K < K1) cp_async_cx(&s_v[e / SU_COLS][e % SU_COLS], &A[(int64_t)r * w1 + K]);
    }
    if (!left)
        for (int e = t; e < nb * nb; e += 4 * SU_COLS)
            cp_async_cx(&s_L[e / nb][e % nb], &A[(int64_t)(c0 + e / nb) * w1 + c0 + e % nb]);
    asm volatile("cp.async.commit_group;\n\tcp.async.wait_group 0;" ::: "memory");
    __syncthreads();
    // the rows that moved: below the panel for every column, in it for the left ones
    for (int e = t; e < 2 * NB * SU_COLS; e += 4 * SU_COLS) {
        const int i = e / SU_COLS, r = s_row[i], K = K0 + e % SU_COLS;
        if (r >= 0 && s_idx[i] != i && (left || i >= NB) && K < K1) A[(int64_t)r * w1 + K] = s_v[s_idx[i]][e % SU_COLS];
    }
    if (left) return;
    const int part = t & 3, col = t >> 2, K = K0 + col;
    const unsigned from = (t & 31) & ~3u;
    cx v[NB / 4];
#pragma unroll
    for (int i = 0; i < NB / 4; ++i) {
        const int q = part + 4 * i;
        v[i] = q < nb && K < K1 ? s_v[s_idx[q]][col] : cx_make(0.0, 0.0);
    }
#pragma unroll
    for (int c = 0; c < NB - 1; ++c) {
        if (c + 1 >= nb) break;
        const cx p = cx_make(__shfl_sync(0xffffffffu, v[c / 4].re, from + (c & 3)),
                             __shfl_sync(0xffffffffu, v[c / 4].im, from + (c & 3)));
#pragma unroll
        for (int i = c / 4; i < NB / 4; ++i) {
            const int q = part + 4 * i;
            if (q > c && q < nb) v[i] = cx_sub(v[i], cx_mul(s_L[q][c], p));
        }
    }
    if (K < K1) {
#pragma unroll
        for (int i = 0; i < NB / 4; ++i)
            if (part + 4 * i < nb) A[(int64_t)(c0 + part + 4 * i) * w1 + K] = v[i];
    }
}
constexpr size_t SU_SMEM = sizeof(cx) * (2 * NB * SU_LD + NB * (NB + 1));

// A22 -= L21 * U12 with per-element in-order accumulation over the panel.
// grid.x = tiles of TT x TT over the trailing block, grid.y = unit.
// The panel blocks stage by cp.async beside the tile's own loads.  32 wide, as
// the Gram's tiles, for their raggedness and the number of CTAs: factor phase
// against 64 x 64 tiles staged first, one N = 255 system 0.65 -> 0.57 ms, 512
// random antennas 10.4 -> 9.4, 20 x 20 mesh 11.4 -> 10.9.  64 wide from
// TRAILING_WIDE_ROWS on, where neither counts and each entry of a staged block
// serves four products instead of two: 46 x 46 mesh (S = 12,972) 448 -> 426 ms,
// 40 x 40 (9840) 214 -> 205, 30 x 30 (5580) 55.1 -> 54.0, 24 x 24 (3600) 21.28
// -> 21.22; the same from 1024 or 3072 rows on, and 20 x 20 (2520) 10.83 = 10.85
// from 2048 on but 10.96 from 1024.
constexpr int TRAILING_WIDE_ROWS = 2048;
template <int TT>
__global__ void __launch_bounds__(256) k_trailing(const UnitDesc *__restrict__ units, int c0,
                                                  cx *abuf, const int32_t *__restrict__ status, const int32_t *__restrict__ order, int base) {
    constexpr int P = TT / 16;
    extern __shared__ cx s_tt[];
    cx(*s_l)[NB + 1] = reinterpret_cast<cx(*)[NB + 1]>(s_tt);
    cx(*s_u)[TT] = reinterpret_cast<cx(*)[TT]>(s_tt + TT * (NB + 1));
    int ui = order[base + blockIdx.y];
    UnitDesc u = units[ui];
    int s = u.s;
    if (c0 + NB >= s || status[ui] != 0) return;  // no trailing block (or a failed unit)
    int r0 = c0 + NB;  // first trailing row/column
    int rows = s - r0, cols = s + 1 - r0;
    int tiles_c = (cols + TT - 1) / TT;
    int tiles_r = (rows + TT - 1) / TT;
    int tile = blockIdx.x;
    if (tile >= tiles_r * tiles_c) return;
    int R0 = r0 + (tile / tiles_c) * TT;
    int K0 = r0 + (tile % tiles_c) * TT;
    int w1 = s + 1;
    cx *A = abuf + u.a_off;
    int tid = threadIdx.x;
    int ty = tid / 16, tx = tid % 16;
    // the panel blocks stage while the tile's own entries load; rows and
    // columns past the end repeat the last one and are not written back
    for (int e = tid; e < TT * NB; e += 256)
        cp_async_cx(&s_l[e / NB][e % NB], &A[(int64_t)min(R0 + e / NB, s - 1) * w1 + c0 + e % NB]);
    for (int e = tid; e < NB * TT; e += 256)
        cp_async_cx(&s_u[e / TT][e % TT], &A[(int64_t)(c0 + e / TT) * w1 + min(K0 + e % TT, s)]);
    asm volatile("cp.async.commit_group;" ::: "memory");
    cx acc[P][P];
#pragma unroll
    for (int a = 0; a < P; ++a)
#pragma unroll
        for (int b = 0; b < P; ++b) {
            int R = R0 + ty + 16 * a, K = K0 + tx + 16 * b;
            acc[a][b] = (R < s && K <= s) ? A[(int64_t)R * w1 + K] : cx_make(0.0, 0.0);
        }
    asm volatile("cp.async.wait_group 0;" ::: "memory");
    __syncthreads();
#pragma unroll (TT == 32 ? 4 : 1)
    for (int q = 0; q < NB; ++q) {
        cx lv[P], uv[P];
#pragma unroll
        for (int a = 0; a < P; ++a) lv[a] = s_l[ty + 16 * a][q];
#pragma unroll
        for (int b = 0; b < P; ++b) uv[b] = s_u[q][tx + 16 * b];
#pragma unroll
        for (int a = 0; a < P; ++a)
#pragma unroll
            for (int b = 0; b < P; ++b) acc[a][b] = cx_sub(acc[a][b], cx_mul(lv[a], uv[b]));
    }
#pragma unroll
    for (int a = 0; a < P; ++a)
#pragma unroll
        for (int b = 0; b < P; ++b) {
            int R = R0 + ty + 16 * a, K = K0 + tx + 16 * b;
            if (R < s && K <= s) A[(int64_t)R * w1 + K] = acc[a][b];
        }
}
template <int TT>
static void launch_trailing(const UnitDesc *units, int n, int rows, int cols, int c0, cx *A, int32_t *status,
                            const int32_t *order, int base, cudaStream_t st) {
    constexpr size_t smem = sizeof(cx) * (TT * (NB + 1) + NB * TT);
    set_smem_limit_once(k_trailing<TT>, (int)smem);
    dim3 g(((rows + TT - 1) / TT) * ((cols + TT - 1) / TT), n);
    k_trailing<TT><<<g, 256, smem, st>>>(units, c0, A, status, order, base);
}

// Back substitution x_i = (b_i - sum_{j>i} a_ij x_j) / a_ii, j ascending.
// The reference's subtraction chain is sequential, and since each row's
// first term needs the x just found, all S^2/2 subtractions form one
// dependent chain; its bound is that count times the latency of a double
// add.  So one warp does nothing but the chain, and two warps form the
// products ahead of it: the U entries arrive by cp.async in pieces of BP
// columns three pieces ahead, and the piece after the one being subtracted
// is multiplied by its x in place.  A row's products start at column i + 2;
// the chain warp itself forms a_{i,i+1} x_{i+1}, the only term whose x is
// new when the row begins.  One barrier per piece.
// Measured, 20 x 20 mesh (S = 2520, 3.2 M subtractions): 48.4 ms with one
// warp that formed and shuffled the products between the subtractions (30
// cycles each) -> 15.9 ms (9.8 cycles; a dependent double add takes 8.2;
// 17.3 with the subtractions in loops of 16 instead of 64).
// 512 random antennas (S up to 700): 3.47 -> 1.06 ms.
// x may alias b (b_in_x: b is read from x): b_i is read before x_i is
// written, and only x_j, j > i, is read after.
constexpr int BP = 256;          // products per piece: 2,000+ cycles of chain per barrier
constexpr int BP_RING = 4;       // pieces: consumed, multiplied, two in flight
constexpr int BP_SLOT = BP + 3;  // then a_ii, a_{i,i+1} and b_i of a row's first piece
constexpr int BS_PROD = 64;      // product threads
constexpr int BS_THREADS = 32 + BS_PROD;
constexpr size_t BS_RING_BYTES = sizeof(cx) * BP_RING * BP_SLOT;
constexpr size_t BS_SMEM_MAX = 226 * 1024;  // x staged in shared memory beside the ring up to S = 13,427

struct PieceCursor {  // columns j0 .. j0 + BP - 1 of row i
    int i, j0;
    __device__ void next(int s) {
        j0 += BP;
        if (j0 >= s) {
            --i;
            j0 = i + 2;
        }
    }
};

// All BS_THREADS threads; ring: BP_RING * BP_SLOT entries of shared memory.
__device__ __forceinline__ void backsub_rows(const cx *A, int s, int w1, const cx *bv, int64_t b_stride,
                                             bool b_in_x, cx *xs, cx *ring) {
    const int tid = threadIdx.x, pt = tid - 32;
    PieceCursor cur{s - 1, s + 1}, ahead = cur;
    int t = 0;  // piece under the chain's hand
    cx x_prev = cx_make(0.0, 0.0), sum = x_prev, diag = x_prev;
    auto load = [&](int piece) {
        cx *slot = ring + (piece % BP_RING) * BP_SLOT;
        if (ahead.i >= 0) {
            const cx *row = A + (int64_t)ahead.i * w1;
            for (int e = pt; e < BP && ahead.j0 + e < s; e += BS_PROD) cp_async_cx(slot + e, row + ahead.j0 + e);
            if (ahead.j0 == ahead.i + 2) {
                if (pt == 0) cp_async_cx(slot + BP, row + ahead.i);
                if (pt == 1 && ahead.i + 1 < s) cp_async_cx(slot + BP + 1, row + ahead.i + 1);
                if (pt == 2 && !b_in_x) cp_async_cx(slot + BP + 2, bv + (int64_t)ahead.i * b_stride);
            }
            ahead.next(s);
        }
        asm volatile("cp.async.commit_group;" ::: "memory");
    };
    auto multiply = [&](int piece, PieceCursor c) {
        cx *slot = ring + (piece % BP_RING) * BP_SLOT;
        asm volatile("cp.async.wait_group 2;" ::: "memory");  // all but the two youngest pieces have landed
        if (c.i < 0) return;
        const int cnt = max(0, min(BP, s - c.j0)), cnt16 = (cnt + 15) & ~15;
        // entries past the row's end are +0: sum - (+0) == sum for every sum
        for (int e = pt; e < cnt16; e += BS_PROD)
            slot[e] = e < cnt ? cx_mul(slot[e], xs[c.j0 + e]) : cx_make(0.0, 0.0);
    };
    if (tid >= 32) {
        for (int q = 0; q < BP_RING - 1; ++q) load(q);
        multiply(0, cur);
    }
    __syncthreads();
    while (cur.i >= 0) {
        if (tid >= 32) {
            load(t + BP_RING - 1);
            PieceCursor nx = cur;
            nx.next(s);
            multiply(t + 1, nx);
        } else {
            const cx *slot = ring + (t % BP_RING) * BP_SLOT;
            const int cnt = (max(0, min(BP, s - cur.j0)) + 15) & ~15;
            if (cur.j0 == cur.i + 2) {
                diag = slot[BP];
                sum = b_in_x ? xs[cur.i] : slot[BP + 2];
                if (cur.i + 1 < s) sum = cx_sub(sum, cx_mul(slot[BP + 1], x_prev));
            }
            // two banks of eight products: one is read while the other is subtracted
            cx p0[8], p1[8];
            auto read8 = [&](cx(&p)[8], int e) {
                const cx *q8 = slot + min(e, BP - 8);  // past the end: not used
#pragma unroll
                for (int q = 0; q < 8; ++q) p[q] = q8[q];
            };
            auto sub16 = [&](int e) {
                read8(p1, e + 8);
#pragma unroll
                for (int q = 0; q < 8; ++q) sum = cx_sub(sum, p0[q]);
                read8(p0, e + 16);
#pragma unroll
                for (int q = 0; q < 8; ++q) sum = cx_sub(sum, p1[q]);
            };
            read8(p0, 0);
            int e = 0;
#pragma unroll 1
            for (; e + 64 <= cnt; e += 64) {
                sub16(e);
                sub16(e + 16);
                sub16(e + 32);
                sub16(e + 48);
            }
#pragma unroll 1
            for (; e < cnt; e += 16) sub16(e);
            if (cur.j0 + BP >= s) {
                x_prev = cx_div(sum, diag);
                if (tid == 0) xs[cur.i] = x_prev;
            }
        }
        cur.next(s);
        ++t;
        __syncthreads();
    }
}

// staged == 0 (systems whose x does not fit in shared memory beside the
// ring): x is built in place in global memory.
__global__ void __launch_bounds__(BS_THREADS) k_backsub(const UnitDesc *__restrict__ units,
                                                        const int32_t *__restrict__ order, const cx *__restrict__ abuf,
                                                        cx *xbuf, const int32_t *__restrict__ status, int staged) {
    extern __shared__ cx s_xs[];
    int ui = order[blockIdx.x];  // tallest first: a tall system's chain is the batch's latency
    UnitDesc u = units[ui];
    if (status[ui] != 0) return;
    int s = u.s, w1 = s + 1;
    const cx *A = abuf + u.a_off;
    cx *xs = staged ? s_xs + BP_RING * BP_SLOT : xbuf + u.x_off;
    backsub_rows(A, s, w1, A + s, w1, false, xs, s_xs);
    if (staged)
        for (int i = threadIdx.x; i < s; i += BS_THREADS) xbuf[u.x_off + i] = xs[i];
}

// Feedpoint rows: v_source = v_vec[idx] * dl, Zin = v_source / I[idx] when
// |I| > 1e-60 (solve_session.rs:911-917).  One CTA per solve; its rows are
// the feed rows of its right-hand side.
__global__ void k_feedpoints(const UnitDesc *__restrict__ solves, const AntDesc *__restrict__ ants,
                             const DevSeg *__restrict__ segs, const int32_t *__restrict__ ibuf,
                             const DevFeed *__restrict__ feeds, const cx *__restrict__ xbuf,
                             const int32_t *__restrict__ status, double *feed_out,
                             const int64_t *__restrict__ feed_row_off) {
    int si = blockIdx.x;
    UnitDesc u = solves[si];
    AntDesc a = ants[u.ant];
    const int32_t *fptr = ibuf + a.fptr_off;
    int f0 = fptr[u.rhs], nf = fptr[u.rhs + 1] - f0;
    for (int q = threadIdx.x; q < nf; q += blockDim.x) {
        DevFeed f = feeds[a.feed_off + f0 + q];
        double *o = feed_out + 7 * (feed_row_off[si] + q);
        if (status[u.sys] != 0) {
            for (int t = 0; t < 7; ++t) o[t] = 0.0;
            continue;
        }
        double dl = segs[a.seg_off + f.seg].len;
        cx vs = cx_make(D_MUL(f.vdl_re, dl), D_MUL(f.vdl_im, dl));
        cx cur = xbuf[u.x_off + f.seg];
        cx zin = cx_norm(cur) > 1e-60 ? cx_div(vs, cur) : vs;
        o[0] = (double)f.seg;
        o[1] = vs.re;
        o[2] = vs.im;
        o[3] = cur.re;
        o[4] = cur.im;
        o[5] = zin.re;
        o[6] = zin.im;
    }
}

// ---------------------------------------------------------------------------
// Further right-hand sides on the factored system (solves with rhs >= 1).
// The reference re-runs the whole elimination for another source; A does
// not depend on the source, so its operations on A repeat exactly and only
// the b column differs.  b = M^H y is formed in the Gram's order; the row
// swaps, the multipliers (stored in L with all later swaps applied, so row
// r of L is the row that ends at position r) and the back substitution then
// give b exactly the sequence of operations the reference's augmented
// column receives.
// ---------------------------------------------------------------------------
__global__ void k_extra_rhs_b(const UnitDesc *__restrict__ solves, const AntDesc *__restrict__ ants,
                              const int32_t *__restrict__ ibuf, const cx *__restrict__ zbuf,
                              const cx *__restrict__ rhs_buf, const double *__restrict__ cos_buf, cx *xbuf,
                              int first_rhs) {
    UnitDesc u = solves[blockIdx.y];
    if (u.rhs < first_rhs) return;
    AntDesc a = ants[u.ant];
    int n = u.n;
    int i = blockIdx.x * blockDim.x + threadIdx.x;
    const cx *z = zbuf + u.z_off;
    const cx *y = rhs_buf + u.rhs_off;
    cx *b = xbuf + u.x_off;
    if (i < n) {
        cx acc = cx_make(0.0, 0.0);
        for (int r = 0; r < n; ++r) acc = cx_add(acc, cx_conj_mul(z[(int64_t)r * n + i], y[r]));
        b[i] = acc;
    } else if (i < n + a.w) {
        int w = i - n;
        const int32_t *wptr = ibuf + a.wptr_off, *wrow = ibuf + a.wrow_off;
        const double *cv = cos_buf + u.cos_off + ((a.hom2 && (w & 1)) ? n : 0);
        cx acc = cx_make(0.0, 0.0);
        for (int q = wptr[w]; q < wptr[w + 1]; ++q) {
            int r = wrow[q];
            acc = cx_add(acc, cx_conj_mul(cx_make(-cv[r], 0.0), y[r]));
        }
        b[i] = acc;
    }
}

__global__ void __launch_bounds__(BS_THREADS) k_extra_rhs_solve(const UnitDesc *__restrict__ solves,
                                                                const cx *__restrict__ abuf,
                                                                const int32_t *__restrict__ piv_buf, cx *xbuf,
                                                                const int32_t *__restrict__ status, int staged,
                                                                int first_rhs) {
    extern __shared__ cx s_bs[];
    UnitDesc u = solves[blockIdx.x];
    if (u.rhs < first_rhs || status[u.sys] != 0) return;
    int s = u.s, w1 = s + 1;
    const cx *A = abuf + u.a_off;
    const int32_t *piv = piv_buf + u.piv_off;
    cx *x = xbuf + u.x_off;
    cx *s_b = staged ? s_bs + BP_RING * BP_SLOT : x;  // unstaged: work in place in global memory
    const int tid = threadIdx.x;
    if (staged)
        for (int i = tid; i < s; i += BS_THREADS) s_b[i] = x[i];
    __syncthreads();
    if (tid == 0)
        for (int c = 0; c < s; ++c) {
            int p = piv[c];
            if (p != c) {
                cx t0 = s_b[c];
                s_b[c] = s_b[p];
                s_b[p] = t0;
            }
        }
    __syncthreads();
    // forward: row r receives b[r] -= f[r][c] * b[c] for c = 0..r-1 in order
    for (int c = 0; c < s; ++c) {
        cx bc = s_b[c];
        for (int r = c + 1 + tid; r < s; r += BS_THREADS)
            s_b[r] = cx_sub(s_b[r], cx_mul(A[(int64_t)r * w1 + c], bc));
        __syncthreads();
    }
    // back substitution, j ascending, as k_backsub (x overwrites b in place)
    backsub_rows(A, s, w1, s_b, 1, true, s_b, s_bs);
    if (staged)
        for (int i = tid; i < s; i += BS_THREADS) x[i] = s_b[i];
}

// ---------------------------------------------------------------------------
// Many right-hand sides on one factorisation (a receive sweep's incidence
// directions), in groups of up to 32 solves of one system: group g =
// (system, first solve, count).  k_extra_rhs_b_group forms M^H y of every
// solve of the group with Z read once per group: thread i keeps the 32
// accumulators of row i, each summed over r ascending exactly as
// k_extra_rhs_b sums it.  k_extra_rhs_solve_group gives each solve one lane
// (16 per block): its right-hand side lives in a shared [s][16] tile, the row swaps, the
// forward elimination (b[r] -= f[r][c] b[c], c ascending) and the back
// substitution (j ascending, then the division) are k_extra_rhs_solve's
// operations in its order, with the factor read warp-uniformly.
// ---------------------------------------------------------------------------
constexpr int RG = 32;  // solves per group
constexpr int SG = 16;  // solves per substitution block: a [s][16] tile, several blocks per SM
constexpr size_t GS_SMEM_MAX = 220 * 1024;  // their dynamic shared memory

__global__ void __launch_bounds__(64) k_extra_rhs_b_group(const UnitDesc *__restrict__ solves,
                                                          const int4 *__restrict__ groups,
                                                          const AntDesc *__restrict__ ants,
                                                          const int32_t *__restrict__ ibuf,
                                                          const cx *__restrict__ zbuf,
                                                          const cx *__restrict__ rhs_buf,
                                                          const double *__restrict__ cos_buf, cx *xbuf) {
    __shared__ cx Y[RG][RG];  // [row in chunk][solve]
    const int4 g = groups[blockIdx.y];
    const UnitDesc u0 = solves[g.y];
    const int n = u0.n, s = u0.s;
    if ((int)(blockIdx.x * blockDim.x) >= s) return;  // the whole block: no barrier is skipped
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    const cx *z = zbuf + u0.z_off;
    cx acc[RG];
#pragma unroll
    for (int d = 0; d < RG; ++d) acc[d] = cx_make(0.0, 0.0);
    for (int r0 = 0; r0 < n; r0 += RG) {
        __syncthreads();
        for (int t = threadIdx.x; t < RG * RG; t += blockDim.x) {
            const int d = t / RG, rr = t % RG;
            Y[rr][d] = (d < g.z && r0 + rr < n) ? rhs_buf[solves[g.y + d].rhs_off + r0 + rr] : cx_make(0.0, 0.0);
        }
        __syncthreads();
        if (i < n) {
            const int rmax = min(RG, n - r0);
            for (int rr = 0; rr < rmax; ++rr) {
                const cx zz = z[(int64_t)(r0 + rr) * n + i];
#pragma unroll
                for (int d = 0; d < RG; ++d) acc[d] = cx_add(acc[d], cx_conj_mul(zz, Y[rr][d]));
            }
        }
    }
    if (i < n) {
#pragma unroll
        for (int d = 0; d < RG; ++d)  // static indices keep acc in registers
            if (d < g.z) xbuf[solves[g.y + d].x_off + i] = acc[d];
    } else if (i < s) {  // a homogeneous column: its rows' -cos (or -sin) values
        const AntDesc a = ants[u0.ant];
        const int w = i - n;
        const int32_t *wptr = ibuf + a.wptr_off, *wrow = ibuf + a.wrow_off;
        const double *cv = cos_buf + u0.cos_off + ((a.hom2 && (w & 1)) ? n : 0);
        for (int d = 0; d < g.z; ++d) {
            const cx *y = rhs_buf + solves[g.y + d].rhs_off;
            cx b = cx_make(0.0, 0.0);
            for (int q = wptr[w]; q < wptr[w + 1]; ++q) {
                const int r = wrow[q];
                b = cx_add(b, cx_conj_mul(cx_make(-cv[r], 0.0), y[r]));
            }
            xbuf[solves[g.y + d].x_off + i] = b;
        }
    }
}

// The factor streams through the lanes in 16-wide row chunks, PD chunks
// ahead of the arithmetic: lane k loads entry c0 + k of a chunk (one
// coalesced access), and the chain receives the entries in column order
// by shuffles.  Forward chunks: rows 1 .. s-1, columns 0 .. r-1; back
// chunks: rows s-1 .. 0, columns i+1 .. s-1 (rows without any skipped).
constexpr int PD = 8;
struct FwdChunks {
    int r, c0;
    __device__ void next(int s) {
        c0 += SG;
        if (c0 >= r) {
            ++r;
            c0 = 0;
        }
        (void)s;
    }
    __device__ bool valid(int s) const { return r < s; }
    __device__ int end(int s) const { return r; }
};
struct BackChunks {
    int r, c0;
    __device__ void norm(int s) {
        while (r >= 0 && c0 >= s) {
            --r;
            c0 = r + 1;
        }
    }
    __device__ void next(int s) {
        c0 += SG;
        norm(s);
    }
    __device__ bool valid(int s) const { return r >= 0; }
    __device__ int end(int s) const { return s; }
};

template <typename Cur>
__device__ __forceinline__ cx chunk_entry(const cx *A, int w1, int s, const Cur &pf, int l) {
    const int c = pf.c0 + l;
    return (pf.valid(s) && c < pf.end(s)) ? A[(int64_t)pf.r * w1 + c] : cx_make(0.0, 0.0);
}

__global__ void __launch_bounds__(SG) k_extra_rhs_solve_group(const UnitDesc *__restrict__ solves,
                                                             const int4 *__restrict__ groups,
                                                             const cx *__restrict__ abuf,
                                                             const int32_t *__restrict__ piv_buf, cx *xbuf,
                                                             const int32_t *__restrict__ status) {
    extern __shared__ cx B[];  // [s][SG], then the diagonal [s], then the pivots (int32 [s])
    const int4 g = groups[blockIdx.x];
    const UnitDesc u0 = solves[g.y];
    if (status[u0.sys] != 0 || (int)(blockIdx.y * SG) >= g.z) return;
    const int s = u0.s, w1 = s + 1, d = blockIdx.y * SG + threadIdx.x, l = threadIdx.x;
    const unsigned mask = (1u << SG) - 1u;
    cx *diag = B + (size_t)s * SG;
    int32_t *pv = reinterpret_cast<int32_t *>(diag + s);
    const cx *A = abuf + u0.a_off;
    const int32_t *piv = piv_buf + u0.piv_off;
    for (int i = l; i < s; i += SG) {
        diag[i] = A[(int64_t)i * w1 + i];
        pv[i] = piv[i];
    }
    const bool live = d < g.z;
    cx *x = xbuf + solves[g.y + (live ? d : 0)].x_off;
    for (int j = 0; j < s; ++j) B[j * SG + l] = live ? x[j] : cx_make(0.0, 0.0);
    __syncwarp(mask);
    for (int c = 0; c < s; ++c) {
        const int p = pv[c];
        if (p != c) {
            const cx t = B[c * SG + l];
            B[c * SG + l] = B[p * SG + l];
            B[p * SG + l] = t;
        }
    }
    // forward elimination row by row: row r receives b[r] -= f[r][c] b[c]
    // for c ascending -- the operations and order of the column sweep, as
    // every b[c] with c < r is final when row r starts
    {
        FwdChunks pf{1, 0};
        cx u[PD];
#pragma unroll
        for (int q = 0; q < PD; ++q) {
            u[q] = chunk_entry(A, w1, s, pf, l);
            if (pf.valid(s)) pf.next(s);
        }
        for (int r = 1; r < s; ++r) {
            cx sum = B[r * SG + l];
            for (int c0 = 0; c0 < r; c0 += SG) {
                const cx uv = u[0];
#pragma unroll
                for (int q = 0; q < PD - 1; ++q) u[q] = u[q + 1];
                u[PD - 1] = chunk_entry(A, w1, s, pf, l);
                if (pf.valid(s)) pf.next(s);
                const int cnt = min(SG, r - c0);
#pragma unroll
                for (int q = 0; q < SG; ++q) {
                    const cx a = cx_make(__shfl_sync(mask, uv.re, q, SG), __shfl_sync(mask, uv.im, q, SG));
                    if (q < cnt) sum = cx_sub(sum, cx_mul(a, B[(c0 + q) * SG + l]));
                }
            }
            B[r * SG + l] = sum;
        }
    }
    // back substitution: j ascending, then the division by the diagonal
    {
        BackChunks pf{s - 1, s};
        pf.norm(s);
        cx u[PD];
#pragma unroll
        for (int q = 0; q < PD; ++q) {
            u[q] = chunk_entry(A, w1, s, pf, l);
            if (pf.valid(s)) pf.next(s);
        }
        for (int i = s - 1; i >= 0; --i) {
            cx sum = B[i * SG + l];
            for (int j0 = i + 1; j0 < s; j0 += SG) {
                const cx uv = u[0];
#pragma unroll
                for (int q = 0; q < PD - 1; ++q) u[q] = u[q + 1];
                u[PD - 1] = chunk_entry(A, w1, s, pf, l);
                if (pf.valid(s)) pf.next(s);
                const int cnt = min(SG, s - j0);
#pragma unroll
                for (int q = 0; q < SG; ++q) {
                    const cx a = cx_make(__shfl_sync(mask, uv.re, q, SG), __shfl_sync(mask, uv.im, q, SG));
                    if (q < cnt) sum = cx_sub(sum, cx_mul(a, B[(j0 + q) * SG + l]));
                }
            }
            B[i * SG + l] = cx_div(sum, diag[i]);
        }
    }
    if (live)
        for (int j = 0; j < s; ++j) x[j] = B[j * SG + l];
}

// Four warps per group of 32 solves (lane = solve): the forward elimination
// as the column sweep (every row r > c receives b[r] -= f[r][c] b[c] at step
// c, rows spread over the warps, the factor staged PC columns at a time in
// shared memory, a barrier per column), the back substitution with each
// 32-column chunk's products formed by all warps and subtracted in ascending
// j by warp 0.  Same operations in the same order per element as
// k_extra_rhs_solve; used while [s][32] + the panel + one product chunk fit.
constexpr int PC = 8;   // factor columns per staged panel
constexpr int CH = 32;  // back-substitution product chunk
constexpr int GW4 = 4;  // warps per block
constexpr int RB = 3;   // row-buffer loads per thread: S <= 3 * 128

size_t solve_group4_smem(int s) { return sizeof(cx) * ((size_t)s * (RG + PC + 2) + (size_t)CH * RG); }

__global__ void __launch_bounds__(GW4 * 32) k_extra_rhs_solve_group4(const UnitDesc *__restrict__ solves,
                                                                    const int4 *__restrict__ groups,
                                                                    const cx *__restrict__ abuf,
                                                                    const int32_t *__restrict__ piv_buf, cx *xbuf,
                                                                    const int32_t *__restrict__ status) {
    extern __shared__ cx sm[];
    const int4 g = groups[blockIdx.x];
    const UnitDesc u0 = solves[g.y];
    if (status[u0.sys] != 0) return;  // uniform over the block
    const int s = u0.s, w1 = s + 1;
    const int d = threadIdx.x & 31, w = threadIdx.x >> 5;
    cx *B = sm;                        // [s][RG]
    cx *Ap = B + (size_t)s * RG;       // [s][PC]: rows of the staged columns
    cx *P = Ap + (size_t)s * PC;       // [CH][RG]
    const cx *A = abuf + u0.a_off;
    const int32_t *piv = piv_buf + u0.piv_off;
    const bool live = d < g.z;
    cx *x = xbuf + solves[g.y + (live ? d : 0)].x_off;
    for (int j = w; j < s; j += GW4) B[j * RG + d] = live ? x[j] : cx_make(0.0, 0.0);
    __syncthreads();
    if (w == 0)
        for (int c = 0; c < s; ++c) {
            const int p = piv[c];
            if (p != c) {
                const cx t = B[c * RG + d];
                B[c * RG + d] = B[p * RG + d];
                B[p * RG + d] = t;
            }
        }
    // forward elimination, column by column
    for (int c0 = 0; c0 < s; c0 += PC) {
        const int pc_n = min(PC, s - c0);
        __syncthreads();  // the previous panel is no longer read
        for (int t = threadIdx.x; t < (s - c0 - 1) * PC; t += blockDim.x) {
            const int r = c0 + 1 + t / PC, q = t % PC;
            if (q < pc_n) Ap[r * PC + q] = A[(int64_t)r * w1 + c0 + q];
        }
        __syncthreads();
        for (int q = 0; q < pc_n; ++q) {
            const int c = c0 + q;
            const cx bc = B[c * RG + d];
            int r = c + 1;
            r += (w - r % GW4 + GW4) % GW4;  // this warp's first row after c
            for (; r < s; r += GW4) B[r * RG + d] = cx_sub(B[r * RG + d], cx_mul(Ap[r * PC + q], bc));
            __syncthreads();
        }
    }
    // back substitution; the factor rows pass through two shared row
    // buffers, row i-1 loaded while row i is processed
    cx *Ar = P + (size_t)CH * RG;  // [2][s]
    for (int t = threadIdx.x; t < s; t += blockDim.x)
        if (t >= s - 1) Ar[t] = A[(int64_t)(s - 1) * w1 + t];
    __syncthreads();
    cx sum = cx_make(0.0, 0.0);
    int cur = 0;
    for (int i = s - 1; i >= 0; --i) {
        cx nxt[RB];
#pragma unroll
        for (int k = 0; k < RB; ++k) {
            const int t = threadIdx.x + k * GW4 * 32;
            nxt[k] = (i > 0 && t >= i - 1 && t < s) ? A[(int64_t)(i - 1) * w1 + t] : cx_make(0.0, 0.0);
        }
        const cx *ar = Ar + (size_t)cur * s;
        if (w == 0) sum = B[i * RG + d];
        for (int j0 = i + 1; j0 < s; j0 += CH) {
            const int cnt = min(CH, s - j0);
            __syncthreads();  // P is free; x[j] for j > i is final
            for (int q = w; q < cnt; q += GW4) P[q * RG + d] = cx_mul(ar[j0 + q], B[(j0 + q) * RG + d]);
            __syncthreads();
            if (w == 0)
                for (int q = 0; q < cnt; ++q) sum = cx_sub(sum, P[q * RG + d]);
        }
        if (w == 0) B[i * RG + d] = cx_div(sum, ar[i]);
        // row i+1's buffer was last read before this row's barriers
#pragma unroll
        for (int k = 0; k < RB; ++k) {
            const int t = threadIdx.x + k * GW4 * 32;
            if (i > 0 && t >= i - 1 && t < s) Ar[(size_t)(cur ^ 1) * s + t] = nxt[k];
        }
        cur ^= 1;
        if (i == s - 1) __syncthreads();  // row s-1 has no chunk barrier before row s-2 reads its buffer
    }
    __syncthreads();
    if (live)
        for (int j = w; j < s; j += GW4) x[j] = B[j * RG + d];
}

// ---------------------------------------------------------------------------
// launch wrappers (host)
// ---------------------------------------------------------------------------
void launch_expand_segments(const DevWire *wires, int nw, DevSeg *segs, cudaStream_t st) {
    if (nw > 0) k_expand_segments<<<nw, 64, 0, st>>>(wires, nw, segs);
}
void launch_hallen_rhs(const UnitDesc *solves, int ns, const AntDesc *ants, const DevSeg *segs,
                       const int32_t *ibuf, const DevSource *srcs, const double *dtab, cx *rhs, double *cosv,
                       double scale, cudaStream_t st) {
    if (ns > 0) k_hallen_rhs<<<ns, 128, 0, st>>>(solves, ants, segs, ibuf, srcs, dtab, rhs, cosv, scale);
}
void launch_planewave_rhs(const UnitDesc *solves, int ns, int max_n, const AntDesc *ants, const DevSeg *segs,
                          const int32_t *ibuf, const double *dtab, cx *x, cx *rhs, double *cosv, double scale,
                          cudaStream_t st) {
    if (ns <= 0 || max_n <= 0) return;
    dim3 g((max_n + 127) / 128, ns < 65535 ? ns : 65535);
    k_planewave_field<<<g, 128, 0, st>>>(solves, ns, ants, segs, ibuf, dtab, x, cosv);
    k_planewave_rhs<<<g, 128, 0, st>>>(solves, ns, ants, segs, ibuf, dtab, cosv, x, rhs, scale);
}
void launch_receive_peaks(const UnitDesc *solves, int ns, const AntDesc *ants, const cx *x, const int32_t *status,
                          double *peak, cudaStream_t st) {
    if (ns > 0) k_receive_peaks<<<ns, 32, 0, st>>>(solves, ants, x, status, peak);
}
void launch_fill_exact(const UnitDesc *units, const AntDesc *ants, const DevSeg *segs,
                       const int4 *tiles, int ntiles, cx *z, cudaStream_t st) {
    if (ntiles > 0) k_fill_exact<<<ntiles, 256, 0, st>>>(units, ants, segs, tiles, z);
}
void launch_fill_exact_flat(const DevSeg *segs, int n, double k, int ground, cx *z, cudaStream_t st) {
    dim3 g((n + 15) / 16, (n + 15) / 16);
    if (n > 0) k_fill_exact_flat<<<g, 256, 0, st>>>(segs, n, k, ground, z);
}
void launch_gram_exact(const UnitDesc *units, int nu, int max_w, const AntDesc *ants, const int4 *gtiles,
                       int ngtiles, const int32_t *ibuf, const DevConstraint *cons,
                       const int32_t *codes, const cx *z, const cx *rhs, const double *cosv, cx *A,
                       cudaStream_t st) {
    if (ngtiles > 0) k_gram_zz<<<ngtiles, 256, 0, st>>>(units, gtiles, z, rhs, A);
    if (nu > 0) {
        dim3 g(max_w > 0 ? max_w : 1, nu);
        k_gram_ccols<<<g, 256, 0, st>>>(units, ants, ibuf, z, rhs, cosv, A);
        k_gram_finish<<<nu, 256, 0, st>>>(units, ants, cons, codes, A);
    }
}

// Raises a kernel's dynamic shared-memory limit once per device: the
// attribute belongs to the kernel in the current device's context, so a
// second GPU needs its own call.  Returns the limit in effect.
int set_smem_limit_once(const void *kernel, int bytes) {
    static std::mutex mu;
    static std::map<std::pair<int, const void *>, int> done;
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess) {
        (void)cudaGetLastError();
        return -1;
    }
    std::lock_guard<std::mutex> lk(mu);
    const auto key = std::make_pair(dev, kernel);
    auto it = done.find(key);
    if (it != done.end()) return it->second;
    int got = -1;
    cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes);
    if (e == cudaSuccess) {
        got = bytes;
    } else {
        (void)cudaGetLastError();  // leave no error behind for the launch checks
        std::fprintf(stderr, "fnec: shared-memory limit %d B refused (%s); kernels fall back to global staging\n",
                     bytes, cudaGetErrorString(e));
        cudaFuncAttributes fa;
        if (cudaFuncGetAttributes(&fa, kernel) == cudaSuccess) got = fa.maxDynamicSharedSizeBytes;
        else (void)cudaGetLastError();
    }
    done[key] = got;
    return got;
}

size_t grid_xchg_bytes() { return sizeof(PanelXchg<cx>) * GRID_PANEL_MAX_UNITS; }
size_t grid_sync_bytes(int steps) { return sizeof(GridSync) * GRID_PANEL_MAX_UNITS * (size_t)(steps > 0 ? steps : 1); }

// Chooses how the panel at column c0 is factored.  Units whose panel
// (s - c0 rows) exceeds thr_rows (plain: the largest cluster's rows; mixed:
// one CTA's shared memory) go to the grid-wide kernel when they are few enough
// to be co-resident; the rest take the form's own kernel for shorter panels.
// Returns the number of grid units
// (0: none; -1: not possible, every unit takes the one-CTA global kernel)
// and the CTAs per grid unit and their shared memory.
int plan_grid_panel(const GridPlan &gp, int c0, int thr_rows, int pnb, size_t elem, const void *kernel,
                    int *G_out, size_t *smem_out) {
    int nl = 0;
    while (nl < (int)gp.s_desc.size() && gp.s_desc[nl] - c0 > thr_rows) ++nl;
    if (nl == 0) return 0;
    if (!gp.grid_on || nl > GRID_PANEL_MAX_UNITS || !gp.d_xchg || !gp.d_sync || gp.sms <= 0) return -1;
    const int m_max = gp.s_desc[0] - c0;
    const size_t cta_cap = 96 * 1024;  // two CTAs per SM
    const int r_cap = (int)(cta_cap / (pnb * elem));
    int G = std::max(1, gp.sms / nl);
    G = std::min(G, (m_max + 31) / 32);
    G = std::max(G, (m_max + r_cap - 1) / r_cap);
    if (G > GRID_PANEL_MAX_CTAS) return -1;
    int R = (m_max + G - 1) / G;
    size_t smem = (size_t)R * pnb * elem;
    int per_sm = 0;
    if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kernel, 256, smem) != cudaSuccess) return -1;
    if ((int64_t)G * nl > (int64_t)per_sm * gp.sms) return -1;
    *G_out = G;
    *smem_out = smem;
    return nl;
}

cudaError_t launch_cooperative(const void *kernel, dim3 grid, dim3 block, void **args, size_t smem,
                               cudaStream_t st) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = grid;
    cfg.blockDim = block;
    cfg.dynamicSmemBytes = smem;
    cfg.stream = st;
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeCooperative;
    at[0].val.cooperative = 1;
    cfg.attrs = at;
    cfg.numAttrs = 1;
    return cudaLaunchKernelExC(&cfg, kernel, args);
}

void step_classes(const GridPlan &gp, int c0, int i_begin, std::vector<StepClass> &out, int i_end) {
    out.clear();
    int i = i_begin, n = i_end < 0 ? (int)gp.s_desc.size() : std::min(i_end, (int)gp.s_desc.size());
    while (i < n && gp.s_desc[i] > c0) {
        const int f = 1 << gp.class_shift;
        int m = gp.s_desc[i] - c0, hi = 64;
        while (hi < m) hi *= f;
        int lo = hi == 64 ? 0 : hi / f;  // the class holds heights (lo, hi]
        StepClass c{i, i, m};
        while (i < n && gp.s_desc[i] - c0 > lo) ++i;  // s descending: the class is a run
        c.i1 = i;
        out.push_back(c);
    }
}

// One cluster per unit, rows dealt evenly over its CTAs.
static void launch_panel_cluster(const UnitDesc *units, int n, int m_max, int c0, cx *A, int32_t *piv, int32_t *status,
                                 const int32_t *order, int base, cudaStream_t st) {
    int nc = 1;
    while (nc * CP_MAX_ROWS < m_max) nc *= 2;
    const int rows = ((m_max + nc - 1) / nc + 31) / 32 * 32;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(n * nc);
    cfg.blockDim = dim3(rows);
    cfg.dynamicSmemBytes = cp_smem(rows);
    cfg.stream = st;
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeClusterDimension;
    at[0].val.clusterDim.x = nc;
    at[0].val.clusterDim.y = at[0].val.clusterDim.z = 1;
    cfg.attrs = at;
    cfg.numAttrs = nc > 1 ? 1 : 0;
    cudaLaunchKernelEx(&cfg, nc > 1 ? k_panel_cluster<true> : k_panel_cluster<false>, units, c0, A, piv, status, order,
                       base, nc);
}

uint64_t launch_factor_exact(const UnitDesc *units, int nu, int max_s, const GridPlan &gp, cx *A,
                             int32_t *piv, int32_t *status, cudaStream_t st) {
    uint64_t L = 0;
    set_smem_limit_once(k_swap_u12, (int)SU_SMEM);  // once per device
    set_smem_limit_once(k_panel_cluster<false>, (int)cp_smem(CP_MAX_ROWS));
    set_smem_limit_once(k_panel_cluster<true>, (int)cp_smem(CP_MAX_ROWS));
    set_smem_limit_once(k_panel_grid, 96 * 1024);
    (void)nu;
    const int thr_rows = CP_MAX_ROWS * CP_MAX_CTAS;
    const int32_t *ord = gp.d_order;
    if (gp.d_sync) cudaMemsetAsync(gp.d_sync, 0, grid_sync_bytes(gp.steps), st);
    std::vector<StepClass> cls;
    for (int c0 = 0; c0 < max_s; c0 += NB) {
        // panels: the tallest units (m > thr_rows) grid-wide or one CTA each
        // from global memory, the rest a cluster each, in size classes so
        // that short panels do not reserve tall panels' memory
        int n_thr = 0;
        while (n_thr < (int)gp.s_desc.size() && gp.s_desc[n_thr] - c0 > thr_rows) ++n_thr;
        if (n_thr > 0) {
            int G = 0;
            size_t gsm = 0;
            bool done = false;
            if (plan_grid_panel(gp, c0, thr_rows, NB, sizeof(cx), (const void *)k_panel_grid, &G, &gsm) == n_thr) {
                PanelXchg<cx> *xg = static_cast<PanelXchg<cx> *>(gp.d_xchg);
                GridSync *gs = static_cast<GridSync *>(gp.d_sync) + (size_t)(c0 / NB) * GRID_PANEL_MAX_UNITS;
                void *args[] = {(void *)&units, (void *)&ord, (void *)&c0, (void *)&A, (void *)&piv,
                                (void *)&status, (void *)&xg, (void *)&gs};
                done = launch_cooperative((const void *)k_panel_grid, dim3(G, n_thr), dim3(256), args, gsm, st) ==
                       cudaSuccess;
                if (!done) (void)cudaGetLastError();  // not co-resident after all
            }
            if (!done) k_panel<<<n_thr, 256, 0, st>>>(units, c0, A, piv, status, ord, 0);
            ++L;
        }
        step_classes(gp, c0, n_thr, cls);
        for (const StepClass &c : cls) {
            launch_panel_cluster(units, c.i1 - c.i0, c.m_max, c0, A, piv, status, ord, c.i0, st);
            ++L;
        }
        // deferred swaps + U12, then the trailing update, by size class
        step_classes(gp, c0, 0, cls);
        for (const StepClass &c : cls) {
            int m = c.m_max;
            int rest = m + 1 - NB;  // columns right of the panel, at least the right-hand side
            if (rest < 1) rest = 1;
            dim3 g1((rest + SU_COLS - 1) / SU_COLS + (c0 + SU_COLS - 1) / SU_COLS, c.i1 - c.i0);
            k_swap_u12<<<g1, 4 * SU_COLS, SU_SMEM, st>>>(units, c0, A, piv, status, ord, c.i0);
            ++L;
            int rows = m - NB;
            if (rows > 0) {
                const auto trailing = rows >= TRAILING_WIDE_ROWS ? launch_trailing<64> : launch_trailing<32>;
                trailing(units, c.i1 - c.i0, rows, rest, c0, A, status, ord, c.i0, st);
                ++L;
            }
        }
    }
    return L;
}
// Dynamic shared memory of the chain kernels for systems of up to max_s
// unknowns: the product ring, and x beside it (*staged) where both fit.
template <typename K>
static size_t backsub_smem(K kernel, int max_s, int *staged) {
    const size_t smem = BS_RING_BYTES + sizeof(cx) * (size_t)max_s;
    *staged = smem <= BS_SMEM_MAX;
    if (*staged) {  // static + dynamic above 48 KB needs the raised limit
        int lim = set_smem_limit_once(kernel, (int)BS_SMEM_MAX);
        if (lim < 0 || (size_t)lim < smem) *staged = 0;
    }
    return *staged ? smem : BS_RING_BYTES;
}

void launch_backsub(const UnitDesc *units, int nu, int max_s, const int32_t *order, const cx *A, cx *x,
                    const int32_t *status, cudaStream_t st) {
    if (nu <= 0) return;
    int staged = 0;
    const size_t smem = backsub_smem(k_backsub, max_s, &staged);
    k_backsub<<<nu, BS_THREADS, smem, st>>>(units, order, A, x, status, staged);
}
// matrix.rs:131-139 add_to_diagonal / add_to_entry: each stamp one
// separately rounded complex add, an entry's stamps in their order (the
// thread at the first stamp of each run applies the run).
__global__ void k_stamps(const DevStamp *__restrict__ stamps, int n, cx *z) {
    const int q = blockIdx.x * blockDim.x + threadIdx.x;
    if (q >= n || !stamps[q].first) return;
    const DevStamp d = stamps[q];
    cx v = z[d.index];
    for (int t = 0; t < d.count; ++t) v = cx_add(v, cx_make(stamps[q + t].re, stamps[q + t].im));
    z[d.index] = v;
}
void launch_stamps(const DevStamp *stamps, int n, cx *z, cudaStream_t st) {
    if (n > 0) k_stamps<<<(n + 255) / 256, 256, 0, st>>>(stamps, n, z);
}
void launch_feedpoints(const UnitDesc *solves, int ns, const AntDesc *ants, const DevSeg *segs,
                       const int32_t *ibuf, const DevFeed *feeds, const cx *x, const int32_t *status,
                       double *feed_out, const int64_t *feed_row_off, cudaStream_t st) {
    if (ns > 0)
        k_feedpoints<<<ns, 32, 0, st>>>(solves, ants, segs, ibuf, feeds, x, status, feed_out, feed_row_off);
}
void launch_extra_rhs_exact(const UnitDesc *solves, int ns, int max_s, const AntDesc *ants, const int32_t *ibuf,
                            const cx *z, const cx *rhs, const double *cosv, const cx *A, const int32_t *piv,
                            cx *x, const int32_t *status, cudaStream_t st, const int4 *groups, int n_groups,
                            int first_rhs) {
    if (ns <= 0) return;
    if (groups && n_groups > 0 && first_rhs == 1) {
        dim3 gb((max_s + 63) / 64, n_groups);
        k_extra_rhs_b_group<<<gb, 64, 0, st>>>(solves, groups, ants, ibuf, z, rhs, cosv, x);
        const size_t smem4 = solve_group4_smem(max_s);
        int lim4 = (smem4 <= GS_SMEM_MAX && max_s <= RB * GW4 * 32)
                       ? set_smem_limit_once(k_extra_rhs_solve_group4, (int)GS_SMEM_MAX)
                       : -1;
        if (lim4 >= 0 && (size_t)lim4 >= smem4) {
            k_extra_rhs_solve_group4<<<n_groups, GW4 * 32, smem4, st>>>(solves, groups, A, piv, x, status);
            return;
        }
        const size_t smem = (sizeof(cx) * (SG + 1) + sizeof(int32_t)) * (size_t)max_s;
        int lim = smem <= GS_SMEM_MAX ? set_smem_limit_once(k_extra_rhs_solve_group, (int)GS_SMEM_MAX) : -1;
        if (lim >= 0 && (size_t)lim >= smem) {
            k_extra_rhs_solve_group<<<dim3(n_groups, RG / SG), SG, smem, st>>>(solves, groups, A, piv, x, status);
            return;
        }
        // a factor too tall for the shared tile: one block per solve on the b vectors formed above
        k_extra_rhs_solve<<<ns, BS_THREADS, BS_RING_BYTES, st>>>(solves, A, piv, x, status, 0, 1);
        return;
    }
    dim3 g((max_s + 127) / 128, ns);
    k_extra_rhs_b<<<g, 128, 0, st>>>(solves, ants, ibuf, z, rhs, cosv, x, first_rhs);
    int staged = 0;
    const size_t smem = backsub_smem(k_extra_rhs_solve, max_s, &staged);
    k_extra_rhs_solve<<<ns, BS_THREADS, smem, st>>>(solves, A, piv, x, status, staged, first_rhs);
}

}  // namespace fnec

// ---------------------------------------------------------------------------
// Self-test of the bounded grid barrier's timeout path
// (fnec_selftest_wait_timeout): every CTA but `absent` takes the barrier;
// the absent CTA returns without arriving, so the others' waits run out
// after wait_ns and each marks the status word FNEC_UNIT_TIMEOUT.  With
// absent < 0 every CTA arrives and the status stays 0.
// ---------------------------------------------------------------------------
namespace fnec {
__global__ void k_grid_barrier_probe(GridSync *gs, int32_t *status, int absent, unsigned long long wait_ns) {
    if ((int)blockIdx.x == absent) return;
    if (!grid_barrier(gs, gridDim.x, 1, wait_ns)) {
        if (threadIdx.x == 0) atomicExch(status, FNEC_UNIT_TIMEOUT);
        return;
    }
}

int selftest_grid_timeout(int32_t device, int32_t ctas, int32_t absent, uint64_t wait_ns, int32_t *unit_status,
                          double *elapsed_ms) {
    if (cudaSetDevice(device) != cudaSuccess) return FNEC_ERR_NO_DEVICE;
    if (ctas < 2 || ctas > 148 || absent >= ctas) return FNEC_ERR_BAD_ARG;
    GridSync *gs = nullptr;
    int32_t *st = nullptr;
    cudaEvent_t e0 = nullptr, e1 = nullptr;
    int rc = FNEC_OK;
    do {
        if (cudaMalloc(&gs, sizeof(GridSync)) != cudaSuccess || cudaMalloc(&st, sizeof(int32_t)) != cudaSuccess) {
            rc = FNEC_ERR_OUT_OF_MEMORY;
            break;
        }
        if (cudaEventCreate(&e0) != cudaSuccess || cudaEventCreate(&e1) != cudaSuccess) {
            rc = FNEC_ERR_CUDA;
            break;
        }
        cudaMemset(gs, 0, sizeof(GridSync));
        cudaMemset(st, 0, sizeof(int32_t));
        unsigned long long w = wait_ns;
        void *args[] = {(void *)&gs, (void *)&st, (void *)&absent, (void *)&w};
        cudaEventRecord(e0, 0);
        if (launch_cooperative((const void *)k_grid_barrier_probe, dim3(ctas), dim3(64), args, 0, 0) != cudaSuccess) {
            (void)cudaGetLastError();
            rc = FNEC_ERR_UNSUPPORTED;
            break;
        }
        cudaEventRecord(e1, 0);
        if (cudaEventSynchronize(e1) != cudaSuccess) {
            rc = FNEC_ERR_CUDA;
            break;
        }
        float ms = 0.f;
        cudaEventElapsedTime(&ms, e0, e1);
        if (elapsed_ms) *elapsed_ms = ms;
        if (unit_status) cudaMemcpy(unit_status, st, sizeof(int32_t), cudaMemcpyDeviceToHost);
    } while (0);
    if (e0) cudaEventDestroy(e0);
    if (e1) cudaEventDestroy(e1);
    cudaFree(gs);
    cudaFree(st);
    return rc;
}
}  // namespace fnec

// ---------------------------------------------------------------------------
// Self-test of the shortened divisions and square root (fnec_test_exact_
// division): every one against the IEEE operation, bit for bit, inside the
// range that its callers guard.
// ---------------------------------------------------------------------------
namespace fnec {
__global__ void k_test_exact_division(const double *av, const double *xv, int n, int32_t *out) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const double a = av[i], x = xv[i];
    auto differ = [](double p, double q) { return __double_as_longlong(p) != __double_as_longlong(q); };
    auto exponent_within = [](double v, int e) {  // 2^-e <= |v| < 2^e
        const int k = (int)((uint32_t)(fnec_libm::lm_hi(v) & 0x7fffffffu) >> 20) - 1023;
        return k >= -e && k < e;
    };
    int bad = 0;
    if (sqrt_recip_domain(x)) {
        const SqrtRecip sr = sqrt_recip(x);
        if (differ(sr.r, D_SQRT(x))) bad |= 1;
        if ((a == 0.0 || exponent_within(a, 400)) && differ(div_by(a, sr), D_DIV(a, sr.r))) bad |= 2;
    }
    if (x > 0.0 && exponent_within(x, 400) && (uint32_t)fnec_libm::lm_bits(x) != 0xffffffffu) {
        const double z = recip_rn(x);
        if (differ(z, D_DIV(1.0, x))) bad |= 4;
        if ((a == 0.0 || exponent_within(a, 400)) && differ(div_by(a, {x, z}), D_DIV(a, x))) bad |= 8;
    }
    const cx num = cx_make(a, x), den = cx_make(x, -a);
    const double ns = D_ADD(D_MUL(den.re, den.re), D_MUL(den.im, den.im));
    const cx p = cp_div(num, den, ns, recip_rn(ns)), q = cx_div(num, den);
    if (differ(p.re, q.re) || differ(p.im, q.im)) bad |= 16;
    out[i] = bad;
}
}  // namespace fnec

extern "C" int fnec_test_exact_division(const double *a, const double *x, uint64_t n, int32_t *out) {
    if (n && (!a || !x || !out)) return FNEC_ERR_BAD_ARG;
    if (n > ((uint64_t)1 << 24)) return FNEC_ERR_TOO_LARGE;
    for (uint64_t i = 0; i < n; ++i)
        if (!std::isfinite(a[i]) || !std::isfinite(x[i])) return FNEC_ERR_BAD_ARG;
    if (n == 0) return FNEC_OK;
    unsigned char *d = nullptr;
    if (cudaMalloc(&d, (2 * sizeof(double) + sizeof(int32_t)) * n) != cudaSuccess) {
        (void)cudaGetLastError();
        return FNEC_ERR_OUT_OF_MEMORY;
    }
    double *da = reinterpret_cast<double *>(d), *dx = da + n;
    int32_t *dout = reinterpret_cast<int32_t *>(dx + n);
    cudaError_t e = cudaMemcpy(da, a, sizeof(double) * n, cudaMemcpyHostToDevice);
    if (e == cudaSuccess) e = cudaMemcpy(dx, x, sizeof(double) * n, cudaMemcpyHostToDevice);
    if (e == cudaSuccess) {
        fnec::k_test_exact_division<<<(unsigned)((n + 255) / 256), 256>>>(da, dx, (int)n, dout);
        e = cudaGetLastError();
    }
    if (e == cudaSuccess) e = cudaMemcpy(out, dout, sizeof(int32_t) * n, cudaMemcpyDeviceToHost);
    cudaFree(d);
    return e == cudaSuccess ? FNEC_OK : FNEC_ERR_CUDA;
}
