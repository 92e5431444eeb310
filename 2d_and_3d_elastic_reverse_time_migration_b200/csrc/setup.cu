// Host set-up shared by every entry point that runs the step kernels: the
// padded-volume geometry, the difference coefficients, the absorbing-boundary
// profiles and the tile rules.  The context path (ertm_api.cu) and the
// no-allocation modelling path (noalloc.cu) both call these, so the two can
// never drift apart.
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>

#include "ertm_internal.cuh"

namespace ertm {

static long long rup(long long v, long long m) { return (v + m - 1) / m * m; }

// Rows per thread of the 2D tile kernels: as many (1, 2 or 4) as still give every SM a
// CTA (64 columns x 4 rows of threads).  More rows per thread share more of the z window
// and re-read fewer halo rows, fewer rows give small grids more CTAs.  Measured on B200, ms
// for 200 steps (R = 4, C-PML, modelling) with 1 / 2 / 4 rows: 168 x 104 1.07 / 1.13 / 1.35,
// 680 x 380 2.16 / 2.01 / 1.60, 1471 x 803 6.18 / 4.89 / 4.40.  With R = 6 the four-row
// kernels' registers leave one CTA less per SM, which costs a grid that streams from HBM
// more than the window saves (4096 x 2048, us per step: 205 / 155 / 165).
static int rows2d(int nx, int nz, int R)
{
    const long long cols = (nx + TX2 - 1) / TX2;
    for (int nr = R > 4 && (long long)nx * nz > (3 << 20) ? 2 : 4; nr > 1; nr /= 2)
        if (cols * ((nz + 4 * nr - 1) / (4 * nr)) >= 148) return nr;
    return 1;
}

Geom make_geom(int nx, int ny, int nz, int R)
{
    Geom g{};
    g.nx = nx;
    g.ny = ny;
    g.nz = nz;
    g.R = R;
    g.two_d = (ny == 1);
    g.tyb = g.two_d ? 1 : TY3;
    g.nr2 = rows2d(nx, nz, R);
    g.hx = XH;
    g.hy = g.two_d ? 0 : R;
    g.hz = R;
    g.px = rup(2LL * g.hx + rup(nx, TX), 32);
    g.py = 2LL * g.hy + rup(ny, g.tyb);
    g.pz = 2LL * g.hz + nz + 1;
    g.sy = g.px;
    g.sz = g.px * g.py;
    g.off0 = g.hz * g.sz + g.hy * g.sy + g.hx;
    g.total = g.px * g.py * g.pz;
    return g;
}

void stencil_coefs(int coef_kind, const float* user, int R, float coef[8])
{
    for (int n = 0; n < 8; n++) coef[n] = 0.f;
    if (coef_kind == ERTM_COEF_USER) {
        for (int n = 0; n <= R && n < 8; n++) coef[n] = user[n];
        return;
    }
    if (coef_kind == ERTM_COEF_REFERENCE12) {
        // the reference's 12-point set (3D_elastic_RTM/zzzzz:202-210)
        const float r12[7] = {0.0f, 1.2213363647f, -0.096931457519f, 0.017447662353f,
                              -0.0029672895159f, 0.00035900539822f, -0.00002184781161f};
        for (int n = 0; n < 7; n++) coef[n] = r12[n];
        return;
    }
    // Taylor weights of the staggered first derivative: sum_n c_n (2n-1)^(2m-1) = delta_m1,
    // solved by Gauss-Jordan elimination with partial pivoting in double
    double A[8][9];
    for (int m = 0; m < R; m++) {
        for (int n = 0; n < R; n++) A[m][n] = std::pow(2.0 * n + 1.0, 2.0 * m + 1.0);
        A[m][R] = (m == 0);
    }
    for (int cc = 0; cc < R; cc++) {
        int p = cc;
        for (int r = cc + 1; r < R; r++)
            if (std::fabs(A[r][cc]) > std::fabs(A[p][cc])) p = r;
        for (int k = 0; k <= R; k++) std::swap(A[cc][k], A[p][k]);
        for (int r = 0; r < R; r++) {
            if (r == cc) continue;
            const double f = A[r][cc] / A[cc][cc];
            for (int k = cc; k <= R; k++) A[r][k] -= f * A[cc][k];
        }
    }
    for (int n = 0; n < R; n++) coef[n + 1] = (float)(A[n][R] / A[n][n]);
}

void cpml_profile(int n, int w0, int w1, int stg, double h, double vmax, double rcoef, double f0,
                  double dts, int i0, int m, float* a, float* b)
{
    // C-PML (Komatitsch & Martin 2007) with kappa = 1: quadratic damping d, alpha
    // falling linearly from pi f0 at the inner edge to 0 at the outer edge;
    // the oracle's orc_cpml_profile computes the same values
    for (int q = 0; q < m; q++) {
        const double p = i0 + q + 0.5 * stg;
        double dist = 0.0, L = 1.0;
        if (w0 > 0 && p < w0 - 1) { dist = (w0 - 1) - p; L = w0; }
        else if (w1 > 0 && p > n - w1) { dist = p - (n - w1); L = w1; }
        if (dist <= 0.0) {
            a[q] = 0.f;
            b[q] = 1.f;
            continue;
        }
        const double Lm = L * h, x = dist * h / Lm;
        const double d = -3.0 * vmax * std::log(rcoef) / (2.0 * Lm) * x * x;
        double al = M_PI * f0 * (1.0 - x);
        if (al < 0) al = 0;
        const double bb = std::exp(-(d + al) * dts);
        b[q] = (float)bb;
        a[q] = (float)(d * (bb - 1.0) / (d + al));
    }
}

void sponge_profile(int n, int w0, int w1, int kind, float coe, int i0, int m, float* v)
{
    // coe_attenuation_3d_new2 (3D_elastic_RTM/3D_zzzzz:261-300): cosine ramp;
    // make_attenuation_new (3D_elastic_RTM/zzzzz:238-280): cubic ramp.  The
    // near-side ramp then the far-side ramp accumulate into a float, as the
    // reference's two loops do.
    const double pai = 3.1415926;   // 3D_zzzzz:1
    for (int q = 0; q < m; q++) {
        const int i = i0 + q;
        float acc = 0.f;
        if (i < w0) {
            float val;
            if (kind == ERTM_BOUNDARY_SPONGE_COS)
                val = (float)(coe * (1.0 - std::cos(pai / 2 * (w0 - i - 1) / (w0 - 1))));
            else {
                const float x = (float)((w0 - 1.0 - i) / (w0 - 1.0));
                val = (float)(coe * std::pow(x * 1.0, 3.0));
            }
            acc += val;
        }
        if (w1 > 0 && i >= n - w1) {
            const int k = i - (n - w1);
            float val;
            if (kind == ERTM_BOUNDARY_SPONGE_COS)
                val = (float)(coe * (1.0 - std::cos(pai / 2 * k / (w1 - 1))));
            else {
                const float x = (float)(k / (w1 - 1.0));
                val = (float)(coe * std::pow(x * 1.0, 3.0));
            }
            acc += val;
        }
        v[q] = acc;
    }
}

// z planes per CTA of the 3D kernels for `tiles` tiles of the x-y plane (of every shot of a
// launch).  From eight waves of CTAs on, balanced chunks of about 32 planes: the time is flat
// from there to 40-48 (480 x 480 x 380, RTM: 235.0, 234.8, 234.6 ms for 32, 40, 48; five
// windows of different sizes in one launch: 120.5, 120.7, 121.5) and grows above (236.1, 245.2
// and 123.5, 128.7 for 64, 96) and below (237.5 and 121.3 for 24).  A smaller launch needs its
// last wave full: the chunk of 4 to 48 planes with the least waves x (planes + start-up),
// start-up being the fill of the z queues and of the ring, about 8 planes' time (151 x 133 x
// 117, modelling, 80 steps: 9.45 ms in chunks of 30 planes, 340 CTAs on 296 places, and 8.19
// in chunks of 39, 255 CTAs; 64 x 64 x 64, RTM, 75 steps: 2.07 ms in chunks of 8, 128 CTAs, and
// 1.78 in chunks of 4).
int choose_kchunk(long long tiles, int nz)
{
    constexpr long long places = CTAS3 * 148;
    const int n32 = std::max(1, (nz + 16) / 32);
    int best = (nz + n32 - 1) / n32;
    if (tiles * n32 >= 8 * places) return best;
    double best_cost = 1e300;
    for (int n = (nz + 47) / 48; n <= (nz + 3) / 4; n++) {
        const int kc = (nz + n - 1) / n, chunks = (nz + kc - 1) / kc;
        const long long waves = (tiles * chunks + places - 1) / places;
        const double cost = (double)waves * (kc + 8);
        if (cost < best_cost) {
            best_cost = cost;
            best = kc;
        }
    }
    return best;
}

long long step_tiles(const Geom& g)
{
    return (long long)((g.nx + TX - 1) / TX) * ((g.ny + TY3 - 1) / TY3);
}

}  // namespace ertm
