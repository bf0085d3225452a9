// green_cells.cuh -- cell integrals of the IGF kernels (phi and E) on the non-negative
// displacements, the real-space half of a Green build.
//
// Near the origin a cell's value is the 8-corner difference of the FP64 primitive
// (osc_get_cgrn_freespace, code/open_spacecharge_mod.f90:648-705).  Away from it the average
// of 1/r and of x/r^3 over the box is its Taylor series about the cell centre,
//   mean f = sum_{ijk} a^2i b^2j c^2k / ((2i+1)! (2j+1)! (2k+1)!) dx^2i dy^2j dz^2k f
// (a, b, c half the cell's edges).  With r^2 = u + v + w (u = x^2 ...) every term of total
// order 2n is a homogeneous integer polynomial of degree n in (u, v, w) over r^(4n+1) (over
// r^(4n+3), times x, for E_x), so the sum to order 8 is one polynomial with 35 coefficients in
// (u, v, w)/r^4 per component.  It needs no log or atan and, unlike the corner difference of
// primitives that grow as r^2, which loses (r/h)^3 of the FP64 round-off, does not cancel.
#pragma once

#include "osc_common.cuh"

namespace osc {

constexpr int kSerN = 4;                       // highest degree (order 8 in 1/r)
constexpr int kSerC = 35;                      // monomials u^i v^j w^k, i + j + k <= 4
constexpr int kSerP = 36;                      // the same, padded to whole 16-byte pairs
// Distance, in half cell diagonals, from which the series is used, by the type of the stored spectra.
// The series' truncation falls as r^-10, the corner difference's round-off in FP64 grows as r^3.  Largest
// errors over the directions, of |E| (series, corners), at 9, 10 and 11: cubes 4.0e-12 1.3e-12, 1.6e-12
// 1.1e-12, 4.9e-13 1.9e-12; cells 1 x 1 x 10 8.2e-11 9.2e-11, 4.4e-11 3.5e-11, 1.3e-11 6.8e-11;
// 1 x 10 x 10 2.3e-11 9.7e-12, 8.0e-12 1.8e-11, 3.1e-12 5.2e-11; 1 x 3 x 10 3.9e-11 9.3e-12, 2.1e-11
// 2.8e-11, 5.5e-12 3.4e-11; 1 x 1 x 50 9.9e-11 7.7e-9 and better from there.  So 11 for FP64: no
// shape of cell has the series where the corners would be the better one.  FP32 spectra keep 6e-8 of
// a value, and 9 spares them near tiles.
template <typename T> constexpr double ser_ratio() { return sizeof(T) == 8 ? 11.0 : 9.0; }

// Position of u^i v^j w^k in Horner order (i, then j, then k), all degrees <= kSerN.
constexpr __host__ __device__ int ser_idx(int i, int j, int k) {
    int p = 0;
    for (int a = 0; a < i; ++a) p += (kSerN - a + 1) * (kSerN - a + 2) / 2;
    for (int b = 0; b < j; ++b) p += kSerN - i - b + 1;
    return p + k;
}

// Homogeneous polynomial of degree n in (u, v, w): coefficient of u^i v^j w^(n-i-j).
struct SerPoly {
    int n;
    double c[kSerN + 1][kSerN + 1];
};
// p.c with one more factor of variable ax (0 u, 1 v, 2 w)
constexpr SerPoly ser_mul(const SerPoly &p, int ax) {
    SerPoly r{p.n + 1, {}};
    for (int i = 0; i <= p.n; ++i)
        for (int j = 0; i + j <= p.n; ++j) r.c[i + (ax == 0)][j + (ax == 1)] += p.c[i][j];
    return r;
}
constexpr SerPoly ser_der(const SerPoly &p, int ax) {
    SerPoly r{p.n - 1, {}};
    for (int i = 0; i <= p.n; ++i)
        for (int j = 0; i + j <= p.n; ++j) {
            const int e = ax == 0 ? i : (ax == 1 ? j : p.n - i - j);
            if (e > 0) r.c[i - (ax == 0)][j - (ax == 1)] += e * p.c[i][j];
        }
    return r;
}
// s p + t q (equal degrees)
constexpr SerPoly ser_lin(double s, const SerPoly &p, double t, const SerPoly &q) {
    SerPoly r{p.n, {}};
    for (int i = 0; i <= p.n; ++i)
        for (int j = 0; i + j <= p.n; ++j) r.c[i][j] = s * p.c[i][j] + t * q.c[i][j];
    return r;
}
constexpr SerPoly ser_r2(const SerPoly &p) {  // times u + v + w
    return ser_lin(1, ser_lin(1, ser_mul(p, 0), 1, ser_mul(p, 1)), 1, ser_mul(p, 2));
}
// d/dx of H / r^(4n+1) is x K / r^(4n+3)
constexpr SerPoly ser_k(const SerPoly &h, int ax) {
    const double m = 4 * h.n + 1;
    if (h.n == 0) return SerPoly{0, {{-h.c[0][0]}}};
    return ser_lin(2, ser_r2(ser_der(h, ax)), -m, h);
}
// d^2/dx^2 of H / r^(4n+1) is H' / r^(4n+5), H' of degree n + 1
constexpr SerPoly ser_d2(const SerPoly &h, int ax) {
    const SerPoly k = ser_k(h, ax);
    SerPoly a = k;
    if (k.n > 0) a = ser_lin(1, k, 2, ser_mul(ser_der(k, ax), ax));
    return ser_lin(1, ser_r2(a), -(4.0 * h.n + 3), ser_mul(k, ax));
}

// t[comp][out][in]: coefficient `out` of component comp (0 phi, 1..3 E) per unit of
// a^2i b^2j c^2k / ((2i+1)! (2j+1)! (2k+1)!), `in` = ser_idx(i, j, k); equal degrees only.
struct SerTab {
    double t[4][kSerC][kSerC];
};
constexpr SerTab ser_table() {
    SerTab s{};
    for (int i = 0; i <= kSerN; ++i) {
        SerPoly hi{0, {{1}}};
        for (int q = 0; q < i; ++q) hi = ser_d2(hi, 0);
        for (int j = 0; i + j <= kSerN; ++j) {
            SerPoly hj = hi;
            for (int q = 0; q < j; ++q) hj = ser_d2(hj, 1);
            for (int k = 0; i + j + k <= kSerN; ++k) {
                SerPoly h = hj;
                for (int q = 0; q < k; ++q) h = ser_d2(h, 2);
                const int in = ser_idx(i, j, k);
                for (int c = 0; c < 4; ++c) {
                    const SerPoly p = c ? ser_k(h, c - 1) : h;
                    for (int a = 0; a <= p.n; ++a)
                        for (int b = 0; a + b <= p.n; ++b)
                            s.t[c][ser_idx(a, b, p.n - a - b)][in] = (c ? -1 : 1) * p.c[a][b];
                }
            }
        }
    }
    return s;
}

// One geometry: cell edges (hz already times gamma), z offset of the kernel (times gamma) and
// the series of its cells.
struct CellGeom {
    double hx, hy, hz, woff, gamma;
    double far2;            // square of the distance from which the series is used
    alignas(16) double coef[4][kSerP];
};

// The values of ncomp components (comps: 0 phi, 1..3 E) of nmem geometries on nx x ny x nzc
// cells: h + (ci * nmem + b) * hstride, [z][y][x].  zwrap 0: the displacements (i, j, k) >= 0.
// zwrap 1: z plane p holds displacement p (p < nz) or p - 2 nz, nzc = 2 nz, plane nz zero.
struct CellArgs {
    int nx, ny, nz, zwrap;
    int ncomp, comps[4];
    int nmem;
    int64_t hstride;
};
// One geometry, by value (its coefficients become immediate operands of the FP64 units).
CellGeom cell_geom(double hx, double hy, double hz, double gamma, double woff, double ratio);
template <typename TH> int launch_green_cells(TH *h, const CellArgs &a, const CellGeom &g, cudaStream_t st);
// nmem geometries from device memory, whose edges and gamma are set; the series of the E
// components are filled in by launch_cell_series first.
int launch_cell_series(CellGeom *g, int n, cudaStream_t st);
int launch_green_cells_batch(float *h, const CellArgs &a, const CellGeom *g, cudaStream_t st);

}  // namespace osc
