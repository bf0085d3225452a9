// green_cells.cu -- cell integrals of the IGF kernels (green_cells.cuh).
#include "green_cells.cuh"

#include <cmath>

#include "osc_igf.cuh"

namespace osc {

static inline int ok() { return cudaGetLastError() == cudaSuccess ? OSC_OK : OSC_E_CUDA; }

static constexpr SerTab kSerHost = ser_table();
__constant__ SerTab kSerDev = ser_table();

// a^2i b^2j c^2k / ((2i+1)! (2j+1)! (2k+1)!)
__host__ __device__ inline double ser_moment(double a2, double b2, double c2, int i, int j, int k) {
    double m = 1.0;
    for (int q = 1; q <= i; ++q) m *= a2 / (2 * q * (2 * q + 1));
    for (int q = 1; q <= j; ++q) m *= b2 / (2 * q * (2 * q + 1));
    for (int q = 1; q <= k; ++q) m *= c2 / (2 * q * (2 * q + 1));
    return m;
}
// Exponents of coefficient m.
__host__ __device__ inline void ser_exp(int m, int &i, int &j, int &k) {
    for (i = 0; i < kSerN && m >= ser_idx(i + 1, 0, 0); ++i) {}
    for (j = 0; j < kSerN - i && m >= ser_idx(i, j + 1, 0); ++j) {}
    k = m - ser_idx(i, j, 0);
}

CellGeom cell_geom(double hx, double hy, double hz, double gamma, double woff, double ratio) {
    CellGeom g;
    g.hx = hx;
    g.hy = hy;
    g.hz = hz;
    g.woff = woff;
    g.gamma = gamma;
    const double a2 = 0.25 * hx * hx, b2 = 0.25 * hy * hy, c2 = 0.25 * hz * hz;
    g.far2 = ratio * ratio * (a2 + b2 + c2);
    // the monomials by degree: a coefficient takes the moments of its own degree only
    for (int n = 0; n <= kSerN; ++n) {
        int at[kSerC], cnt = 0;
        double mom[kSerC];
        for (int i = 0; i <= n; ++i)
            for (int j = 0; i + j <= n; ++j) {
                at[cnt] = ser_idx(i, j, n - i - j);
                mom[cnt++] = ser_moment(a2, b2, c2, i, j, n - i - j);
            }
        for (int c = 0; c < 4; ++c)
            for (int m = 0; m < cnt; ++m) {
                double v = 0;
                for (int q = 0; q < cnt; ++q) v += kSerHost.t[c][at[m]][at[q]] * mom[q];
                g.coef[c][at[m]] = v;
            }
    }
    return g;
}

// The same on the device, one block per geometry: the E components only.
__global__ void __launch_bounds__(128) k_cell_series(CellGeom *__restrict__ gs, double ratio) {
    CellGeom &g = gs[blockIdx.x];
    __shared__ double mom[kSerC];
    __shared__ int deg[kSerC];
    const double a2 = 0.25 * g.hx * g.hx, b2 = 0.25 * g.hy * g.hy, c2 = 0.25 * g.hz * g.hz;
    const int t = threadIdx.x;
    if (t < kSerC) {
        int i, j, k;
        ser_exp(t, i, j, k);
        mom[t] = ser_moment(a2, b2, c2, i, j, k);
        deg[t] = i + j + k;
    }
    __syncthreads();
    if (t < 3 * kSerC) {
        const int c = 1 + t / kSerC, m = t - (c - 1) * kSerC;
        double s = 0;
        for (int q = 0; q < kSerC; ++q)
            if (deg[q] == deg[m]) s += kSerDev.t[c][m][q] * mom[q];
        g.coef[c][m] = s;
    }
    if (t == 0) {
        g.woff = 0.0;
        g.far2 = ratio * ratio * (a2 + b2 + c2);
    }
}
int launch_cell_series(CellGeom *g, int n, cudaStream_t st) {
    if (n <= 0) return OSC_OK;
    k_cell_series<<<n, 128, 0, st>>>(g, ser_ratio<float>());
    return ok();
}

// sum of c[ser_idx(i, j, k)] u^i v^j w^k
__device__ __forceinline__ double ser_eval(const double *c, double u, double v, double w) {
    double s = 0;
#pragma unroll
    for (int i = kSerN; i >= 0; --i) {
        double sj = 0;
#pragma unroll
        for (int j = kSerN - i; j >= 0; --j) {
            double sk = c[ser_idx(i, j, kSerN - i - j)];
#pragma unroll
            for (int k = kSerN - i - j - 1; k >= 0; --k) sk = fma(sk, w, c[ser_idx(i, j, k)]);
            sj = j == kSerN - i ? sk : fma(sj, v, sk);
        }
        s = i == kSerN ? sj : fma(s, u, sj);
    }
    return s;
}

// A CTA of 256 threads owns a tile of 16 x 8 x 4 cells, two cells a thread.  A tile whose nearest cell
// is closer than the series' distance evaluates the primitives of its 17 x 9 x 5 corners in
// shared memory (1.5 per cell) and differences them; the far tiles compute all components at
// once from one 1/r.  On grids of few tiles the components of a near tile go to as many CTAs
// (split; a far tile's other CTAs leave at once), since the chain of one is what the launch
// takes; on larger ones a CTA walks them and no CTA is launched to leave: 128 x 128 x 256 takes
// 106 us with the split and 73 without, 128^3 62 and 44, 48^3 12.8 and 10.8, and 32^3 takes 11 with
// it.  Bound by the FP64 rate: about 150 operations per far cell for three components, against 3 x
// 200 with two logs, an atan, a square root and two divisions each for the primitives of every
// corner, which were also written out and read back: 170 us for the corners of 128 x 128 x 256
// and 71 for their differences.  The tile is small so that the few near tiles, whose chains of
// logs and atans are the longest, spread over the SMs (tiles of 32 x 8 x 4 took 144 us there with
// the split, against 106).
constexpr int CT_X = 16, CT_Y = 8, CT_Z = 4, CT_K = CT_X * CT_Y * CT_Z / 256;

// Component ICOMP of the CT_K far cells of a thread.
template <int ICOMP, typename TH>
__device__ __forceinline__ void far_cells(const double *cf, double fac, const double *lead, const double *u,
                                          const double *v, const double *w, int nk, int zero, TH *out, int64_t plane) {
#pragma unroll
    for (int k = 0; k < CT_K; ++k) {
        const double val = fac * lead[k] * ser_eval(cf, u[k], v[k], w[k]);
        if (k < nk) out[k * plane] = k == zero ? (TH)0 : (TH)val;
    }
}

template <typename TH, bool BATCH>
__global__ void __launch_bounds__(256, 3) k_green_cells(TH *__restrict__ h, CellArgs a, CellGeom g0,
                                                     const CellGeom *__restrict__ gb, bool split) {
    __shared__ double sF[(CT_X + 1) * (CT_Y + 1) * (CT_Z + 1)];
    __shared__ alignas(16) double sc[BATCH ? 4 * kSerP : 2];
    pdl_wait(h);
    pdl_trigger();
    const CellGeom &g = BATCH ? gb[blockIdx.y] : g0;
    const int ntx = (a.nx + CT_X - 1) / CT_X, nty = (a.ny + CT_Y - 1) / CT_Y, ntz = (a.nz + CT_Z - 1) / CT_Z;
    // components of a tile side by side: the near tiles come early for all of them
    const int nci = split ? a.ncomp : 1, ci = blockIdx.x % nci, t = blockIdx.x / nci;
    const int tx = t % ntx, ty = (t / ntx) % nty, tzz = t / (ntx * nty);
    const int half = tzz / ntz;  // zwrap: 1 for the negative displacements
    const int i0 = tx * CT_X, j0 = ty * CT_Y, k0 = (tzz - half * ntz) * CT_Z;
    const int c0 = half ? k0 - a.nz : k0;  // z displacement of the tile's first plane
    const int nz_t = min(CT_Z, a.nz - k0);
    const double hx = g.hx, hy = g.hy, hz = g.hz, woff = g.woff;
    const double wa = c0 * hz + woff, wb = (c0 + nz_t - 1) * hz + woff;
    const double wn = wa * wb <= 0.0 ? 0.0 : fmin(fabs(wa), fabs(wb));
    const double xn = i0 * hx, yn = j0 * hy;
    const bool far = xn * xn + yn * yn + wn * wn >= g.far2;  // NaN: near
    if (far && ci > 0) return;
    const int lx = threadIdx.x % CT_X, ly = (threadIdx.x / CT_X) % CT_Y, lz = threadIdx.x / (CT_X * CT_Y) * CT_K;
    const int i = i0 + lx, j = j0 + ly, nk = nz_t - lz;  // this thread's planes: c0 + lz + [0, min(CT_K, nk))
    const int zero = half ? -a.nz - (c0 + lz) : -1;      // the one at displacement -nz, if any
    const int64_t plane = (int64_t)a.nx * a.ny;
    TH *out = h + (int64_t)blockIdx.y * a.hstride + (int64_t)(half * a.nz + k0 + lz) * plane + (int64_t)j * a.nx + i;
    const int64_t cstride = (int64_t)a.nmem * a.hstride;
    if (!far) {
        const int mx = min(CT_X, a.nx - i0), my = min(CT_Y, a.ny - j0);
#pragma unroll 1
        for (int c = ci; c < a.ncomp; c += nci) {
            const int icomp = a.comps[c];
            const double factor = (icomp == 1 || icomp == 2 ? g.gamma : 1.0) / (hx * hy * hz);
#pragma unroll 1
            for (int q = threadIdx.x; q < (CT_X + 1) * (CT_Y + 1) * (CT_Z + 1); q += 256) {
                const int cx = q % (CT_X + 1), r = q / (CT_X + 1), cy = r % (CT_Y + 1), cz = r / (CT_Y + 1);
                if (cx <= mx && cy <= my && cz <= nz_t)
                    sF[q] = igf_primitive(icomp, (i0 + cx - 0.5) * hx, (j0 + cy - 0.5) * hy,
                                          (c0 + cz - 0.5) * hz + woff) * factor;
            }
            __syncthreads();
            if (i < a.nx && j < a.ny) {
                constexpr int sy = CT_X + 1, sz = sy * (CT_Y + 1);
#pragma unroll
                for (int k = 0; k < CT_K; ++k) {
                    if (k >= nk) break;
                    const double *f0 = sF + lx + sy * ly + sz * (lz + k);
                    double v = +f0[1 + sy + sz];
                    v = v - f0[sy + sz];
                    v = v - f0[1 + sz];
                    v = v - f0[1 + sy];
                    v = v - f0[0];
                    v = v + f0[sz];
                    v = v + f0[sy];
                    v = v + f0[1];
                    out[c * cstride + k * plane] = k == zero ? (TH)0 : (TH)v;
                }
            }
            if (nci == a.ncomp) return;
            __syncthreads();
        }
        return;
    }
    if (BATCH) {  // the coefficients, read by all threads at once
        for (int q = threadIdx.x; q < 4 * kSerP; q += 256) sc[q] = (&g.coef[0][0])[q];
        __syncthreads();
    }
    if (i >= a.nx || j >= a.ny || nk <= 0) return;
    const double x = i * hx, y = j * hy;
    double u[CT_K], v[CT_K], w[CT_K], ri[CT_K], lx3[CT_K], ly3[CT_K], lz3[CT_K];
#pragma unroll
    for (int k = 0; k < CT_K; ++k) {
        const double z = (c0 + lz + k) * hz + woff;
        const double r2 = x * x + y * y + z * z;
        ri[k] = rsqrt(r2);
        const double t2 = ri[k] * ri[k], t4 = t2 * t2, t3 = ri[k] * t2;
        lx3[k] = x * t3;
        ly3[k] = y * t3;
        lz3[k] = z * t3;
        u[k] = x * x * t4;
        v[k] = y * y * t4;
        w[k] = z * z * t4;
    }
    // the component is a compile-time constant of each branch, so that one geometry's
    // coefficients are constant-bank operands
    for (int c = 0; c < a.ncomp; ++c) {
        TH *oc = out + c * cstride;
        switch (a.comps[c]) {
        case 0: far_cells<0, TH>(BATCH ? sc : g0.coef[0], 1.0, ri, u, v, w, nk, zero, oc, plane); break;
        case 1: far_cells<1, TH>(BATCH ? sc + kSerP : g0.coef[1], g.gamma, lx3, u, v, w, nk, zero, oc, plane); break;
        case 2: far_cells<2, TH>(BATCH ? sc + 2 * kSerP : g0.coef[2], g.gamma, ly3, u, v, w, nk, zero, oc, plane); break;
        default: far_cells<3, TH>(BATCH ? sc + 3 * kSerP : g0.coef[3], 1.0, lz3, u, v, w, nk, zero, oc, plane); break;
        }
    }
}

// CTAs of a launch; split where one CTA per component of every tile is still within two waves.
static dim3 cells_grid(const CellArgs &a, bool &split) {
    const int64_t ntx = ceil_div(a.nx, CT_X), nty = ceil_div(a.ny, CT_Y), ntz = ceil_div(a.nz, CT_Z);
    const int64_t nt = ntx * nty * ntz * (a.zwrap ? 2 : 1);
    split = nt * a.ncomp * a.nmem <= 148 * 3 * 2;
    return dim3((unsigned)(nt * (split ? a.ncomp : 1)), (unsigned)a.nmem);
}
template <typename TH> int launch_green_cells(TH *h, const CellArgs &a, const CellGeom &g, cudaStream_t st) {
    if (a.nmem != 1 || a.ncomp < 1 || a.ncomp > 4) return OSC_E_INVALID;
    bool split;
    const dim3 grid = cells_grid(a, split);
    launch_pdl(k_green_cells<TH, false>, grid, dim3(256), 0, st, h, a, g, nullptr, split);
    return ok();
}
template int launch_green_cells<float>(float *, const CellArgs &, const CellGeom &, cudaStream_t);
template int launch_green_cells<double>(double *, const CellArgs &, const CellGeom &, cudaStream_t);
int launch_green_cells_batch(float *h, const CellArgs &a, const CellGeom *g, cudaStream_t st) {
    if (a.nmem < 1 || a.ncomp < 1 || a.ncomp > 4) return OSC_E_INVALID;
    bool split;
    const dim3 grid = cells_grid(a, split);
    launch_pdl(k_green_cells<float, true>, grid, dim3(256), 0, st, h, a, CellGeom{}, g, split);
    return ok();
}

}  // namespace osc
