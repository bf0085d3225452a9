// fft_kernels_impl.cuh -- batched shared-memory FFT kernels for the IGF convolution (sm_100a).
// Included by the fft_*_f32.cu and fft_*_f64.cu files, which instantiate one family of kernels in one
// precision each.
//
// The free-space solve runs as five kernels over HBM (FP32 path, G spectra cached):
//   k_r2c_rows  x: real rho rows -> half spectra (two rows packed per complex line)
//   k_lines     y: forward C2C along y (input window [0,ny))
//   k_zconv     z: forward along z, multiply by the stored Green spectra, inverse along z
//   k_lines     y: inverse C2C along y (output window [0,ny))
//   k_c2r_rows  x: inverse to real rows, epilogue scatters E (and B) to their layouts
// Zero padding of the doubled grid is never stored: loads past the physical window are
// zeros (or, for the static engines, not read at all) and stores cover only the window.
#pragma once
#include <cstdio>
#include <map>
#include <mutex>
#include <type_traits>
#include <utility>

#include "fft_kernels.cuh"
#include "zconv_warp.cuh"
#include "zconv_w512.cuh"
#include "zconv_img.cuh"

namespace osc {

// Line buffers of a kernel that transforms in shared memory (FftRuntime alternates between two).
template <class E> constexpr int eng_bufs() { return E::kLen > 0 ? 1 : 2; }

// f(row, e) for e < len of rows [0, nrows).  Where len is the compile-time LEN, threads walk the flat
// sequence; otherwise whole warps walk a row, so that no index is divided by a length known only
// at run time, at the price of part-empty warps at the ends of rows: the x inverse to planes of
// 16 x 16 x 16 takes 28.9 us with rows of 16 walked by warps, 18.9 flat.
template <int LEN, class F> __device__ __forceinline__ void for_rows(int nrows, int len, F &&f) {
    if constexpr (LEN > 0) {
        if (len == LEN) {
            for (int idx = threadIdx.x; idx < nrows * LEN; idx += blockDim.x) f(idx / LEN, idx % LEN);
            return;
        }
    }
    const int lane = threadIdx.x & 31, nw = blockDim.x >> 5;
#pragma unroll 2
    for (int r = threadIdx.x >> 5; r < nrows; r += nw)
#pragma unroll 2
        for (int e = lane; e < len; e += 32) f(r, e);
}

// ------------------------------------------------------------------------------------
// MODE 0: full transform; 1: input window is the lower half (static engines skip it);
// 2: output window is the lower half and is not flipped (static engines skip the rest).
template <typename T, int NL, bool ROW, class E, int MODE>
__global__ void __launch_bounds__(E::kMaxThreads) k_lines(const cplx<T> *in, cplx<T> *out, LineArgs a,
                                                          const cplx<T> *__restrict__ twg) {
    typedef cplx<T> V;
    extern __shared__ __align__(16) unsigned char smem_raw[];
    V *tw = reinterpret_cast<V *>(smem_raw);
    const int L = E::kLen ? E::kLen : a.p.L;
    V *buf = tw + L;
    constexpr int lstr = NL + 1;
    const int nthreads = blockDim.x, tid = threadIdx.x;
    const int col0 = blockIdx.x * NL;
    const V *src;
    V *dst = out + (int64_t)blockIdx.z * a.out_zstride + (int64_t)blockIdx.y * a.out_pstride;
    load_twiddles(tw, twg, L);
    // rows are copied to shared memory as they are read (128^3 plain FP64 solve, seven x passes: 1120 us
    // with generic loads, 890 this way); columns go to registers first, and either wait does
    if (ROW) pdl_wait_global(in);
    else pdl_wait(in);
    pdl_trigger();
    src = in + (int64_t)blockIdx.z * a.in_zstride + (int64_t)blockIdx.y * a.in_pstride;
    if (!ROW) {
        // columns: the first stage reads global memory, the last stage writes it
        __syncthreads();
        const bool flip = (a.flip_mask >> blockIdx.z) & 1u;
        const T sc = (T)a.scale;
        if constexpr (E::kLen == 0) {
            // a thread stays on one line: its pointers once, flat or plane by plane
            const int l0 = tid % NL;
            int pl = a.flat_lines > 0 ? col0 / a.ncols : (int)blockIdx.y, c = a.flat_lines > 0 ? col0 - pl * a.ncols + l0 : col0 + l0;
            const bool live = a.flat_lines > 0 ? col0 + l0 < a.flat_lines : c < a.ncols;
            if (a.flat_lines > 0 && c >= a.ncols) {
                c -= a.ncols;
                ++pl;
            }
            const V *sp = in + (int64_t)blockIdx.z * a.in_zstride + (int64_t)pl * a.in_pstride + (int64_t)c * a.in_cstride;
            V *dp = out + (int64_t)blockIdx.z * a.out_zstride + (int64_t)pl * a.out_pstride + (int64_t)c * a.out_cstride;
            auto ld = [&](int e, int) -> V {
                return live && e < a.in_len ? sp[(int64_t)e * a.in_estride] : mk<T>(0, 0);
            };
            auto st = [&](int p, int, const V &v) {
                const int e = (flip && p > 0 ? L - p : p) - a.out_lo;
                if (live && e >= 0 && e < a.out_len) dp[(int64_t)e * a.out_estride] = cscale(v, sc);
            };
            E::template run_io<V, NL, false, false>(buf, a.p, tw, a.sign, ld, st);
            return;
        }
        if (a.flat_lines > 0) {
            // tile over the flat line sequence: line col0 + l is column (c0 + l) of plane pl0,
            // or column (c0 + l - ncols) of plane pl0 + 1 (NL <= ncols, so at most one wrap)
            const int pl0 = col0 / a.ncols, c0 = col0 - pl0 * a.ncols;
            const V *src0 = in + (int64_t)blockIdx.z * a.in_zstride + (int64_t)pl0 * a.in_pstride;
            V *dst0 = out + (int64_t)blockIdx.z * a.out_zstride + (int64_t)pl0 * a.out_pstride;
            const int64_t in_wrap = a.in_pstride - (int64_t)a.ncols * a.in_cstride;
            const int64_t out_wrap = a.out_pstride - (int64_t)a.ncols * a.out_cstride;
            auto ld = [&](int e, int l) -> V {
                const int c = c0 + l;
                V v = mk<T>(0, 0);
                if (e < a.in_len && col0 + l < a.flat_lines)
                    v = src0[(int64_t)c * a.in_cstride + (c >= a.ncols ? in_wrap : 0) + (int64_t)e * a.in_estride];
                return v;
            };
            auto st = [&](int p, int l, const V &v) {
                const int c = c0 + l;
                const int e = (flip ? (L - p) % L : p) - a.out_lo;
                if (col0 + l < a.flat_lines && e >= 0 && e < a.out_len)
                    dst0[(int64_t)c * a.out_cstride + (c >= a.ncols ? out_wrap : 0) + (int64_t)e * a.out_estride] =
                        cscale(v, sc);
            };
            E::template run_io<V, NL, MODE == 1, MODE == 2>(buf, a.p, tw, a.sign, ld, st);
            return;
        }
        auto ld = [&](int e, int l) -> V {
            const int col = col0 + l;
            V v = mk<T>(0, 0);
            if (e < a.in_len && col < a.ncols) v = src[(int64_t)col * a.in_cstride + (int64_t)e * a.in_estride];
            return v;
        };
        auto st = [&](int p, int l, const V &v) {
            const int col = col0 + l;
            const int e = (flip ? (L - p) % L : p) - a.out_lo;
            if (col < a.ncols && e >= 0 && e < a.out_len)
                dst[(int64_t)col * a.out_cstride + (int64_t)e * a.out_estride] = cscale(v, sc);
        };
        E::template run_io<V, NL, MODE == 1, MODE == 2>(buf, a.p, tw, a.sign, ld, st);
        return;
    }
    // rows (blocks of contiguous lines); every element of a line is loaded, zeros past in_len
    static_assert(!ROW || E::kLen * NL / E::kEPT % 32 == 0, "for_rows needs whole warps");
    auto put = [&](int c, int e) {
        V v = mk<T>(0, 0);
        const int col = col0 + c;
        if (e < a.in_len && col < a.ncols) v = src[(int64_t)col * a.in_cstride + (int64_t)e * a.in_estride];
        buf[e * lstr + c] = v;
    };
    if constexpr (E::kLen > 0)
        for (int idx = tid; idx < NL * E::kLen; idx += nthreads) put(idx / E::kLen, idx % E::kLen);
    else
        for_rows<0>(NL, L, put);
    __syncthreads();
    const V *res = E::template run<V, NL, false, false>(buf, a.p, tw, a.sign);
    const T sc = (T)a.scale;
    for_rows<0>(NL, a.out_len, [&](int c, int e) {
        const int col = col0 + c;
        const int p = e + a.out_lo, src_e = ((a.flip_mask >> blockIdx.z) & 1u) && p > 0 ? L - p : p;
        if (col < a.ncols)
            dst[(int64_t)col * a.out_cstride + (int64_t)e * a.out_estride] = cscale(res[src_e * lstr + c], sc);
    });
}

// ------------------------------------------------------------------------------------
// Element e of the real input row at p (jn: a quad-grid row with a y neighbour below it).
template <typename TIn>
__device__ __forceinline__ TIn r2c_in(const TIn *__restrict__ p, const R2CArgs &, bool, int e) {
    return p[e];
}
// Quad-grid input of the FP32 deposit: node (i,j) of a plane is the sum of the four
// contributions held at (i,j).x, (i-1,j).y, (i,j-1).z and (i-1,j-1).w, added in that
// fixed order (the order of k_quad_to_nodes, so rho is the same to the bit).
__device__ __forceinline__ float r2c_in(const float4 *__restrict__ p, const R2CArgs &a, bool jn, int e) {
    const float4 *q = p + e;
    float s = __ldca(&q->x);
    if (e > 0) s += __ldca(&q[-1].y);
    if (jn) s += __ldca(&q[-a.in_rstride].z);
    if (e > 0 && jn) s += __ldca(&q[-a.in_rstride - 1].w);
    return s;
}

// resident CTAs the register allocation of k_r2c_rows is bounded for: 4 (32 registers, no
// spills) for the FP32 step's quad-grid input on the 8-values-per-thread engine at L = 256,
// whose loads wait on L2 (35.4 against 40.8 us at 40 registers and 3 CTAs, then with one row of a
// line per thread; 29 us with both); 1 otherwise
template <typename T, typename TIn, class E> constexpr int r2c_minb() {
    return (std::is_same<TIn, float4>::value && E::kLen == 256 && E::kEPT == 8) ? 4 : 1;
}
template <typename T, typename TIn, int NL, class E, bool HIN>
__global__ void __launch_bounds__(E::kMaxThreads, r2c_minb<T, TIn, E>()) k_r2c_rows(const TIn *__restrict__ in, cplx<T> *__restrict__ out,
                                                             R2CArgs a, const cplx<T> *__restrict__ twg) {
    typedef cplx<T> V;
    extern __shared__ __align__(16) unsigned char smem_raw[];
    V *tw = reinterpret_cast<V *>(smem_raw);
    const int L = E::kLen ? E::kLen : a.p.L;
    V *buf = tw + L;
    constexpr int lstr = NL + 1;
    // static engines launch with L*NL/E::kEPT threads: compile-time trip counts below
    const int nthreads = E::kLen ? E::kLen * NL / E::kEPT : (int)blockDim.x, tid = threadIdx.x;
    const int64_t row0 = (int64_t)blockIdx.x * (2 * NL);
    // whether a quad-grid row has a y neighbour: one division per row, not per element
    __shared__ bool jns[2 * NL];
    if (std::is_same<TIn, float4>::value) {
        for (int t = tid; t < 2 * NL; t += nthreads) jns[t] = (row0 + t) % a.qny > 0;
        __syncthreads();
    }
    load_twiddles(tw, twg, L);
    pdl_wait(in);
    pdl_trigger();
    auto elem = [&](int rr, int e) -> T {
        const int64_t row = row0 + rr;
        if (row >= a.nrows || e >= a.nin) return (T)0;
        return (T)r2c_in(in + row * a.in_rstride, a, std::is_same<TIn, float4>::value ? jns[rr] : false, e);
    };
    if constexpr (E::kLen > 0) {
        // a thread carries both rows of a line; all of its loads are issued before any is stored to
        // shared memory
        constexpr int LDL = HIN ? E::kLen / 2 : E::kLen, NT = E::kLen * NL / E::kEPT;
        constexpr int IT = (NL * LDL + NT - 1) / NT;
        V v[IT];
#pragma unroll
        for (int it = 0; it < IT; ++it) {
            const int idx = tid + it * NT, ln = idx / LDL, e = idx - ln * LDL;
            v[it] = mk<T>(0, 0);
            if (idx < NL * LDL) v[it] = mk<T>(elem(2 * ln, e), elem(2 * ln + 1, e));
        }
#pragma unroll
        for (int it = 0; it < IT; ++it) {
            const int idx = tid + it * NT, ln = idx / LDL, e = idx - ln * LDL;
            if (idx < NL * LDL) buf[e * lstr + ln] = v[it];
        }
    } else {
        for_rows<0>(NL, L, [&](int ln, int e) { buf[e * lstr + ln] = mk<T>(elem(2 * ln, e), elem(2 * ln + 1, e)); });
    }
    __syncthreads();
    const V *res = E::template run<V, NL, HIN, false>(buf, a.p, tw, +1);
    auto put = [&](int ln, int k) {
        const int64_t row = row0 + 2 * ln;
        const V Z = res[k * lstr + ln], Zm = res[(k > 0 ? L - k : 0) * lstr + ln];
        V *o = out + row * a.out_rstride + k;
        // (Z + conj Zm)/2 and (Z - conj Zm)/(2i)
        if (row < a.nrows) *o = mk<T>((T)0.5 * (Z.x + Zm.x), (T)0.5 * (Z.y - Zm.y));
        if (row + 1 < a.nrows) o[a.out_rstride] = mk<T>((T)0.5 * (Z.y + Zm.y), (T)0.5 * (Zm.x - Z.x));
    };
    if constexpr (E::kLen > 0) {
        constexpr int nh = E::kLen / 2 + 1;
        for (int idx = tid; idx < NL * nh; idx += nthreads) put(idx / nh, idx % nh);
    } else {
        for_rows<0>(NL, L / 2 + 1, put);
    }
}

// ------------------------------------------------------------------------------------
// Input offset and output grid row of real row r of an x inverse (see C2RArgs::zin).
__device__ __forceinline__ void row_bases(const C2RArgs &a, int64_t r, int64_t &in_off, int64_t &out_row) {
    if (!a.zin) {
        in_off = r * a.in_rstride;
        out_row = r;
        return;
    }
    const int64_t t = r / a.zin_nz, z = r - t * a.zin_nz;  // t = b*ny + y
    const int64_t b = t / a.zin_ny, y = t - b * a.zin_ny;
    in_off = t * a.in_rstride + z;
    out_row = (b * a.zin_nz + z) * a.zin_ny + y;
}

template <typename T>
__device__ __forceinline__ void write_dest(const OutDest &d, int64_t gidx, int x, T val) {
    // vec4 grids also write their unused 4th slot, so every 32-byte sector is written whole
    switch (d.kind) {
    case 0: {
        T *p = reinterpret_cast<T *>(d.ptr) + gidx * 4;
        p[d.slot] = (T)(d.coef * val);
        if (d.slot == 2) p[3] = (T)0;
        break;
    }
    case 1: reinterpret_cast<double *>(d.ptr)[gidx] = d.coef * (double)val; break;
    case 3: reinterpret_cast<double *>(d.ptr)[gidx] += d.coef * (double)val; break;
    case 4: {  // x-pair grid: node n holds (E(n), E(n+1)) as two vec4; the last node's
               // second half is never read and is zeroed
        T *p = reinterpret_cast<T *>(d.ptr);
        const T v = (T)(d.coef * val);
        p[gidx * 8 + d.slot] = v;
        if (d.slot == 2) p[gidx * 8 + 3] = (T)0;
        if (x > 0) {
            p[(gidx - 1) * 8 + 4 + d.slot] = v;
            if (d.slot == 2) p[(gidx - 1) * 8 + 7] = (T)0;
        }
        if (x == d.last_x) {
            p[gidx * 8 + 4 + d.slot] = (T)0;
            if (d.slot == 2) p[gidx * 8 + 7] = (T)0;
        }
        break;
    }
    default: reinterpret_cast<T *>(d.ptr)[gidx] = (T)(d.coef * val); break;
    }
}

template <typename T, int NL, class E, bool HOUT>
__global__ void __launch_bounds__(E::kMaxThreads) k_c2r_rows(const cplx<T> *__restrict__ in, C2RArgs a,
                                                             const cplx<T> *__restrict__ twg) {
    typedef cplx<T> V;
    extern __shared__ __align__(16) unsigned char smem_raw[];
    V *tw = reinterpret_cast<V *>(smem_raw);
    const int L = E::kLen ? E::kLen : a.p.L;
    V *buf = tw + L;
    constexpr int lstr = NL + 1;
    const int nthreads = blockDim.x, tid = threadIdx.x;
    const int64_t row0 = (int64_t)blockIdx.x * (2 * NL);
    const int half = L / 2;
    static_assert(E::kLen * NL / E::kEPT % 32 == 0, "for_rows needs whole warps");
    T *res = reinterpret_cast<T *>(buf + eng_bufs<E>() * L * lstr);  // [3][2*NL][nout] when a.e8 is set
    __shared__ int64_t rin[2 * NL], rout[2 * NL];
    for (int t = tid; t < 2 * NL; t += nthreads) row_bases(a, row0 + t, rin[t], rout[t]);
    const int64_t ies = a.zin ? a.zin_nz : 1;
    load_twiddles(tw, twg, L);
    pdl_wait(in);
    pdl_trigger();
    __syncthreads();
    for (int c = 0; c < a.ncomp; ++c) {
        const V *src = in + (int64_t)c * a.in_cstride;
        auto put = [&](int line, int k) {
            const int64_t ra = row0 + 2 * line, rb = ra + 1;
            const int kk = k <= half ? k : L - k;
            V A = mk<T>(0, 0), B = mk<T>(0, 0);
            if (ra < a.nrows) A = src[rin[2 * line] + kk * ies];
            if (rb < a.nrows) B = src[rin[2 * line + 1] + kk * ies];
            if (k == 0 || k == half) { A.y = 0; B.y = 0; }
            if (k > half) { A.y = -A.y; B.y = -B.y; }
            buf[k * lstr + line] = mk<T>(A.x - B.y, A.y + B.x);
        };
        if (a.zin)  // adjacent lines (adjacent z) fastest for the kz-innermost spectra
            for (int idx = tid; idx < NL * L; idx += nthreads) put(idx % NL, idx / NL);
        else
            for_rows<E::kLen>(NL, L, put);
        __syncthreads();
        const V *fb = E::template run<V, NL, false, HOUT>(buf, a.p, tw, -1);
        for_rows<E::kLen / 2>(2 * NL, a.nout, [&](int rr, int x) {
            const int64_t row = row0 + rr;
            if (row >= a.nrows) return;
            const int xs = ((a.flip_mask >> c) & 1u) && x > 0 ? L - x : x;
            const V z = fb[xs * lstr + (rr >> 1)];
            const T val = (rr & 1) ? z.y : z.x;
            const int64_t gidx = rout[rr] * a.nout + x;
            for (int d = 0; d < a.ndest[c]; ++d) write_dest<T>(a.dest[c][d], gidx, x, val);
            if (a.e8) {
#pragma unroll
                for (int q = 0; q < 3; ++q)
                    if (a.e8_comp[q] == c) res[(q * 2 * NL + rr) * a.nout + x] = val;
            }
        });
        __syncthreads();
    }
    if (a.e8) {
        // x-pair grid rows: node n gets (E(n), E(n+1)), the row's last node (E(n), 0)
        typedef vec4<T> V4;
        V4 *g = reinterpret_cast<V4 *>(a.e8);
        for_rows<E::kLen / 2>(2 * NL, a.nout, [&](int rr, int x) {
            const int64_t row = row0 + rr;
            if (row >= a.nrows) return;
            const int64_t gidx = rout[rr] * a.nout + x;
            const T *r0 = res + rr * a.nout + x;
            const int64_t cs = (int64_t)2 * NL * a.nout;
            V4 lo, hi;
            lo.x = r0[0];
            lo.y = r0[cs];
            lo.z = r0[2 * cs];
            lo.w = (T)0;
            if (x + 1 < a.nout) {
                hi.x = r0[1];
                hi.y = r0[cs + 1];
                hi.z = r0[2 * cs + 1];
            } else {
                hi.x = hi.y = hi.z = (T)0;
            }
            hi.w = (T)0;
            if (a.e8_node) {
                g[gidx] = lo;
            } else {
                g[2 * gidx] = lo;
                g[2 * gidx + 1] = hi;
            }
        });
    }
}

// ------------------------------------------------------------------------------------
// One (kx, ky) column of a stored Green spectrum: g_lookup with everything that does not depend
// on kz worked out once.
template <typename T> struct GColumn {
    const void *p;
    int64_t zs;
    bool realv, iu, symz, neg, zneg;
    __device__ __forceinline__ GColumn(const GSpecDev &g, int kx, int ky, int nxh, int Ny, int ny, int64_t goff) {
        const bool my = g.sym_y && ky > ny;
        const int yy = my ? Ny - ky : ky;
        realv = g.real_valued;
        iu = g.imag_unit;
        symz = g.sym_z;
        neg = my && g.par_y < 0;
        zneg = g.par_z < 0;
        const int64_t at = goff + (int64_t)yy * nxh + kx;
        zs = (int64_t)g.dimy * nxh;
        p = realv ? (const void *)(reinterpret_cast<const T *>(g.data) + at)
                  : (const void *)(reinterpret_cast<const cplx<T> *>(g.data) + at);
    }
    __device__ __forceinline__ cplx<T> times(const cplx<T> &x, int kz, int Nz, int nz) const {
        const bool mz = symz && kz > nz;
        const int64_t at = (int64_t)(mz ? Nz - kz : kz) * zs;
        const bool sg = neg != (mz && zneg);
        if (realv) {
            T s = __ldg(reinterpret_cast<const T *>(p) + at);
            if (sg) s = -s;
            return iu ? mk<T>(-x.y * s, x.x * s) : mk<T>(x.x * s, x.y * s);
        }
        cplx<T> v = __ldg(reinterpret_cast<const cplx<T> *>(p) + at);
        if (sg) { v.x = -v.x; v.y = -v.y; }
        return cmul(x, v);
    }
};

// The z pass of the lengths without a warp engine, NL columns per CTA on the runtime-plan
// engine.  The forward transform reads its columns straight from global memory into its first
// stage; each inverse transform forms its input (spectrum times Green spectrum, plus the image
// term) inside its first stage and writes its last stage straight to global memory.  A thread
// stays on one column, whose Green column and pointers it works out once.
template <typename T, int NL>
__global__ void __launch_bounds__(FftRuntime::kMaxThreads) k_zconv(const cplx<T> *__restrict__ in, cplx<T> *__restrict__ out,
                                                                   ZConvArgs a, const cplx<T> *__restrict__ twg,
                                                                   const cplx<T> *__restrict__ tw_rt) {
    typedef cplx<T> V;
    extern __shared__ __align__(16) unsigned char smem_raw[];
    V *tw = reinterpret_cast<V *>(smem_raw);
    const int L = a.p.L;
    V *rhat = tw + L;
    constexpr int lstr = NL + 1;
    V *buf = rhat + L * lstr;
    const int l0 = threadIdx.x % NL, col = blockIdx.x * NL + l0, colc = min(col, a.ncols - 1);
    const bool live = col < a.ncols;
    const int ky = colc / a.nxh, kx = colc - ky * a.nxh;
    in += blockIdx.y * a.in_bstride + colc;
    out += blockIdx.y * a.out_bstride + (int64_t)colc * a.out_colstride;
    const int64_t goff = blockIdx.y * a.g_bstride;
    load_twiddles(tw, twg, L);
    pdl_wait(in);
    pdl_trigger();
    __syncthreads();
    auto ld_in = [&](int e, int) -> V { return live && e < a.nz ? in[(int64_t)e * a.in_estride] : mk<T>(0, 0); };
    auto st_rhat = [&](int e, int l, const V &v) { rhat[e * lstr + l] = v; };
    FftRuntime::template run_io<V, NL, false, false>(buf, a.p, tw, +1, ld_in, st_rhat);
    for (int o = 0; o < a.nout; ++o) {
        const int gd = a.gdir[o], gi = a.gimg[o];
        const GColumn<T> cd(a.g[gd >= 0 ? gd : 0], kx, ky, a.nxh, a.Ny, a.ny, goff);
        V *dst = out + (int64_t)o * a.out_cstride;
        auto st_out = [&](int e, int, const V &v) {
            if (e < a.nz && live) dst[(int64_t)e * a.out_estride] = v;
        };
        if (gi < 0) {
            auto ld_mul = [&](int e, int l) -> V {
                return gd >= 0 ? cd.times(rhat[e * lstr + l], e, L, a.nz) : mk<T>(0, 0);
            };
            FftRuntime::template run_io<V, NL, false, false>(buf, a.p, tw, -1, ld_mul, st_out);
        } else {
            const GColumn<T> ci(a.g[gi], kx, ky, a.nxh, a.Ny, a.ny, goff);
            const T icoef = (T)a.img_coef[o];
            auto ld_mul = [&](int e, int l) -> V {
                V S = gd >= 0 ? cd.times(rhat[e * lstr + l], e, L, a.nz) : mk<T>(0, 0);
                // spectrum of -rho flipped in z: -w^((nz-1) kz) * rho_hat(-kz)
                const V rm = rhat[(e > 0 ? L - e : 0) * lstr + l];
                // (nz-1)*kz < 2^21: 32-bit index arithmetic
                const V ph = __ldg(tw_rt + (int)(((unsigned)a.img_phase_mul * (unsigned)e) % (unsigned)L));
                V ri = cmul(ph, rm);
                ri.x = -ri.x * icoef;
                ri.y = -ri.y * icoef;
                return cadd(S, ci.times(ri, e, L, a.nz));
            };
            FftRuntime::template run_io<V, NL, false, false>(buf, a.p, tw, -1, ld_mul, st_out);
        }
    }
}

// x inverse of the FP32 step: three E components of 2*NLC real rows each go through one
// transform batch of 3*NLC complex lines, and every output node of the window x < L/2 is
// written as one 32-byte x-pair (E(x), E(x+1)) with a single 256-bit store.  Requires the
// static engine for L, nout = L/2, no index flips and no other destinations.
__device__ __forceinline__ void st_pair(float4 *p, const float4 &lo, const float4 &hi) {
    asm volatile("st.global.v8.f32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8};" ::"l"(p), "f"(lo.x), "f"(lo.y), "f"(lo.z),
                 "f"(lo.w), "f"(hi.x), "f"(hi.y), "f"(hi.z), "f"(hi.w)
                 : "memory");
}
__device__ __forceinline__ void st_node(double4 *p, double x, double y, double z) {
    asm volatile("st.global.v4.f64 [%0], {%1,%2,%3,%4};" ::"l"(p), "d"(x), "d"(y), "d"(z), "d"(0.0) : "memory");
}
// Node x of the two real rows (row, row + 1) that came out as one complex line per component:
// z0 at x and, for x-pairs, z1 at x + 1 (0 past the end).
template <typename T>
__device__ __forceinline__ void e8_rows(const C2RArgs &a, const cplx<T> (&z0)[3], const cplx<T> (&z1)[3], int64_t row,
                                        const int64_t *rout, int nout, int x) {
    if constexpr (sizeof(T) == 4) {
        float4 *g = reinterpret_cast<float4 *>(a.e8);
        if (row < a.nrows)
            st_pair(g + 2 * (rout[0] * nout + x), make_float4(z0[0].x, z0[1].x, z0[2].x, 0.f),
                    make_float4(z1[0].x, z1[1].x, z1[2].x, 0.f));
        if (row + 1 < a.nrows)
            st_pair(g + 2 * (rout[1] * nout + x), make_float4(z0[0].y, z0[1].y, z0[2].y, 0.f),
                    make_float4(z1[0].y, z1[1].y, z1[2].y, 0.f));
    } else {
        double4 *g = reinterpret_cast<double4 *>(a.e8);
        if (row < a.nrows) st_node(g + rout[0] * nout + x, z0[0].x, z0[1].x, z0[2].x);
        if (row + 1 < a.nrows) st_node(g + rout[1] * nout + x, z0[0].y, z0[1].y, z0[2].y);
    }
}
template <typename T, class E> constexpr int c2r_e8_nlc() {
    return (E::kLen <= 128 ? 16 : (E::kLen <= 256 ? 8 : 4)) / (sizeof(T) == 8 ? 2 : 1);
}

// FP32: x-pair nodes (E(x), E(x+1)) with one 256-bit store; FP64: nodes (Ex, Ey, Ez, 0)
// with one 256-bit store.
template <typename T, int NLC, class E>
__global__ void __launch_bounds__(E::kLen * 3 * NLC / E::kEPT, sizeof(T) == 4 ? 3 : 1) k_c2r_e8(const cplx<T> *__restrict__ in, C2RArgs a,
                                                                      const cplx<T> *__restrict__ twg) {
    typedef cplx<T> V;
    constexpr int L = E::kLen, NLT = 3 * NLC, lstr = NLT + 1, half = L / 2, nout = L / 2;
    constexpr int nthreads = L * NLT / E::kEPT;
    extern __shared__ __align__(16) unsigned char smem_raw[];
    V *tw = reinterpret_cast<V *>(smem_raw);
    V *buf = tw + L;
    const int tid = threadIdx.x;
    const int64_t row0 = (int64_t)blockIdx.x * (2 * NLC);
    __shared__ int64_t rin[2 * NLC], rout[2 * NLC];
    for (int t = tid; t < 2 * NLC; t += nthreads) row_bases(a, row0 + t, rin[t], rout[t]);
    const int64_t ies = a.zin ? a.zin_nz : 1;
    load_twiddles(tw, twg, L);
    pdl_wait(in);
    pdl_trigger();
    __syncthreads();
    // line = two real rows A + iB; each stored value k <= L/2 is read once and also gives
    // the line's value at L-k (from the conjugates)
    constexpr int nk = half + 1, IT = (NLT * nk + nthreads - 1) / nthreads;
    auto slot_of = [&](int idx, int &c, int &line, int &k) {
        if (a.zin) {  // rows (adjacent z) fastest: coalesced reads of the kz-innermost spectra
            k = idx / NLT;
            const int rem = idx - k * NLT;
            c = rem / NLC;
            line = rem - c * NLC;
        } else {
            c = idx / (NLC * nk);
            const int rem = idx - c * (NLC * nk);
            line = rem / nk;
            k = rem - line * nk;
        }
    };
    // all of a thread's loads are issued before any is stored to shared memory
    V A[IT], B[IT];
#pragma unroll
    for (int it = 0; it < IT; ++it) {
        const int idx = tid + it * nthreads;
        A[it] = mk<T>(0, 0);
        B[it] = mk<T>(0, 0);
        if (idx < NLT * nk) {
            int c, line, k;
            slot_of(idx, c, line, k);
            const V *src = in + (int64_t)a.e8_comp[c] * a.in_cstride;
            const int64_t ra = row0 + 2 * line, rb = ra + 1;
            if (ra < a.nrows) A[it] = src[rin[2 * line] + k * ies];
            if (rb < a.nrows) B[it] = src[rin[2 * line + 1] + k * ies];
        }
    }
#pragma unroll
    for (int it = 0; it < IT; ++it) {
        const int idx = tid + it * nthreads;
        if (idx < NLT * nk) {
            int c, line, k;
            slot_of(idx, c, line, k);
            V a0 = A[it], b0 = B[it];
            if (k == 0 || k == half) { a0.y = 0; b0.y = 0; }
            buf[k * lstr + c * NLC + line] = mk<T>(a0.x - b0.y, a0.y + b0.x);
            if (k > 0 && k < half) buf[(L - k) * lstr + c * NLC + line] = mk<T>(a0.x + b0.y, b0.x - a0.y);
        }
    }
    __syncthreads();
    E::template run<V, NLT, false, true>(buf, a.p, tw, -1);
    for (int idx = tid; idx < NLC * nout; idx += nthreads) {
        const int ln = idx / nout, x = idx - ln * nout;
        V z0[3], z1[3];
#pragma unroll
        for (int c = 0; c < 3; ++c) {
            z0[c] = buf[x * lstr + c * NLC + ln];
            if constexpr (sizeof(T) == 4) z1[c] = x + 1 < nout ? buf[(x + 1) * lstr + c * NLC + ln] : mk<T>(0, 0);
        }
        e8_rows<T>(a, z0, z1, row0 + 2 * ln, &rout[2 * ln], nout, x);
    }
}

// The same on the runtime-plan engine, for the lengths without a static one.
template <typename T, int NLC>
__global__ void __launch_bounds__(FftRuntime::kMaxThreads) k_c2r_e8_rt(const cplx<T> *__restrict__ in, C2RArgs a,
                                                                       const cplx<T> *__restrict__ twg) {
    typedef cplx<T> V;
    constexpr int NLT = 3 * NLC, lstr = NLT + 1;
    const int L = a.p.L, half = L / 2, nout = half;
    extern __shared__ __align__(16) unsigned char smem_raw[];
    V *tw = reinterpret_cast<V *>(smem_raw);
    V *buf = tw + L;
    const int tid = threadIdx.x;
    const int64_t row0 = (int64_t)blockIdx.x * (2 * NLC);
    __shared__ int64_t rin[2 * NLC], rout[2 * NLC];
    for (int t = tid; t < 2 * NLC; t += blockDim.x) row_bases(a, row0 + t, rin[t], rout[t]);
    const int64_t ies = a.zin ? a.zin_nz : 1;
    load_twiddles(tw, twg, L);
    pdl_wait(in);
    pdl_trigger();
    __syncthreads();
    auto put = [&](int ln, int k) {  // ln = c * NLC + line
        const int c = ln / NLC, line = ln - c * NLC;
        const V *src = in + (int64_t)a.e8_comp[c] * a.in_cstride;
        const int64_t ra = row0 + 2 * line, rb = ra + 1;
        V A = mk<T>(0, 0), B = mk<T>(0, 0);
        if (ra < a.nrows) A = src[rin[2 * line] + k * ies];
        if (rb < a.nrows) B = src[rin[2 * line + 1] + k * ies];
        if (k == 0 || k == half) { A.y = 0; B.y = 0; }
        buf[k * lstr + ln] = mk<T>(A.x - B.y, A.y + B.x);
        if (k > 0 && k < half) buf[(L - k) * lstr + ln] = mk<T>(A.x + B.y, B.x - A.y);
    };
    if (a.zin)
#pragma unroll 4
        for (int idx = tid; idx < NLT * (half + 1); idx += blockDim.x) put(idx % NLT, idx / NLT);
    else
        for_rows<0>(NLT, half + 1, put);
    __syncthreads();
    const V *res = FftRuntime::template run<V, NLT, false, true>(buf, a.p, tw, -1);
    for_rows<0>(NLC, nout, [&](int ln, int x) {
        V z0[3], z1[3];
#pragma unroll
        for (int c = 0; c < 3; ++c) {
            z0[c] = res[x * lstr + c * NLC + ln];
            if constexpr (sizeof(T) == 4) z1[c] = x + 1 < nout ? res[(x + 1) * lstr + c * NLC + ln] : mk<T>(0, 0);
        }
        e8_rows<T>(a, z0, z1, row0 + 2 * ln, &rout[2 * ln], nout, x);
    });
}

// Even/odd real line transforms (Green spectra): two real lines per complex line, the
// parity extension formed in the load, the halves separated after the transform.  TC is
// the arithmetic type (and that of the twiddles), TI the input's, TO the output's.
template <typename TC, typename TI, typename TO, int NL, class E, bool LDE, bool STK>
__global__ void __launch_bounds__(E::kMaxThreads) k_sym_lines(const TI *__restrict__ in, TO *__restrict__ out,
                                                              SymArgs a, const cplx<TC> *__restrict__ twg) {
    typedef cplx<TC> V;
    extern __shared__ __align__(16) unsigned char smem_raw[];
    __shared__ int64_t bin[2 * NL], bout[2 * NL];
    __shared__ int podd[2 * NL];
    V *tw = reinterpret_cast<V *>(smem_raw);
    const int L = E::kLen ? E::kLen : a.p.L;
    V *buf = tw + L;
    constexpr int lstr = NL + 1;
    const int nthreads = blockDim.x, tid = threadIdx.x;
    const int64_t r0 = (int64_t)blockIdx.x * (2 * NL);
    const int n = a.n;
    for (int t = tid; t < 2 * NL; t += nthreads) {  // line start offsets, once per line
        // members start on even lines, so that no two of them (phi and E differ by orders of
        // magnitude) share a complex line
        const int64_t r = r0 + t, npq2 = (a.npq + 1) & ~(int64_t)1, bi = r / npq2, rl = r - bi * npq2;
        int64_t oi = -1, oo = -1;
        int odd = 0;
        if (bi < a.nb && rl < a.npq) {
            const int64_t pi = rl / a.nq, qi = rl - pi * a.nq;
            oi = bi * a.in_bs + pi * a.in_ps + qi * a.in_qs;
            oo = bi * a.out_bs + pi * a.out_ps + qi * a.out_qs;
            odd = bi >= a.odd_lo && bi < a.odd_hi;
        }
        bin[t] = oi;
        bout[t] = oo;
        podd[t] = odd;
    }
    load_twiddles(tw, twg, L);
    pdl_wait(in);
    pdl_trigger();
    __syncthreads();
    if constexpr (E::kLen > 0) {
        // static engine (L = 2n known, L*NL/E::kEPT threads): each thread first loads its share of
        // the n+1 distinct values of every line pair into registers (all loads in flight), then
        // writes each pair of values at e and its parity image at L-e
        constexpr int nh = E::kLen / 2, NK = nh + 1, TOT = NL * NK;
        constexpr int NT = E::kLen * NL / E::kEPT, IT = (TOT + NT - 1) / NT;
        V v[IT];
#pragma unroll
        for (int it = 0; it < IT; ++it) {
            const int idx = tid + it * NT;
            v[it] = mk<TC>(0, 0);
            if (idx < TOT) {
                const int ln = LDE ? idx / NK : idx % NL, e = LDE ? idx - ln * NK : idx / NL;
                const int64_t o0 = bin[2 * ln], o1 = bin[2 * ln + 1];
                if (o0 >= 0 && e != nh) v[it].x = (TC)in[o0 + (int64_t)e * a.in_es];
                if (o1 >= 0 && e != nh) v[it].y = (TC)in[o1 + (int64_t)e * a.in_es];
            }
        }
#pragma unroll
        for (int it = 0; it < IT; ++it) {
            const int idx = tid + it * NT;
            if (idx < TOT) {
                const int ln = LDE ? idx / NK : idx % NL, e = LDE ? idx - ln * NK : idx / NL;
                buf[e * lstr + ln] = v[it];
                if (e > 0 && e < nh)
                    buf[(E::kLen - e) * lstr + ln] = podd[2 * ln] ? mk<TC>(-v[it].x, -v[it].y) : v[it];
            }
        }
    } else {
        // each of the n+1 distinct values is read once and written at e and at L - e
        auto put = [&](int ln, int e) {
            const int64_t o0 = bin[2 * ln], o1 = bin[2 * ln + 1];
            V v = mk<TC>(0, 0);
            if (o0 >= 0 && e != n) v.x = (TC)in[o0 + (int64_t)e * a.in_es];
            if (o1 >= 0 && e != n) v.y = (TC)in[o1 + (int64_t)e * a.in_es];
            buf[e * lstr + ln] = v;
            if (e > 0 && e < n) buf[(L - e) * lstr + ln] = podd[2 * ln] ? mk<TC>(-v.x, -v.y) : v;
        };
        if (LDE) for_rows<0>(NL, n + 1, put);
        else
#pragma unroll 4
            for (int idx = tid; idx < NL * (n + 1); idx += nthreads) put(idx % NL, idx / NL);
    }
    __syncthreads();
    const V *res = E::template run<V, NL, false, false>(buf, a.p, tw, +1);
    const int nk = n + 1;
    // both lines of a pair have the same parity (members start on even lines)
    auto fin = [&](int ln, int k) {
        const int64_t o0 = bout[2 * ln], o1 = bout[2 * ln + 1];
        const V Z = res[k * lstr + ln], Zm = res[(k > 0 ? L - k : 0) * lstr + ln];
        const bool odd = podd[2 * ln];
        const TC hf = (TC)0.5;
        const TC s0 = !odd ? hf * (Z.x + Zm.x) : hf * (Z.y - Zm.y);
        const TC s1 = !odd ? hf * (Z.y + Zm.y) : hf * (Zm.x - Z.x);
        if (o0 >= 0) out[o0 + (int64_t)k * a.out_es] = (TO)(s0 * (TC)a.scale);
        if (o1 >= 0) out[o1 + (int64_t)k * a.out_es] = (TO)(s1 * (TC)a.scale);
    };
    if (!STK)
        for (int idx = tid; idx < NL * nk; idx += nthreads) fin(idx % NL, idx / NL);
    else if constexpr (E::kLen > 0)
        for (int idx = tid; idx < NL * (E::kLen / 2 + 1); idx += nthreads)
            fin(idx / (E::kLen / 2 + 1), idx % (E::kLen / 2 + 1));
    else
        for_rows<0>(NL, nk, fin);
}

// z transforms of the Green columns that are not even or odd in z (ZLineArgs): two real columns per
// complex line, FP64.  Reads and, with zpitch 0, writes walk adjacent columns; the kz-innermost
// store walks k.
template <typename TO, int NL, class E>
__global__ void __launch_bounds__(E::kMaxThreads) k_green_zlines(const double *__restrict__ in, cplx<TO> *__restrict__ out,
                                                                 ZLineArgs a, const double2 *__restrict__ twg,
                                                                 const double2 *__restrict__ tw_rt) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    __shared__ int64_t bin[2 * NL], bout[2 * NL];
    __shared__ bool bim[2 * NL];
    double2 *tw = reinterpret_cast<double2 *>(smem_raw);
    const int L = E::kLen ? E::kLen : a.p.L;
    double2 *buf = tw + L;
    constexpr int lstr = NL + 1;
    const int nthreads = blockDim.x, tid = threadIdx.x;
    for (int t = tid; t < 2 * NL; t += nthreads) {
        // members start on even lines (as in k_sym_lines)
        const int64_t r = (int64_t)blockIdx.x * (2 * NL) + t, nq2 = (a.nq + 1) & ~(int64_t)1;
        const int64_t b = r / nq2, q = r - b * nq2;
        const bool live = b < a.nb && q < a.nq;
        bin[t] = live ? b * a.in_bs + q : -1;
        bout[t] = b * a.out_bs + q * (a.zpitch > 0 ? a.zpitch : 1);
        bim[t] = (a.imag >> b) & 1u;
    }
    load_twiddles(tw, twg, L);
    pdl_wait(in);
    pdl_trigger();
    __syncthreads();
#pragma unroll 4
    for (int idx = tid; idx < 2 * NL * L; idx += nthreads) {
        const int rr = idx % (2 * NL), p = idx / (2 * NL);
        const double v = bin[rr] >= 0 ? in[bin[rr] + (int64_t)p * a.nq] : 0.0;
        reinterpret_cast<double *>(&buf[p * lstr + (rr >> 1)])[rr & 1] = v;
    }
    __syncthreads();
    const double2 *res = E::template run<double2, NL, false, false>(buf, a.p, tw, +1);
    auto put = [&](int rr, int k) {
        if (bin[rr] < 0) return;
        const double2 Z = res[k * lstr + (rr >> 1)], Zm = res[(k > 0 ? L - k : 0) * lstr + (rr >> 1)];
        double2 v = (rr & 1) == 0 ? make_double2(0.5 * (Z.x + Zm.x), 0.5 * (Z.y - Zm.y))
                                  : make_double2(0.5 * (Z.y + Zm.y), 0.5 * (Zm.x - Z.x));
        if (bim[rr]) v = make_double2(-v.y, v.x);
        if (a.fold >= 0) {  // fold, k < 2^11: 32-bit index arithmetic
            const double2 ph = __ldg(tw_rt + (int)(((unsigned)a.fold * (unsigned)k) % (unsigned)L));
            v = make_double2(-(v.x * ph.x - v.y * ph.y), -(v.x * ph.y + v.y * ph.x));
        }
        out[bout[rr] + (a.zpitch > 0 ? (int64_t)k : (int64_t)k * a.nq)] =
            mk<TO>((TO)(v.x * a.scale), (TO)(v.y * a.scale));
    };
    if (a.zpitch > 0) {
        for (int idx = tid; idx < 2 * NL * a.dimz; idx += nthreads) put(idx / a.dimz, idx % a.dimz);
    } else {
        for (int idx = tid; idx < 2 * NL * a.dimz; idx += nthreads) put(idx % (2 * NL), idx / (2 * NL));
    }
}

// ------------------------------------------------------------------------------------
// Launchers.  Shared memory above 48 KB needs the opt-in attribute, set per kernel.
// The attribute is set once per kernel, device and size (a lookup instead of a driver call
// on every launch of the many small launches of a batch).
// prefer_smem: the SM's storage is split in favour of shared memory even where one CTA needs little
// (the runtime engine's kernels, whose CTAs per SM are bounded by their line buffers).  A kernel started
// by launch_pdl otherwise comes up with the split of the kernel that is still running.
template <typename K> inline int set_smem(K kern, size_t bytes, bool prefer_smem = false) {
    if (bytes > 227 * 1024) return OSC_E_INVALID;
    // with the kernel's static arrays within the 48 KB that need no opt-in
    if (bytes <= 46 * 1024 && !prefer_smem) return OSC_OK;
    static std::mutex mu;
    static std::map<std::pair<const void *, int>, size_t> done;
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess) return OSC_E_CUDA;
    const auto key = std::make_pair(reinterpret_cast<const void *>(kern), dev);
    std::lock_guard<std::mutex> lk(mu);
    auto it = done.find(key);
    if (it != done.end() && it->second >= bytes) return OSC_OK;
    if (cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes) != cudaSuccess ||
        (prefer_smem && cudaFuncSetAttribute(kern, cudaFuncAttributePreferredSharedMemoryCarveout,
                                             cudaSharedmemCarveoutMaxShared) != cudaSuccess))
        return OSC_E_CUDA;
    done[key] = bytes;
    return OSC_OK;
}
inline int launch_ok() { return cudaGetLastError() == cudaSuccess ? OSC_OK : OSC_E_CUDA; }

// Lines per CTA of a runtime-plan kernel: the widest of nl (descending) whose nbuf line buffers of
// L (nl + 1) elements, twiddles and `extra` bytes a line leave several CTAs per SM, else the
// widest that fits (8 at most); 0 when none does.
inline int pick_nl_rt(int L, const int *nl, int nnl, size_t elem, int nbuf, size_t extra = 0) {
    auto need = [&](int n) { return (size_t)nbuf * L * (n + 1) * elem + L * elem + extra * n; };
    for (int i = 0; i < nnl; ++i)
        if (need(nl[i]) <= 56 * 1024) return nl[i];
    for (int i = 0; i < nnl; ++i)
        if (nl[i] <= 8 && need(nl[i]) <= 226 * 1024) return nl[i];
    return 0;
}
// Threads and dynamic shared memory of a kernel on engine E with NL lines.
template <class E> inline int eng_threads(const FFTPlan &p, int NL) {
    return E::kLen > 0 ? fft_threads(p.L, NL, E::kEPT) : mix_threads(p, NL);
}
template <class E, typename T> inline size_t eng_smem(int L, int NL) {
    return sizeof(cplx<T>) * ((size_t)L + (size_t)eng_bufs<E>() * L * (NL + 1));
}

// Calls f(std::integral_constant<int, NL>) for the engine's lines per CTA.  Static engines use a
// compile-time NL, the widest that fits; runtime plans MAXNL, 8 or MINNL (pick_nl_rt).
template <typename T, class E, int MAXNL, int MINNL, bool HALVES, class F>
inline int with_nl(int L, F &&f, int nl_div = 0, size_t extra = 0) {
    if constexpr (E::kLen > 0) {
        (void)L;
        (void)extra;
        constexpr int NL1 = nl_static(E::kLen, sizeof(T) == 4 ? 16 : 8, (int)sizeof(cplx<T>), 1, 100 * 1024, E::kEPT);
        // the autotuner's alternative tile: half the lines per CTA (more, smaller CTAs)
        constexpr int NLH = NL1 >= 4 && ((E::kLen * (NL1 / 2)) % E::kEPT) == 0 ? NL1 / 2 : NL1;
        if constexpr (HALVES && NLH != NL1)
            if (nl_div == 2) return f(std::integral_constant<int, NLH>{});
        return f(std::integral_constant<int, NL1>{});
    } else {
        constexpr int nls[3] = {MAXNL, 8, MINNL};
        switch (pick_nl_rt(L, nls, 3, sizeof(cplx<T>), eng_bufs<E>(), extra)) {
        case MAXNL: return f(std::integral_constant<int, MAXNL>{});
        case MINNL: return f(std::integral_constant<int, MINNL>{});
        case 0: return OSC_E_FFT_SIZE;
        default: return f(std::integral_constant<int, 8>{});
        }
    }
}

template <typename T, int NL, bool ROW, class E, int MODE>
inline int launch_lines_k(const cplx<T> *in, cplx<T> *out, const LineArgs &a, int nplanes, int ncomp, const cplx<T> *tw,
                          cudaStream_t st) {
    const int L = a.p.L;
    const int nt = eng_threads<E>(a.p, NL);
    const size_t sm = eng_smem<E, T>(L, NL);
    auto kern = k_lines<T, NL, ROW, E, MODE>;
    int rc = set_smem(kern, sm, E::kLen == 0);
    if (rc) return rc;
    // the flat tiling needs a column layout, at most one plane wrap per tile and int line indices
    const bool flat = !ROW && a.flat_lines > 0 && a.ncols >= NL && (int64_t)a.ncols * nplanes < (1ll << 30);
    LineArgs af = a;
    af.flat_lines = flat ? a.ncols * nplanes : 0;
    dim3 grid(flat ? (unsigned)ceil_div(af.flat_lines, NL) : (unsigned)ceil_div(a.ncols, NL),
              flat ? 1u : (unsigned)nplanes, (unsigned)ncomp);
    launch_pdl(kern, dim3(grid), dim3(nt), sm, st, in, out, af, tw);
    return launch_ok();
}

template <typename T>
int launch_lines(const cplx<T> *in, cplx<T> *out, const LineArgs &a, int nplanes, int ncomp, bool row_mode,
                 const TwPair<cplx<T>> &tw, cudaStream_t st) {
    const int L = a.p.L;
    return dispatch_fft_len<T>(L, [&](auto eng) -> int {
        using E = decltype(eng);
        const cplx<T> *twe = tw.st;
        return with_nl<T, E, sizeof(T) == 4 ? 16 : 8, 2, true>(L, [&](auto nlc) -> int {
            constexpr int NL = decltype(nlc)::value;
            if constexpr (E::kLen * NL / E::kEPT % 32 == 0)  // whole warps (the widest tile always is)
                if (row_mode) return launch_lines_k<T, NL, true, E, 0>(in, out, a, nplanes, ncomp, twe, st);
            if constexpr (E::kLen > 0) {
                if (2 * a.in_len == L && a.out_len == L && a.out_lo == 0)
                    return launch_lines_k<T, NL, false, E, 1>(in, out, a, nplanes, ncomp, twe, st);
                if (a.in_len == L && 2 * a.out_len == L && a.out_lo == 0 && a.flip_mask == 0)
                    return launch_lines_k<T, NL, false, E, 2>(in, out, a, nplanes, ncomp, twe, st);
            }
            return launch_lines_k<T, NL, false, E, 0>(in, out, a, nplanes, ncomp, twe, st);
        }, row_mode ? 0 : a.nl_div);
    });
}

template <typename T, typename TIn>
int launch_r2c_rows(const TIn *in, cplx<T> *out, const R2CArgs &a, const TwPair<cplx<T>> &tw, cudaStream_t st) {
    const int L = a.p.L;
    // the FP32 x transform at L = 256 runs faster with 8 values per thread (the other FP32
    // passes at 256 do not); same radices as the 16-value engine, so the same twiddle table
    auto dispatch = [&](auto &&f) -> int {
        if constexpr (sizeof(T) == 4)
            if (L == 256) return f(FftStatic8<256, 8, 8, 4>{});
        return dispatch_fft_len<T>(L, f);
    };
    return dispatch([&](auto eng) -> int {
        using E = decltype(eng);
        const cplx<T> *twe = tw.st;
        return with_nl<T, E, 8, 2, true>(L, [&](auto nlc) -> int {
            constexpr int NL = decltype(nlc)::value;
            const int nt = eng_threads<E>(a.p, NL);
            const size_t sm = eng_smem<E, T>(L, NL);
            const unsigned nblk = (unsigned)ceil_div(a.nrows, 2 * NL);
            if (E::kLen > 0 && 2 * a.nin == L) {
                auto kern = k_r2c_rows<T, TIn, NL, E, true>;
                int rc = set_smem(kern, sm);
                if (rc) return rc;
                launch_pdl(kern, dim3(nblk), dim3(nt), sm, st, in, out, a, twe);
            } else {
                auto kern = k_r2c_rows<T, TIn, NL, E, false>;
                int rc = set_smem(kern, sm, E::kLen == 0);
                if (rc) return rc;
                launch_pdl(kern, dim3(nblk), dim3(nt), sm, st, in, out, a, twe);
            }
            return launch_ok();
        }, a.nl_div);
    });
}

template <typename T>
int launch_c2r_rows(const cplx<T> *in, const C2RArgs &a, const TwPair<cplx<T>> &tw, cudaStream_t st) {
    const int L = a.p.L;
    // FP32 x-pairs or FP64 nodes: the specialised kernel; other combinations: generic
    if (a.e8 && (a.e8_node != 0) == (sizeof(T) == 8)) {
        bool e8_only = a.e8 && a.ncomp <= 3 && a.flip_mask == 0 && 2 * a.nout == L &&
                       reinterpret_cast<uintptr_t>(a.e8) % 32 == 0;
        for (int c = 0; c < a.ncomp && e8_only; ++c) e8_only = a.ndest[c] == 0;
        if (e8_only) {
            const int rc = dispatch_fft_len<T>(L, [&](auto eng) -> int {
                using E = decltype(eng);
                if constexpr (E::kLen > 0) {
                    auto go = [&](auto nlcc) -> int {
                        constexpr int NLC = decltype(nlcc)::value;
                        constexpr int nt = E::kLen * 3 * NLC / E::kEPT;
                        const size_t sm = sizeof(cplx<T>) * ((size_t)E::kLen + (size_t)E::kLen * (3 * NLC + 1));
                        auto kern = k_c2r_e8<T, NLC, E>;
                        int r = set_smem(kern, sm);
                        if (r) return r;
                        launch_pdl(kern, dim3((unsigned)ceil_div(a.nrows, 2 * NLC)), dim3(nt), sm, st, in, a, tw.st);
                        return launch_ok();
                    };
                    constexpr int NLC = c2r_e8_nlc<T, E>();
                    // the autotuner's alternative tile: half the rows per CTA
                    constexpr int NLH = NLC >= 2 && (E::kLen * 3 * (NLC / 2)) % E::kEPT == 0 ? NLC / 2 : NLC;
                    if (a.nl_div == 2 && NLH != NLC) return go(std::integral_constant<int, NLH>{});
                    return go(std::integral_constant<int, NLC>{});
                }
                else {
                    auto go = [&](auto nlcc) -> int {
                        constexpr int NLC = decltype(nlcc)::value;
                        const size_t sm = eng_smem<E, T>(L, 3 * NLC);
                        auto kern = k_c2r_e8_rt<T, NLC>;
                        int r = set_smem(kern, sm, true);
                        if (r) return r;
                        launch_pdl(kern, dim3((unsigned)ceil_div(a.nrows, 2 * NLC)), dim3(mix_threads(a.p, 3 * NLC)), sm, st, in, a, tw.st);
                        return launch_ok();
                    };
                    if (eng_smem<E, T>(L, 12) <= 75 * 1024) return go(std::integral_constant<int, 4>{});
                    if (eng_smem<E, T>(L, 3) <= 200 * 1024) return go(std::integral_constant<int, 1>{});
                    return -1;  // too long for three lines at once: the generic kernel
                }
            });
            if (rc != -1) return rc;
        }
    }
    return dispatch_fft_len<T>(L, [&](auto eng) -> int {
        using E = decltype(eng);
        const cplx<T> *twe = tw.st;
        return with_nl<T, E, 8, 1, false>(L, [&](auto nlc) -> int {
            constexpr int NL = decltype(nlc)::value;
            const int nt = eng_threads<E>(a.p, NL);
            const size_t sm = eng_smem<E, T>(L, NL) +
                              (a.e8 ? sizeof(T) * 3 * 2 * NL * (size_t)a.nout : 0);
            const unsigned nblk = (unsigned)ceil_div(a.nrows, 2 * NL);
            if (E::kLen > 0 && 2 * a.nout == L && a.flip_mask == 0) {
                auto kern = k_c2r_rows<T, NL, E, true>;
                int rc = set_smem(kern, sm);
                if (rc) return rc;
                launch_pdl(kern, dim3(nblk), dim3(nt), sm, st, in, a, twe);
            } else {
                auto kern = k_c2r_rows<T, NL, E, false>;
                int rc = set_smem(kern, sm, E::kLen == 0);
                if (rc) return rc;
                launch_pdl(kern, dim3(nblk), dim3(nt), sm, st, in, a, twe);
            }
            return launch_ok();
        }, 0, a.e8 ? sizeof(T) * 3 * 2 * (size_t)a.nout : 0);
    });
}

template <typename T, int W, int MODE, int L, int... Rs>
inline int launch_zconv_warp_k(const cplx<T> *in, cplx<T> *out, const ZConvArgs &a, const TwPair<cplx<T>> &tw,
                               cudaStream_t st) {
    const size_t sm = zconv_warp_smem<T>(L, W, MODE, MODE == ZW_SUM ? a.nsum : a.nout, a.g[0].zpitch);
    auto kern = k_zconv_warp<T, W, MODE, L, Rs...>;
    int rc = set_smem(kern, sm);
    if (rc) return rc;
    // summed inputs: the members are the inputs of one output, read by every CTA
    const unsigned gy = MODE == ZW_SUM ? 1u : (unsigned)(a.nbatch > 0 ? a.nbatch : 1);
    const dim3 grid((unsigned)ceil_div(a.ncols, W), gy);
    launch_pdl(kern, dim3(grid), dim3(W * 32), sm, st, in, out, a, tw.wt, tw.rt);
    return launch_ok();
}
template <typename T, int MODE, int L, int... Rs>
inline int launch_zconv_warp(WarpFft<L, Rs...>, const cplx<T> *in, cplx<T> *out, const ZConvArgs &a,
                             const TwPair<cplx<T>> &tw, cudaStream_t st) {
    return launch_zconv_warp_k<T, zw_warps<T>(), MODE, L, Rs...>(in, out, a, tw, st);
}

// Staged Green columns need real spectra, even/odd in z, one common 16-byte column pitch
// (one column per output, or per input when the inputs are summed).
template <typename T> inline bool zconv_can_stage(const ZConvArgs &a) {
    const int zp = a.g[0].zpitch;
    if (zp <= 0 || (zp * sizeof(T)) % 16) return false;
    const int ns = a.nsum > 0 ? a.nsum : a.nout;
    for (int o = 0; o < ns; ++o) {
        const int gd = a.gdir[o];
        if (gd < 0 || a.gimg[o] >= 0) return false;
        const GSpecDev &g = a.g[gd];
        if (!g.real_valued || !g.sym_z || !g.zinner || g.zpitch != zp || g.dimz > zp) return false;
        if (reinterpret_cast<uintptr_t>(g.data) % 16) return false;
    }
    return zconv_warp_smem<T>(a.p.L, zw_warps<T>(), ZW_STAGED, ns, zp) <= 100 * 1024;
}

// The image z pass: every output has a staged-compatible direct spectrum and a herm_img
// image spectrum, each kind with one 16-byte column pitch; kz-innermost output.
template <typename T> inline bool zconv_img_can(const ZConvArgs &a) {
    if (a.nout < 1 || a.nsum > 0 || a.out_estride != 1 || a.g_bstride != 0) return false;
    const int zp = a.g[a.gdir[0] >= 0 ? a.gdir[0] : 0].zpitch, zpi = a.g[a.gimg[0] >= 0 ? a.gimg[0] : 0].zpitch;
    if ((zp * sizeof(T)) % 16 || (zpi * sizeof(cplx<T>)) % 16) return false;
    for (int o = 0; o < a.nout; ++o) {
        const int gd = a.gdir[o], gi = a.gimg[o];
        if (gd < 0 || gi < 0) return false;
        const GSpecDev &d = a.g[gd], &m = a.g[gi];
        if (!d.real_valued || !d.sym_z || !d.sym_y || !d.zinner || d.zpitch != zp || d.dimz > zp) return false;
        if (!m.herm_img || !m.sym_y || !m.zinner || m.zpitch != zpi || m.dimz != a.nz + 1 || m.dimz > zpi) return false;
        if (reinterpret_cast<uintptr_t>(d.data) % 16 || reinterpret_cast<uintptr_t>(m.data) % 16) return false;
    }
    return zconv_img_smem<T>(a.p.L, a.nout, zp, zpi) <= 200 * 1024;
}
// The same kernel without images (the staged free-space product, Green columns shared by
// the rows ky and Ny - ky): staged spectra, all even/odd in y, kz-innermost output; batched
// members (blockIdx.y) may carry their own spectra g_bstride elements apart.
template <typename T> inline bool zconv_pair_can(const ZConvArgs &a) {
    if (a.nout < 1 || a.nsum > 0 || a.out_estride != 1) return false;
    for (int o = 0; o < a.nout; ++o)
        if (a.gdir[o] < 0 || !a.g[a.gdir[o]].sym_y) return false;
    return zconv_img_smem<T>(a.p.L, a.nout, a.g[a.gdir[0]].zpitch, 0) <= 200 * 1024;
}
template <typename T, bool IMG, int L, int... Rs>
inline int launch_zconv_img(WarpFft<L, Rs...>, const cplx<T> *in, cplx<T> *out, const ZConvArgs &a,
                            const TwPair<cplx<T>> &tw, cudaStream_t st) {
    const size_t sm = zconv_img_smem<T>(L, a.nout, a.g[a.gdir[0]].zpitch, IMG ? a.g[a.gimg[0]].zpitch : 0);
    auto kern = k_zconv_img<T, IMG, L, Rs...>;
    int rc = set_smem(kern, sm);
    if (rc) return rc;
    const int nkp = (a.nxh + 1) / 2;
    const dim3 grid((unsigned)(nkp * (a.ny + 1)), (unsigned)(a.nbatch > 0 ? a.nbatch : 1));
    launch_pdl(kern, dim3(grid), dim3(ZI_WARPS * 32), sm, st, in, out, a, tw.wt);
    return launch_ok();
}

inline int launch_zconv_w512(const float2 *in, float2 *out, const ZConvArgs &a, const float2 *rt, cudaStream_t st) {
    constexpr int W = 4;
    const size_t sm = zconv_w512_smem<W>(a.nout, a.g[0].zpitch);
    auto kern = k_zconv_w512<W>;
    int rc = set_smem(kern, sm);
    if (rc) return rc;
    const dim3 grid((unsigned)ceil_div(a.ncols, W), (unsigned)(a.nbatch > 0 ? a.nbatch : 1));
    launch_pdl(kern, dim3(grid), dim3(W * 32), sm, st, in, out, a, rt);
    return launch_ok();
}

template <typename T>
int launch_zconv(const cplx<T> *in, cplx<T> *out, const ZConvArgs &a, const TwPair<cplx<T>> &tw,
                 cudaStream_t st) {
    const int L = a.p.L;
    // a column range of a z slab runs on the radix warp engine only
    const bool whole = a.col_base == 0 && (int64_t)a.ncols == (int64_t)a.nxh * a.Ny;
    const bool warp = zconv_warp_ok(L, a.nz, (int)sizeof(T)) && (a.ng < 1 || a.g[0].zinner);
    if (a.col_base != 0 && (!warp || a.nsum > 0)) return OSC_E_UNSUPPORTED;
    if (warp) {
        for (int i = 0; i < a.ng; ++i)
            if (!a.g[i].zinner) return OSC_E_INVALID;  // spectra stored for the other z pass
        bool img = false, herm = false;
        for (int o = 0; o < a.nout; ++o) {
            img |= a.gimg[o] >= 0;
            herm |= a.gimg[o] >= 0 && a.g[a.gimg[o]].herm_img;
        }
        if (tw.wt == tw.rt) return OSC_E_INVALID;
        if (herm) {  // image spectra stored for the image z pass: no other kernel reads them
            if (!whole || !zconv_img_ok(L, a.nz, (int)sizeof(T)) || !zconv_img_can<T>(a))
                return OSC_E_INVALID;
            return dispatch_warp_len(L, [&](auto eng) -> int {
                using E = decltype(eng);
                if constexpr (E::kLen > 0) {
                    constexpr int nb = E::kLen / E::kRad[0];
                    if constexpr (nb % 32 == 0 || nb < 32) return launch_zconv_img<T, true>(eng, in, out, a, tw, st);
                }
                return OSC_E_INVALID;
            });
        }
        const bool staged = !img && zconv_can_stage<T>(a);
        if (a.nsum > 0 && (img || !staged || a.nout != 1)) return OSC_E_UNSUPPORTED;
        if constexpr (sizeof(T) == 4) {
            if (L == 512 && staged && a.nsum == 0 && a.out_estride == 1 && a.engine == ZCONV_EXCHANGE && whole &&
                zconv_w512_smem<4>(a.nout, a.g[0].zpitch) <= 100 * 1024)
                return launch_zconv_w512(in, out, a, tw.rt, st);
        }
        // The staged product with Green columns shared by the rows ky and Ny - ky wherever it applies,
        // unless the caller asks for another engine: it reads half the spectra, and is never the
        // slower one.  Paired against one warp per column (us), FP32: 16^3 8.6 10.6, 64^3 18.9 24.4,
        // 64 x 64 x 96 27.1 31.1, 128^3 76.2 81.7, 192 x 192 x 64 113 148, 128 x 128 x 256 138.5 143.9
        // (one exchange 155); FP64: 32^3 10.6 16.9, 128^3 128 137, 96^3 72 97, 128 x 128 x 256 287 326.
        const bool pair = staged && a.engine == ZCONV_PAIRED && whole && zconv_img_ok(L, a.nz, (int)sizeof(T)) &&
                          zconv_pair_can<T>(a);
        return dispatch_warp_len(L, [&](auto eng) -> int {
            using E = decltype(eng);
            if constexpr (E::kLen > 0) {
                constexpr int nb = E::kLen / E::kRad[0];
                if constexpr (nb % 32 == 0 || nb < 32)
                    if (pair) return launch_zconv_img<T, false>(eng, in, out, a, tw, st);
                if (a.nsum > 0) return launch_zconv_warp<T, ZW_SUM>(eng, in, out, a, tw, st);
                if (img) return launch_zconv_warp<T, ZW_IMAGE>(eng, in, out, a, tw, st);
                if (staged) return launch_zconv_warp<T, ZW_STAGED>(eng, in, out, a, tw, st);
                return launch_zconv_warp<T, ZW_DIRECT>(eng, in, out, a, tw, st);
            }
            return OSC_E_INVALID;
        });
    }
    if (a.nsum > 0) return OSC_E_UNSUPPORTED;  // summed inputs: warp engine lengths only
    for (int i = 0; i < a.ng; ++i)
        if (a.g[i].zinner) return OSC_E_INVALID;
    auto go = [&](auto nlc) -> int {
        constexpr int NL = decltype(nlc)::value;
        const size_t sm = sizeof(cplx<T>) * ((size_t)L + (size_t)(a.p.nst > 2 ? 3 : 2) * L * (NL + 1));
        auto kern = k_zconv<T, NL>;
        int rc = set_smem(kern, sm, true);
        if (rc) return rc;
        const dim3 nblk((unsigned)ceil_div(a.ncols, NL), (unsigned)(a.nbatch > 0 ? a.nbatch : 1));
        launch_pdl(kern, dim3(nblk), dim3(mix_threads(a.p, NL)), sm, st, in, out, a, tw.st, tw.rt);
        return launch_ok();
    };
    const int nls[2] = {8, 1};
    switch (pick_nl_rt(L, nls, 2, sizeof(cplx<T>), a.p.nst > 2 ? 3 : 2)) {
    case 8: return go(std::integral_constant<int, 8>{});
    case 1: return go(std::integral_constant<int, 1>{});
    default: return OSC_E_FFT_SIZE;
    }
}

template <typename TC, typename TI, typename TO>
int launch_sym_lines(const TI *in, TO *out, const SymArgs &a, const TwPair<cplx<TC>> &tw, bool row_load,
                     bool k_fast_store, cudaStream_t st) {
    const int L = a.p.L;
    if (L != 2 * a.n) return OSC_E_INVALID;
    return dispatch_fft_len<TC>(L, [&](auto eng) -> int {
        using E = decltype(eng);
        const cplx<TC> *twe = tw.st;
        // static engines: up to 16 line pairs per CTA, so the short lines of small batch
        // groups still give CTAs of several warps
        auto with_sym_nl = [&](auto &&f) -> int {
            if constexpr (E::kLen > 0) {
                constexpr int NL1 = nl_static(E::kLen, 16, (int)sizeof(cplx<TC>), 1, 100 * 1024, E::kEPT);
                // the autotuner's alternative tiles: a half or a quarter of the line pairs per
                // CTA (more CTAs for grids whose line count fills barely more than one wave)
                constexpr int NL2 = NL1 >= 4 && (E::kLen * (NL1 / 2)) % E::kEPT == 0 ? NL1 / 2 : NL1;
                constexpr int NL4 = NL2 >= 4 && (E::kLen * (NL2 / 2)) % E::kEPT == 0 ? NL2 / 2 : NL2;
                if (a.nl_div == 4 && NL4 != NL1) return f(std::integral_constant<int, NL4>{});
                if (a.nl_div >= 2 && NL2 != NL1) return f(std::integral_constant<int, NL2>{});
                return f(std::integral_constant<int, NL1>{});
            } else {
                return with_nl<TC, E, 8, 2, false>(L, f);
            }
        };
        return with_sym_nl([&](auto nlc) -> int {
            constexpr int NL = decltype(nlc)::value;
            const int nt = eng_threads<E>(a.p, NL);
            const size_t sm = eng_smem<E, TC>(L, NL);
            const unsigned nblk = (unsigned)ceil_div(((a.npq + 1) & ~(int64_t)1) * a.nb, 2 * NL);
            auto go = [&](auto kern) -> int {
                int rc = set_smem(kern, sm, E::kLen == 0);
                if (rc) return rc;
                launch_pdl(kern, dim3(nblk), dim3(nt), sm, st, in, out, a, twe);
                return launch_ok();
            };
            if (row_load) return k_fast_store ? go(k_sym_lines<TC, TI, TO, NL, E, true, true>)
                                              : go(k_sym_lines<TC, TI, TO, NL, E, true, false>);
            return k_fast_store ? go(k_sym_lines<TC, TI, TO, NL, E, false, true>)
                                : go(k_sym_lines<TC, TI, TO, NL, E, false, false>);
        });
    });
}

template <typename TO>
int launch_green_zlines(const double *in, cplx<TO> *out, const ZLineArgs &a, const TwPair<cplx<double>> &tw,
                        cudaStream_t st) {
    const int L = a.p.L;
    return dispatch_fft_len<double>(L, [&](auto eng) -> int {
        using E = decltype(eng);
        return with_nl<double, E, 8, 2, false>(L, [&](auto nlc) -> int {
            constexpr int NL = decltype(nlc)::value;
            auto kern = k_green_zlines<TO, NL, E>;
            const size_t sm = eng_smem<E, double>(L, NL);
            int rc = set_smem(kern, sm, E::kLen == 0);
            if (rc) return rc;
            const unsigned nblk = (unsigned)ceil_div(((a.nq + 1) & ~(int64_t)1) * a.nb, 2 * NL);
            launch_pdl(kern, dim3(nblk), dim3(eng_threads<E>(a.p, NL)), sm, st, in, out, a, tw.st, tw.rt);
            return launch_ok();
        });
    });
}

}  // namespace osc
