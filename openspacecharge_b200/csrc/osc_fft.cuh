// osc_fft.cuh -- shared-memory Stockham FFT building blocks for sm_100a.
//
// A CTA transforms NL independent lines of length L that sit interleaved in shared memory:
// element e of line l is buf[e*lstr + l] with lstr = NL+1 (odd, so the 8/16-byte complex
// accesses of a warp spread over all banks).  Threads are mapped line-fastest, so the NL
// lanes that share a butterfly index touch consecutive words.  Each stage is an in-place
// mixed-radix Stockham step: every thread loads the R inputs of its butterflies (with the
// stage twiddle), the CTA synchronises, then every thread writes its R outputs to their
// autosorted positions.  The CTA has L*NL/FFT_EPT threads, so each thread owns FFT_EPT
// complex values per stage and all butterflies of a stage fit in registers.
//
// Two engines share these stages.  FftStatic<L, R...> fixes the radix sequence at compile
// time (every index is a shift or a constant multiply) and reads its twiddles from a
// per-stage table laid out [stage][k][r-1], so the lanes of a warp read consecutive words.
// Its first stage can skip the zero upper half of the input (forward transforms of the
// zero-padded doubled grid) and its last stage can skip the upper half of the output
// (inverse transforms whose physical window is the lower half).  FftRuntime follows a
// runtime radix plan for any other 2^a 3^b 5^c length: radices up to 16, so that the lengths
// up to 240 take two stages and most others three, the same per-stage twiddle table, and two
// line buffers that the stages alternate between (one barrier per stage).  A step on 45 x 36 x 50
// (lengths 90, 72, 100) took 339 us on radices 8, 4, 2, 3, 5 in place, and takes 211.
//
// Twiddles are computed on the host in FP64 and rounded once for FP32; sign -1 uses the
// conjugate.  Convention: X[k] = sum_j x[j] exp(sign*2*pi*i*j*k/L), unnormalised -- the sign
// convention of the reference's ccfft3d / Singleton sfft (code/fft_interface_mod.f90:96).
#pragma once

#include "osc_common.cuh"

namespace osc {

constexpr int FFT_MAX_STAGES = 12;
constexpr int FFT_EPT = 16;
constexpr int FFT_MAX_LEN = 2048;

struct FFTPlan {
    int L;
    int nst;
    int radix[FFT_MAX_STAGES];
};

// Host: radix plan for L = 2^a 3^b 5^c with the fewest stages, and of those the smallest sum
// of radices, an even radix first (its upper half of zero-padded input is zero).  Returns false
// for other lengths, odd lengths or L > FFT_MAX_LEN.
bool make_fft_plan(int L, FFTPlan &p);
// Threads of a CTA that transforms NL lines of length L.
inline int fft_threads(int L, int NL, int ept = FFT_EPT) { return (L * NL) / ept; }

template <typename V> __device__ __forceinline__ V tw_get(const V *tw, int m, int sign) {
    V w = tw[m];
    if (sign < 0) w.y = -w.y;
    return w;
}

// Small DFTs in registers: y[q] = sum_r v[r] exp(s*2*pi*i*r*q/R).
template <int R> struct Dft;

template <> struct Dft<2> {
    template <typename V> __device__ __forceinline__ static void run(V *v, int) {
        V a = v[0], b = v[1];
        v[0] = cadd(a, b);
        v[1] = csub(a, b);
    }
};

template <> struct Dft<4> {
    template <typename V> __device__ __forceinline__ static void run(V *v, int s) {
        V apc = cadd(v[0], v[2]), amc = csub(v[0], v[2]);
        V bpd = cadd(v[1], v[3]), bmd = csub(v[1], v[3]);
        V jb = cmul_si(bmd, s);
        v[0] = cadd(apc, bpd);
        v[1] = cadd(amc, jb);
        v[2] = csub(apc, bpd);
        v[3] = csub(amc, jb);
    }
};

template <> struct Dft<8> {
    template <typename V> __device__ __forceinline__ static void run(V *v, int s) {
        typedef decltype(v[0].x) T;
        const T h = (T)0.70710678118654752440084436210485;  // cos(pi/4)
        V a[4], b[4];
#pragma unroll
        for (int r = 0; r < 4; ++r) {
            a[r] = cadd(v[r], v[r + 4]);
            b[r] = csub(v[r], v[r + 4]);
        }
        // b_r *= w8^r, w8 = exp(s*i*pi/4)
        {
            V t = b[1];  // * h(1 + s i)
            V u;
            u.x = h * (t.x - (T)s * t.y);
            u.y = h * (t.y + (T)s * t.x);
            b[1] = u;
            b[2] = cmul_si(b[2], s);
            t = b[3];  // * h(-1 + s i)
            u.x = h * (-t.x - (T)s * t.y);
            u.y = h * (-t.y + (T)s * t.x);
            b[3] = u;
        }
        Dft<4>::run(a, s);
        Dft<4>::run(b, s);
#pragma unroll
        for (int q = 0; q < 4; ++q) {
            v[2 * q] = a[q];
            v[2 * q + 1] = b[q];
        }
    }
};

// Radix 16 by decimation in frequency: X[2q] is the 8-point DFT of a_r = v_r + v_{r+8},
// X[2q+1] the 8-point DFT of b_r = (v_r - v_{r+8}) w16^r, w16 = exp(s i pi/8).
template <> struct Dft<16> {
    template <typename V> __device__ __forceinline__ static void run(V *v, int s) {
        typedef decltype(v[0].x) T;
        const T c1 = (T)0.92387953251128675612818318939679;  // cos(pi/8)
        const T s1 = (T)0.38268343236508977172845998403040;  // sin(pi/8)
        const T h = (T)0.70710678118654752440084436210485;   // cos(pi/4)
        const T sg = (T)s;
        V a[8], b[8];
#pragma unroll
        for (int r = 0; r < 8; ++r) {
            a[r] = cadd(v[r], v[r + 8]);
            b[r] = csub(v[r], v[r + 8]);
        }
        // b_r *= cos(r pi/8) + s i sin(r pi/8)
        auto rot = [&](V &t, T cr, T sr) {
            const V u = t;
            t.x = cr * u.x - sg * sr * u.y;
            t.y = cr * u.y + sg * sr * u.x;
        };
        rot(b[1], c1, s1);
        rot(b[2], h, h);
        rot(b[3], s1, c1);
        b[4] = cmul_si(b[4], s);
        rot(b[5], -s1, c1);
        rot(b[6], -h, h);
        rot(b[7], -c1, s1);
        Dft<8>::run(a, s);
        Dft<8>::run(b, s);
#pragma unroll
        for (int q = 0; q < 8; ++q) {
            v[2 * q] = a[q];
            v[2 * q + 1] = b[q];
        }
    }
};

template <> struct Dft<3> {
    template <typename V> __device__ __forceinline__ static void run(V *v, int s) {
        typedef decltype(v[0].x) T;
        const T h = (T)0.86602540378443864676372317075294;  // sin(2 pi/3)
        V a = v[0], t = cadd(v[1], v[2]), d = csub(v[1], v[2]);
        V m;
        m.x = a.x - (T)0.5 * t.x;
        m.y = a.y - (T)0.5 * t.y;
        V jd;
        jd.x = -(T)s * h * d.y;
        jd.y = (T)s * h * d.x;
        v[0] = cadd(a, t);
        v[1] = cadd(m, jd);
        v[2] = csub(m, jd);
    }
};

template <> struct Dft<5> {
    template <typename V> __device__ __forceinline__ static void run(V *v, int s) {
        typedef decltype(v[0].x) T;
        const T c1 = (T)0.30901699437494742410229341718282;   // cos(2 pi/5)
        const T c2 = (T)-0.80901699437494742410229341718282;  // cos(4 pi/5)
        const T s1 = (T)0.95105651629515357211643933337938;   // sin(2 pi/5)
        const T s2 = (T)0.58778525229247312916870595463907;   // sin(4 pi/5)
        const V x0 = v[0];
        const V a1 = cadd(v[1], v[4]), b1 = csub(v[1], v[4]);
        const V a2 = cadd(v[2], v[3]), b2 = csub(v[2], v[3]);
        V p1, p2, q1, q2;
        p1.x = x0.x + c1 * a1.x + c2 * a2.x;
        p1.y = x0.y + c1 * a1.y + c2 * a2.y;
        p2.x = x0.x + c2 * a1.x + c1 * a2.x;
        p2.y = x0.y + c2 * a1.y + c1 * a2.y;
        q1.x = s1 * b1.x + s2 * b2.x;
        q1.y = s1 * b1.y + s2 * b2.y;
        q2.x = s2 * b1.x - s1 * b2.x;
        q2.y = s2 * b1.y - s1 * b2.y;
        const V j1 = cmul_si(q1, s), j2 = cmul_si(q2, s);
        v[0] = cadd(x0, cadd(a1, a2));
        v[1] = cadd(p1, j1);
        v[4] = csub(p1, j1);
        v[2] = cadd(p2, j2);
        v[3] = csub(p2, j2);
    }
};

// N = N1 N2 coprime by the prime-factor map, without twiddles: input N2 n1 + N1 n2, output the k
// with k = k1 mod N1 and k = k2 mod N2.
constexpr int crt_index(int n1, int n2, int k1, int k2) {
    int k = 0;
    while (k % n1 != k1 || k % n2 != k2) ++k;
    return k;
}
template <int N1, int N2> struct DftPfa {
    template <typename V> __device__ __forceinline__ static void run(V *v, int s) {
        V t[N1][N2];
#pragma unroll
        for (int n2 = 0; n2 < N2; ++n2) {
            V a[N1];
#pragma unroll
            for (int n1 = 0; n1 < N1; ++n1) a[n1] = v[(N2 * n1 + N1 * n2) % (N1 * N2)];
            Dft<N1>::run(a, s);
#pragma unroll
            for (int n1 = 0; n1 < N1; ++n1) t[n1][n2] = a[n1];
        }
#pragma unroll
        for (int k1 = 0; k1 < N1; ++k1) {
            Dft<N2>::run(t[k1], s);
#pragma unroll
            for (int k2 = 0; k2 < N2; ++k2) v[crt_index(N1, N2, k1, k2)] = t[k1][k2];
        }
    }
};
template <> struct Dft<6> : DftPfa<2, 3> {};
template <> struct Dft<10> : DftPfa<2, 5> {};
template <> struct Dft<12> : DftPfa<4, 3> {};
template <> struct Dft<15> : DftPfa<3, 5> {};

template <> struct Dft<9> {
    template <typename V> __device__ __forceinline__ static void run(V *v, int s) {
        typedef decltype(v[0].x) T;
        // cos and sin of 2 pi m / 9, m = 1, 2, 4
        const T c1 = (T)0.76604444311897803520239265055542, s1 = (T)0.64278760968653932632264340990726;
        const T c2 = (T)0.17364817766693034885171662676931, s2 = (T)0.98480775301220805936674302458952;
        const T c4 = (T)-0.93969262078590838405410927732473, s4 = (T)0.34202014332566873304409961468226;
        const T sg = (T)s;
        V t[3][3];
#pragma unroll
        for (int n = 0; n < 3; ++n) {
            t[n][0] = v[n];
            t[n][1] = v[n + 3];
            t[n][2] = v[n + 6];
            Dft<3>::run(t[n], s);
        }
        auto rot = [&](V &x, T cr, T sr) {
            const V u = x;
            x.x = cr * u.x - sg * sr * u.y;
            x.y = cr * u.y + sg * sr * u.x;
        };
        rot(t[1][1], c1, s1);
        rot(t[1][2], c2, s2);
        rot(t[2][1], c2, s2);
        rot(t[2][2], c4, s4);
#pragma unroll
        for (int k = 0; k < 3; ++k) {
            V a[3] = {t[0][k], t[1][k], t[2][k]};
            Dft<3>::run(a, s);
            v[k] = a[0];
            v[k + 3] = a[1];
            v[k + 6] = a[2];
        }
    }
};

// ---- runtime-plan engine ----------------------------------------------------------------
// One Stockham stage over NL interleaved lines from ld(e, line) to st(e, line, v), which must
// not overlap unless a butterfly's inputs are its outputs.  A thread takes butterfly after
// butterfly; with blockDim a multiple of NL its line is threadIdx.x % NL in all of them.
template <typename V, int R, int NL, bool FIRST, class LD, class ST>
__device__ __forceinline__ void mix_stage_r(int L, int Ns, const V *tw, int sign, const LD &ld, const ST &st) {
    const int nb = L / R, total = nb * NL;
    // j / Ns by multiplication: exact while j Ns < 2^20 (j < L / R <= 1024)
    const unsigned magic = FIRST ? 0u : ((1u << 20) + (unsigned)Ns - 1u) / (unsigned)Ns;
    for (int b = threadIdx.x; b < total; b += blockDim.x) {
        const int line = b % NL, j = b / NL;
        const int q = FIRST ? j : (int)(((unsigned)j * magic) >> 20), k = FIRST ? 0 : j - q * Ns;
        V v[R];
#pragma unroll
        for (int r = 0; r < R; ++r) v[r] = ld(j + r * nb, line);
        if (!FIRST) {
            const V *t = tw + (Ns - 1) + k * (R - 1) - 1;
#pragma unroll
            for (int r = 1; r < R; ++r) v[r] = cmul(v[r], tw_get(t, r, sign));
        }
        Dft<R>::run(v, sign);
        const int d = q * Ns * R + k;
#pragma unroll
        for (int r = 0; r < R; ++r) st(d + r * Ns, line, v[r]);
    }
}
template <typename V, int NL, bool FIRST, class LD, class ST>
__device__ __forceinline__ void mix_stage(int R, int L, int Ns, const V *tw, int sign, const LD &ld, const ST &st) {
    switch (R) {
    case 2: mix_stage_r<V, 2, NL, FIRST>(L, Ns, tw, sign, ld, st); break;
    case 3: mix_stage_r<V, 3, NL, FIRST>(L, Ns, tw, sign, ld, st); break;
    case 4: mix_stage_r<V, 4, NL, FIRST>(L, Ns, tw, sign, ld, st); break;
    case 5: mix_stage_r<V, 5, NL, FIRST>(L, Ns, tw, sign, ld, st); break;
    case 6: mix_stage_r<V, 6, NL, FIRST>(L, Ns, tw, sign, ld, st); break;
    case 8: mix_stage_r<V, 8, NL, FIRST>(L, Ns, tw, sign, ld, st); break;
    case 9: mix_stage_r<V, 9, NL, FIRST>(L, Ns, tw, sign, ld, st); break;
    case 10: mix_stage_r<V, 10, NL, FIRST>(L, Ns, tw, sign, ld, st); break;
    case 12: mix_stage_r<V, 12, NL, FIRST>(L, Ns, tw, sign, ld, st); break;
    case 15: mix_stage_r<V, 15, NL, FIRST>(L, Ns, tw, sign, ld, st); break;
    default: mix_stage_r<V, 16, NL, FIRST>(L, Ns, tw, sign, ld, st); break;
    }
}

// ---- compile-time engine ------------------------------------------------------------------
// MODE 0: full stage; 1: first stage whose upper input half is zero (not read);
// 2: last stage whose upper output half is not needed (not written).
template <typename V, int R, int NL, int L, int Ns, int MODE, int EPT>
__device__ __forceinline__ void stage_ct(V *buf, const V *tw, int sign) {
    constexpr int lstr = NL + 1;
    constexpr int MAXB = (EPT + R - 1) / R;
    constexpr int nb = L / R;
    constexpr int total = nb * NL;
    constexpr int nthreads = L * NL / EPT;
    constexpr int toff = Ns - 1;  // this stage's block of the per-stage twiddle table
    constexpr bool half_in = MODE == 1 && (R % 2 == 0);
    constexpr bool half_out = MODE == 2 && (R % 2 == 0);
    const int tid = threadIdx.x;
    V v[MAXB][R];
#pragma unroll
    for (int q = 0; q < MAXB; ++q) {
        const int b = tid + q * nthreads;
        if (total % nthreads == 0 || b < total) {
            const int line = b % NL, j = b / NL, k = j % Ns;
#pragma unroll
            for (int r = 0; r < R; ++r) {
                V x;
                if (half_in && r >= R / 2) {
                    x.x = 0;
                    x.y = 0;
                } else {
                    x = buf[(j + r * nb) * lstr + line];
                    if (r && Ns > 1) x = cmul(x, tw_get(tw, toff + k * (R - 1) + (r - 1), sign));
                }
                v[q][r] = x;
            }
            Dft<R>::run(v[q], sign);
        }
    }
    __syncthreads();
#pragma unroll
    for (int q = 0; q < MAXB; ++q) {
        const int b = tid + q * nthreads;
        if (total % nthreads == 0 || b < total) {
            const int line = b % NL, j = b / NL, k = j % Ns;
            const int idxD = (j / Ns) * Ns * R + k;
#pragma unroll
            for (int r = 0; r < R; ++r)
                if (!half_out || r < R / 2) buf[(idxD + r * Ns) * lstr + line] = v[q][r];
        }
    }
    __syncthreads();
}

template <typename V, int NL, int L, int Ns, bool HIN, bool HOUT, int EPT, int R, int... Rest>
__device__ __forceinline__ void fft_ct(V *buf, const V *tw, int sign) {
    constexpr bool last = sizeof...(Rest) == 0;
    constexpr int mode = (Ns == 1 && HIN) ? 1 : ((last && HOUT) ? 2 : 0);
    stage_ct<V, R, NL, L, Ns, mode, EPT>(buf, tw, sign);
    if constexpr (!last) fft_ct<V, NL, L, Ns * R, false, HOUT, EPT, Rest...>(buf, tw, sign);
}

// Stage with explicit input and output functors: ld(e, line) -> V and st(e, line, V).
// The first stage of a transform can read straight from global memory (or compute its
// input, e.g. a spectral product) and the last stage can write straight to global memory,
// which saves two shared-memory passes per transform.
template <typename V, int R, int NL, int L, int Ns, bool HALF_IN, bool HALF_OUT, int EPT, class LD, class ST>
__device__ __forceinline__ void stage_io(const LD &ld, const ST &st, const V *tw, int sign) {
    constexpr int MAXB = (EPT + R - 1) / R;
    constexpr int nb = L / R;
    constexpr int total = nb * NL;
    constexpr int nthreads = L * NL / EPT;
    constexpr int toff = Ns - 1;
    constexpr bool half_in = HALF_IN && (R % 2 == 0);
    constexpr bool half_out = HALF_OUT && (R % 2 == 0);
    const int tid = threadIdx.x;
    V v[MAXB][R];
#pragma unroll
    for (int q = 0; q < MAXB; ++q) {
        const int b = tid + q * nthreads;
        if (total % nthreads == 0 || b < total) {
            const int line = b % NL, j = b / NL, k = j % Ns;
#pragma unroll
            for (int r = 0; r < R; ++r) {
                V x;
                if (half_in && r >= R / 2) {
                    x.x = 0;
                    x.y = 0;
                } else {
                    x = ld(j + r * nb, line);
                    if (r && Ns > 1) x = cmul(x, tw_get(tw, toff + k * (R - 1) + (r - 1), sign));
                }
                v[q][r] = x;
            }
            Dft<R>::run(v[q], sign);
        }
    }
    __syncthreads();
#pragma unroll
    for (int q = 0; q < MAXB; ++q) {
        const int b = tid + q * nthreads;
        if (total % nthreads == 0 || b < total) {
            const int line = b % NL, j = b / NL, k = j % Ns;
            const int idxD = (j / Ns) * Ns * R + k;
#pragma unroll
            for (int r = 0; r < R; ++r)
                if (!half_out || r < R / 2) st(idxD + r * Ns, line, v[q][r]);
        }
    }
    __syncthreads();
}

template <int... Rs> struct Radices {};

template <typename V, int NL, int L, int Ns, bool HIN, bool HOUT, int EPT, int R, int... Rest, class LD, class ST>
__device__ __forceinline__ void fft_io_rec(Radices<R, Rest...>, V *buf, const V *tw, int sign, const LD &ld,
                                           const ST &st) {
    constexpr bool first = Ns == 1, last = sizeof...(Rest) == 0;
    constexpr int lstr = NL + 1;
    auto sld = [buf](int e, int l) -> V { return buf[e * lstr + l]; };
    auto sst = [buf](int e, int l, const V &x) { buf[e * lstr + l] = x; };
    if constexpr (first && last) stage_io<V, R, NL, L, Ns, HIN, HOUT, EPT>(ld, st, tw, sign);
    else if constexpr (first) stage_io<V, R, NL, L, Ns, HIN, false, EPT>(ld, sst, tw, sign);
    else if constexpr (last) stage_io<V, R, NL, L, Ns, false, HOUT, EPT>(sld, st, tw, sign);
    else stage_io<V, R, NL, L, Ns, false, false, EPT>(sld, sst, tw, sign);
    if constexpr (!last) fft_io_rec<V, NL, L, Ns * R, HIN, HOUT, EPT>(Radices<Rest...>{}, buf, tw, sign, ld, st);
}

// FFT engines.  FftRuntime CTAs are capped at 256 threads so the radix-16 stages keep their
// registers; FftStatic CTAs at 512.  HIN/HOUT only change the static engine.
//
// run_io(buf, plan, tw, sign, ld, st): transform with input ld(e, line) (asked only for
// e < L/2 when HIN) and output st(e, line, v) (called only for e < L/2 when HOUT; storers
// must themselves ignore indices outside their window).  buf is the working buffer; ld may
// read another shared buffer.  run(buf, ...): transform of the lines in buf, returns the buffer
// that holds the result.  FftRuntime's working buffer is two line buffers, the second after
// the first (one is enough for run_io with at most two stages).
struct FftRuntime {
    static constexpr int kLen = 0;
    static constexpr int kEPT = FFT_EPT;
    static constexpr int kMaxThreads = 256;
    static constexpr int kNst = 0;
    static constexpr int kRad[1] = {0};
    template <typename V, int NL, bool HIN, bool HOUT>
    __device__ __forceinline__ static V *run(V *buf, const FFTPlan &p, const V *tw, int sign) {
        constexpr int lstr = NL + 1;
        V *a = buf, *b = buf + p.L * lstr;
        int Ns = 1;
        for (int s = 0; s < p.nst; ++s) {
            auto ld = [a](int e, int l) -> V { return a[e * lstr + l]; };
            auto st = [b](int e, int l, const V &x) { b[e * lstr + l] = x; };
            if (s == 0) mix_stage<V, NL, true>(p.radix[s], p.L, Ns, tw, sign, ld, st);
            else mix_stage<V, NL, false>(p.radix[s], p.L, Ns, tw, sign, ld, st);
            __syncthreads();
            Ns *= p.radix[s];
            V *t = a;
            a = b;
            b = t;
        }
        return a;
    }
    template <typename V, int NL, bool HIN, bool HOUT, class LD, class ST>
    __device__ __forceinline__ static void run_io(V *buf, const FFTPlan &p, const V *tw, int sign, const LD &ld,
                                                  const ST &st) {
        constexpr int lstr = NL + 1;
        V *a = buf, *b = buf + p.L * lstr;
        {
            auto sst = [a](int e, int l, const V &x) { a[e * lstr + l] = x; };
            mix_stage<V, NL, true>(p.radix[0], p.L, 1, tw, sign, ld, sst);
        }
        __syncthreads();
        int Ns = p.radix[0];
        for (int s = 1; s + 1 < p.nst; ++s) {
            auto sld = [a](int e, int l) -> V { return a[e * lstr + l]; };
            auto sst = [b](int e, int l, const V &x) { b[e * lstr + l] = x; };
            mix_stage<V, NL, false>(p.radix[s], p.L, Ns, tw, sign, sld, sst);
            __syncthreads();
            Ns *= p.radix[s];
            V *t = a;
            a = b;
            b = t;
        }
        auto sld = [a](int e, int l) -> V { return a[e * lstr + l]; };
        if (p.nst > 1) {
            mix_stage<V, NL, false>(p.radix[p.nst - 1], p.L, Ns, tw, sign, sld, st);
        } else {
            for (int idx = threadIdx.x; idx < NL * p.L; idx += blockDim.x) st(idx / NL, idx % NL, sld(idx / NL, idx % NL));
        }
        __syncthreads();
    }
};
// Threads of a runtime-plan CTA for `lines` lines: about one butterfly each in the stage with the
// most, whole warps, at most 256.
inline int mix_threads(const FFTPlan &p, int lines) {
    int r = p.radix[0];
    for (int s = 1; s < p.nst; ++s) r = p.radix[s] < r ? p.radix[s] : r;
    const int n = (p.L / r * lines + 31) / 32 * 32;
    return n < 64 ? 64 : (n > FftRuntime::kMaxThreads ? FftRuntime::kMaxThreads : n);
}
// Static engine with EPT_ complex values per thread and stage (L*NL/EPT_ threads per CTA).
template <int EPT_, int L_, int... Rs> struct FftStaticT {
    static constexpr int kLen = L_;
    static constexpr int kEPT = EPT_;
    static constexpr int kMaxThreads = 512;
    static constexpr int kNst = sizeof...(Rs);
    static constexpr int kRad[sizeof...(Rs)] = {Rs...};
    template <typename V, int NL, bool HIN, bool HOUT>
    __device__ __forceinline__ static V *run(V *buf, const FFTPlan &, const V *tw, int sign) {
        fft_ct<V, NL, L_, 1, HIN, HOUT, EPT_, Rs...>(buf, tw, sign);
        return buf;
    }
    template <typename V, int NL, bool HIN, bool HOUT, class LD, class ST>
    __device__ __forceinline__ static void run_io(V *buf, const FFTPlan &, const V *tw, int sign, const LD &ld,
                                                  const ST &st) {
        fft_io_rec<V, NL, L_, 1, HIN, HOUT, EPT_>(Radices<Rs...>{}, buf, tw, sign, ld, st);
    }
};
// FP32 transforms: 16 values per thread.  FP64: 8 (half the registers of the same bytes),
// with radices of at most 8 so that every thread owns a butterfly in every stage.
template <int L_, int... Rs> using FftStatic = FftStaticT<FFT_EPT, L_, Rs...>;
template <int L_, int... Rs> using FftStatic8 = FftStaticT<8, L_, Rs...>;

// Lines per CTA for a static engine: the largest NL <= nl_max with a whole number of
// threads, at most 512 threads, and nbuf line buffers within budget bytes of shared memory.
constexpr int nl_static(int L, int nl_max, int elem_bytes, int nbuf, int budget = 100 * 1024, int ept = FFT_EPT) {
    int nl = nl_max;
    while (nl > 2 && ((L * nl) % ept != 0 || (L * nl) / ept > 512 ||
                      nbuf * L * (nl + 1) * elem_bytes + L * elem_bytes > budget))
        nl /= 2;
    return nl;
}

// Calls f(engine) with the static engine for L when there is one, else FftRuntime.  T is
// the real type of the transform: FP64 transforms use 8 values per thread and radices up to
// 8; FP32 transforms 8 values per thread up to L = 192 (the many short lines of batched
// small grids) and 16 from L = 256 (where the 8-value engines measured slower).
template <typename T, class F> inline int dispatch_fft_len(int L, F &&f) {
    if constexpr (sizeof(T) == 8) {
        switch (L) {
        case 32: return f(FftStatic8<32, 8, 4>{});
        case 64: return f(FftStatic8<64, 8, 8>{});
        case 96: return f(FftStatic8<96, 8, 4, 3>{});
        case 128: return f(FftStatic8<128, 8, 4, 4>{});
        case 192: return f(FftStatic8<192, 8, 8, 3>{});
        case 256: return f(FftStatic8<256, 8, 8, 4>{});
        case 384: return f(FftStatic8<384, 8, 8, 2, 3>{});
        case 512: return f(FftStatic8<512, 8, 8, 8>{});
        default: return f(FftRuntime{});
        }
    } else {
        switch (L) {
        case 32: return f(FftStatic8<32, 8, 4>{});
        case 64: return f(FftStatic8<64, 8, 8>{});
        case 96: return f(FftStatic8<96, 8, 4, 3>{});
        case 128: return f(FftStatic8<128, 8, 4, 4>{});
        case 192: return f(FftStatic8<192, 8, 8, 3>{});
        case 256: return f(FftStatic<256, 8, 8, 4>{});
        case 384: return f(FftStatic<384, 8, 8, 2, 3>{});
        case 512: return f(FftStatic<512, 8, 8, 8>{});
        default: return f(FftRuntime{});
        }
    }
}

// Radix sequences of the warp-per-column engine of the z pass (first radix == last radix,
// even); WarpNone for lengths without one.
template <int L_, int... Rs> struct WarpFft {
    static constexpr int kLen = L_;
    static constexpr int kNst = sizeof...(Rs);
    static constexpr int kRad[sizeof...(Rs)] = {Rs...};
};
struct WarpNone {
    static constexpr int kLen = 0;
    static constexpr int kNst = 0;
    static constexpr int kRad[1] = {0};
};
// 192 as 8 3 8: 55.7 us for the z pass of 96^3 in FP32 against 61.9 as 4 4 3 4 (FP64 97 against 113), and
// its first stage has whole rounds of butterflies, which pairing its rows needs.  96 as 4 6 4 is
// slower than as below (48^3: 23.0 against 18.9, FP64 29.1 against 26.2).
template <class F> inline int dispatch_warp_len(int L, F &&f) {
    switch (L) {
    case 32: return f(WarpFft<32, 4, 2, 4>{});
    case 64: return f(WarpFft<64, 4, 4, 4>{});
    case 96: return f(WarpFft<96, 4, 2, 3, 4>{});
    case 128: return f(WarpFft<128, 4, 8, 4>{});
    case 192: return f(WarpFft<192, 8, 3, 8>{});
    case 256: return f(WarpFft<256, 8, 4, 8>{});
    case 384: return f(WarpFft<384, 4, 8, 3, 4>{});
    case 512: return f(WarpFft<512, 8, 8, 8>{});
    default: return f(WarpNone{});
    }
}

// Twiddle tables of one length: rt[m] = exp(2 pi i m/L); st is the per-stage table
// ([stage][k][r-1], L-1 entries) of the static engine, or of the runtime plan when the length
// has no static engine; wt the same for the warp engine of the z pass (or rt).
template <typename V> struct TwPair {
    const V *rt;
    const V *st;
    const V *wt;
};

// Stage the twiddle table of length n into shared memory.
template <typename V> __device__ __forceinline__ void load_twiddles(V *tw_s, const V *tw_g, int n) {
    const int nthreads = blockDim.x * blockDim.y;
    const int tid = threadIdx.x + blockDim.x * threadIdx.y;
    for (int m = tid; m < n; m += nthreads) tw_s[m] = tw_g[m];
}

}  // namespace osc
