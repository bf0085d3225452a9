// fft_plan.cu -- radix plans of the transform lengths and the lengths each z pass covers.
#include <mutex>

#include "fft_kernels.cuh"

namespace osc {

namespace {
// Fewest radices whose product is m (in non-increasing order from `from`), then the smallest
// sum; best holds the best plan so far.
void plan_search(int m, int from, int *cur, int n, int sum, int *best, int &best_n, int &best_sum) {
    static const int rad[] = {16, 15, 12, 10, 9, 8, 6, 5, 4, 3, 2};
    if (m == 1) {
        if (n < best_n || (n == best_n && sum < best_sum)) {
            best_n = n;
            best_sum = sum;
            for (int i = 0; i < n; ++i) best[i] = cur[i];
        }
        return;
    }
    if (n >= best_n || n >= FFT_MAX_STAGES) return;
    for (int i = from; i < 11; ++i)
        if (m % rad[i] == 0) {
            cur[n] = rad[i];
            plan_search(m / rad[i], i, cur, n + 1, sum + rad[i], best, best_n, best_sum);
        }
}

FFTPlan search(int L) {
    FFTPlan p{};
    p.L = L;
    int cur[FFT_MAX_STAGES], n = FFT_MAX_STAGES + 1, sum = 0;
    plan_search(L, 0, cur, 0, 0, p.radix, n, sum);
    p.nst = n > FFT_MAX_STAGES ? 0 : n;
    for (int i = 0; i < p.nst; ++i)
        if (p.radix[i] % 2 == 0) {
            const int r = p.radix[i];
            p.radix[i] = p.radix[0];
            p.radix[0] = r;
            break;
        }
    return p;
}
}  // namespace

// The plan of a length depends on nothing else, so it is searched for once per process.
bool make_fft_plan(int L, FFTPlan &p) {
    if (L < 2 || L > FFT_MAX_LEN || (L % 2) != 0) return false;
    static std::once_flag once[FFT_MAX_LEN / 2 + 1];
    static FFTPlan plans[FFT_MAX_LEN / 2 + 1];
    std::call_once(once[L / 2], [L] { plans[L / 2] = search(L); });
    p = plans[L / 2];
    return p.nst > 0;
}

// The warp-per-column z pass (FP32 and FP64) for the lengths of the warp registry.
bool zconv_warp_ok(int L, int nz, int elem_bytes) {
    if ((elem_bytes != 4 && elem_bytes != 8) || 2 * nz != L) return false;
    return dispatch_warp_len(L, [](auto eng) -> int { return decltype(eng)::kLen > 0 ? 1 : 0; }) != 0;
}
bool zconv_zinner(int L, int nz, int elem_bytes, bool staged, int64_t columns) {
    return zconv_warp_ok(L, nz, elem_bytes) && (staged || L >= 96 || columns * elem_bytes <= 28 * 1024);
}
bool zconv_img_ok(int L, int nz, int elem_bytes) {
    if (!zconv_warp_ok(L, nz, elem_bytes)) return false;
    return dispatch_warp_len(L, [](auto eng) -> int {
               using E = decltype(eng);
               if constexpr (E::kLen > 0) {
                   constexpr int nb = E::kLen / E::kRad[0];
                   return nb % 32 == 0 || nb < 32 ? 1 : 0;
               }
               return 0;
           }) != 0;
}

}  // namespace osc
