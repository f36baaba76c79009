// float32 instantiations of the runtime-length passes, and the choice of their radices.
#include <cmath>

#include "qpd_any.cuh"

namespace qpd {

// Fewest and cheapest stages: the factorisation into radices 2..17 of least summed cost, a stage costing about
// 8 instructions per value for its loads, stores, twiddle and addressing besides its butterfly.  An odd radix
// goes first: its outputs land an odd number of rows apart, on different banks.
bool any_stages(long long N, AnyStages* p) {
    // arithmetic per value of each butterfly (real operations, halved)
    static const double cost[kMaxBfly + 1] = {0, 0, 1, 3, 2, 4.5, 4, 6.5, 3.5, 6, 5.5, 9, 5, 8, 7.5, 7.5, 5.2, 11};
    AnyStages best;
    double least = 1e30;
    if (N < 1 || N > (1 << 20)) return false;
    int cur[kAnyStages];
    auto search = [&](auto&& self, int m, int from, int n, double c) -> void {
        if (c >= least) return;
        if (m == 1) {
            least = c;
            best.n = n;
            for (int i = 0; i < n; i++) best.R[i] = cur[i];
            return;
        }
        if (n == kAnyStages) return;
        for (int R = from; R >= 2; R--)
            if (m % R == 0) {
                cur[n] = R;
                self(self, m / R, R, n + 1, c + cost[R] + 8.0);
            }
    };
    search(search, (int)N, kMaxBfly, 0, 0.0);
    if (least > 1e29) return false;
    for (int i = 0; i < best.n; i++)
        if (best.R[i] % 2) {
            const int r = best.R[i];
            for (int j = i; j > 0; j--) best.R[j] = best.R[j - 1];
            best.R[0] = r;
            break;
        }
    best.N = (int)N;
    int Ns = 1;
    for (int i = 0; i < best.n; i++) {
        if (i) best.ntw += Ns * any_tw_row(best.R[i]);
        Ns *= best.R[i];
    }
    *p = best;
    return true;
}

void any_twiddles(const AnyStages& p, double2* tw) {
    int Ns = 1;
    for (int i = 0; i < p.n; i++) {
        const int R = p.R[i], row = any_tw_row(R);
        if (i)
            for (int k = 0; k < Ns; k++, tw += row)
                for (int r = 1; r <= row; r++) {
                    const double t = 2.0 * M_PI * (double)((long long)r * k) / ((double)Ns * R);
                    tw[r - 1] = r < R ? make_double2(std::cos(t), -std::sin(t)) : make_double2(1.0, 0.0);
                }
        Ns *= R;
    }
}

QPD_ANY_INSTANTIATE(float)
}  // namespace qpd
