// Host-only test driver: for each engine read from stdin, the CTA shapes its lag launches would get
// (hist_pick_shape) and how many of its launches build_hist_table refuses, for
// tests/test_lag_hist_shape.py. Calls no CUDA API.
//
// Input, one engine per line: compat batch R n0_step count_step ntau, then taus[ntau] ascending. Launches of
// every count_step-th frame count (and the largest, and the largest but one) at every n0_step-th start
// frame from the first to one turn of the ring past the longest lag; compat: every start block.
// Output: EB of the shape (0: none), launches tried, refused; the same of the pairs of batches.
#include <iostream>

#include "lag_hist_host.hpp"

using namespace ddm;

static HistInput launch(const std::vector<int> &taus, bool compat, int R, long long n0, int nreg, int nsub) {
    const int T = static_cast<int>(taus.size()), tau_max = taus.back(), c = nreg * nsub;
    auto slot = [&](long long f) { return f < 0 ? -1 : static_cast<int>(f % R); };
    HistInput in;
    in.nreg = nreg;
    in.nsub = nsub;
    for (int i = 0; i < T; i++) {
        in.ent_acc.push_back(compat ? i : T - 1 - i);
        in.ent_w.push_back(compat ? taus[i] : tau_max - taus[T - 1 - i]);
    }
    for (int p = 0; p < c + tau_max; p++)
        // compat: a second block that starts anywhere, and a few frames never written
        in.pos.push_back(compat ? (p % 97 == 96 ? -1 : slot(p < c + tau_max / 2 ? n0 + p : 7 * n0 + p)) : slot(n0 - tau_max + p));
    for (int j = 0; j < c; j++) in.reg.push_back(compat ? in.pos[j] : slot(n0 + j));
    return in;
}

int main() {
    int compat, batch, R, n0_step, count_step, ntau;
    while (std::cin >> compat >> batch >> R >> n0_step >> count_step >> ntau) {
        std::vector<int> taus(ntau);
        for (int &t : taus) std::cin >> t;
        for (int nsub = 1; nsub <= (compat ? 1 : 2); nsub++) {
            const HistShape s = hist_pick_shape(hist_steady(taus, batch, nsub, R, compat), compat);
            long long tried = 0, refused = 0;
            for (long long n0 = 0; s.EB && n0 <= taus.back() + R; n0 += n0_step)
                for (int c = nsub == 2 ? batch : 1; c <= batch; c++) {
                    if (c < batch - 1 && (c - 1) % count_step != 0) continue;
                    HistTable t;
                    tried++;
                    refused += !build_hist_table(launch(taus, compat, R, n0, c, nsub), s, &t).empty();
                }
            std::cout << s.EB << " " << tried << " " << refused << (nsub == 1 && !compat ? " " : "\n");
        }
    }
    return 0;
}
