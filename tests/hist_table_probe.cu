// Host-only test driver: runs the resident-history lag kernel's table builder
// (build_hist_table) on launch descriptions read from stdin and prints each table, so that
// tests/test_lag_hist.py can check them on the CPU. Calls no CUDA API.
//
// Input, one case per line: EB CW buffers x_buffers nreg nsub ntau npos, then reg[nreg * nsub], ent_acc[ntau],
// ent_w[ntau], pos[npos]. Output, one line per case: smem, frames, then the table's ints, or
// "ERR <message>".
#include <iostream>
#include <string>

#include "lag_hist_host.hpp"

int main() {
    int EB, CW, buffers, x_buffers, ntau, npos;
    ddm::HistInput in;
    while (std::cin >> EB >> CW >> buffers >> x_buffers >> in.nreg >> in.nsub >> ntau >> npos) {
        in.reg.resize(in.nreg * in.nsub);
        in.ent_acc.resize(ntau);
        in.ent_w.resize(ntau);
        in.pos.resize(npos);
        for (auto *v : {&in.reg, &in.ent_acc, &in.ent_w, &in.pos})
            for (int &x : *v) std::cin >> x;
        ddm::HistTable t;
        const ddm::HistShape shape{EB, CW, buffers, x_buffers != 0};
        const std::string err = ddm::build_hist_table(in, shape, &t);
        if (!err.empty()) {
            std::cout << "ERR " << err << "\n";
            continue;
        }
        std::cout << t.smem << " " << t.frames;
        for (int v : t.ints) std::cout << " " << v;
        std::cout << "\n";
    }
    return 0;
}
