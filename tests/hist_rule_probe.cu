// Host-only test driver: for each "E scales tau_max chunk" on stdin, whether the engine leaves its lag launches to
// the ring kernel (hist_leave_to_ring). Calls no CUDA API.
#include <iostream>

#include "lag_hist_host.hpp"

int main() {
    long long E;
    int scales, tau_max, chunk;
    while (std::cin >> E >> scales >> tau_max >> chunk) std::cout << ddm::hist_leave_to_ring(E, scales, tau_max, chunk) << "\n";
    return 0;
}
