// Answers of the library's dispatch rules (sc_lbm_b200/csrc/routes.h), one line
// per question on standard input.
#include <iostream>
#include <string>

#include "routes.h"

using namespace sclbm;

int main()
{
    std::string what;
    while (std::cin >> what) {
        size_t nx, ny;
        int p, sms, n, K, keep;
        if (what == "single") { // depth, and whether one step goes by tiles
            std::cin >> nx >> ny >> p >> sms;
            K = single_depth(nx, ny, (sclbm_precision)p, sms);
            std::cout << K << ' ' << single_pays(nx, ny, (sclbm_precision)p, K, 1) << '\n';
        } else if (what == "launches") {
            std::cin >> n >> K >> keep;
            std::cout << single_launches(n, K, keep != 0) << '\n';
        } else if (what == "flat") { // one node per thread rather than the register tile
            std::cin >> nx >> ny >> p >> keep;
            std::cout << flat_beats_tile(nx, ny, (sclbm_precision)p, keep != 0) << '\n';
        } else if (what == "rows") { // bands of this height in pairs
            std::cin >> p >> n >> K >> keep >> sms; // height, units, solid nodes
            std::cout << two_rows_pay((sclbm_precision)p, n, K, keep != 0, sms) << '\n';
        } else if (what == "warp") { // rows of strips, thousandths of their columns, SMs
            std::cin >> n >> K >> sms;
            std::cout << batch_two_beats_warp(n, K / 1000.0, sms) << '\n';
        } else if (what == "batch64") { // thousands of nodes, thousandths full, changes per 1000 nodes
            std::cin >> nx >> K >> n;
            std::cout << batch_flat_beats_ring(1000.0 * (double)nx, K / 1000.0, n / 1000.0) << '\n';
        } else {
            return 1;
        }
    }
    return 0;
}
