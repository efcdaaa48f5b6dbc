// Prints the cells per tile (ablate_b200/csrc/fv_setup.hpp) and the face pass's CTAs per SM for every
// "owned cells, species, SMs" triple of the command line; compiled with g++ by tests/test_tile_rule.py.
#include <cstdio>
#include <cstdlib>

#include "fv_setup.hpp"

int main(int argc, char** argv) {
    for (int i = 1; i + 2 < argc; i += 3) {
        const int ns = std::atoi(argv[i + 1]);
        std::printf("%d %d\n", abl::tile_cell_count(std::atoll(argv[i]), ns, std::atoi(argv[i + 2])), abl::face_pass_ctas(ns));
    }
    return 0;
}
