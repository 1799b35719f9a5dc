// Which plan of corner blocks a frame gets from a buffer that refuses some sizes (no GPU needed): one line per answer.
#include <cstdio>
#include <cstdlib>
#include <vector>

#include "../megamol_gb300/csrc/ao_internal.h"

using namespace p2v;

// argv: the largest size that the buffer grants, the error it answers with above that
int main(int argc, char** argv) {
    if (argc != 3)
        return 2;
    const size_t limit = std::strtoull(argv[1], nullptr, 10);
    const cudaError_t refused = (cudaError_t) std::atoi(argv[2]);
    ConeParams cp{};
    cp.ncones = 8;
    cp.nsteps = 32;
    cp.nlevels = 3;
    for (int k = 0; k < cp.nsteps; ++k) {
        cp.t[k] = 0.01f + 0.02f * (float) k;
        cp.lod[k] = 2.0f * (float) k / 31.0f;
    }
    for (int l = 0; l < cp.nlevels; ++l)
        for (int a = 0; a < 3; ++a) {
            cp.lv[l].d[a] = 64 >> l;
            cp.lv[l].fd[a] = (float) (64 >> l);
        }
    std::vector<size_t> asked;
    auto room = [&](size_t bytes) {
        asked.push_back(bytes);
        return bytes <= limit ? cudaSuccess : refused;
    };
    ConeBlocks cb;
    const cudaError_t e = fit_cone_blocks(cp, true, 100000, room, cb);
    int blocked = 0;
    for (int l = 0; l < cp.nlevels; ++l)
        blocked += cb.lv[l].sxy != 0u;
    std::printf("{\"error\": %d, \"nblocks\": %u, \"blocked\": %d, \"wlo\": %.9g, \"whi\": %.9g, \"asked\": [", (int) e,
                cb.nblocks, blocked, cb.wlo, cb.whi);
    for (size_t k = 0; k < asked.size(); ++k)
        std::printf("%s%zu", k ? ", " : "", asked[k]);
    std::printf("]}\n");
    return 0;
}
