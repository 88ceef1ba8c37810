// Test-only: the count-only ply's check of the moves it generates
// (movegen.cuh, moves_as_counted), compiled for the host.
#include <stdint.h>

#include "../../perft_gpu_b200/csrc/movegen.cuh"

namespace pg {
void build_tables();
}

using namespace pg;

namespace {
struct CountSink {
    u32 n;
    void room(int) {}
    void operator()(u32) { n++; }
};
}  // namespace

extern "C" {

int lc_init(void)
{
    build_tables();
    return 0;
}

// The check for pos, with `extra` moves too many generated.
int lc_agrees(const uint64_t pos[6], uint32_t counted, int extra)
{
    const Board b = from_pos48(pos);
    QuietCtx q;
    quiet_setup(flip_board(b), q);
    quiet_flip(q);
    CountSink s{0};
    u32 quiet = 0, replies = 0;
    gen_moves_quiet<SV_KOGGE>(b, q, s, quiet, replies);
    return moves_as_counted(counted, quiet + s.n + (u32)extra);
}
}
