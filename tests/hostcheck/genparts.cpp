// Test-only: generation in parts and with quiet moves counted as sets
// (movegen.cuh, gen_part and gen_moves_quiet) compiled for the host.
#include <stdint.h>

#include "../../perft_gpu_b200/csrc/movegen.cuh"

namespace pg {
void build_tables();
}

using namespace pg;

namespace {
struct ListSink {
    u32 *out;
    u32 n, reserved;
    void room(int k) { reserved += (u32)k; }
    void operator()(u32 m)
    {
        if (n < 256) out[n] = m;
        n++;
    }
};
}  // namespace

extern "C" {

int gp_init(void)
{
    build_tables();
    return 0;
}

// Children of pos made from its parts; the number of moves, -1 when it is not
// the position's move count, -2 when a part emitted more or fewer moves than
// it asked room for.
int gp_children(const uint64_t pos[6], uint64_t *out)
{
    const Board b = from_pos48(pos);
    MoveCtx c;
    const u32 n = count_moves_fused<SV_KOGGE>(b, -1, -1, 0, 0, &c);
    u32 moves[256];
    ListSink s{moves, 0, 0};
    for (int p = 0; p < GEN_PARTS; p++) {
        gen_part(b, c, p, s);
        if (s.n != s.reserved) return -2;
    }
    if (s.n != n || n > 256) return -1;
    for (u32 i = 0; i < n; i++) to_pos48(make_child(b, moves[i]), out + 6 * i);
    return (int)n;
}

// Replies to every move of pos, the quiet ones from the position alone
// (gen_moves_quiet) and the rest one by one; nQuiet: how many were quiet.
// -1 when the moves are not all accounted for.
int64_t gp_replies(const uint64_t pos[6], uint32_t *nQuiet)
{
    const Board b = from_pos48(pos);
    QuietCtx q;
    quiet_setup(flip_board(b), q);
    quiet_flip(q);
    u32 moves[256], replies = 0;
    ListSink s{moves, 0, 0};
    *nQuiet = 0;
    gen_moves_quiet<SV_KOGGE>(b, q, s, *nQuiet, replies);
    if (s.n != s.reserved || s.n + *nQuiet != count_moves<SV_KOGGE>(b)) return -1;
    int64_t total = replies;
    for (u32 i = 0; i < s.n; i++) total += count_moves<SV_KOGGE>(make_child(b, moves[i]));
    return total;
}
}
