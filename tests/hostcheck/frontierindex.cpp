// Test-only: the index of a deep search's frontier boards (host.cpp,
// BoardIndex), built for a position's frontier, and how far its boards lie
// from their first slots.
#include "../../perft_gpu_b200/csrc/host.cpp"

int pg::engine_batch_host(const u64 *, const uint8_t *, u32, u64 *) { return PERFT_ERR_NO_DEVICE; }

extern "C" int fi_probes(const uint64_t pos[6], uint32_t plies, uint64_t *boards, uint64_t *probes, uint64_t *longest)
{
    build_tables();
    const Board b = from_pos48(pos);
    Frontier f;
    f.build(b, legal_moves(b), plies);
    BoardIndex ix;
    std::vector<BoardKey> list;
    for (const BoardKey &k : f.boards) ix.id_of(list, k);
    if (list.size() != f.boards.size()) return -1;
    *boards = list.size();
    *probes = *longest = 0;
    const size_t mask = ix.slots.size() - 1;
    for (size_t i = 0; i < list.size(); i++) {
        const size_t at = ix.slot_of(list, list[i]);
        if (ix.slots[at] != i) return -2;
        const u64 n = ((at - ix.home(list[i])) & mask) + 1;
        *probes += n;
        *longest = std::max<u64>(*longest, n);
    }
    return 0;
}
