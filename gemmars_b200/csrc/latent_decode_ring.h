// How latent_decode_kernel (latent_attention_mma.cu) shares out an SM's shared memory, as plain C++: the kernel, its launcher
// and a host program ask the same function.
#pragma once
#include <cstddef>

namespace latent_ring {

constexpr int KT = 32;              // keys of a tile
constexpr int MAX_SEQS = 1024;      // sequences of a step
constexpr size_t ROOM = 227 * 1024;

constexpr int warps_of(int rank) { return rank <= 128 ? 1 : (rank <= 256 ? 2 : 4); }      // warps that share 16 rows

struct Ring {
  int teams, stages;                // teams of warps that take the tiles in turn; tiles in flight (0: the rows are too wide)
  int share;                        // floats that 16 rows of a team share: the scores' parts, the warps' maxima, the weights
  int floats;                       // all teams' shares, or, if more, the teams' results as they meet
  size_t stage_bytes, smem;
};

// A place in the ring belongs to one team: whoever waits for a tile has then had the tile before it in that place, so that
// a parity never stands for the phase before the last (copies may arrive out of their order).  So the stages are a
// multiple of the teams, two for each at least, and as many teams work as that leaves (wide rows, or many heads, make
// few stages): of rows of 256 + 64 four teams, of 256 + 96 two.
constexpr Ring ring(int rank, int rot, int groups) {
  const int split = warps_of(rank), boxes = (rank + rot + 63) / 64;
  Ring r{};
  r.stage_bytes = (size_t)boxes * KT * 128;
  r.share = split > 1 ? split * 16 * (KT + 8) + split * 16 + 16 * (KT + 8) / 2 : 0;
  for (int teams = split * groups == 1 ? 4 : 8 / (split * groups); teams > 0; teams /= 2) {
    const int meet = (teams - 1) * split * groups * (rank / split / 2 + 4) * 32, shares = teams * groups * r.share;
    const int floats = shares > meet ? shares : meet;
    const size_t rest = (size_t)floats * 4 + 512 + MAX_SEQS * 4 + 1024;
    const int fit = (int)((ROOM - rest) / r.stage_bytes), stages = (fit > 16 ? 16 : fit) / teams * teams;
    if (stages < 2 * teams) continue;
    r.teams = teams;
    r.stages = stages;
    r.floats = floats;
    r.smem = 1024 + (size_t)stages * r.stage_bytes + (size_t)floats * 4 + 2 * (size_t)stages * 8 + 16 + (size_t)(MAX_SEQS + 1) * 4;
    return r;
  }
  return r;
}

}  // namespace latent_ring
