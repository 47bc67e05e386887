// How the tensor-core GEMV on NF4 weights shares a matrix out over its CTAs (two slots an SM).  Host arithmetic only.
#pragma once

#include <stdint.h>

#include <algorithm>

namespace rewb {

struct Nf4Split {
  int slabs;   // f32 slabs that the launch leaves
  int span;    // 0: `slabs` CTAs along K for each tile of 128 features; otherwise equal shares of all 128 x 64 blocks, `span` to a CTA
};

// CTAs along K of one tile each
inline int nf4_tile_split(int sms, int64_t K, int64_t N) {
  const int64_t tiles = (N + 127) / 128, KB = K / 64;
  const int64_t ks = std::min(std::max<int64_t>(1, 2 * sms / tiles), std::max<int64_t>(1, KB / 4));
  return (int)std::max<int64_t>(1, std::min<int64_t>(ks, 16));
}

// ... or, where those leave a fifth of the slots empty, equal shares of all blocks: a CTA's share ends one tile and begins the next.
// 4096 x 28672 has 224 tiles for 296 slots: one CTA an SM works for 64 blocks while its neighbours' two work for 128.  Four rows
// 33.3 us a launch, 28.5 with shares of 49 blocks.  most: slabs that the caller has room for; shares that need more of them give way
// to whole tiles.
inline Nf4Split nf4_split(int sms, int64_t K, int64_t N, int64_t most) {
  const int64_t tiles = (N + 127) / 128, KB = K / 64, slots = 2 * sms, ks = nf4_tile_split(sms, K, N);
  const int64_t span = std::max<int64_t>(4, (tiles * KB + slots - 1) / slots), slabs = (KB + span - 1) / span + 1;
  if (span <= KB && slabs <= std::min<int64_t>(most, 16) && tiles * ks * 5 < slots * 4 && (tiles * KB + span - 1) / span > tiles * ks)
    return {(int)slabs, (int)span};
  return {(int)std::max<int64_t>(1, std::min(ks, most)), 0};
}

}  // namespace rewb
