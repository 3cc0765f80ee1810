// zchunks.h — the automatic z chunk: planes of one work item of the
// z-marching kernels, for a model stepped on its own and for a model that is
// advanced together with others.  Host code without CUDA calls.
#pragma once

#include <algorithm>
#include <cstdint>

namespace sgfd {

inline int chunk_of(int nz, int64_t chunks) {   // planes of each of `chunks` equal chunks
    return (int)std::max<int64_t>(1, (nz + chunks - 1) / chunks);
}

// A model on its own, `tiles` tiles of nz planes on a GPU of `sms` SMs.  A
// chunk starts by filling the z queues and the first stages: two to three
// planes' time in a lone short wave (64^3, launches included), 0.3 planes' on
// a filled GPU (150^3: 196.6 us per step with 2-plane chunks, 182.1 with 4,
// 175.6 with 8).  Long chunks waste least of it; short ones fill the GPU
// when the grid has few tiles.  One wave is three CTAs on every SM (measured
// with 32 x 8 tiles, ms per step, FP32):
//   * every tile fits one wave with chunks of at most 14 planes: the shortest
//     such chunk (64^3: 2 planes 0.0226, 14 planes 0.0697; 80^3: 5 planes
//     0.0436, 14 planes 0.0711; 60 x 60 x 400: 13 planes 0.111, 8 0.122;
//     where one wave needs longer chunks several waves are faster: 120^3
//     16 planes 0.1261, 8 planes 0.1226);
//   * fewer than 16 waves of 16-plane chunks: about four waves, 8 to 16
//     planes (150^3: 8 planes 0.2161, 16 planes 0.2210; 300 x 200 x 100:
//     12 planes 0.3443, 8 planes 0.3480, 16 planes 0.3497; 200^3 flat from 8
//     to 16, 0.424 to 0.430);
//   * larger grids: 16 waves, at most 48 planes (24, 32 and 48 planes within
//     1 % on the 394^3 grid, 48 planes 2 % faster than 24 on 522^3).
// The 64 x 8 tiles (pair) run two CTAs on an SM, so their one wave is that
// (ms per step, FP32 then FP16: 90^3 4 planes 0.0997, 0.124, 6 planes 0.0815,
// 0.0991; 130^3 FP16 9 planes 0.276, 14 planes 0.243); the other lines count
// CTAs and stay.  With 16-bit storage (half) each tap of theirs is converted
// as it is read and a chunk's start-up is dearer: 16 planes where such chunks
// make two waves of a grid of at least 64 planes (180^3 8 planes 0.687, 16
// planes 0.650; 157 x 333 x 91 8 planes 0.612, evened out to 14 0.583; below
// two waves 140^3 8 planes 0.392, 15 0.453, and on flat grids 1000 x 300 x 30
// 8 planes 0.645, 10 0.697), evened out if the last would hold one or two.
inline int solo_chunk(int tiles, int nz, int sms, bool pair = false, bool half = false) {
    const int wave = 3 * sms;
    auto waves = [&](int w) { return chunk_of(nz, ((int64_t)w * wave + tiles - 1) / tiles); };
    const int per_tile = (pair ? 2 : 3) * sms / tiles;   // chunks of every tile that one wave holds
    const int single = per_tile > 0 ? chunk_of(nz, per_tile) : nz;
    const int n16 = (nz + 15) / 16;
    int zc;
    if (single <= 14) zc = single;
    else if (waves(16) >= 16) zc = std::min(48, waves(16));
    else if (pair && half && nz >= 64 && (int64_t)tiles * n16 >= 4 * sms)
        zc = (nz - 1) % 16 < 2 ? chunk_of(nz, n16) : 16;
    else zc = std::min(16, std::max(8, waves(4)));
    return std::max(1, std::min(zc, nz));
}

// One model of a batch whose graph replays advance all models side by side,
// `all` tiles of all models: the models fill the GPU together, so chunks
// shorter than about 2.5 waves of all their work items need only pay more
// start-ups.  Never shorter than the model's own chunk, and at most 16 planes
// unless that is longer.  wave: CTAs of the model's kernel that the GPU holds
// at once.  us per step with the solo chunk and with this one, FP32: 64 models
// of 36 to 44 cells an edge 263 and 175, 32 of 48 to 70 414 and 327, 12 of 64
// 175 and 153, 8 of 150 1201 and 1147 (2 of 64, 16 of 28: the solo chunk, 28.5
// and 22.7).
// pairs: the kernels take planes in pairs (16-bit storage, 32 x 8 tiles): even
// chunks, since an odd one's last plane costs as much as two, and at most 8
// planes; chunks of 6 planes and more stay (FP16: 64 models of 36 to 44 491 and
// 340, 12 of 64 250 and 227; 8 of 100 540 at 8 planes, 565 at 16; 3 of 90 149
// at 6, 154 at 8).
inline int graph_batch_chunk(int own, int64_t all, int nz, int wave, bool pairs) {
    if (pairs && own >= 6) return own;
    const int64_t items = ((int64_t)wave * 5 + 1) / 2;
    int zc = std::max(own, std::min(pairs ? 8 : 16, chunk_of(nz, (items + all - 1) / all)));
    if (pairs && zc != own) zc += zc & 1;
    return std::max(1, std::min(zc, nz));
}

// One model of a persistent batch: `ctas` CTAs take the work items of all
// models, so the line is at one item per CTA where chunks of at most 14 planes
// allow that, else at two and chunks of at most 16 planes (a model whose own
// chunk is longer keeps it).  Rounded so that the items do not exceed the line:
// 2 of 100 cells an edge at 8 chunks per tile, 1.95 items per CTA, 130 us per
// step, at 9 chunks 136.  us per step with the solo chunk and with this one: 64
// models of 36 to 44 cells an edge 408 and 226, 32 of 48 to 70 565 and 418, 12
// of 64 238 and 208, 2 of 64 45.7 and 40.4, 2 of 150 373 and 365.
inline int persistent_chunk(int own, int64_t all, int nz, int ctas) {
    if (own > 16) return own;
    const int64_t one = ctas / all, two = std::max<int64_t>(1, 2 * (int64_t)ctas / all);   // chunks of every tile
    const int single = one > 0 ? chunk_of(nz, one) : nz;
    const int zc = one > 0 && single <= 14 ? single : std::min(16, chunk_of(nz, two));
    return std::max(1, std::min(zc, nz));
}

}  // namespace sgfd
