// mgp_stage.cuh -- how a persistent CTA walks over its tiles with one staging
// buffer that bulk copies fill (mgp_sweep.cu).  Plain control flow, so that it
// also compiles for the host with a barrier of its own.
#pragma once

#ifdef __CUDACC__
#define MGP_STAGE_FN __device__ __forceinline__
#else
#define MGP_STAGE_FN inline
#endif

namespace mgp {

// What became of a tile: stored with another one to follow, stored as the last,
// or given up because its copies did not arrive in time.
enum TileEnd { TILE_MORE, TILE_LAST, TILE_LOST };

// Every thread of the CTA makes the walk.  place(it) places the tile after this
// one, it alternating between the two places kept; wait(parity) waits, bounded,
// for the barrier phase of this tile's copies; tile(it) works on the tile, has
// the next one's copies issued, and ends the same in every thread.  After
// TILE_LOST nothing has been stored or issued and the tile's copies may still be
// in flight: drain(parity) waits (bounded) for that same phase before the CTA may
// leave, whichever tile it was.  (The opposite parity would not wait at all: the
// phase before it is complete.)
template <class Place, class Wait, class Tile, class Drain>
MGP_STAGE_FN void walk_tiles(Place place, Wait wait, Tile tile, Drain drain) {
    unsigned parity = 0;
#ifdef __CUDACC__
#pragma unroll 1
#endif
    for (int it = 0;; it ^= 1) {
        place(it);
        wait(parity);
        const TileEnd end = tile(it);
        if (end == TILE_LOST) drain(parity);
        if (end != TILE_MORE) return;
        parity ^= 1;
    }
}

}  // namespace mgp
