// Tilings of the resident time loops, and those of the fourth-order stencils
// (resident8.cu has the eighth-order ones).
#include "resident_launch.cuh"

#include <algorithm>

namespace pyfwi {

template cudaError_t launch_fwd_resident_r<2>(FwdResArgs &a, cudaStream_t s);
template cudaError_t launch_adj_resident_r<2>(AdjResArgs &a, cudaStream_t s);
template cudaError_t launch_exact_resident_r<2>(AdjResArgs &a, cudaStream_t s);
template cudaError_t launch_rev_resident_r<2>(RevResArgs &a, cudaStream_t s);
extern template cudaError_t launch_rev_resident_r<4>(RevResArgs &a, cudaStream_t s);
extern template cudaError_t launch_fwd_resident_r<4>(FwdResArgs &a, cudaStream_t s);
extern template cudaError_t launch_adj_resident_r<4>(AdjResArgs &a, cudaStream_t s);
extern template cudaError_t launch_exact_resident_r<4>(AdjResArgs &a, cudaStream_t s);

namespace {

template <int R>
bool fits(int th, int nq, int rb, int ctas, const Lines &lines, ResLoop loop)
{
    using S = ResShape<R>;
    const int halo = (th + 4 * R) * (nq + 2 * S::HG) - th * nq, slots = res_slots(R, lines, th, nq);
    return th <= S::TH && nq <= S::NQ && (th / rb) * nq <= RES_THREADS && halo <= RES_HALO &&
           ctas * frame_count(th, nq, 2 * R, S::HG) <= RES_MAX_STRIPS && slots <= RES_MAX_SLOTS &&
           (loop == RES_FORWARD ||
            (loop == RES_EXACT ? exact_res_floats<R>(rb) : adj_res_floats<R>(rb)) + RES_SLOT_FLOATS * (size_t)slots <= RES_MAX_FLOATS);
}

static_assert(FWD_RES_FLOATS<2, 3> <= RES_MAX_FLOATS && FWD_RES_FLOATS<4, 3> <= RES_MAX_FLOATS && REV_RES_FLOATS<2, 3> <= RES_MAX_FLOATS &&
                  REV_RES_FLOATS<4, 3> <= RES_MAX_FLOATS,
              "the forward and reverse-time loops fit on an SM");

}  // namespace

// The tiling with the least modelled time of `shots` shots, in launches of c
// shots each on sms / c tiles.  Few rows per block make a step short but a
// launch small; many let one launch hold four times the cells.  The model of a
// step (us) is a fit to launches of both orders on grids of 140 x 140 to 560 x
// 1060 cells, each run with 1, 2 and 3 rows and 1 to 8 shots per launch; it is
// within 7 % of all that come near their grid's best.  Measured, forward / adjoint, per step of all shots: 8
// shots of 240 x 440 take 12.6 / 16.0 us with 1 row and two shots at a time,
// 13.6 / 17.1 with 2 rows and two, 10.8 / 17.0 with 3 rows and four; 8 of 140 x
// 140 in one launch 3.15 / 3.36 with 1 row, 4.31 / 7.47 with 3.
bool resident_tiles(const Grid &g, int R, const Lines &lines, int shots, int sms, ResLoop loop, ResTiles *out, double *us)
{
    struct Cost {
        double step, row, warp_row, ring, row3;  // fixed; per row; per warp of blocks and row; per warp of ring items; with 3 rows
    };
    constexpr Cost COST[2][2] = {{{1.463, 0.368, 0.013, 0.3, 0.737}, {1.335, 0.545, 0.060, 0.3, 2.460}},
                                 {{1.806, 0.258, 0.090, 0.3, 1.090}, {1.280, 0.721, 0.196, 0.3, 3.239}}};
    const Cost &k = COST[R > 2][loop != RES_FORWARD];
    const int ncg = (g.tnx + 3) / 4, hg = R <= 2 ? 1 : 2;
    double best = 0;
    if (g.tnz < 4 * R || g.tnx < 4 * R) return false;
    for (int rb = 1; rb <= (loop == RES_EXACT ? RES_EXACT_ROWS : 3); ++rb) {
        const int nbz = (g.tnz + rb - 1) / rb;
        for (int c = 1; c <= std::min(shots, sms); ++c) {
            const int most = sms / c, waves = (shots + c - 1) / c;
            if (c > 1 && (shots + c - 2) / (c - 1) == waves) continue;  // as many launches with fewer shots each
            for (int gz = 1; gz <= most && (gz == 1 || nbz / gz * rb >= 2 * R); ++gz) {
                const int gx = std::min(most / gz, std::max(1, ncg / hg));
                const int bz = (nbz + gz - 1) / gz, nq = (ncg + gx - 1) / gx, th = rb * bz;
                if (!(R == 2 ? fits<2>(th, nq, rb, c * gz * gx, lines, loop) : fits<4>(th, nq, rb, c * gz * gx, lines, loop)))
                    continue;
                const double ring = (double)(th + 2 * R) * (nq + 2) - (double)th * nq;
                const double cost = waves * (k.step + rb * (k.row + k.warp_row * bz * nq / 32.0) + k.ring * ring / 32.0 +
                                             (rb == 3 ? k.row3 : 0.0));
                if (best == 0 || cost < best) {
                    best = cost;
                    *out = {gz, gx, c, rb, nbz, ncg, bz, nq};
                }
            }
        }
    }
    if (us) *us = best;
    return best > 0;
}

// With many shots in a launch the step kernels run at the memory's rate, while a
// resident launch holds so few shots that its latency does not shrink with their
// number.  So the time of a step (us) is modelled for both: the resident loops' as
// resident_tiles does, the step kernels' as a fixed part and a rate in
// ps per cell and shot of whole tiles, which measured (64 shots unless said, us per step, step kernels / on chip):
//   sets, eighth order, forward and backward: 340 x 540 602 / 647, 300 x 500 475 / 587, 190 x 940 555 / 603; tiles
//     of 8 rows 240 x 440 430 / 313, 280 x 440 505 / 515.  Fourth order is always faster on chip: 340 x 540
//     436 / 313, 8 shots of 560 x 1060 181 / 121, and the model finds no grid where it would not be.
//   states, forward: fourth order 520 x 560 216 / 250, 340 x 540 148 / 147, eighth 340 x 540 255 / 300; tiles of
//     8 rows 240 x 440 102 / 82 and 206 / 152.  Backward with energy terms always on chip: 1204 / 594, 1655 / 569.
//   checkpoints, backward, fourth order: 520 x 560 735 / 1053, 16 shots of it 211 / 267, of 240 x 440
//     82 / 87, 4 of 560 x 1060 110 / 112, 1 of it 31 / 26, 10 of 240 x 440 53 / 48; eighth order 340 x 540
//     1487 / 1016.
void resident_pays(const Grid &g, int R, const Lines &lines, int shots, int rows, ResStore store, int chunk, bool energy,
                   bool *fwd, bool *bwd)
{
    const bool eighth = R > 2, large = rows > 8;
    const double cells = 1e-6 * g.tnz * g.tnx * shots,
                 tiles = 1e-6 * ((g.tnx + 31) / 32 * 32) * ((g.tnz + rows - 1) / rows * rows) * shots;
    ResTiles tl;
    double f = 0, b = 0;
    *fwd = *bwd = true;
    if (store == RES_OF_SETS && !eighth) return;
    *fwd = resident_tiles(g, R, lines, shots, RES_MAX_CTAS, RES_FORWARD, &tl, &f);
    *bwd = resident_tiles(g, R, lines, shots, RES_MAX_CTAS, RES_ADJOINT, &tl, &b);
    if (store == RES_OF_SETS) {  // both passes or neither
        *fwd = *bwd = *fwd && *bwd && f + b <= 8 + (large ? 46.5 : 62.5) * tiles;
        return;
    }
    // a loop that writes every state takes 6 % more than one with sets, one that writes few 10 % less
    *fwd = *fwd && f * (store == RES_OF_STATES ? 1.06 : 0.9) <= 4 + (eighth ? (large ? 20.8 : 30) : (large ? 11.6 : 14.8)) * tiles;
    if (store == RES_OF_STATES || energy) return;
    // reverse-time loop, forming the sets and the launches of a chunk, adjoint loop
    *bwd = *bwd && chunk > 0 &&
           f + b + (12 + 60.0 / chunk) * cells + 8.0 / chunk <= 9 + (eighth ? 120 : large ? 38 : 42) * tiles;
}

cudaError_t launch_fwd_resident(FwdResArgs &a, int R, cudaStream_t s)
{
    return R == 2 ? launch_fwd_resident_r<2>(a, s) : launch_fwd_resident_r<4>(a, s);
}

cudaError_t launch_rev_resident(RevResArgs &a, int R, cudaStream_t s)
{
    return R == 2 ? launch_rev_resident_r<2>(a, s) : launch_rev_resident_r<4>(a, s);
}

cudaError_t launch_exact_resident(AdjResArgs &a, int R, cudaStream_t s)
{
    return R == 2 ? launch_exact_resident_r<2>(a, s) : launch_exact_resident_r<4>(a, s);
}

cudaError_t launch_adj_resident(AdjResArgs &a, int R, cudaStream_t s)
{
    return R == 2 ? launch_adj_resident_r<2>(a, s) : launch_adj_resident_r<4>(a, s);
}

}  // namespace pyfwi
