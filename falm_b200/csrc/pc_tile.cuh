// Tile geometry of the fused half iterations (pc_mv.cuh) and the number of z
// planes of their blocks.  Plain host C++, without CUDA.
#pragma once

namespace fb {

template <typename T>
struct PCTile {
    static constexpr int H = 4;                                   // halo: stages after the first
    static constexpr int NW = sizeof(T) == 4 ? 16 : 12, NT = 32 * NW;
    static constexpr int TX = 64, TY = 2 * NW, OX = TX - 2 * H, OY = TY - 2 * H;
    static constexpr int NS = sizeof(T) == 4 ? 4 : 3;             // planes of the operand ring
    // FP32: every stage with the operations of sor_point() and dot7p() in their order, so that an iterate has the bits of the
    // stand-alone stream kernels (an FP32 recursion with restarts is sensitive to a consistent operator: sharing stage 3's sum with
    // the product, as FP64 does, left the same error per application but 4 times the error after five restarts)
    static constexpr bool SEQ = sizeof(T) == 4;
    static constexpr bool CSM = sizeof(T) == 8;                   // the cells' diagonals and weights kept in shared memory (registers are full)
    static constexpr int XP = TX / 2 + 2, EPL = (TY + 2) * XP;    // a stage's plane: pairs and rows with a border
    static constexpr int KMAX = 96, ZPL = KMAX + 2 * H + 8;       // planes of a chunk; staged z coefficients
    template <int NF> static constexpr int smem() {
        return (NS * NF * 2 * NT * 2 + 8 * EPL + 4 * ZPL + 4 * NT + (CSM ? 8 * NT : 0)) * (int)sizeof(T);
    }
    static int tiles_x(int n) { return n <= TX ? 1 : (n - 2 * H + OX - 1) / OX; }
    static int tiles_y(int n) { return n <= TY ? 1 : (n - 2 * H + OY - 1) / OY; }
};

// z planes per CTA of a half iteration on nx x ny x nz cells: the chunk that
// minimises waves x (planes + the eight of the pipeline's fill + about six for the
// start and the reduction); one CTA is resident per SM.  0: even the longest chunk
// gives more blocks than the reduction workspace has slots (max_blocks), on wide
// shallow grids (FP64 8192 x 8192 x 4: 75264 tiles).
template <typename T>
int pc_chunk(int nx, int ny, int nz, int sm_count, int max_blocks) {
    using L = PCTile<T>;
    const long long tiles = (long long)L::tiles_x(nx) * L::tiles_y(ny);
    const int hi = nz < L::KMAX ? nz : L::KMAX, lo = nz < 2 ? nz : 2;
    int best = 0;
    long long best_t = -1;
    for (int kc = hi; kc >= lo; kc--) {
        const long long ctas = tiles * ((nz + kc - 1) / kc);
        if (ctas > max_blocks) break;
        const long long t = ((ctas + sm_count - 1) / sm_count) * (kc + 2 * L::H + 6);
        if (best_t < 0 || t < best_t) { best_t = t; best = kc; }
    }
    return best;
}

}  // namespace fb
