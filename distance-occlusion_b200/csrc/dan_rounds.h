// dan_rounds.h -- how many rounds the Danielsson block iteration (k_dan_blocks.cu)
// can take, for the kernel's limit.  Plain C++, so that the CPU tests compile it.
#pragma once

namespace dolk {

// A phase of `nchain` slices of h rows, cut into nx blocks along x, is a serial
// chain of pieces: per slice every row going down and every row going up, per
// row a pass to the right and one to the left, per pass a piece per x block.  A
// round makes at least one more piece final: the block that owns the first
// piece that is not has only final inputs for it, and either runs on them or
// has already run on the same ones.  One more round finds that nothing
// changed.  (A limit per block, 4 * blocks + 8, held while rows were whole;
// with x blocks a side cell per row and pass is a piece of its own, and
// caller's deltas of a few dozen cells ran out of it: 65 x 8 x 2 in 67 of 1000
// random fields, that is, 4 blocks and 24 rounds.)  Rounds stay below 2^28: a block's
// state word holds the round above four bits.
inline int dan_max_rounds(long long nchain, long long h, long long nx)
{
    const long long cap = (1LL << 28) - 2;
    const long long rows = nchain * h;   // below 2^62: both are ints
    if (rows > cap / 4 || rows * 4 > cap / nx) return (int)cap;
    return (int)(rows * 4 * nx) + 2;
}

// Rounds after which the serial walk takes a caller's field over.  A field of
// seeds settles within about nc + nk + nx rounds (one seed in a corner: 72 of 73 on
// 1024 x 1024, 501 of 509 on 20 x 20 x 1000); seeds with offsets of part of a cell took
// up to 172 (of 81, 300 x 200 x 40) and, images, 100 (of 80, 2000 x 500).  Arbitrary
// components may take as many rounds as the chain is long: 256^3 of components up
// to 2000 4.9 s, 0.49 with this budget (the walk alone takes 0.3).
inline int dan_round_budget(int dim, long long nchain, long long h, long long nc, long long nk, long long nx)
{
    const long long spread = nc + nk + nx;
    const long long budget = dim == 3 ? 6 * spread + 64 : spread + spread / 2 + 32;
    const int most = dan_max_rounds(nchain, h, nx);
    return budget < most ? (int)budget : most;
}

}  // namespace dolk
