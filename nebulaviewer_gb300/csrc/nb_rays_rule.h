// Where the ionizing rays may take the march without clamps (cast_ray1 in nb_rays.cu).  Plain C++: the
// host test compiles it alone.
#pragma once

// Along the part of a ray that lies a cell inside the box the corners of a sample are gathered unclamped, so
// the part's approximate ends and the sample's float position must together stay within the half cell to
// spare.  Both are off by a few roundings of the way from the star, which is nsteps dr at the most: the
// ends 7 x 2^-24 of it (difference, reciprocals, products), the position 3 x 2^-24, and 3 x 2^-24 of the box.
// 2^18 cells of way and 2^16 of box come to 0.17 of a cell.  Besides, cells, samples and the index of a
// corner are exact in the march's floats and 32-bit integers, the box has a part a cell from its faces, and
// the cell size keeps every product and quotient of positions normal.
inline bool nb_march_unclamped(int nx, int ny, int nz, int nsteps, float dr, float dx) {
    const int most = 1 << 16;
    return nx >= 4 && ny >= 4 && nz >= 4 && nx <= most && ny <= most && nz <= most &&
           (long long)nx * ny * nz < (1LL << 31) && nsteps <= (1 << 22) && dx > 1e-12f && dx < 1e12f &&
           (double)nsteps * dr <= 262144.0 * dx;
}
