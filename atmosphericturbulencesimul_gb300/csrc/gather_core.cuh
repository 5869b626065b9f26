// gather_core.cuh -- bicubic window sampling of a TMA-loaded screen tile.
// Host-compilable (__host__ __device__) so that the tile geometry can be
// checked by the CPU emulation against the oracle's per-pixel sampling.
#pragma once
#include "engine.cuh"

namespace atmwfs {

// Keys (a = -1/2) cubic convolution weights for taps at -1, 0, 1, 2.
AW_HD void keys_weights(float t, float w[4])
{
    const float t2 = t * t, t3 = t2 * t;
    w[0] = 0.5f * (-t3 + 2.0f * t2 - t);
    w[1] = 0.5f * (3.0f * t3 - 5.0f * t2 + 2.0f);
    w[2] = 0.5f * (-3.0f * t3 + 4.0f * t2 + t);
    w[3] = 0.5f * (t3 - t2);
}

struct TileGeom {
    int xs, ys, d;
    float fx, fy;
};

// Tile origin of layer position p for a CTA whose first row is y0, in the
// pass orientation (orient 1 exchanges the roles of the two screen axes).
AW_HD TileGeom tile_geom(LayerPos p, int orient, int y0)
{
    TileGeom g;
    const int ix = orient ? p.iy : p.ix;
    const int iy = orient ? p.ix : p.iy;
    g.fx = orient ? p.fy : p.fx;
    g.fy = orient ? p.fx : p.fy;
    g.xs = (ix + kPadX - 1) & ~3;
    g.d = ix + kPadX - 1 - g.xs;
    g.ys = iy + y0 + kPadY - 1;
    return g;
}

// Element (row r, column c) of a TMA tile made of NBOX boxes of kBoxW x TROWS.
template <int TROWS>
AW_HD int tile_index(int r, int c) { return ((c >> 5) * TROWS + r) * kBoxW + (c & (kBoxW - 1)); }

// Interpolate columns x .. x + 3 (x a multiple of 4) of one layer for the CTA's
// RR rows: per tile row four horizontal cubic sums from two or three aligned
// 16-byte reads, then the vertical cubic slides down the columns.  Reading
// four columns at once takes 3 shared reads per tile row where single columns
// took 16, which bounded the window kernels.  D = the tile's column offset
// g.d.  Calls emit(r, v0, v1, v2, v3) for every row.
template <int RR, int D, typename F>
AW_HD void gather_quad_d(const float* tile, const float wx[4], const float wy[4], int x, F emit)
{
    constexpr int TROWS = RR + 3;
    constexpr int NQ = D + 7 > 8 ? 3 : 2;
    float h[4][4];  // [tile row mod 4][column]
    AW_UNROLL
    for (int b = 0; b < TROWS; b++) {
        float t[4 * NQ];
        AW_UNROLL
        for (int q = 0; q < NQ; q++) {
            const float4 v = *reinterpret_cast<const float4*>(tile + tile_index<TROWS>(b, x + 4 * q));
            t[4 * q] = v.x;
            t[4 * q + 1] = v.y;
            t[4 * q + 2] = v.z;
            t[4 * q + 3] = v.w;
        }
        AW_UNROLL
        for (int k = 0; k < 4; k++)
            h[b & 3][k] = wx[0] * t[D + k] + wx[1] * t[D + k + 1] + wx[2] * t[D + k + 2] + wx[3] * t[D + k + 3];
        if (b < 3) continue;
        const int r = b - 3;
        float v[4];
        AW_UNROLL
        for (int k = 0; k < 4; k++)
            v[k] = wy[0] * h[r & 3][k] + wy[1] * h[(r + 1) & 3][k] + wy[2] * h[(r + 2) & 3][k] + wy[3] * h[b & 3][k];
        emit(r, v[0], v[1], v[2], v[3]);
    }
}

template <int RR, typename F>
AW_HD void gather_quad(const float* tile, const TileGeom& g, const float wx[4], const float wy[4], int x, F emit)
{
    switch (g.d) {  // the same in the whole CTA
        case 0: gather_quad_d<RR, 0>(tile, wx, wy, x, emit); break;
        case 1: gather_quad_d<RR, 1>(tile, wx, wy, x, emit); break;
        case 2: gather_quad_d<RR, 2>(tile, wx, wy, x, emit); break;
        default: gather_quad_d<RR, 3>(tile, wx, wy, x, emit); break;
    }
}

// Interpolate one layer for the CTA's RR rows; thread tid walks quads of
// columns.  Calls emit(r, x, value) for every pixel.
template <int N, int RR, int NT, typename F>
AW_HD void gather_tile(const float* tile, const TileGeom& g, float sc, int tid, F emit)
{
    float wx[4], wy[4];
    keys_weights(g.fx, wx);
    keys_weights(g.fy, wy);
    for (int x = 4 * tid; x < N; x += 4 * NT)
        gather_quad<RR>(tile, g, wx, wy, x, [&](int r, float v0, float v1, float v2, float v3) {
            emit(r, x, v0 * sc);
            emit(r, x + 1, v1 * sc);
            emit(r, x + 2, v2 * sc);
            emit(r, x + 3, v3 * sc);
        });
}

}  // namespace atmwfs
