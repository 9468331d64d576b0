// sesgb_grid.cuh -- device helpers of the uniform neighbour grids.
#pragma once
#include "sesgb_internal.h"

namespace sesgb
{
    constexpr float kRel = 1.0f / 65536.0f; // relative half-width of the float32 error bands

    __device__ __forceinline__ int3 fine_cell( const FineGrid & g, float x, float y, float z )
    {
        int cx = (int)floorf( ( x - g.origin.x ) / g.h );
        int cy = (int)floorf( ( y - g.origin.y ) / g.h );
        int cz = (int)floorf( ( z - g.origin.z ) / g.h );
        cx     = cx < 0 ? 0 : ( cx >= g.dims.x ? g.dims.x - 1 : cx );
        cy     = cy < 0 ? 0 : ( cy >= g.dims.y ? g.dims.y - 1 : cy );
        cz     = cz < 0 ? 0 : ( cz >= g.dims.z ? g.dims.z - 1 : cz );
        return make_int3( cx, cy, cz );
    }
    __device__ __forceinline__ uint32_t fine_key( const FineGrid & g, int3 c )
    {
        return ( (uint32_t)c.z * (uint32_t)g.dims.y + (uint32_t)c.y ) * (uint32_t)g.dims.x + (uint32_t)c.x;
    }

    // The 25 rows of a span-2 stencil (cells of at least half the largest pair cutoff) around
    // atom position p, each cut to the x-range that can hold a neighbour of the atom: a
    // neighbour j lies within cut = R_i + R_max (+ margins) of p, so a row (y, z) whose cells
    // keep |dy|, |dz| >= ey, ez from p only needs x within sqrt(cut^2 - ey^2 - ez^2) of p.
    // Lane r < 25 computes row r; the rows' first items and exclusive prefixes go to shared
    // memory (start[25], pre[26] with pre[25] = total), and the total is returned. A cell two
    // beyond the atom's own along any axis starts at least 2h >= the largest pair cutoff away.
    __device__ __forceinline__ uint32_t stencil_rows_span2( const FineGrid & g, const uint32_t * cellStart, float4 p,
                                                            float cut, uint32_t * start, uint32_t * pre )
    {
        const uint32_t lane = lane_id();
        const int3     c    = fine_cell( g, p.x, p.y, p.z );
        uint32_t       st = 0, len = 0;
        if ( lane < 25u )
        {
            const int y = c.y + (int)( lane % 5u ) - 2;
            const int z = c.z + (int)( lane / 5u ) - 2;
            if ( y >= 0 && z >= 0 && y < g.dims.y && z < g.dims.z )
            {
                const float ylo = g.origin.y + (float)y * g.h, zlo = g.origin.z + (float)z * g.h;
                const float ey  = fmaxf( 0.f, fmaxf( ylo - p.y, p.y - ( ylo + g.h ) ) );
                const float ez  = fmaxf( 0.f, fmaxf( zlo - p.z, p.z - ( zlo + g.h ) ) );
                const float w2  = cut * cut - ey * ey - ez * ez;
                if ( w2 >= 0.f )
                {
                    const float w  = sqrtf( w2 ) + 0.01f;
                    int         x0 = (int)floorf( ( p.x - w - g.origin.x ) / g.h );
                    int         x1 = (int)floorf( ( p.x + w - g.origin.x ) / g.h );
                    x0             = max( x0, max( c.x - 2, 0 ) );
                    x1             = min( x1, min( c.x + 2, g.dims.x - 1 ) );
                    if ( x0 <= x1 )
                    {
                        st  = cellStart[ fine_key( g, make_int3( x0, y, z ) ) ];
                        len = cellStart[ fine_key( g, make_int3( x1, y, z ) ) + 1 ] - st;
                    }
                }
            }
        }
        uint32_t       total;
        const uint32_t ex = warp_exclusive_sum( len, total );
        if ( lane < 25u )
        {
            start[ lane ] = st;
            pre[ lane ]   = ex;
        }
        if ( lane == 0 )
            pre[ 25 ] = total;
        __syncwarp();
        return total;
    }
    // cell-item index of stencil item f (f < total): the last row whose prefix is <= f
    __device__ __forceinline__ uint32_t row_item_span2( const uint32_t * start, const uint32_t * pre, uint32_t f )
    {
        uint32_t r = 0;
#pragma unroll
        for ( uint32_t step = 16; step > 0; step >>= 1 )
            if ( r + step < 25u && pre[ r + step ] <= f )
                r += step;
        return start[ r ] + ( f - pre[ r ] );
    }
} // namespace sesgb
