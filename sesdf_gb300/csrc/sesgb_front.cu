// sesgb_front.cu -- the head of a small build in one block.
//
// A build of a few thousand atoms is bound by its chain of launches, not by the work in them: the reference-grid hash, the
// radix sort (two passes of histogram, scan and scatter), the gather and the neighbour grid (size, zero, count, scan,
// scatter) are 13 to 16 launches of 2 to 5 us each. With a molecule's sort keys, permutation and cell counters in the
// shared memory of one SM the same steps are phases of one kernel:
//
//   k_front         hash and largest radius, stable sort by hash (up to two passes of 6 bits: ranks of equal digits by
//                   warp match masks, a (digit, warp) matrix scanned by the block), gather, neighbour grid
//   k_front_probes  the grid of the singular probes: size, count, scan, scatter
//
// The cells of a grid are as many as shared memory holds (106,496 counters of 16 bits, 53,248 of 32 bits); a sparser
// molecule's grid is coarsened to fit, as the general path coarsens it to its capacity. Neighbour lists do not depend on
// the cells. Atoms of equal hash keep their order, and the order of a cell's items is free on both paths.
#include <algorithm>

#include "sesgb_device.cuh"
#include "sesgb_grid.cuh"
#include "sesgb_stages.cuh"

namespace sesgb
{
    namespace
    {
        constexpr uint32_t kThreads    = 1024;
        constexpr uint32_t kCells16    = 106496; // counters of 16 bits: an atom's rank in a cell stays below 2^14
        constexpr uint32_t kCells32    = 53248;
        constexpr uint32_t kFrontSmem  = kCells16 * 2u + 16u;
        constexpr int      kDigitBits  = 6;
        constexpr uint32_t kDigits     = 1u << kDigitBits;
        constexpr uint32_t kIndexBits  = 14; // of an atom's index; keys of kFrontBits above
        static_assert( kFrontAtoms <= 8u * kThreads && kFrontAtoms <= 1u << kIndexBits && kFrontBits <= 2 * kDigitBits, "packed sort items" );

        // block-wide exclusive sum of one value per thread (32 warps)
        __device__ __forceinline__ uint32_t block_sum( uint32_t v, uint32_t * warpSums )
        {
            uint32_t       wt;
            const uint32_t x = warp_exclusive_sum( v, wt );
            if ( lane_id() == 31u )
                warpSums[ threadIdx.x >> 5 ] = wt;
            __syncthreads();
            if ( threadIdx.x < 32u )
            {
                uint32_t t;
                warpSums[ threadIdx.x ] = warp_exclusive_sum( warpSums[ threadIdx.x ], t );
            }
            __syncthreads();
            return x + warpSums[ threadIdx.x >> 5 ];
        }

        // cells of edge cutoff / span over the reference grid's box, coarsened until at most cap
        __device__ FineGrid fit_grid( const GridRef & gr, float cutoff, int span, uint32_t cap )
        {
            const float ex = gr.cell.x * gr.size, ey = gr.cell.y * gr.size, ez = gr.cell.z * gr.size;
            FineGrid    g;
            g.origin = gr.origin;
            g.h      = cutoff / (float)span;
            g.span   = span;
            for ( int it = 0; it < 200; it++ )
            {
                g.dims = make_int3( max( 1, (int)ceilf( ex / g.h ) ), max( 1, (int)ceilf( ey / g.h ) ), max( 1, (int)ceilf( ez / g.h ) ) );
                if ( (uint64_t)g.dims.x * g.dims.y * g.dims.z <= cap )
                    break;
                g.h *= 1.1f;
            }
            g.cells = (uint32_t)( (uint64_t)g.dims.x * g.dims.y * g.dims.z );
            return g;
        }

        // I atoms per thread: warp w holds atoms 32 I w + 32 r + lane, r < I, so that the rounds of a warp keep their order.
        // One SM's issue rate bounds it: 14 us at 2,000 atoms, 29 at 6,007 (49 at 11,638, with 16 per thread), against 13 to 16
        // launches of 2 to 5 us each. Build of 2,000 atoms: 182.5 -> 158.7 us, of 6,007 with a 2.4 A probe: 434.9 -> 418.5 us.
        template<int I>
        __global__ void __launch_bounds__( kThreads ) k_front( Build b, int bits )
        {
            pdl_begin();
            extern __shared__ __align__( 16 ) uint32_t sh[];
            __shared__ uint32_t hist[ kDigits * 32 ];
            __shared__ uint32_t warpSums[ 32 ];
            __shared__ FineGrid grid;
            __shared__ int      sRmax;
            __shared__ uint32_t sOutside;
            const uint32_t tid = threadIdx.x, lane = lane_id(), warp = tid >> 5, n = b.n;
            const uint32_t base = warp * 32u * I + lane;
            if ( tid < sizeof( DeviceCounts ) / 4u )
                reinterpret_cast<uint32_t *>( b.counts )[ tid ] = 0u;
            if ( tid == 0u )
            {
                sRmax    = 0;
                sOutside = 0u;
            }
            __syncthreads();
            uint32_t item[ I ];
            float    rmax    = 0.f;
            uint32_t outside = 0u;
#pragma unroll
            for ( int r = 0; r < I; r++ )
            {
                const uint32_t i = base + 32u * r;
                item[ r ]        = 0xffffffffu;
                if ( i < n )
                {
                    const float4 a = b.atomsIn[ i ];
                    const int3   p = ref_grid_position( b.grid, a.x, a.y, a.z );
                    outside += p.x < 0 || p.y < 0 || p.z < 0 || p.x >= b.grid.size || p.y >= b.grid.size || p.z >= b.grid.size;
                    item[ r ] = ( ref_grid_hash( b.grid, p ) << kIndexBits ) | i;
                    rmax      = fmaxf( rmax, a.w );
                }
            }
            const int      rm = __reduce_max_sync( 0xffffffffu, __float_as_int( rmax ) );
            const uint32_t om = __reduce_add_sync( 0xffffffffu, outside );
            if ( lane == 0u )
            {
                atomicMax( &sRmax, rm );
                if ( om )
                    atomicAdd( &sOutside, om );
            }
            // stable sort by hash
            for ( int shift = 0; shift < bits; shift += kDigitBits )
            {
                hist[ tid ]              = 0u;
                hist[ tid + kThreads ] = 0u;
                __syncthreads();
                uint32_t rank[ I ];
#pragma unroll
                for ( int r = 0; r < I; r++ )
                {
                    const bool     valid = base + 32u * r < n;
                    const uint32_t digit = valid ? ( item[ r ] >> ( kIndexBits + shift ) ) & ( kDigits - 1u ) : kDigits;
                    const uint32_t peers = __match_any_sync( 0xffffffffu, digit );
                    const uint32_t slot  = digit * 32u + warp;
                    rank[ r ]            = valid ? hist[ slot ] + __popc( peers & lanemask_lt() ) : 0u;
                    __syncwarp();
                    if ( valid && ( peers & lanemask_lt() ) == 0u )
                        hist[ slot ] += __popc( peers );
                    __syncwarp();
                }
                __syncthreads();
                {
                    const uint32_t a = hist[ 2u * tid ], c = hist[ 2u * tid + 1u ];
                    const uint32_t e = block_sum( a + c, warpSums );
                    hist[ 2u * tid ]      = e;
                    hist[ 2u * tid + 1u ] = e + a;
                }
                __syncthreads();
#pragma unroll
                for ( int r = 0; r < I; r++ )
                    if ( base + 32u * r < n )
                        sh[ hist[ ( ( item[ r ] >> ( kIndexBits + shift ) ) & ( kDigits - 1u ) ) * 32u + warp ] + rank[ r ] ] = item[ r ];
                __syncthreads();
#pragma unroll
                for ( int r = 0; r < I; r++ )
                    if ( base + 32u * r < n )
                        item[ r ] = sh[ base + 32u * r ];
            }
            // neighbour grid
            __syncthreads();
            if ( tid == 0u )
            {
                const float rmaxAll   = __int_as_float( sRmax );
                grid                  = fit_grid( b.grid, 2.f * ( rmaxAll + b.rp ) + 0.01f, b.nbrSpan, min( b.capCells, kCells16 ) );
                b.fine[ 0 ]           = grid;
                b.counts->rmax        = rmaxAll;
                b.counts->outside     = sOutside;
                b.counts->fineCells   = grid.cells;
                b.counts->fineCell    = grid.h;
            }
            __syncthreads();
            const FineGrid g     = grid;
            const uint32_t words = g.cells / 2u + 1u; // of the counters 0 .. cells
            for ( uint32_t w = tid; w < words; w += kThreads )
                sh[ w ] = 0u;
            __syncthreads();
#pragma unroll
            for ( int r = 0; r < I; r++ )
            {
                const uint32_t s = base + 32u * r;
                if ( s < n )
                {
                    const uint32_t i = item[ r ] & ( ( 1u << kIndexBits ) - 1u );
                    const float4   a = b.atomsIn[ i ];
                    b.atoms[ s ]     = a;
                    b.perm[ s ]      = i;
                    b.keys[ s ]      = item[ r ] >> kIndexBits;
                    const uint32_t key = fine_key( g, fine_cell( g, a.x, a.y, a.z ) );
                    const uint32_t up  = ( key & 1u ) * 16u;
                    const uint32_t old = atomicAdd( sh + ( key >> 1 ), 1u << up );
                    item[ r ]          = ( key << kIndexBits ) | ( ( old >> up ) & 0xffffu );
                }
            }
            __syncthreads();
            {
                // an odd number of words per thread: no bank conflicts
                const uint32_t each = ( ( words + kThreads - 1u ) / kThreads ) | 1u;
                const uint32_t w0 = min( tid * each, words ), w1 = min( w0 + each, words );
                uint32_t       sum = 0u;
                for ( uint32_t w = w0; w < w1; w++ )
                    sum += ( sh[ w ] & 0xffffu ) + ( sh[ w ] >> 16 );
                uint32_t e = block_sum( sum, warpSums );
                for ( uint32_t w = w0; w < w1; w++ )
                {
                    const uint32_t c = sh[ w ], hi = e + ( c & 0xffffu );
                    sh[ w ] = e | ( hi << 16 );
                    e       = hi + ( c >> 16 );
                }
            }
            __syncthreads();
            for ( uint32_t c = tid; c <= g.cells; c += kThreads )
                b.cellStart[ c ] = ( sh[ c >> 1 ] >> ( ( c & 1u ) * 16u ) ) & 0xffffu;
#pragma unroll
            for ( int r = 0; r < I; r++ )
            {
                const uint32_t s = base + 32u * r;
                if ( s < n )
                {
                    const uint32_t key = item[ r ] >> kIndexBits;
                    const uint32_t idx = ( ( sh[ key >> 1 ] >> ( ( key & 1u ) * 16u ) ) & 0xffffu ) + ( item[ r ] & ( ( 1u << kIndexBits ) - 1u ) );
                    b.cellItems[ idx ] = s;
                    b.cellPos[ idx ]   = b.atoms[ s ];
                }
            }
        }

        __global__ void __launch_bounds__( kThreads ) k_front_probes( Build b, float cutoff )
        {
            pdl_begin();
            extern __shared__ __align__( 16 ) uint32_t sh[];
            __shared__ uint32_t warpSums[ 32 ];
            __shared__ FineGrid grid;
            const uint32_t tid = threadIdx.x, Q = min( b.counts->Q, b.capProbes );
            if ( tid == 0u )
            {
                grid                = fit_grid( b.grid, cutoff, 1, min( b.capCells, kCells32 ) );
                b.fine[ 0 ]         = grid;
                b.counts->fineCells = grid.cells;
                b.counts->fineCell  = grid.h;
            }
            __syncthreads();
            const FineGrid g = grid;
            for ( uint32_t w = tid; w <= g.cells; w += kThreads )
                sh[ w ] = 0u;
            __syncthreads();
            for ( uint32_t q = tid; q < Q; q += kThreads )
            {
                const float4 p = b.probePos[ q ];
                atomicAdd( sh + fine_key( g, fine_cell( g, p.x, p.y, p.z ) ), 1u );
            }
            __syncthreads();
            {
                const uint32_t words = g.cells + 1u, each = ( ( words + kThreads - 1u ) / kThreads ) | 1u;
                const uint32_t w0 = min( tid * each, words ), w1 = min( w0 + each, words );
                uint32_t       sum = 0u;
                for ( uint32_t w = w0; w < w1; w++ )
                    sum += sh[ w ];
                uint32_t e = block_sum( sum, warpSums );
                for ( uint32_t w = w0; w < w1; w++ )
                {
                    const uint32_t c = sh[ w ];
                    sh[ w ]          = e;
                    e += c;
                }
            }
            __syncthreads();
            for ( uint32_t c = tid; c <= g.cells; c += kThreads )
                b.cellStart[ c ] = sh[ c ];
            __syncthreads(); // the starts become cursors
            for ( uint32_t q = tid; q < Q; q += kThreads )
            {
                float4         p   = b.probePos[ q ];
                const uint32_t idx = atomicAdd( sh + fine_key( g, fine_cell( g, p.x, p.y, p.z ) ), 1u );
                // w: the sort key of the probe in its neighbours' lists
                p.w                = __uint_as_float( ref_grid_hash( b.grid, ref_grid_position( b.grid, p.x, p.y, p.z ) ) );
                b.cellItems[ idx ] = q;
                b.cellPos[ idx ]   = p;
            }
        }
    } // namespace

    bool small_front( const Build & b, int bits ) { return b.nMol <= 1 && b.n > 0 && b.n <= kFrontAtoms && bits <= kFrontBits; }

    void launch_front( const Build & b, int bits, cudaStream_t s )
    {
        if ( b.n <= 2u * kThreads )
            pdl_launch( k_front<2>, 1, kThreads, kFrontSmem, s, b, bits );
        else if ( b.n <= 4u * kThreads )
            pdl_launch( k_front<4>, 1, kThreads, kFrontSmem, s, b, bits );
        else
            pdl_launch( k_front<8>, 1, kThreads, kFrontSmem, s, b, bits );
        count_launches( 1 );
    }
    void launch_front_probes( const Build & b, float cutoff, cudaStream_t s )
    {
        pdl_launch( k_front_probes, 1, kThreads, kFrontSmem, s, b, cutoff );
        count_launches( 1 );
    }
    cudaError_t configure_front()
    {
        const void * kernels[] = { (const void *)k_front<2>, (const void *)k_front<4>, (const void *)k_front<8>,
                                   (const void *)k_front_probes };
        cudaError_t  e         = cudaSuccess;
        for ( const void * k : kernels )
            if ( e == cudaSuccess )
                e = cudaFuncSetAttribute( k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kFrontSmem );
        return e;
    }
} // namespace sesgb
