// sesgb_cavities.cu -- components of the probe-accessible space on the GPU (no counterpart in the
// reference, whose exterior-only build keeps every probe, cavities included:
// sesdf/src/ssesdf/ssesdf.cu:133-187).
//
// E = probe-centre positions outside every SAS sphere (radius R = r + rp). Its component that touches
// the border of a box around the SAS is the exterior; every other one is a cavity. E is sampled at
// the centres of a voxel grid of spacing h (origin lo = min(c - R) - 2h, dims = ceil((hi - lo) / h) + 1,
// hi = max(c + R) + 2h, index v = (ix * ny + iy) * nz + iz) and its 6-connected components are labelled:
//   k_cav_bounds   min and max of c -+ R over the atoms (double, as ordered 64-bit keys)
//   k_cav_raster   one warp per atom, a lane per (ix, iy) column of its bounding box: the run of voxel
//                  centres inside the SAS sphere along z, set in an occupancy bit grid with one atomicOr
//                  per 32-voxel word. The voxel test is ((dx^2 + dy^2) + dz^2) < R^2 in double
//                  precision, dx = (lo_x + ix h) - c_x; the ends of the run are found in float32 relative to
//                  the atom, and the exact test decides the voxels within the float32 error of the sphere.
//   k_cav_runs     the nodes of the union-find are the runs of accessible voxels along z, each at its first
//                  voxel v: label[v] = v
//   k_cav_union    runs joined across y and x: lock-free union-find (one merge per pair of overlapping
//                  runs, where their overlap begins) in which a root is only ever linked under a
//                  smaller one (atomicMin), with path halving in every find, so the root of a component
//                  ends as its smallest voxel index
//   k_cav_flatten  label of a run = its root; a bit per voxel and a count per 32 voxels of the roots
//   k_cav_rank     components are numbered in the order of their first voxel in index order (the numbering of a
//                  raster-order labelling): the exclusive count of roots before it, left at the root as -2 - k
//   k_cav_resolve  every run's first voxel takes its root's code; border flag per component
//   k_cav_labels   label[v] = 1 + the number of its root; voxel count per component, the number of components
//                  that touch the border
// The passes over the grid up to k_cav_resolve take a word of 32 voxels per thread and find the few run or overlap starts
// in it with bit operations.
//   k_cav_probes   each probe: the label of the nearest accessible voxel centre among the 5^3 around its
//                  nearest voxel (first minimum in (ox, oy, oz) order), 0 when there is none
// Every loop that follows parent links is bounded (a chain only ever points to smaller indices); a
// kernel that meets its bound sets an error flag instead of looping on.
#include <cstring>

#include "sesgb_stages.cuh"

namespace sesgb
{
    namespace
    {
        constexpr uint32_t kCavMaxFind = 1u << 28; // parent links followed at most (a chain is shorter than V)

        inline uint32_t cav_blocks( uint64_t n, uint32_t threads, uint32_t cap = 152u * 16u )
        {
            const uint64_t b = ( n + threads - 1 ) / threads;
            return (uint32_t)( b < cap ? ( b ? b : 1 ) : cap );
        }

        __device__ __forceinline__ double sq( double x ) { return __dmul_rn( x, x ); }

        // a double as an unsigned key of the same order, and back
        __host__ __device__ __forceinline__ unsigned long long double_key( double v )
        {
            unsigned long long u;
            memcpy( &u, &v, 8 );
            return u >> 63 ? ~u : u | 1ull << 63;
        }

        // keys[0..2]: smallest c - R, keys[3..5]: largest c + R, per axis (memset to 0xff and 0 before)
        __global__ void __launch_bounds__( 256 ) k_cav_bounds( const float4 * atoms, uint32_t n, double rp, unsigned long long * keys )
        {
            unsigned long long m[ 6 ] = { ~0ull, ~0ull, ~0ull, 0ull, 0ull, 0ull };
            for ( uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x )
            {
                const float4 a = atoms[ i ];
                const double R = __dadd_rn( (double)a.w, rp );
                const double c[ 3 ] = { (double)a.x, (double)a.y, (double)a.z };
                for ( int k = 0; k < 3; k++ )
                {
                    m[ k ]     = min( m[ k ], double_key( __dsub_rn( c[ k ], R ) ) );
                    m[ 3 + k ] = max( m[ 3 + k ], double_key( __dadd_rn( c[ k ], R ) ) );
                }
            }
            for ( int k = 0; k < 6; k++ )
                for ( int o = 16; o > 0; o >>= 1 )
                {
                    const unsigned long long v = __shfl_xor_sync( 0xffffffffu, m[ k ], o );
                    m[ k ]                     = k < 3 ? min( m[ k ], v ) : max( m[ k ], v );
                }
            if ( ( threadIdx.x & 31u ) < 6u )
            {
                const int          k = (int)( threadIdx.x & 31u );
                unsigned long long v = m[ 0 ];
                for ( int q = 1; q < 6; q++ )
                    v = k == q ? m[ q ] : v;
                if ( k < 3 )
                    atomicMin( keys + k, v );
                else
                    atomicMax( keys + k, v );
            }
        }

        // voxel centre (index i) inside the sphere: the exact double test of the host labelling
        __device__ __forceinline__ bool cav_inside( const CavGrid & g, double a, int iz, double cz, double R2 )
        {
            const double dz = __dsub_rn( __dadd_rn( g.lo[ 2 ], __dmul_rn( (double)iz, g.h ) ), cz );
            return __dadd_rn( a, sq( dz ) ) < R2;
        }

        __device__ __forceinline__ void cav_set_run( uint32_t * bits, uint32_t v0, uint32_t v1 )
        {
            for ( uint32_t w = v0 >> 5; w <= v1 >> 5; w++ )
            {
                const uint32_t lo = w << 5;
                const uint32_t a  = v0 > lo ? v0 - lo : 0u;
                const uint32_t b  = min( v1 - lo, 31u );
                atomicOr( bits + w, ( 0xffffffffu << a ) & ( 0xffffffffu >> ( 31u - b ) ) );
            }
        }

        // ends of a column's run that float32 leaves open, by the exact test: first and last inside of [za, zb]
        __device__ __noinline__ int cav_end_d( const CavGrid & g, const float4 & at, int ix, int iy, int z0, int z1, int step )
        {
            const double R2 = sq( __dadd_rn( (double)at.w, g.rp ) );
            const double dx = __dsub_rn( __dadd_rn( g.lo[ 0 ], __dmul_rn( (double)ix, g.h ) ), (double)at.x );
            const double dy = __dsub_rn( __dadd_rn( g.lo[ 1 ], __dmul_rn( (double)iy, g.h ) ), (double)at.y );
            const double a  = __dadd_rn( sq( dx ), sq( dy ) );
            for ( int iz = z0; iz != z1 + step; iz += step )
                if ( cav_inside( g, a, iz, (double)at.z, R2 ) )
                    return iz;
            return -1;
        }

        constexpr uint32_t kRasterAtoms = 32; // atoms of a block of k_cav_raster, probes of one of k_cav_probes

        // A block takes 32 atoms: a thread per atom and axis finds the box of voxels in double precision, then a warp
        // takes an atom at a time. Bound by its atomics and the columns' float32 arithmetic. An FP64
        // instruction occupies its scheduler's pipe for 64 cycles whatever the lanes hold: with every column's run ends in
        // double precision, and every lane working out the box, 705 us for 20,000 atoms on a 0.5 A grid, 27 us now.
        __global__ void __launch_bounds__( 256 ) k_cav_raster( const float4 * atoms, uint32_t n, CavGrid g, double invh64, uint32_t * bits )
        {
            __shared__ int   sLo[ 3 ][ kRasterAtoms ], sHi[ 3 ][ kRasterAtoms ];
            __shared__ float sD0[ 3 ][ kRasterAtoms ], sCm[ 3 ][ kRasterAtoms ];
            const uint32_t lane = threadIdx.x & 31u, warp = threadIdx.x >> 5;
            const uint32_t first0 = blockIdx.x * kRasterAtoms;
            if ( warp < 3u && first0 + lane < n )
            {
                const float4 at = atoms[ first0 + lane ];
                const int    a  = (int)warp;
                const double c  = (double)( a == 0 ? at.x : a == 1 ? at.y : at.z );
                const double R  = __dadd_rn( (double)at.w, g.rp );
                const double t  = __dsub_rn( c, g.lo[ a ] );
                // voxels with |d| <= R along this axis; the margin is the error of the voxel coordinates
                const float  cm     = fmaxf( fabsf( (float)c ), fabsf( (float)g.lo[ a ] ) );
                const double margin = (double)( 1e-3f + 1e-14f * cm * (float)invh64 );
                const int    lo     = max( (int)ceil( ( t - R ) * invh64 - margin ), 0 );
                sLo[ a ][ lane ]    = lo;
                sHi[ a ][ lane ]    = (int)fmin( floor( ( t + R ) * invh64 + margin ), (double)g.dims[ a ] - 1.0 );
                // centre of voxel lo relative to the atom
                sD0[ a ][ lane ] = (float)__dsub_rn( __dadd_rn( g.lo[ a ], __dmul_rn( (double)lo, g.h ) ), c );
                sCm[ a ][ lane ] = cm;
            }
            __syncthreads();
            const float h = (float)g.h, invh = 1.f / h;
            for ( uint32_t k = warp; k < kRasterAtoms && first0 + k < n; k += blockDim.x >> 5 )
            {
                const float4 at = atoms[ first0 + k ];
                const int    lo[ 3 ] = { sLo[ 0 ][ k ], sLo[ 1 ][ k ], sLo[ 2 ][ k ] }, hi[ 3 ] = { sHi[ 0 ][ k ], sHi[ 1 ][ k ], sHi[ 2 ][ k ] };
                const float  d0[ 3 ] = { sD0[ 0 ][ k ], sD0[ 1 ][ k ], sD0[ 2 ][ k ] };
                const float  cm = fmaxf( sCm[ 0 ][ k ], fmaxf( sCm[ 1 ][ k ], sCm[ 2 ][ k ] ) );
                const float  R = at.w + (float)g.rp, R2 = R * R;
                // bound of the error of dx^2 + dy^2 + dz^2 - R^2 with |d| <= S: float32's (1.8e-6 S^2 by adding up the
                // roundings), and that of the voxel coordinates far from the origin. Voxels are 0.05 to 100 A and a
                // sphere spans at most 2^28 of them: S is at most 330 voxels.
                const float S  = R + 2.f * h;
                const float eb = 2.5e-6f * S * S + 1e-14f * S * cm;
                const int   ny = hi[ 1 ] - lo[ 1 ] + 1;
                const int   cols = max( hi[ 0 ] - lo[ 0 ] + 1, 0 ) * max( ny, 0 );
                const float invy = 1.f / (float)max( ny, 1 ); // (exact: fewer than 2^19 columns)
                for ( int col = (int)lane; col < cols; col += 32 )
                {
                    const int   cx = (int)( ( (float)col + 0.5f ) * invy ), cy = col - cx * ny;
                    const int   ix = lo[ 0 ] + cx, iy = lo[ 1 ] + cy;
                    const float dx = d0[ 0 ] + (float)cx * h, dy = d0[ 1 ] + (float)cy * h;
                    const float a = dx * dx + dy * dy, rem = R2 - a;
                    if ( rem < -eb )
                        continue;
                    // the run of centres with |dz| < w; x0, x1: its ends in voxels from lo, tol: their error
                    const float w   = sqrtf( fmaxf( rem, 0.f ) );
                    const float x0  = ( -w - d0[ 2 ] ) * invh, x1 = ( w - d0[ 2 ] ) * invh;
                    const float tol = 1e-6f * S * invh + eb * invh / w;
                    int         first = max( lo[ 2 ] + (int)ceilf( x0 ), lo[ 2 ] ), last = min( lo[ 2 ] + (int)floorf( x1 ), hi[ 2 ] );
                    if ( rem <= 4.f * eb || fabsf( x0 - rintf( x0 ) ) < tol || fabsf( x1 - rintf( x1 ) ) < tol )
                    {
                        const float we = sqrtf( fmaxf( rem + eb, 0.f ) );
                        const int   za = max( lo[ 2 ] + (int)ceilf( ( -we - d0[ 2 ] ) * invh - 1e-3f ), lo[ 2 ] );
                        const int   zb = min( lo[ 2 ] + (int)floorf( ( we - d0[ 2 ] ) * invh + 1e-3f ), hi[ 2 ] );
                        first          = za <= zb ? cav_end_d( g, at, ix, iy, za, zb, 1 ) : -1;
                        last           = first >= 0 ? cav_end_d( g, at, ix, iy, zb, first, -1 ) : -1;
                        if ( first < 0 )
                            continue;
                    }
                    if ( first > last )
                        continue;
                    const uint32_t row = ( (uint32_t)ix * g.dims[ 1 ] + (uint32_t)iy ) * g.dims[ 2 ];
                    cav_set_run( bits, row + (uint32_t)first, row + (uint32_t)last );
                }
            }
        }

        // (a grid has at most 2^28 voxels: 32-bit indices)
        __device__ __forceinline__ bool cav_free( const uint32_t * bits, uint32_t v ) { return !( ( bits[ v >> 5 ] >> ( v & 31u ) ) & 1u ); }

        // free voxels among the 32 from v on (v may end past the grid)
        __device__ __forceinline__ uint32_t cav_free32( const uint32_t * bits, uint32_t v, uint32_t V )
        {
            if ( v >= V )
                return 0u;
            const uint32_t w = v >> 5, last = ( V - 1u ) >> 5;
            const uint32_t b = __funnelshift_r( bits[ w ], w < last ? bits[ w + 1 ] : 0u, v & 31u );
            return ~b & ( V - v >= 32u ? 0xffffffffu : ( 1u << ( V - v ) ) - 1u );
        }

        // of the 32 voxels from v on: firsts, the first voxels of a row; mask: those with a next row in the same plane
        __device__ __forceinline__ void cav_rows32( const CavGrid & g, uint32_t v, uint32_t & firsts, uint32_t & mask )
        {
            const uint32_t nz = g.dims[ 2 ];
            uint32_t       col = v / nz, iy = col % g.dims[ 1 ], at = 0u, iz = v - col * nz;
            firsts = mask = 0u;
            while ( at < 32u )
            {
                if ( iz == 0u )
                    firsts |= 1u << at;
                const uint32_t n = min( nz - iz, 32u - at );
                if ( iy + 1u < g.dims[ 1 ] )
                    mask |= ( n == 32u ? 0xffffffffu : ( 1u << n ) - 1u ) << at;
                at += n;
                iz = 0u;
                iy = iy + 1u == g.dims[ 1 ] ? 0u : iy + 1u;
            }
        }

        __global__ void __launch_bounds__( 128 ) k_cav_runs( const uint32_t * bits, CavGrid g, uint32_t * runs, int32_t * L )
        {
            const uint32_t V = g.dims[ 2 ] * g.dims[ 1 ] * g.dims[ 0 ], words = ( V + 31u ) / 32u;
            for ( uint32_t w = blockIdx.x * blockDim.x + threadIdx.x; w < words; w += gridDim.x * blockDim.x )
            {
                const uint32_t v0 = 32u * w, f = cav_free32( bits, v0, V );
                uint32_t       m = 0u;
                if ( f )
                {
                    uint32_t firsts, mask;
                    cav_rows32( g, v0, firsts, mask );
                    const uint32_t before = ( f << 1 ) | ( w > 0u && cav_free( bits, v0 - 1u ) ? 1u : 0u );
                    m                     = f & ( firsts | ~before );
                }
                runs[ w ] = m;
                for ( ; m; m &= m - 1u )
                {
                    const uint32_t v = v0 + (uint32_t)__ffs( (int)m ) - 1u;
                    L[ v ]           = (int32_t)v;
                }
            }
        }

        // first voxel of the run of free voxel v: the last start up to v
        __device__ __forceinline__ int32_t cav_start( const uint32_t * runs, uint32_t v )
        {
            uint32_t w = v >> 5, x = runs[ w ] & ( 0xffffffffu >> ( 31u - ( v & 31u ) ) );
            while ( !x )
                x = runs[ --w ];
            return (int32_t)( 32u * w + 31u ) - __clz( (int)x );
        }

        // root of v, halving the path on the way (labels only decrease: every write keeps an ancestor)
        __device__ __forceinline__ int32_t cav_find( int32_t * L, int32_t v, uint32_t * err )
        {
            for ( uint32_t s = 0; s < kCavMaxFind; s++ )
            {
                const int32_t p = __ldcg( L + v );
                if ( p == v )
                    return v;
                const int32_t gp = __ldcg( L + p );
                if ( gp == p )
                    return p;
                atomicMin( L + v, gp );
                v = gp;
            }
            atomicOr( err, 1u );
            return v;
        }

        __device__ __forceinline__ void cav_merge( int32_t * L, int32_t a, int32_t b, uint32_t * err )
        {
            for ( uint32_t s = 0; s < kCavMaxFind; s++ )
            {
                a = cav_find( L, a, err );
                b = cav_find( L, b, err );
                if ( a == b )
                    return;
                if ( a > b )
                {
                    const int32_t t = a;
                    a               = b;
                    b               = t;
                }
                // link the larger root under the smaller one; done unless b stopped being a root meanwhile
                const int32_t old = atomicMin( L + b, a );
                if ( old == b )
                    return;
                b = old;
            }
            atomicOr( err, 2u );
        }

        // Bound by the latency of the finds. A thread per voxel took 73 us for 20,000 atoms on a 0.5 A grid, 33 us now
        __global__ void __launch_bounds__( 128 ) k_cav_union( const uint32_t * bits, const uint32_t * runs, CavGrid g, int32_t * L, uint32_t * err )
        {
            const uint32_t nz = g.dims[ 2 ], nyz = g.dims[ 1 ] * nz, V = nyz * g.dims[ 0 ], words = ( V + 31u ) / 32u;
            for ( uint32_t w = blockIdx.x * blockDim.x + threadIdx.x; w < words; w += gridDim.x * blockDim.x )
            {
                const uint32_t v0 = 32u * w, f = cav_free32( bits, v0, V );
                if ( !f )
                    continue;
                uint32_t firsts, mask;
                cav_rows32( g, v0, firsts, mask );
                for ( int axis = 0; axis < 2; axis++ )
                {
                    const uint32_t d = axis == 0 ? nz : nyz;
                    const uint32_t o = f & cav_free32( bits, v0 + d, V ) & ( axis == 0 ? mask : 0xffffffffu );
                    // a neighbouring run is joined once, where its overlap with v's run begins
                    uint32_t before = o << 1;
                    if ( ( o & 1u ) && !( firsts & 1u ) && cav_free( bits, v0 - 1u ) && cav_free( bits, v0 - 1u + d ) )
                        before |= 1u;
                    for ( uint32_t m = o & ( firsts | ~before ); m; m &= m - 1u )
                    {
                        const uint32_t v = v0 + (uint32_t)__ffs( (int)m ) - 1u;
                        cav_merge( L, cav_start( runs, v ), cav_start( runs, v + d ), err );
                    }
                }
            }
        }

        __global__ void __launch_bounds__( 128 ) k_cav_flatten( const uint32_t * runs, uint32_t V, int32_t * L, uint32_t * rootBits,
                                                                uint32_t * rootCount, uint32_t * err )
        {
            const uint32_t words = ( V + 31u ) / 32u;
            for ( uint32_t w = blockIdx.x * blockDim.x + threadIdx.x; w < words; w += gridDim.x * blockDim.x )
            {
                uint32_t roots = 0u;
                for ( uint32_t m = runs[ w ]; m; m &= m - 1u )
                {
                    const int32_t v = (int32_t)( 32u * w ) + __ffs( (int)m ) - 1;
                    const int32_t r = cav_find( L, v, err );
                    if ( r == v )
                        roots |= m & ( 0u - m );
                    else
                        __stcg( L + v, r );
                }
                rootBits[ w ]  = roots;
                rootCount[ w ] = (uint32_t)__popc( roots );
            }
        }

        // first[w]: roots before word w; first[words]: their number. Zeroes the components' records.
        __global__ void __launch_bounds__( 128 ) k_cav_rank( uint32_t V, int32_t * L, const uint32_t * rootBits, const uint32_t * first,
                                                             uint32_t rootCap, uint32_t * voxels, uint8_t * border, uint32_t * scalars )
        {
            const uint32_t words = ( V + 31u ) / 32u;
            const uint32_t total = first[ words ];
            if ( blockIdx.x == 0 && threadIdx.x == 0 )
            {
                voxels[ 0 ]  = 0u;
                border[ 0 ]  = 0u;
                scalars[ 0 ] = total;
                if ( total > rootCap )
                    atomicOr( scalars + 1, 4u );
            }
            for ( uint32_t w = blockIdx.x * blockDim.x + threadIdx.x; w < words; w += gridDim.x * blockDim.x )
            {
                uint32_t k = first[ w ];
                for ( uint32_t m = rootBits[ w ]; m; m &= m - 1u, k++ )
                {
                    L[ 32u * w + (uint32_t)__ffs( (int)m ) - 1u ] = -2 - (int32_t)k;
                    if ( k < rootCap )
                    {
                        voxels[ k + 1 ] = 0u;
                        border[ k + 1 ] = 0u;
                    }
                }
            }
        }

        __global__ void __launch_bounds__( 128 ) k_cav_resolve( const uint32_t * bits, const uint32_t * runs, CavGrid g, int32_t * L,
                                                                const uint32_t * scalars, uint8_t * border )
        {
            if ( scalars[ 1 ] )
                return; // an error: the records do not hold the components
            const uint32_t nz = g.dims[ 2 ], V = nz * g.dims[ 1 ] * g.dims[ 0 ], words = ( V + 31u ) / 32u;
            bool           one = false; // most of the border is the first component's: set once per block
            for ( uint32_t w = blockIdx.x * blockDim.x + threadIdx.x; w < words; w += gridDim.x * blockDim.x )
                for ( uint32_t m = runs[ w ]; m; m &= m - 1u )
                {
                    const uint32_t v = 32u * w + (uint32_t)__ffs( (int)m ) - 1u;
                    int32_t        p = L[ v ];
                    if ( p >= 0 )
                    {
                        // voxel 0 can only be the first root: most runs are its, and would all load from it
                        p      = p == 0 ? -2 : L[ p ];
                        L[ v ] = p;
                    }
                    const int32_t lab = -1 - p;
                    if ( lab == 1 && one )
                        continue;
                    const uint32_t col = v / nz, iz = v - col * nz, ix = col / g.dims[ 1 ], iy = col - ix * g.dims[ 1 ];
                    const uint32_t end = ( col + 1u ) * nz - 1u; // a run that ends with its row
                    if ( ix == 0 || iy == 0 || iz == 0 || ix + 1 == g.dims[ 0 ] || iy + 1 == g.dims[ 1 ]
                         || ( cav_free( bits, end ) && cav_start( runs, end ) == (int32_t)v ) )
                    {
                        if ( lab == 1 )
                            one = true;
                        else
                            border[ lab ] = 1;
                    }
                }
            if ( __syncthreads_or( one ) && threadIdx.x == 0u )
                border[ 1 ] = 1;
        }

        // Bound by the writes of the labels. A lane takes four voxels; a voxel's run starts in its word or is the one
        // that reaches into the word. Most accessible voxels are the first component's: its count is kept to the end, one
        // atomic per block (one per warp, all to one address, took most of the former kernel's
        // 133 us for 20,000 atoms on a 0.5 A grid; 17 us now).
        __global__ void __launch_bounds__( 256 ) k_cav_labels( const uint32_t * bits, const uint32_t * runs, uint32_t V, int32_t * L, uint32_t * voxels,
                                                               const uint8_t * border, uint32_t * scalars )
        {
            if ( scalars[ 1 ] )
                return;
            const uint32_t quads = ( V + 3u ) / 4u, total = scalars[ 0 ], stride = gridDim.x * blockDim.x;
            const uint32_t lane = threadIdx.x & 31u;
            uint32_t       ones = 0, borders = 0;
            for ( uint32_t k = 1u + blockIdx.x * blockDim.x + threadIdx.x; k <= total; k += stride )
                borders += border[ k ];
            // every lane runs the same number of iterations, so that the votes below see full warps
            for ( uint32_t base = blockIdx.x * blockDim.x; base < quads; base += stride )
            {
                const uint32_t q = base + threadIdx.x, v = 4u * q, at = v & 31u;
                int            lab[ 4 ] = { 0, 0, 0, 0 };
                if ( q < quads )
                {
                    const uint32_t f = ~bits[ q >> 3 ] >> at & ( V - v >= 4u ? 15u : ( 1u << ( V - v ) ) - 1u );
                    if ( f )
                    {
                        const uint32_t starts = runs[ q >> 3 ], inner = starts >> at & 15u;
                        // a start's value is the code of its component, or already its label
                        int32_t run = -1;
                        if ( f & ~inner & 1u )
                        {
                            run = L[ cav_start( runs, v ) ];
                            run = run < 0 ? -1 - run : run;
                        }
#pragma unroll
                        for ( int i = 0; i < 4; i++ )
                        {
                            if ( inner >> i & 1u )
                            {
                                run = L[ v + (uint32_t)i ];
                                run = run < 0 ? -1 - run : run;
                            }
                            lab[ i ] = f >> i & 1u ? run : 0;
                        }
                    }
                }
                __syncwarp();
                if ( q < quads ) // (the labels' allocation is a multiple of four)
                    __stcg( reinterpret_cast<int4 *>( L ) + q, make_int4( lab[ 0 ], lab[ 1 ], lab[ 2 ], lab[ 3 ] ) );
                bool more = false;
                for ( int i = 0; i < 4; i++ )
                {
                    ones += lab[ i ] == 1;
                    more |= lab[ i ] > 1;
                }
                if ( __any_sync( 0xffffffffu, more ) )
                    for ( int i = 0; i < 4; i++ )
                    {
                        // the other components' counts, one atomic per distinct label of the warp
                        const uint32_t peers = __match_any_sync( 0xffffffffu, lab[ i ] );
                        if ( lab[ i ] > 1 && lane == (uint32_t)( __ffs( (int)peers ) - 1 ) )
                            atomicAdd( voxels + lab[ i ], (uint32_t)__popc( peers ) );
                    }
            }
            __shared__ uint32_t sum[ 2 ];
            if ( threadIdx.x < 2u )
                sum[ threadIdx.x ] = 0u;
            __syncthreads();
            ones    = __reduce_add_sync( 0xffffffffu, ones );
            borders = __reduce_add_sync( 0xffffffffu, borders );
            if ( lane == 0u && ones )
                atomicAdd( sum, ones );
            if ( lane == 0u && borders )
                atomicAdd( sum + 1, borders );
            __syncthreads();
            if ( threadIdx.x == 0u && sum[ 0 ] )
                atomicAdd( voxels + 1, sum[ 0 ] );
            if ( threadIdx.x == 0u && sum[ 1 ] )
                atomicAdd( scalars + 2, sum[ 1 ] );
        }

        // A warp per probe, a lane per (ox, oy). The labels around a probe are nearly always those of one component, and the
        // FP64 pipe is what the distances would wait for (42 us for the 31,000 probes of 20,000 atoms with every distance
        // in double precision, 29 us now): they are taken only where the labels differ.
        // (as in k_cav_raster, a block first takes a thread per probe and axis.)
        __global__ void __launch_bounds__( 256 ) k_cav_probes( const float4 * probes, uint32_t k, CavGrid g, const int32_t * L, int32_t * out )
        {
            __shared__ int sBase[ 3 ][ kRasterAtoms ];
            const uint32_t lane = threadIdx.x & 31u, warp = threadIdx.x >> 5;
            const uint32_t first0 = blockIdx.x * kRasterAtoms;
            if ( warp < 3u && first0 + lane < k )
            {
                const float4 pf = probes[ first0 + lane ];
                const int    a  = (int)warp;
                sBase[ a ][ lane ] = (int)rint( __ddiv_rn( __dsub_rn( (double)( a == 0 ? pf.x : a == 1 ? pf.y : pf.z ), g.lo[ a ] ), g.h ) );
            }
            __syncthreads();
            for ( uint32_t i = warp; i < kRasterAtoms && first0 + i < k; i += blockDim.x >> 5 )
            {
                const uint32_t q = first0 + i;
                const float4   pf = probes[ q ];
                const float    p[ 3 ] = { pf.x, pf.y, pf.z };
                const int      base[ 3 ] = { sBase[ 0 ][ i ], sBase[ 1 ][ i ], sBase[ 2 ][ i ] };
                auto square = [ & ]( int a, int v ) { return sq( __dsub_rn( __dadd_rn( g.lo[ a ], __dmul_rn( (double)v, g.h ) ), (double)p[ a ] ) ); };
                const int      ix = min( max( base[ 0 ] + (int)( lane / 5u ) - 2, 0 ), (int)g.dims[ 0 ] - 1 );
                const int      iy = min( max( base[ 1 ] + (int)( lane % 5u ) - 2, 0 ), (int)g.dims[ 1 ] - 1 );
                const uint32_t row = ( (uint32_t)ix * g.dims[ 1 ] + (uint32_t)iy ) * g.dims[ 2 ];
                int            iz[ 5 ];
                int32_t        l[ 5 ];
                uint32_t       least = 0xffffffffu, most = 0u; // labels > 0
#pragma unroll
                for ( int o = 0; o < 5; o++ )
                {
                    iz[ o ] = min( max( base[ 2 ] + o - 2, 0 ), (int)g.dims[ 2 ] - 1 );
                    l[ o ]  = lane < 25u ? L[ row + (uint32_t)iz[ o ] ] : 0;
                }
#pragma unroll
                for ( int o = 0; o < 5; o++ )
                    if ( l[ o ] > 0 )
                    {
                        least = min( least, (uint32_t)l[ o ] );
                        most  = max( most, (uint32_t)l[ o ] );
                    }
                least       = __reduce_min_sync( 0xffffffffu, least );
                most        = __reduce_max_sync( 0xffffffffu, most );
                int32_t lab = (int32_t)most;
                if ( most && least != most )
                {
                    double       best = 1e300;
                    const double dxy  = __dadd_rn( square( 0, ix ), square( 1, iy ) );
                    lab               = 0;
                    for ( int o = 0; o < 5; o++ )
                        if ( l[ o ] > 0 )
                        {
                            const double d = __dadd_rn( dxy, square( 2, iz[ o ] ) );
                            if ( d < best )
                            {
                                best = d;
                                lab  = l[ o ];
                            }
                        }
                    // first minimum: the lower lane on a tie (distances are in the order of their bits)
                    const unsigned long long key = lab > 0 ? (unsigned long long)__double_as_longlong( best ) : ~0ull;
                    const uint32_t hi = __reduce_min_sync( 0xffffffffu, (uint32_t)( key >> 32 ) );
                    const uint32_t lo = __reduce_min_sync( 0xffffffffu, (uint32_t)( key >> 32 ) == hi ? (uint32_t)key : 0xffffffffu );
                    const uint32_t at = __ballot_sync( 0xffffffffu, key == ( (unsigned long long)hi << 32 | lo ) );
                    lab               = __shfl_sync( 0xffffffffu, lab, __ffs( (int)at ) - 1 );
                }
                if ( lane == 0u )
                    out[ q ] = lab;
            }
        }
    } // namespace

    void launch_cavity_bounds( const Build & b, double rp, unsigned long long * keys, cudaStream_t s )
    {
        cudaMemsetAsync( keys, 0xff, 3 * sizeof( unsigned long long ), s );
        cudaMemsetAsync( keys + 3, 0, 3 * sizeof( unsigned long long ), s );
        k_cav_bounds<<<cav_blocks( b.n, 256, 152u ), 256, 0, s>>>( b.atoms, b.n, rp, keys );
        count_launches( 1 );
    }
    double cavity_bound( unsigned long long key )
    {
        const unsigned long long u = key >> 63 ? key & ~( 1ull << 63 ) : ~key;
        double                   v;
        std::memcpy( &v, &u, 8 );
        return v;
    }

    void launch_cavities( const Build & b, const CavGrid & g, const CavBuffers & c, uint32_t rootCap, const float4 * probes, uint32_t k,
                          int32_t * probeLabel, cudaStream_t s )
    {
        const uint32_t V = g.dims[ 0 ] * g.dims[ 1 ] * g.dims[ 2 ], words = ( V + 31u ) / 32u;
        cudaMemsetAsync( c.bits, 0, sizeof( uint32_t ) * words, s );
        cudaMemsetAsync( c.scalars, 0, sizeof( uint32_t ) * 3, s );
        if ( b.n )
            k_cav_raster<<<( b.n + kRasterAtoms - 1 ) / kRasterAtoms, 256, 0, s>>>( b.atoms, b.n, g, 1.0 / g.h, c.bits );
        const uint32_t blocks = cav_blocks( words, 128 );
        k_cav_runs<<<blocks, 128, 0, s>>>( c.bits, g, c.runs, c.labels );
        k_cav_union<<<blocks, 128, 0, s>>>( c.bits, c.runs, g, c.labels, c.scalars + 1 );
        k_cav_flatten<<<blocks, 128, 0, s>>>( c.runs, V, c.labels, c.rootBits, c.rootCount, c.scalars + 1 );
        exclusive_scan( c.rootCount, c.rootCount, words, nullptr, nullptr, c.scan, s );
        k_cav_rank<<<blocks, 128, 0, s>>>( V, c.labels, c.rootBits, c.rootCount, rootCap, c.voxels, c.border, c.scalars );
        k_cav_resolve<<<blocks, 128, 0, s>>>( c.bits, c.runs, g, c.labels, c.scalars, c.border );
        k_cav_labels<<<cav_blocks( ( V + 3u ) / 4u, 256, 152u * 8u ), 256, 0, s>>>( c.bits, c.runs, V, c.labels, c.voxels, c.border, c.scalars );
        count_launches( b.n ? 7 : 6 );
        if ( k && probeLabel )
        {
            k_cav_probes<<<( k + kRasterAtoms - 1 ) / kRasterAtoms, 256, 0, s>>>( probes, k, g, c.labels, probeLabel );
            count_launches( 1 );
        }
    }
} // namespace sesgb
