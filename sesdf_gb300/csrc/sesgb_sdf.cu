// sesgb_sdf.cu -- signed distance to the SES at query points, its adjoint, and the headless image.
//
// Definition (project-written; the reference has no SDF). E is the set of
// probe-centre positions that overlap no atom: outside every SAS sphere
// (radius R_i = r_i + rp). With T = rp + kSdfBand:
//   x outside the SAS:  sdf = min_i (|x - c_i| - r_i), clamped to kSdfBand;
//   x inside the SAS:   sdf = rp - min(T, dist(x, dE)).
// dE is the SAS surface: the accessible parts of the SAS spheres, the arcs of
// the visible circles and the probe positions. The nearest point of dE is the
// radial projection of x on a sphere, the nearest point of a circle (any one
// where x lies on its axis), or a probe, whichever is nearest among those that
// lie on dE (not strictly inside another SAS sphere); only atoms with
// |x - c_i| <= R_i + T can carry one.
// The gradient with respect to the atoms follows the active primitive: the
// sphere or atom distance directly, a circle point and a probe by the
// Lagrange / implicit-function rule for points constrained to |p - c_m| = R_m.
//
// Two searches give every value, the same to the last bit. The general search (sdf_query_pass, a
// warp per query) examines the atoms within reach in the order of their lower bound, every
// visible circle of each, with the accessibility of every candidate point settled in double
// precision where float32 cannot. The tile search (sdf_tile_search, a lane per query or a
// few) takes up to 32 neighbouring queries at once: it screens the probes, the accessible
// arcs and the atoms around them, gathered once into shared memory; the distances of the
// nearest few primitives then come from the general search's own expressions, and where more
// than one lies within the float32 error of the smallest, the order in which the general
// search meets them decides as it does there.
#include <algorithm>
#include <cfloat>
#include <cmath>
#include <type_traits>

#include "../../include/sesgb.h"
#include "sesgb_grid.cuh"
#include "sesgb_stages.cuh"

namespace sesgb
{
    namespace
    {
        // Cells of half the reach of a query (rmax + 2 rp + band) with, in this order in one
        // array: the atoms, the probes, the arcs (cells each) and the queries (sub sub-cells a cell);
        // for the general search alone the atoms and the queries.
        struct SdfIndex
        {
            FineGrid         grid;
            uint32_t         sub;     // sub-cells of a cell that order the queries: 8 (octants) or 1
            uint32_t         items;   // kinds of items before the queries: 3, or 1 (atoms)
            uint32_t         outside; // atoms outside the grid's box: whole stencil rows
            float            rmax;
            const uint32_t * start;   // (3 + sub) cells + 1
            const float4 *   pos;     // atom (x, y, z, r; r < 0 without accessible surface), probe (x, y, z, 0), arc ball (centre, radius)
            const uint32_t * id;      // sorted atom (bit 31: no accessible direction), probe, arc, query
            const uint2 *    arcs;    // circle (i, j), i < j, of every arc
            const uint32_t * open;    // per sorted atom: 256 bins of directions, those that may be accessible (direction_bin); null without arcs
            const uint32_t * flags;   // [0] arcs, [1] queries listed for the general search, [2] 1: the arcs did not fit
        };

        // The distances that decide and give the values, every operation rounded as written (fused
        // multiply-adds included), so that each kernel that evaluates one gets the same bits.
        __device__ __forceinline__ float sdf_dot( float3 a, float3 b )
        {
            return __fmaf_rn( a.z, b.z, __fmaf_rn( a.x, b.x, __fmul_rn( a.y, b.y ) ) );
        }
        __device__ __forceinline__ float3 sdf_sub( float3 a, float4 b )
        {
            return make_float3( __fsub_rn( a.x, b.x ), __fsub_rn( a.y, b.y ), __fsub_rn( a.z, b.z ) );
        }
        // |x - c|
        __device__ __forceinline__ float sdf_distance( float3 x, float4 c )
        {
            const float3 d = sdf_sub( x, c );
            return __fsqrt_rn( sdf_dot( d, d ) );
        }

        // Nearest point q of circle (i, j) to x and its distance; nj = (c_j, R_j). -1: no circle; 0: x on the
        // axis (q the centre, dist that of any point); 1: next to it, where x - c hardly has a direction; 2 otherwise.
        // turn: the radius over the distance of x from the axis, by which an error of x - c moves q.
        __device__ __forceinline__ int sdf_circle_point( float3 x, float4 ci, float Ri, float4 nj, float & dist, float3 & q, float & turn )
        {
            const float3 d  = make_float3( __fsub_rn( nj.x, ci.x ), __fsub_rn( nj.y, ci.y ), __fsub_rn( nj.z, ci.z ) );
            const float  dd = sdf_dot( d, d ), Ri2 = __fmul_rn( Ri, Ri );
            const float  tt = __fdiv_rn( __fadd_rn( __fmaf_rn( -nj.w, nj.w, Ri2 ), dd ), __fmul_rn( 2.f, dd ) );
            const float  r2 = __fmaf_rn( -__fmul_rn( tt, tt ), dd, Ri2 );
            if ( !( r2 > 0.f ) )
                return -1;
            const float  r   = __fsqrt_rn( r2 );
            const float  inv = rsqrtf( dd );
            const float3 n   = make_float3( __fmul_rn( d.x, inv ), __fmul_rn( d.y, inv ), __fmul_rn( d.z, inv ) );
            const float3 c   = make_float3( __fmaf_rn( d.x, tt, ci.x ), __fmaf_rn( d.y, tt, ci.y ), __fmaf_rn( d.z, tt, ci.z ) );
            const float3 w   = make_float3( __fsub_rn( x.x, c.x ), __fsub_rn( x.y, c.y ), __fsub_rn( x.z, c.z ) );
            const float  h   = sdf_dot( w, n );
            const float3 v   = make_float3( __fmaf_rn( -h, n.x, w.x ), __fmaf_rn( -h, n.y, w.y ), __fmaf_rn( -h, n.z, w.z ) );
            const float  rho = __fsqrt_rn( sdf_dot( v, v ) );
            if ( !( rho > 1e-6f ) )
            {
                q    = c;
                dist = __fsqrt_rn( __fmaf_rn( h, h, r2 ) );
                return 0;
            }
            const float s = __fdiv_rn( r, rho ), e = __fsub_rn( rho, r );
            turn          = s;
            q             = make_float3( __fmaf_rn( v.x, s, c.x ), __fmaf_rn( v.y, s, c.y ), __fmaf_rn( v.z, s, c.z ) );
            dist          = __fsqrt_rn( __fmaf_rn( h, h, __fmul_rn( e, e ) ) );
            return rho > 1e-3f ? 2 : 1;
        }

        constexpr int   kSdfWarps = 4;   // warps per block (one query per warp)
        constexpr int   kSdfList   = 256; // atoms within reach held per query
        constexpr int   kSdfStaged = 128; // neighbour slots staged in shared memory

        enum SdfKind : int
        {
            kSdfClampInside = 0, // deeper than T below dE
            kSdfAtom        = 1, // outside the SAS: nearest vdW sphere
            kSdfClampOutside = 2,
            kSdfSphere      = 3, // radial projection on an accessible SAS sphere patch
            kSdfCircle      = 4, // nearest point of an accessible arc
            kSdfProbe       = 5, // probe position (vertex of dE)
        };

        struct SdfHit
        {
            int    kind;
            int    a, b, c; // sorted atom ids
            float3 q;       // point of dE (or of the vdW sphere)
            float  value;
        };

        struct SdfSmem
        {
            unsigned long long key[ kSdfList ];   // (delta bits << 32) | atom
            float4             nb[ kSdfStaged ];   // neighbourhood of the atom being examined: (c_k, R_k)
            uint16_t           near[ kNbrBuf ];    // its slots whose SAS sphere comes within the current best of x
            uint8_t            vis[ kNbrBuf ];     // status of its circles
            uint32_t           rowStart[ 25 ], rowPre[ 26 ]; // the stencil's rows
        };

        // neighbour slot s of atom i as (c_k, R_k): staged slots from shared memory
        __device__ __forceinline__ float4 sdf_nb( const Build & b, const SdfSmem & sm, size_t row, uint32_t s )
        {
            if ( s < (uint32_t)kSdfStaged )
                return sm.nb[ s ];
            const float4 c = b.atoms[ b.nbr[ row + s ] ];
            return make_float4( c.x, c.y, c.z, c.w + b.rp );
        }

        __device__ __forceinline__ void warp_min_hit( float & best, int & owner )
        {
            // smallest candidate distance, lowest lane on ties
            for ( int o = 16; o > 0; o >>= 1 )
            {
                const float ob = __shfl_xor_sync( 0xffffffffu, best, o );
                const int   oo = __shfl_xor_sync( 0xffffffffu, owner, o );
                if ( ob < best || ( ob == best && oo < owner ) )
                {
                    best  = ob;
                    owner = oo;
                }
            }
        }

        // Float32 error bound of |q - c_k|^2 - R_k^2 for a point q computed in absolute float32
        // coordinates: a few ulps of the coordinates (at most qQ / 4, the query's largest coordinate
        // plus its reach) on every coordinate, times 2 |q - c_k| (taken as R_k: the bound matters only
        // where |q - c_k| is close to R_k), plus the rounding of the squares. Inside it the test is
        // taken again in double precision.
        constexpr float kHiddenBand = 3.8147e-6f;
        __device__ __forceinline__ float hidden_band( float qQ, float d2, float Rk, float scale = kHiddenBand )
        {
            return scale * ( d2 + Rk * ( Rk + qQ ) + 1.f );
        }

        // point q (double) strictly inside the SAS sphere of atom k, in double precision
        __device__ __noinline__ bool point_inside_d( const Build & b, d3 q, uint32_t k )
        {
            const float4 ck = b.atoms[ k ];
            const double Rk = (double)ck.w + (double)b.rp;
            const double dx = q.x - (double)ck.x, dy = q.y - (double)ck.y, dz = q.z - (double)ck.z;
            return dx * dx + dy * dy + dz * dz < Rk * Rk;
        }

        // The radial projection of x on the SAS sphere of i, in double precision, strictly inside the
        // SAS sphere of one of this lane's near neighbours (lanes take every 32nd)
        __device__ __noinline__ bool sphere_point_hidden_d( const Build & b, const SdfSmem & sm, size_t row, uint32_t nn,
                                                            uint32_t i, float3 x, uint32_t lane )
        {
            const float4 ci = b.atoms[ i ];
            const d3     wd = D3( (double)x.x - (double)ci.x, (double)x.y - (double)ci.y, (double)x.z - (double)ci.z );
            const double Rd = (double)ci.w + (double)b.rp;
            const double sc = Rd / sqrt( wd.x * wd.x + wd.y * wd.y + wd.z * wd.z );
            const d3     qd = D3( (double)ci.x + wd.x * sc, (double)ci.y + wd.y * sc, (double)ci.z + wd.z * sc );
            bool         hd = false;
            for ( uint32_t e = lane; e < nn; e += 32 )
                hd = hd || point_inside_d( b, qd, b.nbr[ row + sm.near[ e ] ] );
            return hd;
        }

        // The nearest point of circle (i, neighbour slot s) to x, in double precision, strictly inside
        // the SAS sphere of a near neighbour of i other than that of slot s
        __device__ __noinline__ bool circle_point_hidden_d( const Build & b, const SdfSmem & sm, size_t row, uint32_t nn,
                                                            uint32_t i, uint32_t s, float3 x )
        {
            const float4 ai = b.atoms[ i ], aj = b.atoms[ b.nbr[ row + s ] ];
            const double Ri = (double)ai.w + (double)b.rp, Rj = (double)aj.w + (double)b.rp;
            const d3     d  = D3( (double)aj.x - (double)ai.x, (double)aj.y - (double)ai.y, (double)aj.z - (double)ai.z );
            const double dd = d.x * d.x + d.y * d.y + d.z * d.z;
            const double tt = ( Ri * Ri - Rj * Rj + dd ) / ( 2.0 * dd );
            const double r2 = Ri * Ri - tt * tt * dd;
            if ( !( r2 > 0.0 ) )
                return false;
            const double r   = sqrt( r2 );
            const double inv = 1.0 / sqrt( dd );
            const d3     n   = D3( d.x * inv, d.y * inv, d.z * inv );
            const d3     c   = D3( (double)ai.x + d.x * tt, (double)ai.y + d.y * tt, (double)ai.z + d.z * tt );
            const d3     w   = D3( (double)x.x - c.x, (double)x.y - c.y, (double)x.z - c.z );
            const double h   = w.x * n.x + w.y * n.y + w.z * n.z;
            const d3     v   = D3( w.x - h * n.x, w.y - h * n.y, w.z - h * n.z );
            const double rho = sqrt( v.x * v.x + v.y * v.y + v.z * v.z );
            if ( !( rho > 0.0 ) )
                return false;
            const d3 q = D3( c.x + v.x * ( r / rho ), c.y + v.y * ( r / rho ), c.z + v.z * ( r / rho ) );
            for ( uint32_t e = 0; e < nn; e++ )
            {
                const uint32_t k = sm.near[ e ];
                if ( k != s && point_inside_d( b, q, b.nbr[ row + k ] ) )
                    return true;
            }
            return false;
        }

        // A point of circle (i, neighbour slot s), all as far from x, lies in no SAS sphere of a near neighbour of i other than
        // that of slot s: in double precision. An uncovered arc ends where a sphere meets the circle, in a point that no
        // other one holds.
        __device__ __noinline__ bool circle_open_d( const Build & b, const SdfSmem & sm, size_t row, uint32_t nn, uint32_t i, uint32_t s )
        {
            const float4 ai = b.atoms[ i ], aj = b.atoms[ b.nbr[ row + s ] ];
            const double Ri = (double)ai.w + (double)b.rp, Rj = (double)aj.w + (double)b.rp;
            const d3     d  = D3( (double)aj.x - (double)ai.x, (double)aj.y - (double)ai.y, (double)aj.z - (double)ai.z );
            const double dd = ddot( d, d ), tt = ( Ri * Ri - Rj * Rj + dd ) / ( 2.0 * dd ), r2 = Ri * Ri - tt * tt * dd;
            if ( !( r2 > 0.0 ) )
                return true;
            const double r = sqrt( r2 );
            const d3     n = dmul( d, 1.0 / sqrt( dd ) ), c = dadd( D3( ai ), dmul( d, tt ) );
            bool         cut = false;
            for ( uint32_t e = 0; e < nn; e++ )
            {
                const uint32_t k = sm.near[ e ];
                if ( k == s )
                    continue;
                // hidden where A + B cos(phi - phi_k) > 0, phi_k the direction v of c_k from the axis
                const float4 ak = b.atoms[ b.nbr[ row + k ] ];
                const double Rk = (double)ak.w + (double)b.rp;
                const d3     w  = dsub( D3( ak ), c );
                const double h  = ddot( w, n );
                const d3     v  = dsub( w, dmul( n, h ) );
                const double l = sqrt( ddot( v, v ) ), A = Rk * Rk - ddot( w, w ) - r2, B = 2.0 * r * l;
                if ( A > B )
                    return false;
                if ( !( A > -B ) || !( l > 0.0 ) )
                    continue;
                cut            = true;
                const double cs = -A / B, sn = sqrt( fmax( 0.0, ( 1.0 - cs ) * ( 1.0 + cs ) ) );
                const d3     u = dmul( v, r * cs / l ), t = dmul( dcross( n, v ), r * sn / l );
                for ( int side = 0; side < 2; side++ )
                {
                    const d3 q    = dadd( c, side ? dsub( u, t ) : dadd( u, t ) );
                    bool     open = true;
                    for ( uint32_t o = 0; o < nn && open; o++ )
                    {
                        const float4 ao = b.atoms[ b.nbr[ row + sm.near[ o ] ] ];
                        const double Ro = (double)ao.w + (double)b.rp;
                        const d3     y  = dsub( q, D3( ao ) );
                        // (by more than rounding: spheres of a lattice meet in one point)
                        open = o == e || sm.near[ o ] == s || !( ddot( y, y ) < Ro * Ro * ( 1.0 - 1e-11 ) );
                    }
                    if ( open )
                        return true;
                }
            }
            return !cut;
        }

        // The general search: one query, the whole warp; the hit is valid in every lane. A point of dE
        // within the float32 error of another SAS sphere is decided in double precision with kExact;
        // without, the query is only marked (exact set, in every lane) and its hit means nothing.
        template<bool kExact>
        __device__ __forceinline__ SdfHit sdf_query_pass( const Build & b, const SdfIndex & ix, float3 x, SdfSmem & sm, float band,
                                                          uint32_t & overflow, bool & exact )
        {
            const uint32_t lane      = lane_id();
            bool           exactLane = false;
            exact                    = false;
            // 4 x (largest coordinate of any point of dE this query examines)
            const float qQ = 4.f * ( fmaxf( fabsf( x.x ), fmaxf( fabsf( x.y ), fabsf( x.z ) ) ) + 12.f );
            const float    T    = b.rp + band;
            // the atoms of the 5 x 5 x 5 cells around x, rows cut to the reach (whole rows where atoms lie
            // outside the grid's box and sit in its border cells)
            const uint32_t total = stencil_rows_span2( ix.grid, ix.start, make_float4( x.x, x.y, x.z, 0.f ),
                                                       ix.outside ? 3e18f : ix.rmax + b.rp + T + 0.01f, sm.rowStart, sm.rowPre );
            SdfHit hit;
            hit.a = hit.b = hit.c = -1;
            hit.q                 = x;
            hit.kind              = kSdfClampOutside;
            hit.value             = band;
            if ( total == 0u )
                return hit; // no atom near (most steps of most rays)
            // atoms within reach; minima of |x - c| - R (SAS) and |x - c| - r (vdW)
            uint32_t nl = 0;
            float    smin = 3.4e38f, vmin = 3.4e38f;
            int      vatom = 0x7fffffff;
            for ( uint32_t base = 0; base < total; base += 32 )
            {
                const uint32_t f    = base + lane;
                bool           keep = false;
                uint32_t       i    = 0;
                float          dl   = 0.f;
                if ( f < total )
                {
                    const uint32_t idx = row_item_span2( sm.rowStart, sm.rowPre, f );
                    i                  = ix.id[ idx ] & 0x7fffffffu;
                    const float4 c     = ix.pos[ idx ];
                    const float  ra    = fabsf( c.w );
                    const float  L     = sdf_distance( x, c );
                    const float  R     = ra + b.rp;
                    if ( L <= R + T )
                    {
                        smin = fminf( smin, L - R );
                        const float v = L - ra;
                        if ( v < vmin || ( v == vmin && (int)i < vatom ) )
                        {
                            vmin  = v;
                            vatom = (int)i;
                        }
                        dl = fabsf( L - R );
                        // fully buried atoms carry no point of dE: only the bounds above use them
                        keep = !signbit( c.w );
                    }
                }
                const uint32_t mk = __ballot_sync( 0xffffffffu, keep );
                const uint32_t at = nl + __popc( mk & lanemask_lt() );
                if ( keep && at < (uint32_t)kSdfList )
                    sm.key[ at ] = ( (unsigned long long)__float_as_uint( dl ) << 32 ) | i;
                nl += __popc( mk );
            }
            if ( nl > (uint32_t)kSdfList )
            {
                overflow = 1;
                nl       = kSdfList;
            }
            for ( int o = 16; o > 0; o >>= 1 )
            {
                smin          = fminf( smin, __shfl_xor_sync( 0xffffffffu, smin, o ) );
                const float v = __shfl_xor_sync( 0xffffffffu, vmin, o );
                const int   a = __shfl_xor_sync( 0xffffffffu, vatom, o );
                if ( v < vmin || ( v == vmin && a < vatom ) )
                {
                    vmin  = v;
                    vatom = a;
                }
            }
            if ( !( smin < 0.f ) )
            {
                // outside the SAS (or nothing within reach)
                if ( vatom != 0x7fffffff && vmin <= band )
                {
                    hit.kind  = kSdfAtom;
                    hit.a     = vatom;
                    hit.value = vmin;
                }
                return hit;
            }
            __syncwarp();
            float best  = T;
            hit.kind    = kSdfClampInside;
            // x lies in a SAS sphere with R - |x - c| = -smin: every point of dE is at least that far
            const float floorD = -smin;
            if ( !( floorD < T ) )
            {
                hit.value = b.rp - T;
                return hit;
            }
            // probes (vertices of dE, never hidden) first: an early upper bound for the search
            {
                float  cand = 3.4e38f;
                int    pa = -1, pb = -1, pc = -1;
                float3 pq = x;
                // lane per atom: its probe chunk
                for ( uint32_t e0 = lane; e0 < nl; e0 += 32 )
                {
                    const uint32_t i     = (uint32_t)sm.key[ e0 ];
                    const uint32_t chunk = b.chunkStart[ i ], len = b.chunkLen[ i ];
                    for ( uint32_t e = 0; e < len; e++ )
                    {
                        const int4 cid = b.stageCid[ chunk + e ];
                        if ( cid.w == 0 )
                            continue;
                        const float4 p    = b.stagePos[ chunk + e ];
                        const float  dist = sdf_distance( x, p );
                        // (of equal distances the lowest atom's, the first of its chunk: the list's order differs from call to call)
                        if ( dist < cand || ( dist == cand && (int)i < pa ) )
                        {
                            const int4 ids = b.stageIds[ chunk + e ];
                            cand           = dist;
                            pa             = ids.x;
                            pb             = ids.y;
                            pc             = ids.z;
                            pq             = make_float3( p.x, p.y, p.z );
                        }
                    }
                }
                float wbest = cand;
                for ( int o = 16; o > 0; o >>= 1 )
                    wbest = fminf( wbest, __shfl_xor_sync( 0xffffffffu, wbest, o ) );
                if ( wbest < best )
                {
                    const uint32_t key   = cand == wbest ? (uint32_t)pa : 0xffffffffu;
                    const uint32_t first = __reduce_min_sync( 0xffffffffu, key );
                    const int      owner = __ffs( (int)__ballot_sync( 0xffffffffu, key == first ) ) - 1;
                    best     = wbest;
                    hit.kind = kSdfProbe;
                    hit.a    = __shfl_sync( 0xffffffffu, pa, owner );
                    hit.b    = __shfl_sync( 0xffffffffu, pb, owner );
                    hit.c    = __shfl_sync( 0xffffffffu, pc, owner );
                    hit.q.x  = __shfl_sync( 0xffffffffu, pq.x, owner );
                    hit.q.y  = __shfl_sync( 0xffffffffu, pq.y, owner );
                    hit.q.z  = __shfl_sync( 0xffffffffu, pq.z, owner );
                }
            }
            // atoms in ascending |x - c| - R order (the lower bound of all their candidates),
            // each picked by a warp minimum over the ones left, until the bound reaches best
            for ( uint32_t t = 0; t < nl; t++ )
            {
                unsigned long long key = ~0ull;
                uint32_t           at  = 0;
                for ( uint32_t e = lane; e < nl; e += 32 )
                    if ( sm.key[ e ] < key )
                    {
                        key = sm.key[ e ];
                        at  = e;
                    }
                for ( int o = 16; o > 0; o >>= 1 )
                {
                    const unsigned long long ok = __shfl_xor_sync( 0xffffffffu, key, o );
                    const uint32_t           oa = __shfl_xor_sync( 0xffffffffu, at, o );
                    if ( ok < key )
                    {
                        key = ok;
                        at  = oa;
                    }
                }
                const float dl = __uint_as_float( (uint32_t)( key >> 32 ) );
                if ( !( dl < best ) || !( floorD < best ) )
                    break; // every candidate of this and the remaining atoms is at least dl away
                __syncwarp();
                if ( lane == 0 )
                    sm.key[ at ] = ~0ull; // taken
                const uint32_t i   = (uint32_t)key;
                const float4   ci  = b.atoms[ i ];
                const float    Ri  = ci.w + b.rp;
                const uint32_t ni  = b.nbrCount[ i ];
                const size_t   row = (size_t)i * b.cap;
                // stage N(i); a point q with |x - q| < best can only lie inside the SAS
                // sphere of a neighbour k with |x - c_k| - R_k < best: those are the "near" ones
                uint32_t nn = 0;
                for ( uint32_t s0 = 0; s0 < ni; s0 += 32 )
                {
                    const uint32_t s    = s0 + lane;
                    bool           near = false;
                    if ( s < ni )
                    {
                        sm.vis[ s ]     = b.status[ row + s ];
                        const float4 ck = b.atoms[ b.nbr[ row + s ] ];
                        const float  Rk = ck.w + b.rp;
                        if ( s < (uint32_t)kSdfStaged )
                            sm.nb[ s ] = make_float4( ck.x, ck.y, ck.z, Rk );
                        const float Lk  = sqrtf( ( x.x - ck.x ) * ( x.x - ck.x ) + ( x.y - ck.y ) * ( x.y - ck.y ) + ( x.z - ck.z ) * ( x.z - ck.z ) );
                        near            = Lk - Rk < best;
                    }
                    const uint32_t mk = __ballot_sync( 0xffffffffu, near );
                    if ( near )
                        sm.near[ nn + __popc( mk & lanemask_lt() ) ] = (uint16_t)s;
                    nn += __popc( mk );
                }
                __syncwarp();
                // candidates of this atom, one per lane at most, reduced at the end
                float  cand = 3.4e38f;
                int    ck = 0, cb = -1, cc = -1;
                float3 cq = x;
                // radial projection on sphere i
                {
                    const float3 w = make_float3( x.x - ci.x, x.y - ci.y, x.z - ci.z );
                    const float  L = sqrtf( w.x * w.x + w.y * w.y + w.z * w.z );
                    if ( L > 0.f )
                    {
                        const float3 q = make_float3( ci.x + w.x * ( Ri / L ), ci.y + w.y * ( Ri / L ), ci.z + w.z * ( Ri / L ) );
                        bool         hidden = false, unsure = false;
                        for ( uint32_t e = lane; e < nn; e += 32 )
                        {
                            const float4 nk = sdf_nb( b, sm, row, sm.near[ e ] );
                            const float  dx = q.x - nk.x, dy = q.y - nk.y, dz = q.z - nk.z;
                            const float  d2 = dx * dx + dy * dy + dz * dz;
                            const float  m  = d2 - nk.w * nk.w;
                            const float  eb = hidden_band( qQ, d2, nk.w );
                            hidden          = hidden || m < -eb;
                            unsure          = unsure || !( fabsf( m ) > eb );
                        }
                        bool hid = __any_sync( 0xffffffffu, hidden );
                        // a neighbour's sphere passes within the float32 error of the point: the point
                        // and the test in double precision
                        if ( !hid && __any_sync( 0xffffffffu, unsure ) )
                        {
                            if constexpr ( kExact )
                                hid = __any_sync( 0xffffffffu, sphere_point_hidden_d( b, sm, row, nn, i, x, lane ) );
                            else
                                exactLane = true;
                        }
                        if ( !hid && lane == 0 )
                        {
                            cand = dl;
                            ck   = kSdfSphere;
                            cq   = q;
                        }
                    }
                }
                // nearest points of the visible circles of i
                for ( uint32_t s0 = 0; s0 < ni; s0 += 32 )
                {
                    const uint32_t s = s0 + lane;
                    if ( s >= ni || sm.vis[ s ] == 0 )
                        continue;
                    const float4 nj = sdf_nb( b, sm, row, s );
                    {
                        // every point of circle (i, j) is on sphere j too: |x - c_j| - R_j bounds it
                        const float Lj = sqrtf( ( x.x - nj.x ) * ( x.x - nj.x ) + ( x.y - nj.y ) * ( x.y - nj.y ) + ( x.z - nj.z ) * ( x.z - nj.z ) );
                        if ( !( fabsf( Lj - nj.w ) < best ) )
                            continue;
                    }
                    float        dist, turn;
                    float3       q;
                    const int    at = sdf_circle_point( x, ci, Ri, nj, dist, q, turn );
                    if ( at < 0 )
                        continue;
                    if ( at > 0 )
                    {
                        if ( !( dist < cand ) || !( dist < best ) )
                            continue;
                        // x - c is off by up to 1.1e-7 coordinates + 1.2e-6, across the axis, and q by turn times that: 2 R_k times this is
                        // 0.014 turn of hidden_band
                        bool        hidden = false, unsure = at == 1;
                        const float wide = kHiddenBand * ( 1.f + 0.03f * turn );
                        for ( uint32_t e = 0; at > 1 && e < nn && !hidden; e++ )
                        {
                            const uint32_t k = sm.near[ e ];
                            if ( k == s )
                                continue;
                            const float4 nk = sdf_nb( b, sm, row, k );
                            const float  dx = q.x - nk.x, dy = q.y - nk.y, dz = q.z - nk.z;
                            const float  d2 = dx * dx + dy * dy + dz * dz;
                            const float  m  = d2 - nk.w * nk.w;
                            const float  eb = hidden_band( qQ, d2, nk.w, wide );
                            hidden          = m < -eb;
                            unsure          = unsure || !( fabsf( m ) > eb );
                        }
                        if ( !hidden && unsure )
                        {
                            if constexpr ( kExact )
                                hidden = circle_point_hidden_d( b, sm, row, nn, i, s, x );
                            else
                                exactLane = true;
                        }
                        if ( hidden )
                            continue;
                    }
                    else
                    {
                        // x on the axis: every point of the circle is as near. A visible circle is one that no single
                        // sphere buries; several together may
                        if ( !( dist < cand ) || !( dist < best ) )
                            continue;
                        if constexpr ( kExact )
                        {
                            if ( !circle_open_d( b, sm, row, nn, i, s ) )
                                continue;
                        }
                        else
                            exactLane = true;
                    }
                    cand = dist;
                    ck   = kSdfCircle;
                    cb   = (int)b.nbr[ row + s ];
                    cq   = q;
                }
                float wbest = cand;
                int   owner = (int)lane;
                warp_min_hit( wbest, owner );
                if ( wbest < best )
                {
                    best     = wbest;
                    hit.kind = __shfl_sync( 0xffffffffu, ck, owner );
                    hit.a    = (int)i;
                    hit.b    = __shfl_sync( 0xffffffffu, cb, owner );
                    hit.c    = __shfl_sync( 0xffffffffu, cc, owner );
                    hit.q.x  = __shfl_sync( 0xffffffffu, cq.x, owner );
                    hit.q.y  = __shfl_sync( 0xffffffffu, cq.y, owner );
                    hit.q.z  = __shfl_sync( 0xffffffffu, cq.z, owner );
                }
                __syncwarp();
            }
            hit.value = b.rp - best;
            exact     = __any_sync( 0xffffffffu, exactLane );
            return hit;
        }
        __device__ __noinline__ SdfHit sdf_query_exact( const Build & b, const SdfIndex & ix, float3 x, SdfSmem & sm, float band,
                                                        uint32_t & overflow )
        {
            bool marked;
            return sdf_query_pass<true>( b, ix, x, sm, band, overflow, marked );
        }
        // The float32 pass. Its whole hit is kept alive: without the parts that a caller does not read, the compiler arranges
        // the loops over the neighbours so that one query took 3.1 ms instead of 2.1 (20,000 atoms, 2.9 A probe).
        __device__ __forceinline__ SdfHit sdf_query_float( const Build & b, const SdfIndex & ix, float3 x, SdfSmem & sm, float band,
                                                           uint32_t & overflow, bool & exact )
        {
            const SdfHit h = sdf_query_pass<false>( b, ix, x, sm, band, overflow, exact );
            asm volatile( "" ::"r"( h.a ), "r"( h.b ), "r"( h.c ), "f"( h.q.x ), "f"( h.q.y ), "f"( h.q.z ) );
            return h;
        }

        __device__ __forceinline__ void add_grad( float * g, uint32_t atom, float gx, float gy, float gz, float gr )
        {
            atomicAdd( g + 4 * atom + 0, gx );
            atomicAdd( g + 4 * atom + 1, gy );
            atomicAdd( g + 4 * atom + 2, gz );
            atomicAdd( g + 4 * atom + 3, gr );
        }

        // d sdf / d (c, r) of the active primitive, scaled by gs, into g (sorted order)
        __device__ __noinline__ void sdf_gradient( const Build & b, const SdfHit & h, float3 x, float gs, float * g )
        {
            if ( h.kind == kSdfAtom || h.kind == kSdfSphere )
            {
                // sdf = |x - c_a| - r_a (outside the SAS, or x inside sphere a); the
                // opposite sign when x lies outside sphere a but inside another
                const float4 c = b.atoms[ h.a ];
                const float3 w = make_float3( x.x - c.x, x.y - c.y, x.z - c.z );
                const float  L = sqrtf( w.x * w.x + w.y * w.y + w.z * w.z );
                if ( !( L > 0.f ) )
                    return;
                float sgn = -1.f;
                if ( h.kind == kSdfSphere && L > c.w + b.rp )
                    sgn = 1.f;
                add_grad( g, (uint32_t)h.a, gs * sgn * w.x / L, gs * sgn * w.y / L, gs * sgn * w.z / L, gs * sgn );
                return;
            }
            if ( h.kind != kSdfCircle && h.kind != kSdfProbe )
                return;
            // The multipliers of the constraints |p - c_k|^2 = R_k^2 that hold the point p: a 2x2
            // (circle) or 3x3 (probe) system that is nearly singular when the constraint normals
            // are nearly parallel (two circle centres nearly aligned with p, a probe near the plane
            // of its three centres), where float32 would show in the gradient. Solved in double
            // precision from the float32 values (their differences are exact in double); one lane
            // per query, so the FP64 pipe's rate does not matter.
            const float3 pf = h.q;
            const d3     p  = D3( (double)pf.x, (double)pf.y, (double)pf.z );
            const d3     dv = D3( (double)x.x - p.x, (double)x.y - p.y, (double)x.z - p.z );
            const double D  = sqrt( dv.x * dv.x + dv.y * dv.y + dv.z * dv.z );
            if ( !( D > 0.0 ) )
                return;
            const d3  u = D3( dv.x / D, dv.y / D, dv.z / D );
            const int m = h.kind == kSdfCircle ? 2 : 3;
            const int ids[ 3 ] = { h.a, h.b, h.c };
            d3        a[ 3 ];
            double    R[ 3 ];
            for ( int k = 0; k < m; k++ )
            {
                const float4 c = b.atoms[ ids[ k ] ];
                a[ k ]         = D3( 2.0 * ( p.x - (double)c.x ), 2.0 * ( p.y - (double)c.y ), 2.0 * ( p.z - (double)c.z ) );
                R[ k ]         = (double)c.w + (double)b.rp;
            }
            // multipliers w: sum_k w_k a_k = u (least squares for the circle, exact for the probe)
            double w[ 3 ] = { 0.0, 0.0, 0.0 };
            if ( m == 2 )
            {
                const double g00 = a[ 0 ].x * a[ 0 ].x + a[ 0 ].y * a[ 0 ].y + a[ 0 ].z * a[ 0 ].z;
                const double g01 = a[ 0 ].x * a[ 1 ].x + a[ 0 ].y * a[ 1 ].y + a[ 0 ].z * a[ 1 ].z;
                const double g11 = a[ 1 ].x * a[ 1 ].x + a[ 1 ].y * a[ 1 ].y + a[ 1 ].z * a[ 1 ].z;
                const double r0  = a[ 0 ].x * u.x + a[ 0 ].y * u.y + a[ 0 ].z * u.z;
                const double r1  = a[ 1 ].x * u.x + a[ 1 ].y * u.y + a[ 1 ].z * u.z;
                const double det = g00 * g11 - g01 * g01;
                if ( !( fabs( det ) > 0.0 ) )
                    return;
                w[ 0 ] = ( r0 * g11 - r1 * g01 ) / det;
                w[ 1 ] = ( r1 * g00 - r0 * g01 ) / det;
            }
            else
            {
                // columns a_0, a_1, a_2: Cramer's rule
                const d3     c12 = dcross( a[ 1 ], a[ 2 ] );
                const double det = ddot( a[ 0 ], c12 );
                if ( !( fabs( det ) > 0.0 ) )
                    return;
                w[ 0 ] = ddot( u, c12 ) / det;                    // det[u, a1, a2]
                w[ 1 ] = ddot( a[ 0 ], dcross( u, a[ 2 ] ) ) / det; // det[a0, u, a2]
                w[ 2 ] = ddot( dcross( a[ 0 ], a[ 1 ] ), u ) / det; // det[a0, a1, u]
            }
            // sdf = rp - D: d sdf / d c_k = w_k a_k, d sdf / d r_k = 2 w_k R_k
            for ( int k = 0; k < m; k++ )
                add_grad( g, (uint32_t)ids[ k ], (float)( gs * w[ k ] * a[ k ].x ), (float)( gs * w[ k ] * a[ k ].y ),
                          (float)( gs * w[ k ] * a[ k ].z ), (float)( gs * 2.0 * w[ k ] * R[ k ] ) );
        }

        // ---- index: accessible arcs, and the cells of atoms, probes, arcs and queries ------------
        constexpr int   kArcWarps  = 8;
        constexpr int   kArcStaged = 128;   // neighbours staged in shared memory
        constexpr float kArcHalf   = 1.f;   // half length of an arc piece (A), about
        constexpr float kArcBall   = 1.05f; // largest ball of one; a larger one sends every query to the general search
        constexpr float kArcStep   = 6.283185307f / 64.f;

        // Directions in 16 x 16 bins of the octahedral map (a unit vector scaled to |x| + |y| + |z| = 1, the
        // lower half folded over the corners of the square).
        __device__ __forceinline__ uint32_t direction_bin( f3 v )
        {
            const float s = __fdividef( 1.f, fabsf( v.x ) + fabsf( v.y ) + fabsf( v.z ) );
            float       x = v.x * s, y = v.y * s;
            if ( v.z < 0.f )
            {
                const float t = copysignf( 1.f - fabsf( y ), x );
                y             = copysignf( 1.f - fabsf( x ), y );
                x             = t;
            }
            const int ix = min( max( (int)floorf( x * 8.f + 8.f ), 0 ), 15 ), iy = min( max( (int)floorf( y * 8.f + 8.f ), 0 ), 15 );
            return (uint32_t)( iy * 16 + ix );
        }
        __device__ __forceinline__ bool direction_open( const uint32_t * open, uint32_t atom, f3 v )
        {
            const uint32_t bin = direction_bin( v );
            return open[ 8u * (size_t)atom + ( bin >> 5 ) ] >> ( bin & 31u ) & 1u;
        }
        // unit vector of a point of the square [-1, 1]^2
        __device__ __forceinline__ f3 direction_of( float x, float y )
        {
            const float z = 1.f - fabsf( x ) - fabsf( y );
            f3          v = F3( x, y, z );
            if ( z < 0.f )
            {
                v.x = copysignf( 1.f - fabsf( y ), x );
                v.y = copysignf( 1.f - fabsf( x ), y );
            }
            return normalize( v );
        }

        // What of every atom's SAS sphere and circles can be accessible. A warp per atom with an
        // accessible patch:
        //  - its directions in 256 bins, a lane per bin: the bins that no single neighbour's SAS sphere covers
        //    whole by a clear margin, first on 8 x 8 bins, then the quarters of the open ones. 98 % of the
        //    spheres of a globule is hidden, and this settles most radial projections with one look-up (of 17.6
        //    a query 5.6 passed 64 bins alone, 0.1 are accessible). Without `quarters` (few queries, which would
        //    not earn the time back) a coarse bin stands for its four;
        //  - the accessible arcs of its visible circles (i, j), i < j, as pieces in balls of at most about
        //    kArcHalf, a lane per circle: the circle's 64 bins of angle, less those inside a neighbour's
        //    SAS sphere by a clear margin. Three quarters of the partial circles are covered by their
        //    neighbours together and leave no arc, so that a query meets ~3 pieces an atom instead of
        //    ~20 circles.
        // Issue-bound (few circles an atom: 7 of 32 lanes).
        __global__ void __launch_bounds__( 32 * kArcWarps ) k_sdf_arcs( Build b, float4 * balls, uint2 * arcs, uint32_t capArcs,
                                                                        uint32_t * openBins, bool quarters, uint32_t * flags )
        {
            __shared__ float4   rel[ kArcWarps ][ kArcStaged ];
            __shared__ uint16_t list[ kArcWarps ][ kNbrBuf ];
            __shared__ float4   caps[ kArcWarps ][ kArcStaged ]; // cap of directions that a neighbour hides: axis, cosine
            __shared__ float    capSin[ kArcWarps ][ kArcStaged ];
            __shared__ float4   bins[ 64 + 256 ]; // centre of every bin of directions, cosine of its farthest corner: coarse, fine
            __shared__ uint32_t openWords[ kArcWarps ][ 8 ];
            __shared__ uint8_t  openList[ kArcWarps ][ 64 ];
            const uint32_t      warp = threadIdx.x >> 5, lane = lane_id();
            const uint32_t      i = blockIdx.x * kArcWarps + warp;
            for ( uint32_t t = threadIdx.x; t < 64u + 256u; t += 32u * kArcWarps )
            {
                const uint32_t side = t < 64u ? 8u : 16u, q = t < 64u ? t : t - 64u;
                const float    e    = 1.f / (float)side; // half a bin
                const float    x = ( (float)( 2u * ( q % side ) + 1u ) ) * e - 1.f, y = ( (float)( 2u * ( q / side ) + 1u ) ) * e - 1.f;
                const f3       u  = direction_of( x, y );
                float          cb = 1.f;
                for ( int k = 0; k < 4; k++ )
                    cb = fminf( cb, dot( u, direction_of( x + ( k & 1 ? e : -e ), y + ( k & 2 ? e : -e ) ) ) );
                bins[ t ] = make_float4( u.x, u.y, u.z, cb - 1e-3f );
            }
            __syncthreads();
            if ( i >= b.n )
                return;
            const uint32_t ni = min( b.nbrCount[ i ], (uint32_t)kNbrBuf );
            if ( b.visCnt[ i ] == 0 && ni > 0 )
                return; // no accessible patch: its bins are never read
            const size_t   row = (size_t)i * b.cap;
            const float4   ai  = b.atoms[ i ];
            const float    Ri  = ai.w + b.rp, invRi = 1.f / Ri;
            auto           neighbour = [ & ]( uint32_t k ) {
                const float4 a = b.atoms[ b.nbr[ row + k ] ];
                const f3     d = F3( a.x - ai.x, a.y - ai.y, a.z - ai.z );
                const float  R = a.w + b.rp;
                // x on the SAS sphere of i lies inside the SAS sphere of k where x . d_k > K_k
                return make_float4( d.x, d.y, d.z, 0.5f * ( ( Ri * Ri + dot( d, d ) ) - R * R ) );
            };
            auto cap_of = [ & ]( float4 q ) {
                const float dd = q.x * q.x + q.y * q.y + q.z * q.z, inv = rsqrtf( dd );
                return dd > 0.f ? make_float4( q.x * inv, q.y * inv, q.z * inv, fmaxf( q.w * inv * invRi, -1.f ) )
                                : make_float4( 0.f, 0.f, 1.f, 2.f );
            };
            auto     sin_of = []( float c ) { return sqrtf( fmaxf( 0.f, ( 1.f - c ) * ( 1.f + c ) ) ); };
            uint32_t nc = 0;
            for ( uint32_t s0 = 0; s0 < ni; s0 += 32 )
            {
                const uint32_t s    = s0 + lane;
                bool           mine = false;
                if ( s < ni )
                {
                    mine = b.status[ row + s ] != 0 && b.nbr[ row + s ] > i;
                    if ( s < (uint32_t)kArcStaged )
                    {
                        rel[ warp ][ s ]    = neighbour( s );
                        caps[ warp ][ s ]   = cap_of( rel[ warp ][ s ] );
                        capSin[ warp ][ s ] = sin_of( caps[ warp ][ s ].w );
                    }
                }
                const uint32_t mk = __ballot_sync( 0xffffffffu, mine );
                if ( mine )
                    list[ warp ][ nc + __popc( mk & lanemask_lt() ) ] = (uint16_t)s;
                nc += __popc( mk );
            }
            __syncwarp();
            {
                // a cone of cosine u.w lies in a cap of cosine c where its axis is within acos(c) - acos(u.w) of
                // the cap's
                auto covered = [ & ]( float4 u ) {
                    const float sb = sin_of( u.w );
                    for ( uint32_t k = 0; k < ni; k++ )
                    {
                        const bool   staged = k < (uint32_t)kArcStaged;
                        const float4 q      = staged ? caps[ warp ][ k ] : cap_of( neighbour( k ) );
                        const float  sc     = staged ? capSin[ warp ][ k ] : sin_of( q.w );
                        if ( u.x * q.x + u.y * q.y + u.z * q.z > q.w * u.w + sc * sb + 1e-3f && q.w < u.w )
                            return true;
                    }
                    return false;
                };
                uint32_t coarse = 0;
                if ( lane < 8u )
                    openWords[ warp ][ lane ] = 0;
                // lanes 0-31 take bins 0-31, then 32-63, then the quarters of the open ones
                for ( uint32_t t0 = 0; t0 < 64u + 4u * coarse; t0 += 32 )
                {
                    const uint32_t t    = t0 + lane;
                    const bool     fine = t0 >= 64u;
                    uint32_t       bin  = t;
                    if ( fine && t < 64u + 4u * coarse )
                    {
                        const uint32_t c = openList[ warp ][ ( t - 64u ) >> 2 ];
                        bin              = ( 2u * ( c >> 3 ) + ( t >> 1 & 1u ) ) * 16u + 2u * ( c & 7u ) + ( t & 1u );
                    }
                    const bool     open = t < 64u + 4u * coarse && ( ( fine && !quarters ) || !covered( bins[ fine ? 64u + bin : bin ] ) );
                    const uint32_t mk   = __ballot_sync( 0xffffffffu, open );
                    if ( fine && open )
                        atomicOr( &openWords[ warp ][ bin >> 5 ], 1u << ( bin & 31u ) );
                    if ( !fine )
                    {
                        if ( open )
                            openList[ warp ][ coarse + __popc( mk & lanemask_lt() ) ] = (uint8_t)bin;
                        coarse += __popc( mk );
                    }
                    __syncwarp();
                }
                const uint32_t word = lane < 8u ? openWords[ warp ][ lane ] : 0u;
                if ( lane < 8u )
                    openBins[ 8u * (size_t)i + lane ] = word;
                if ( !__any_sync( 0xffffffffu, word != 0u ) )
                    return; // no direction left: no arc either
            }
            const float margin = 1e-3f + 1e-6f * fmaxf( fabsf( ai.x ), fmaxf( fabsf( ai.y ), fabsf( ai.z ) ) );
            for ( uint32_t c0 = 0; c0 < nc; c0 += 32 )
            {
                const bool mine = c0 + lane < nc;
                uint32_t   j    = 0;
                f3         c = F3( 0.f, 0.f, 0.f ), e1 = c, e2 = c;
                float      r      = 0.f;
                uint64_t   open   = 0; // bins that may hold accessible points
                uint32_t   most   = 64, turn = 0, pieces = 0;
                if ( mine )
                {
                    const uint32_t s  = list[ warp ][ c0 + lane ];
                    j                 = b.nbr[ row + s ];
                    const float4 q    = neighbour( s );
                    const f3     dj   = F3( q.x, q.y, q.z );
                    const float  dd   = dot( dj, dj );
                    c                 = dj * ( q.w / dd );
                    const float r2    = Ri * Ri - dot( c, c );
                    r                 = r2 > 0.f ? sqrtf( r2 ) : 0.f;
                    const f3    n     = dj * rsqrtf( dd );
                    const float ax = fabsf( n.x ), ay = fabsf( n.y ), az = fabsf( n.z );
                    const f3    t  = ( ax <= ay && ax <= az ) ? F3( 1.f, 0.f, 0.f ) : ( ay <= az ? F3( 0.f, 1.f, 0.f ) : F3( 0.f, 0.f, 1.f ) );
                    e1             = normalize( cross( n, t ) );
                    e2             = cross( n, e1 );
                    uint64_t hidden = 0;
                    // a complete circle, and one too small for its angles to mean much, stays whole
                    if ( b.status[ row + s ] == 1 && r > 0.1f )
                    {
                        // the neighbours that touch the circle (lists of up to 64), or all
                        const bool masked = ni <= 64u && b.pairOff[ i ] + s < b.capPairs;
                        uint64_t   rest   = masked ? b.touch[ b.pairOff[ i ] + s ] & ~( 1ull << s ) : 0ull;
                        for ( uint32_t k = 0; ~hidden; k++ )
                        {
                            if ( masked )
                            {
                                if ( !rest )
                                    break;
                                k = (uint32_t)__ffsll( (long long)rest ) - 1u;
                                rest &= rest - 1u;
                            }
                            if ( k >= ni )
                                break;
                            if ( k == s )
                                continue;
                            const float4 qk = k < (uint32_t)kArcStaged ? rel[ warp ][ k ] : neighbour( k );
                            const f3     dk = F3( qk.x, qk.y, qk.z );
                            const float  a  = dot( c, dk );
                            const float  p1 = r * dot( e1, dk ), p2 = r * dot( e2, dk );
                            const float  B  = sqrtf( p1 * p1 + p2 * p2 );
                            // hidden where a + B cos(phi - phi_k) > K_k
                            const float v = ( qk.w - a ) + 4.f * kRel * ( fabsf( a ) + fabsf( qk.w ) + B + 1.f );
                            if ( !( v < B ) )
                                continue;
                            if ( v <= -B )
                            {
                                hidden = ~0ull;
                                break;
                            }
                            const float half = bin_atan2( sqrtf( ( B - v ) * ( B + v ) ), v ) - 1e-3f, mid = bin_atan2( p2, p1 );
                            const int   s0   = (int)ceilf( ( mid - half ) * ( 1.f / kArcStep ) );
                            const int   len  = (int)floorf( ( mid + half ) * ( 1.f / kArcStep ) ) - s0;
                            if ( len >= 64 )
                                hidden = ~0ull;
                            else if ( len > 0 )
                            {
                                const uint64_t m  = ( 1ull << len ) - 1ull;
                                const uint32_t sh = (uint32_t)s0 & 63u;
                                hidden |= ( m << sh ) | ( sh ? m >> ( 64u - sh ) : 0ull );
                            }
                        }
                    }
                    open = ~hidden;
                    if ( hidden && open )
                    {
                        // turned so that no run of open bins passes the end
                        turn = (uint32_t)__ffsll( (long long)hidden );
                        turn &= 63u;
                        open = turn ? ( open >> turn ) | ( open << ( 64u - turn ) ) : open;
                    }
                    most = r > kArcHalf ? max( 1, (int)( 2.f * asinf( kArcHalf / r ) * ( 1.f / kArcStep ) ) ) : 64u;
                    if ( !( r > 0.1f ) )
                        most = 64u;
                }
                // runs of open bins in pieces of at most `most` bins: counted, then written
                auto runs = [ & ]( auto piece ) {
                    uint64_t w = open;
                    while ( w )
                    {
                        const uint32_t s   = (uint32_t)__ffsll( (long long)w ) - 1u;
                        const uint64_t up  = ~( w >> s );
                        const uint32_t len = up ? (uint32_t)__ffsll( (long long)up ) - 1u : 64u;
                        for ( uint32_t o = 0; o < len; o += most )
                            piece( s + o, min( most, len - o ) );
                        w = s + len >= 64u ? 0ull : w & ( ~0ull << ( s + len ) );
                    }
                };
                runs( [ & ]( uint32_t, uint32_t ) { pieces++; } );
                uint32_t total;
                uint32_t at   = warp_exclusive_sum( pieces, total );
                uint32_t base = 0;
                if ( lane == 0 && total )
                    base = atomicAdd( &flags[ 0 ], total );
                at += __shfl_sync( 0xffffffffu, base, 0 );
                runs( [ & ]( uint32_t s, uint32_t len ) {
                    if ( at >= capArcs )
                    {
                        flags[ 2 ] = 1u;
                        at++;
                        return;
                    }
                    const float half = 0.5f * (float)len * kArcStep + 1e-3f;
                    float       h = r, x = 0.f, y = 0.f;
                    if ( half < 1.5f )
                    {
                        float sn, cs, s1, c1;
                        __sincosf( half, &s1, &c1 );
                        __sincosf( ( (float)( ( s + turn ) & 63u ) + 0.5f * (float)len ) * kArcStep, &sn, &cs );
                        h = r * s1;
                        x = r * c1 * cs;
                        y = r * c1 * sn;
                    }
                    if ( !( h + margin < kArcBall ) ) // spheres of tens of A, or coordinates of 10^4 A
                        flags[ 2 ] = 1u;
                    const f3 p  = c + e1 * x + e2 * y;
                    balls[ at ] = make_float4( ai.x + p.x, ai.y + p.y, ai.z + p.z, h + margin );
                    arcs[ at ]  = make_uint2( i, j );
                    at++;
                } );
            }
        }

        struct SdfItems
        {
            const float4 *  balls;
            const float *   queries;
            uint32_t        m, capArcs;
            uint32_t *      count; // per cell; the rank of every item in its cell
            uint32_t *      rank;
            float4 *        pos;
            uint32_t *      id;
        };

        // Counting sort of atoms, probes, arcs and queries into their cells, in two passes: the count
        // (its atomics give every item its rank), and after the scan the placement.
        template<bool kPlace>
        __global__ void __launch_bounds__( 256 ) k_sdf_bin( Build b, SdfIndex ix, SdfItems it )
        {
            const uint32_t I = ix.items == 3u ? min( b.counts->I, b.capProbes ) : 0u, A = min( ix.flags[ 0 ], it.capArcs );
            const uint32_t n0 = b.n, n1 = n0 + I, n2 = n1 + A, total = n2 + it.m;
            for ( uint32_t t = blockIdx.x * blockDim.x + threadIdx.x; t < total; t += gridDim.x * blockDim.x )
            {
                float4   p;
                uint32_t own = t, seg = 0;
                if ( t < n0 )
                {
                    p = b.atoms[ t ];
                    // the sign of the radius marks an atom without any accessible surface (neighbours
                    // present, every circle buried); bit 31 of the id one with every bin of its directions covered too
                    if ( b.visCnt[ t ] == 0 && b.nbrCount[ t ] > 0 )
                    {
                        p.w = -p.w;
                        own |= 0x80000000u;
                    }
                    else if ( ix.open )
                    {
                        const uint4 * o = reinterpret_cast<const uint4 *>( ix.open ) + 2u * (size_t)t;
                        const uint4   u = o[ 0 ], v = o[ 1 ];
                        if ( ( u.x | u.y | u.z | u.w | v.x | v.y | v.z | v.w ) == 0u )
                            own |= 0x80000000u;
                    }
                }
                else if ( t < n1 )
                {
                    own = t - n0;
                    seg = 1;
                    p   = b.probePos[ own ];
                    p.w = 0.f;
                }
                else if ( t < n2 )
                {
                    own = t - n1;
                    seg = 2;
                    p   = it.balls[ own ];
                }
                else
                {
                    own = t - n2;
                    seg = ix.items;
                    p   = make_float4( it.queries[ 3 * (size_t)own ], it.queries[ 3 * (size_t)own + 1 ], it.queries[ 3 * (size_t)own + 2 ], 0.f );
                }
                const int3 c   = fine_cell( ix.grid, p.x, p.y, p.z );
                uint32_t   key = seg * ix.grid.cells + fine_key( ix.grid, c );
                if ( t >= n2 && ix.sub == 8u )
                {
                    const FineGrid & g   = ix.grid;
                    const uint32_t   oct = ( p.x - g.origin.x >= ( (float)c.x + 0.5f ) * g.h ? 1u : 0u ) |
                                         ( p.y - g.origin.y >= ( (float)c.y + 0.5f ) * g.h ? 2u : 0u ) |
                                         ( p.z - g.origin.z >= ( (float)c.z + 0.5f ) * g.h ? 4u : 0u );
                    key = seg * g.cells + fine_key( g, c ) * 8u + oct;
                }
                if ( !kPlace )
                    it.rank[ t ] = atomicAdd( &it.count[ key ], 1u );
                else
                {
                    const uint32_t at = ix.start[ key ] + it.rank[ t ];
                    it.id[ at ]       = own;
                    if ( t < n2 )
                        it.pos[ at ] = p;
                }
            }
        }

        // ---- tile search -----------------------------------------------------------------------
        constexpr int   kTileAtoms = 256;  // atoms around a tile
        constexpr int   kTileItems = 192;  // probes or arcs held at a time
        constexpr float kTileEdge  = 4.f;  // queries of one tile lie within this of its first one

        struct TileSmem
        {
            float4   atom[ kTileAtoms ]; // centre relative to the tile's origin, R
            uint32_t id[ kTileAtoms ];   // sorted atom; bit 31: no accessible direction
            float4   item[ kTileItems ]; // relative position, ball radius
            uint32_t itemId[ kTileItems ];
            uint32_t near[ kTileAtoms / 32 ][ 32 ]; // per query: atoms whose SAS sphere comes within its best distance
            uint32_t rowStart[ 32 ], rowPre[ 33 ];
        };
        union SdfScratch
        {
            SdfSmem  query;
            TileSmem tile;
        };

        // A primitive that can be the nearest: its distance by the general search's expressions (the
        // smaller of a circle's two), SdfKind, and probe, atom or circle (i, j).
        struct SdfCand
        {
            float d;
            int   kind, a, b;
        };
        // the nearest three so far, and the smallest distance of one that found no place
        struct SdfBest
        {
            SdfCand c0, c1, c2;
            float   dropped;
            __device__ __forceinline__ bool holds( int kind, int a, int b ) const
            {
                return ( c0.kind == kind && c0.a == a && c0.b == b ) || ( c1.kind == kind && c1.a == a && c1.b == b ) ||
                       ( c2.kind == kind && c2.a == a && c2.b == b );
            }
            __device__ __forceinline__ void insert( SdfCand n, float tol )
            {
                if ( !( n.d <= c0.d + tol ) || holds( n.kind, n.a, n.b ) )
                    return;
                if ( !( n.d < c2.d ) )
                {
                    dropped = fminf( dropped, n.d );
                    return;
                }
                dropped = fminf( dropped, c2.d );
                c2      = n;
                if ( c2.d < c1.d )
                {
                    const SdfCand t = c1;
                    c1              = c2;
                    c2              = t;
                }
                if ( c1.d < c0.d )
                {
                    const SdfCand t = c0;
                    c0              = c1;
                    c1              = t;
                }
            }
            // the candidates of the G lanes of one query, in all of them
            __device__ __forceinline__ void combine( uint32_t G, float tol )
            {
                for ( uint32_t o = 1; o < G; o <<= 1 )
                {
                    SdfCand n[ 3 ] = { c0, c1, c2 };
                    for ( int k = 0; k < 3; k++ )
                    {
                        n[ k ].d    = __shfl_xor_sync( 0xffffffffu, n[ k ].d, o );
                        n[ k ].kind = __shfl_xor_sync( 0xffffffffu, n[ k ].kind, o );
                        n[ k ].a    = __shfl_xor_sync( 0xffffffffu, n[ k ].a, o );
                        n[ k ].b    = __shfl_xor_sync( 0xffffffffu, n[ k ].b, o );
                    }
                    dropped = fminf( dropped, __shfl_xor_sync( 0xffffffffu, dropped, o ) );
                    for ( int k = 0; k < 3; k++ )
                        insert( n[ k ], tol );
                }
            }
        };

        // q inside the SAS sphere of an atom near the query, other than sorted atoms i0 and i1: 1 yes, 0 no, -1
        // closer to one than float32 tells
        __device__ __noinline__ int tile_hidden( const TileSmem & sm, uint32_t query, uint32_t na, f3 q, float eb, uint32_t i0, uint32_t i1 )
        {
            bool unsure = false;
            for ( uint32_t w = 0; w * 32u < na; w++ )
                for ( uint32_t bits = sm.near[ w ][ query ]; bits; bits &= bits - 1u )
                {
                    const uint32_t k = w * 32u + (uint32_t)__ffs( (int)bits ) - 1u;
                    const float4   p = sm.atom[ k ];
                    const f3       v = F3( q.x - p.x, q.y - p.y, q.z - p.z );
                    const float    m = dot( v, v ) - p.w * p.w;
                    if ( m > eb )
                        continue;
                    const uint32_t id = sm.id[ k ] & 0x7fffffffu;
                    if ( id == i0 || id == i1 )
                        continue;
                    if ( m < -eb )
                        return 1;
                    unsure = true;
                }
            return unsure ? -1 : 0;
        }

        // x's radial projection on the SAS sphere of i (j < 0), or its nearest point on circle (i, j), strictly
        // inside the SAS sphere of one of the query's near atoms: in double precision, against the atoms that
        // the float32 point q does not clear by eb
        __device__ __noinline__ bool near_point_hidden_d( const Build & b, const TileSmem & sm, uint32_t query, uint32_t na, float3 x, int i,
                                                          int j, f3 q, float eb )
        {
            const float4 ai = b.atoms[ i ];
            const double Ri = (double)ai.w + (double)b.rp;
            d3           p;
            if ( j < 0 )
            {
                const d3     w  = D3( (double)x.x - (double)ai.x, (double)x.y - (double)ai.y, (double)x.z - (double)ai.z );
                const double sc = Ri / sqrt( w.x * w.x + w.y * w.y + w.z * w.z );
                p               = D3( (double)ai.x + w.x * sc, (double)ai.y + w.y * sc, (double)ai.z + w.z * sc );
            }
            else
            {
                const float4 aj  = b.atoms[ j ];
                const double Rj  = (double)aj.w + (double)b.rp;
                const d3     d   = D3( (double)aj.x - (double)ai.x, (double)aj.y - (double)ai.y, (double)aj.z - (double)ai.z );
                const double dd  = d.x * d.x + d.y * d.y + d.z * d.z;
                const double tt  = ( Ri * Ri - Rj * Rj + dd ) / ( 2.0 * dd );
                const double r2  = Ri * Ri - tt * tt * dd;
                const double inv = 1.0 / sqrt( dd );
                const d3     n   = D3( d.x * inv, d.y * inv, d.z * inv );
                const d3     c   = D3( (double)ai.x + d.x * tt, (double)ai.y + d.y * tt, (double)ai.z + d.z * tt );
                const d3     w   = D3( (double)x.x - c.x, (double)x.y - c.y, (double)x.z - c.z );
                const double h   = w.x * n.x + w.y * n.y + w.z * n.z;
                const d3     v   = D3( w.x - h * n.x, w.y - h * n.y, w.z - h * n.z );
                const double rho = sqrt( v.x * v.x + v.y * v.y + v.z * v.z );
                if ( !( r2 > 0.0 ) || !( rho > 0.0 ) )
                    return false;
                const double sc = sqrt( r2 ) / rho;
                p               = D3( c.x + v.x * sc, c.y + v.y * sc, c.z + v.z * sc );
            }
            for ( uint32_t w = 0; w * 32u < na; w++ )
                for ( uint32_t bits = sm.near[ w ][ query ]; bits; bits &= bits - 1u )
                {
                    const uint32_t k  = w * 32u + (uint32_t)__ffs( (int)bits ) - 1u;
                    const float4   a  = sm.atom[ k ];
                    const f3       v  = F3( q.x - a.x, q.y - a.y, q.z - a.z );
                    const int      id = (int)( sm.id[ k ] & 0x7fffffffu );
                    if ( !( dot( v, v ) - a.w * a.w > eb ) && id != i && id != j && point_inside_d( b, p, (uint32_t)id ) )
                        return true;
                }
            return false;
        }

        // Of probes p and q at the same float32 distance from x, whether p is taken: where they are as far in double precision too
        // (by symmetry), by their atoms, then as they were found, as the general search does; else p if `lower`.
        __device__ __noinline__ bool probe_first( const Build & b, float3 x, int p, int q, bool lower )
        {
            const d3     xd = D3( (double)x.x, (double)x.y, (double)x.z );
            const d3     u = dsub( D3( b.probePos[ p ] ), xd ), v = dsub( D3( b.probePos[ q ] ), xd );
            const double du = ddot( u, u ), dv = ddot( v, v );
            if ( fabs( du - dv ) > 1e-12 * du )
                return lower;
            const int4 a = b.probeIds[ p ], c = b.probeIds[ q ];
            if ( a.x != c.x )
                return a.x < c.x;
            if ( a.y != c.y )
                return a.y < c.y;
            return a.z != c.z ? a.z < c.z : p < q;
        }

        // slot of target in an ascending neighbour row that holds it
        __device__ __forceinline__ uint32_t slot_of( const uint32_t * row, uint32_t len, uint32_t target )
        {
            uint32_t lo = 0, hi = len;
            while ( lo < hi )
            {
                const uint32_t mid = ( lo + hi ) >> 1;
                if ( row[ mid ] < target )
                    lo = mid + 1;
                else
                    hi = mid;
            }
            return lo;
        }

        // The general search's outcome among up to three candidates that lie within the float32 error of
        // the smallest distance (no other one can matter there): probes first, then atom by atom in the order of
        // ||x - c| - R| (its own projection and circles compete with the distance held so far, strictly), until
        // that bound or the depth of x reaches the distance held. False for a circle around x (x on its axis).
        __device__ __noinline__ bool sdf_decide( const Build & b, float3 x, const SdfCand * cand, int count, float T, float depth, SdfHit & hit )
        {
            float best = T;
            hit.kind   = kSdfClampInside;
            hit.value  = b.rp - T;
            int    atom[ 6 ], other[ 6 ], events = 0;
            float  dl[ 6 ], dlOther[ 6 ], dist[ 6 ];
            float3 q[ 6 ];
            for ( int k = 0; k < count; k++ )
            {
                const SdfCand c = cand[ k ];
                if ( c.kind == kSdfProbe )
                {
                    if ( c.d < best )
                    {
                        const float4 p  = b.probePos[ c.a ];
                        const int4   id = b.probeIds[ c.a ];
                        best            = c.d;
                        hit.kind        = kSdfProbe;
                        hit.a           = id.x;
                        hit.b           = id.y;
                        hit.c           = id.z;
                        hit.q           = make_float3( p.x, p.y, p.z );
                    }
                }
                else if ( c.kind == kSdfSphere )
                {
                    atom[ events ]    = c.a;
                    other[ events ]   = -1;
                    dl[ events ]      = c.d;
                    dlOther[ events ] = 0.f;
                    dist[ events ]    = c.d;
                    q[ events++ ]     = x;
                }
                else if ( c.kind == kSdfCircle )
                {
                    const float4 ci = b.atoms[ c.a ], cj = b.atoms[ c.b ];
                    const float  Ri = ci.w + b.rp, Rj = cj.w + b.rp;
                    const float  di = fabsf( sdf_distance( x, ci ) - Ri ), dj = fabsf( sdf_distance( x, cj ) - Rj );
#pragma unroll 1
                    for ( int e = 0; e < 2; e++ )
                    {
                        const float4 u = e ? cj : ci, o = e ? ci : cj;
                        float        turn;
                        const int    at =
                            sdf_circle_point( x, u, u.w + b.rp, make_float4( o.x, o.y, o.z, o.w + b.rp ), dist[ events ], q[ events ], turn );
                        if ( at == 0 )
                            return false;
                        if ( at < 0 )
                            continue;
                        atom[ events ]    = e ? c.b : c.a;
                        other[ events ]   = e ? c.a : c.b;
                        dl[ events ]      = e ? dj : di;
                        dlOther[ events ] = e ? di : dj;
                        events++;
                    }
                }
            }
            float lastDl   = -1.f;
            int   lastAtom = -1;
            for ( int turn = 0; turn < events; turn++ )
            {
                // the next atom
                int a = -1;
                for ( int e = 0; e < events; e++ )
                    if ( ( dl[ e ] > lastDl || ( dl[ e ] == lastDl && atom[ e ] > lastAtom ) ) &&
                         ( a < 0 || dl[ e ] < dl[ a ] || ( dl[ e ] == dl[ a ] && atom[ e ] < atom[ a ] ) ) )
                        a = e;
                if ( a < 0 || !( dl[ a ] < best ) || !( depth < best ) )
                    break;
                lastDl   = dl[ a ];
                lastAtom = atom[ a ];
                int win  = -1;
                for ( int e = 0; e < events; e++ )
                {
                    if ( atom[ e ] != lastAtom || ( other[ e ] >= 0 && !( dlOther[ e ] < best ) ) || !( dist[ e ] < best ) )
                        continue;
                    if ( win >= 0 && dist[ e ] == dist[ win ] )
                    {
                        // its own projection first, then the circles by lane (slot mod 32), then slot
                        const uint32_t * row = b.nbr + (size_t)lastAtom * b.cap;
                        auto             key = [ & ]( int k ) {
                            if ( other[ k ] < 0 )
                                return 0u;
                            const uint32_t s = slot_of( row, b.nbrCount[ lastAtom ], (uint32_t)other[ k ] );
                            return 1u + ( ( s & 31u ) << 16 | s >> 5 );
                        };
                        if ( key( e ) < key( win ) )
                            win = e;
                    }
                    else if ( win < 0 || dist[ e ] < dist[ win ] )
                        win = e;
                }
                if ( win >= 0 )
                {
                    best     = dist[ win ];
                    hit.kind = other[ win ] < 0 ? kSdfSphere : kSdfCircle;
                    hit.a    = lastAtom;
                    hit.b    = other[ win ];
                    hit.c    = -1;
                    hit.q    = q[ win ];
                }
            }
            hit.value = b.rp - best;
            return true;
        }

        // root of a squared distance for the screens (2 ulp)
        __device__ __forceinline__ float screen_sqrt( float d2 ) { return d2 * rsqrtf( fmaxf( d2, 1e-30f ) ); }

        // Up to eight entries of a byte each, a lane's own: candidates wait there until all lanes of the warp
        // take one together (taken as they are met, in a few lanes at a time, their loops over the
        // atoms near a query ran one after another).
        struct ByteQueue
        {
            unsigned long long w;
            int                n;
            __device__ __forceinline__ void push( uint32_t v ) { w |= (unsigned long long)v << ( 8 * n++ ); }
            __device__ __forceinline__ uint32_t pop()
            {
                const uint32_t v = (uint32_t)w & 255u;
                w >>= 8;
                n--;
                return v;
            }
        };

        __device__ __forceinline__ float warp_min( float v )
        {
            for ( int o = 16; o > 0; o >>= 1 )
                v = fminf( v, __shfl_xor_sync( 0xffffffffu, v, o ) );
            return v;
        }
        __device__ __forceinline__ float warp_max( float v ) { return -warp_min( -v ); }

        // The items of segment seg whose own ball (radius w of an arc; the atoms' w is their radius and counts as
        // none) comes within radius of the box [lo, hi]: number `first` on, at most `cap` of them, to pos
        // (relative to org) and ids in shared memory. Returns how many there are. One copy of this, and of
        // each stage below, in a kernel: inlined wherever a lambda was called, the tile search did not
        // fit the instruction cache (7 of 13 stall cycles of the image, 2 of 9 of the queries).
        __device__ __noinline__ uint32_t tile_gather( const SdfIndex & ix, uint32_t seg, f3 lo, f3 hi, f3 org, float radius, TileSmem & sm,
                                                      float4 * pos, uint32_t * ids, uint32_t first, uint32_t cap )
        {
            const uint32_t   lane = lane_id();
            const FineGrid & g    = ix.grid;
            const float      pad  = radius + ( seg == 2u ? kArcBall : 0.f );
            const int3       c0   = fine_cell( g, lo.x - pad, lo.y - pad, lo.z - pad ), c1 = fine_cell( g, hi.x + pad, hi.y + pad, hi.z + pad );
            const uint32_t   ny = (uint32_t)( c1.y - c0.y + 1 ), rows = ny * (uint32_t)( c1.z - c0.z + 1 );
            const uint32_t * start = ix.start + seg * g.cells;
            uint32_t         held  = 0;
            for ( uint32_t r0 = 0; r0 < rows; r0 += 32 )
            {
                const uint32_t r  = r0 + lane;
                uint32_t       st = 0, len = 0;
                if ( r < rows )
                {
                    // the row's cells within reach of the box (the border cells also hold what lies beyond them)
                    const int   y = c0.y + (int)( r % ny ), z = c0.z + (int)( r / ny );
                    const float y0 = y > 0 ? g.origin.y + (float)y * g.h : -3e38f, y1 = y + 1 < g.dims.y ? g.origin.y + (float)( y + 1 ) * g.h : 3e38f;
                    const float z0 = z > 0 ? g.origin.z + (float)z * g.h : -3e38f, z1 = z + 1 < g.dims.z ? g.origin.z + (float)( z + 1 ) * g.h : 3e38f;
                    const float ey = fmaxf( fmaxf( lo.y - y1, y0 - hi.y ), 0.f ), ez = fmaxf( fmaxf( lo.z - z1, z0 - hi.z ), 0.f );
                    const float w2 = ( pad + 0.01f ) * ( pad + 0.01f ) - ey * ey - ez * ez;
                    if ( w2 >= 0.f )
                    {
                        const float w  = sqrtf( w2 ) + 0.01f;
                        const int   x0 = max( c0.x, min( (int)floorf( ( lo.x - w - g.origin.x ) / g.h ), g.dims.x - 1 ) ),
                                  x1 = min( c1.x, max( (int)floorf( ( hi.x + w - g.origin.x ) / g.h ), 0 ) );
                        if ( x0 <= x1 )
                        {
                            st  = start[ fine_key( g, make_int3( x0, y, z ) ) ];
                            len = start[ fine_key( g, make_int3( x1, y, z ) ) + 1 ] - st;
                        }
                    }
                }
                uint32_t       total;
                const uint32_t pre = warp_exclusive_sum( len, total );
                __syncwarp();
                sm.rowStart[ lane ] = st;
                sm.rowPre[ lane ]   = pre;
                __syncwarp();
                // 64 items at a time, their loads in flight together
                for ( uint32_t f0 = 0; f0 < total; f0 += 64 )
                {
                    float4   p[ 2 ];
                    uint32_t id[ 2 ];
                    bool     keep[ 2 ];
#pragma unroll
                    for ( int h = 0; h < 2; h++ )
                    {
                        const uint32_t f = f0 + 32u * h + lane;
                        p[ h ]           = make_float4( 3e18f, 0.f, 0.f, 0.f );
                        id[ h ]          = 0;
                        if ( f < total )
                        {
                            uint32_t q = 0;
#pragma unroll
                            for ( uint32_t step = 16; step > 0; step >>= 1 )
                                if ( sm.rowPre[ q + step ] <= f )
                                    q += step;
                            const uint32_t at = sm.rowStart[ q ] + ( f - sm.rowPre[ q ] );
                            p[ h ]            = ix.pos[ at ];
                            id[ h ]           = ix.id[ at ];
                        }
                    }
#pragma unroll
                    for ( int h = 0; h < 2; h++ )
                    {
                        const float4 c  = p[ h ];
                        const float  dx = fmaxf( fmaxf( lo.x - c.x, c.x - hi.x ), 0.f ), dy = fmaxf( fmaxf( lo.y - c.y, c.y - hi.y ), 0.f ),
                                    dz = fmaxf( fmaxf( lo.z - c.z, c.z - hi.z ), 0.f );
                        const float reach = radius + ( seg == 2u ? c.w : 0.f );
                        keep[ h ]         = dx * dx + dy * dy + dz * dz <= reach * reach;
                        const uint32_t mk = __ballot_sync( 0xffffffffu, keep[ h ] );
                        const uint32_t at = held + __popc( mk & lanemask_lt() );
                        if ( keep[ h ] && at >= first && at - first < cap )
                        {
                            pos[ at - first ] = make_float4( c.x - org.x, c.y - org.y, c.z - org.z, c.w );
                            ids[ at - first ] = id[ h ];
                        }
                        held += __popc( mk );
                    }
                }
            }
            __syncwarp();
            return held;
        }

        // the atoms within radius of the box, with their SAS radius
        __device__ __noinline__ uint32_t tile_atoms( const SdfIndex & ix, f3 lo, f3 hi, f3 org, float radius, float rp, TileSmem & sm )
        {
            const uint32_t na = tile_gather( ix, 0u, lo, hi, org, radius, sm, sm.atom, sm.id, 0u, kTileAtoms );
            for ( uint32_t k = lane_id(); k < min( na, (uint32_t)kTileAtoms ); k += 32 )
                sm.atom[ k ].w = fabsf( sm.atom[ k ].w ) + rp;
            __syncwarp();
            return na;
        }

        // Signed distance at the query of every lane with `want` (G lanes of the warp, side by side,
        // share one query and give the same x and want); hit valid in all of them. exact: left to the
        // general search. All lanes of the warp call.
        //
        // Every screen is in float32 relative to the tile's origin. tol bounds, generously, the difference
        // between a screened distance and the general search's float32 one (roundings at the size of the
        // coordinates there, of the tile's extent here), and between a lower bound and a distance there: only
        // primitives within tol of the smallest distance bear on the outcome, whatever order the general search
        // examines the atoms in, and sdf_decide settles those.
        __device__ __forceinline__ void sdf_tile_search( const Build & b, const SdfIndex & ix, float3 x, bool want, uint32_t G, TileSmem & sm,
                                                         float band, SdfHit & hit, bool & exact )
        {
            const uint32_t lane = lane_id(), sub = lane & ( G - 1u ), query = lane / G;
            const float    T = b.rp + band, Rmax = ix.rmax + b.rp;
            exact            = false;
            hit.kind         = kSdfClampOutside;
            hit.a = hit.b = hit.c = -1;
            hit.q                 = x;
            hit.value             = band;
            {
                // farther from the grid's box, which holds every centre, than any vdW sphere within the
                // band reaches (or not a number): outside
                const FineGrid & g = ix.grid;
                const float      ux = x.x - g.origin.x, uy = x.y - g.origin.y, uz = x.z - g.origin.z;
                const float      f  = ix.rmax + band + 1.f;
                want = want && ux > -f && uy > -f && uz > -f && ux < (float)g.dims.x * g.h + f && uy < (float)g.dims.y * g.h + f &&
                       uz < (float)g.dims.z * g.h + f;
            }
            float edge = kTileEdge;
            for ( uint32_t pending = __ballot_sync( 0xffffffffu, want ); pending; )
            {
                // the pending queries near the first one
                const int   lead = __ffs( (int)pending ) - 1;
                const float lx = __shfl_sync( 0xffffffffu, x.x, lead ), ly = __shfl_sync( 0xffffffffu, x.y, lead ),
                            lz = __shfl_sync( 0xffffffffu, x.z, lead );
                const bool mine = ( pending >> lane & 1u ) && fabsf( x.x - lx ) <= edge && fabsf( x.y - ly ) <= edge && fabsf( x.z - lz ) <= edge;
                const uint32_t taken = __ballot_sync( 0xffffffffu, mine );
                pending &= ~taken;
                // more atoms around them than shared memory holds: again with a smaller tile, and in the end
                // (a much denser molecule than a protein) by the general search
                auto crowded = [ & ]() {
                    edge *= 0.5f;
                    if ( edge > 0.2f )
                        pending |= taken;
                    else
                    {
                        edge  = kTileEdge;
                        exact = exact || mine;
                    }
                };
                const float inf = __int_as_float( 0x7f800000 );
                const f3    lo  = F3( warp_min( mine ? x.x : inf ), warp_min( mine ? x.y : inf ), warp_min( mine ? x.z : inf ) );
                const f3    hi  = F3( warp_max( mine ? x.x : -inf ), warp_max( mine ? x.y : -inf ), warp_max( mine ? x.z : -inf ) );
                const f3    org = ( lo + hi ) * 0.5f;
                const f3    xr  = F3( x.x - org.x, x.y - org.y, x.z - org.z );
                const float ext = fmaxf( hi.x - lo.x, fmaxf( hi.y - lo.y, hi.z - lo.z ) ) + Rmax + T + 1.f; // largest relative coordinate
                const float far = fmaxf( fmaxf( fmaxf( fabsf( lo.x ), fabsf( hi.x ) ), fmaxf( fabsf( lo.y ), fabsf( hi.y ) ) ),
                                         fmaxf( fabsf( lo.z ), fabsf( hi.z ) ) ) + Rmax + T + 1.f;
                const float tol = 3e-7f * far + 1e-6f * ext;
                const float eb  = 3e-6f * ext * ( Rmax + 1.f ); // band of |q - c|^2 - R^2

                // atoms: the smallest two |x - c| - R
                float    radius = ix.rmax + fmaxf( band, b.rp ) + tol + 0.01f;
                uint32_t na     = tile_atoms( ix, lo, hi, org, radius, b.rp, sm );
                if ( na > (uint32_t)kTileAtoms )
                {
                    crowded();
                    continue;
                }
                float    smin = inf, smin2 = inf;
                int      satom = -1;
                if ( mine )
                    for ( uint32_t k = sub; k < na; k += G )
                    {
                        const float4 p = sm.atom[ k ];
                        const f3     v = F3( xr.x - p.x, xr.y - p.y, xr.z - p.z );
                        const float  s = screen_sqrt( dot( v, v ) ) - p.w;
                        smin2          = fminf( smin2, fmaxf( s, smin ) );
                        satom          = s < smin ? (int)k : satom;
                        smin           = fminf( s, smin );
                    }
                for ( uint32_t o = 1; o < G; o <<= 1 )
                {
                    const float s1 = __shfl_xor_sync( 0xffffffffu, smin, o ), s2 = __shfl_xor_sync( 0xffffffffu, smin2, o );
                    const int   sa = __shfl_xor_sync( 0xffffffffu, satom, o );
                    smin2          = fminf( fminf( smin2, s2 ), fmaxf( smin, s1 ) );
                    satom          = s1 < smin ? sa : satom;
                    smin           = fminf( smin, s1 );
                }
                float depth  = -smin; // of x in the SAS spheres
                bool  inside = false;
                if ( mine && smin < fmaxf( band - b.rp, 0.f ) + tol )
                {
                    const int id = (int)( sm.id[ satom ] & 0x7fffffffu );
                    if ( smin2 > smin + tol )
                    {
                        // one atom has both minima: as the general search takes them
                        const float4 c = b.atoms[ id ];
                        const float  L = sdf_distance( x, c );
                        depth          = ( c.w + b.rp ) - L;
                        hit.a          = id;
                        hit.value      = L - c.w;
                    }
                    else
                    {
                        float s = inf, v = inf;
                        for ( uint32_t k = 0; k < na; k++ )
                        {
                            const float4 p = sm.atom[ k ];
                            const f3     w = F3( xr.x - p.x, xr.y - p.y, xr.z - p.z );
                            if ( screen_sqrt( dot( w, w ) ) - p.w > smin + 2.f * tol )
                                continue;
                            const int    i = (int)( sm.id[ k ] & 0x7fffffffu );
                            const float4 c = b.atoms[ i ];
                            const float  L = sdf_distance( x, c );
                            s              = fminf( s, L - ( c.w + b.rp ) );
                            if ( L - c.w < v || ( L - c.w == v && i < hit.a ) )
                            {
                                v     = L - c.w;
                                hit.a = i;
                            }
                        }
                        depth     = -s;
                        hit.value = v;
                    }
                    inside   = depth > 0.f;
                    hit.kind = kSdfAtom;
                    if ( inside || !( hit.value <= band ) )
                    {
                        hit.kind  = inside ? kSdfClampInside : kSdfClampOutside;
                        hit.a     = -1;
                        hit.value = inside ? b.rp - T : band;
                        inside    = inside && depth < T;
                    }
                }
                if ( !__any_sync( 0xffffffffu, inside ) )
                {
                    edge = kTileEdge;
                    continue;
                }

                // probes (vertices of dE, never hidden)
                SdfBest best;
                best.c0      = { T, kSdfClampInside, -1, -1 };
                best.c1      = { inf, -1, -1, -1 };
                best.c2      = best.c1;
                best.dropped = inf;
                {
                    float d0 = inf, d1 = inf, d2 = inf; // squared distances of the nearest three
                    int   p0 = -1, p1 = -1, p2 = -1;
                    for ( uint32_t first = 0, total = 1; first < total; first += kTileItems )
                    {
                        __syncwarp();
                        total               = tile_gather( ix, 1u, lo, hi, org, T + tol, sm, sm.item, sm.itemId, first, kTileItems );
                        const uint32_t held = min( total - first, (uint32_t)kTileItems );
                        if ( inside )
                            for ( uint32_t k = sub; k < held && total; k += G )
                            {
                                const float4 p = sm.item[ k ];
                                const f3     v = F3( xr.x - p.x, xr.y - p.y, xr.z - p.z );
                                const float  d = dot( v, v );
                                if ( d < d2 )
                                {
                                    const int id = (int)sm.itemId[ k ];
                                    d2           = fmaxf( d, d1 );
                                    p2           = d < d1 ? p1 : id;
                                    p1           = d < d0 ? p0 : ( d < d1 ? id : p1 );
                                    d1           = fmaxf( fminf( d, d1 ), d0 );
                                    p0           = d < d0 ? id : p0;
                                    d0           = fminf( d, d0 );
                                }
                            }
                    }
                    // the general search takes the nearest one, by its own distances where the screened ones do not
                    // tell (a distance carries a few roundings of its own size only); of equal ones as probe_first says
                    const float near = 5e-7f * ext;
                    float       dp   = p0 >= 0 ? sdf_distance( x, b.probePos[ p0 ] ) : inf;
                    if ( screen_sqrt( d1 ) <= dp + near )
                        for ( int e = 0; e < 2; e++ )
                        {
                            const int q = e ? p2 : p1;
                            if ( q < 0 || screen_sqrt( e ? d2 : d1 ) > dp + near )
                                continue;
                            if ( e )
                                best.dropped = 0.f; // (a fourth one would not be seen)
                            const float d = sdf_distance( x, b.probePos[ q ] );
                            if ( d < dp || ( d == dp && probe_first( b, x, q, p0, false ) ) )
                                p0 = q;
                            dp = fminf( d, dp );
                        }
                    for ( uint32_t o = 1; o < G; o <<= 1 )
                    {
                        const float d = __shfl_xor_sync( 0xffffffffu, dp, o );
                        const int   q = __shfl_xor_sync( 0xffffffffu, p0, o );
                        best.dropped  = fminf( best.dropped, __shfl_xor_sync( 0xffffffffu, best.dropped, o ) );
                        if ( d < dp || ( d == dp && q >= 0 && q != p0 && probe_first( b, x, q, p0, q < p0 ) ) )
                            p0 = q;
                        dp = fminf( d, dp );
                    }
                    if ( p0 >= 0 )
                        best.insert( { dp, kSdfProbe, p0, -1 }, tol );
                }

                // per query the atoms that can hold or hide a point of dE: such a point, within the best distance of
                // x, can only lie in a SAS sphere that comes as near
                const float cut  = best.c0.d + tol;
                const float need = Rmax + warp_max( inside ? cut : 0.f ) + 0.01f;
                if ( need > radius )
                {
                    __syncwarp();
                    na = tile_atoms( ix, lo, hi, org, need, b.rp, sm );
                    if ( na > (uint32_t)kTileAtoms )
                    {
                        crowded();
                        continue;
                    }
                }
                for ( uint32_t w = 0; w * 32u < na; w++ )
                {
                    uint32_t bits = 0;
                    if ( inside )
                        for ( uint32_t k = w * 32u + sub; k < min( na, w * 32u + 32u ); k += G )
                        {
                            const float4 p = sm.atom[ k ];
                            const f3     v = F3( xr.x - p.x, xr.y - p.y, xr.z - p.z );
                            const float  r = cut + p.w, d = dot( v, v );
                            bits |= ( d < r * r ? 1u : 0u ) << ( k & 31u );
                        }
                    for ( uint32_t o = 1; o < G; o <<= 1 )
                        bits |= __shfl_xor_sync( 0xffffffffu, bits, o );
                    if ( sub == 0 )
                        sm.near[ w ][ query ] = bits;
                }
                __syncwarp();

                // radial projections on the SAS spheres
                {
                    ByteQueue wait { 0ull, 0 };
                    // a lane's own atoms of every 32: each G-th
                    const uint32_t own = ( G < 32u ? 0xffffffffu / ( ( 1u << G ) - 1u ) : 1u ) << sub;
                    uint32_t       w = 0, left = inside ? 1u : 0u; // left: words to go
                    uint32_t       bits = inside ? sm.near[ 0 ][ query ] & own : 0u;
                    while ( true )
                    {
                        // atoms that may hold the nearest accessible point
                        while ( __any_sync( 0xffffffffu, left != 0u ) && !__any_sync( 0xffffffffu, wait.n == 8 ) )
                        {
                            if ( left && !bits )
                            {
                                w++;
                                left = w * 32u < na ? 1u : 0u;
                                bits = left ? sm.near[ w ][ query ] & own : 0u;
                            }
                            if ( bits )
                            {
                                const uint32_t k  = w * 32u + (uint32_t)__ffs( (int)bits ) - 1u;
                                const uint32_t id = sm.id[ k ];
                                bits &= bits - 1u;
                                if ( !( id >> 31 ) )
                                {
                                    const float4 p  = sm.atom[ k ];
                                    const f3     v  = F3( xr.x - p.x, xr.y - p.y, xr.z - p.z );
                                    const float  L  = screen_sqrt( dot( v, v ) );
                                    const float  dl = fabsf( L - p.w );
                                    // (nothing accessible is nearer than the depth of x)
                                    if ( dl <= best.c0.d + tol && dl >= depth - 2.f * tol &&
                                         ( L < 1e-2f || direction_open( ix.open, id, v ) ) )
                                        wait.push( k );
                                }
                            }
                        }
                        if ( !__any_sync( 0xffffffffu, wait.n > 0 ) )
                            break;
                        // their projections
                        while ( __any_sync( 0xffffffffu, wait.n > 0 ) )
                        {
                            if ( wait.n == 0 )
                                continue;
                            const uint32_t k  = wait.pop();
                            const uint32_t id = sm.id[ k ];
                            const float4   p  = sm.atom[ k ];
                            const f3       v  = F3( xr.x - p.x, xr.y - p.y, xr.z - p.z );
                            const float    L  = screen_sqrt( dot( v, v ) );
                            if ( fabsf( L - p.w ) > best.c0.d + tol )
                                continue;
                            // near its centre the direction of x is not known well enough
                            const float sc = __fdividef( p.w, fmaxf( L, 1e-6f ) );
                            const f3    q  = F3( p.x + v.x * sc, p.y + v.y * sc, p.z + v.z * sc );
                            const int   h  = L > 0.3f ? tile_hidden( sm, query, na, q, eb, id, id ) : -1;
                            if ( h > 0 )
                                continue;
                            const float4 c = b.atoms[ id ];
                            const float  D = sdf_distance( x, c );
                            // (x the centre: the general search takes no projection)
                            if ( D > 0.f && ( h == 0 || !near_point_hidden_d( b, sm, query, na, x, (int)id, -1, q, L > 0.3f ? eb : inf ) ) )
                                best.insert( { fabsf( D - ( c.w + b.rp ) ), kSdfSphere, (int)id, -1 }, tol );
                        }
                    }
                    best.combine( G, tol );
                }

                // accessible arcs
                {
                    ByteQueue met { 0ull, 0 }, wait { 0ull, 0 };
                    // circle of item k: its atoms, the screened distance, the nearest point q and the band of its
                    // accessibility tests (infinite: not known well enough for float32); false where it cannot matter
                    auto geometry = [ & ]( uint32_t k, uint2 & ij, f3 & q, float & ec ) {
                        const float4 p = sm.item[ k ];
                        ij             = ix.arcs[ sm.itemId[ k ] ];
                        if ( best.holds( kSdfCircle, (int)ij.x, (int)ij.y ) )
                            return false;
                        const float4 ci = b.atoms[ ij.x ], cj = b.atoms[ ij.y ];
                        const float  Ri = ci.w + b.rp, Rj = cj.w + b.rp;
                        const f3     d  = F3( cj.x - ci.x, cj.y - ci.y, cj.z - ci.z );
                        const f3     e  = F3( ( ci.x - org.x ) - xr.x, ( ci.y - org.y ) - xr.y, ( ci.z - org.z ) - xr.z ); // c_i - x
                        const float  dd = dot( d, d );
                        const float  tt = __fdividef( Ri * Ri - Rj * Rj + dd, 2.f * dd );
                        const float  r2 = Ri * Ri - tt * tt * dd;
                        q               = xr;
                        ec              = inf;
                        if ( !( r2 > 0.09f ) ) // a small circle: its radius carries the rounding of nearly equal numbers
                            return true;
                        const float r   = screen_sqrt( r2 );
                        const f3    n   = d * rsqrtf( dd );
                        const f3    cc  = e + d * tt; // centre - x
                        const float hh  = dot( cc, n );
                        const f3    u   = n * hh - cc; // from the axis to x
                        const float rho = screen_sqrt( dot( u, u ) );
                        const float ds  = screen_sqrt( hh * hh + ( rho - r ) * ( rho - r ) );
                        if ( ds > best.c0.d + tol || ds < depth - 2.f * tol )
                            return false;
                        if ( !( rho > 0.02f ) )
                            return true;
                        const float sc = __fdividef( r, rho );
                        const f3    w  = cc + u * sc; // q - x
                        // q - ball centre: the point belongs to this piece
                        const f3 o = F3( xr.x + w.x - p.x, xr.y + w.y - p.y, xr.z + w.z - p.z );
                        q          = xr + w;
                        ec         = eb * ( 1.f + 0.2f * sc );
                        return dot( o, o ) <= ( p.w + 1e-3f ) * ( p.w + 1e-3f );
                    };
                    const float reach = warp_max( inside ? best.c0.d + tol : 0.f );
                    for ( uint32_t first = 0, total = 1; first < total; first += kTileItems )
                    {
                        __syncwarp();
                        total               = tile_gather( ix, 2u, lo, hi, org, reach, sm, sm.item, sm.itemId, first, kTileItems );
                        const uint32_t held = total ? min( total - first, (uint32_t)kTileItems ) : 0u;
                        uint32_t       k0   = 0;
                        while ( true )
                        {
                            // pieces whose ball comes near enough
                            for ( ; k0 < held && !__any_sync( 0xffffffffu, met.n == 8 ); k0 += G )
                            {
                                const uint32_t k = k0 + sub;
                                if ( inside && k < held )
                                {
                                    const float4 p   = sm.item[ k ];
                                    const f3     v   = F3( xr.x - p.x, xr.y - p.y, xr.z - p.z );
                                    const float  cut = best.c0.d + tol + p.w;
                                    if ( dot( v, v ) <= cut * cut )
                                        met.push( k );
                                }
                            }
                            // whose circle's nearest point lies in them and near enough
                            while ( __any_sync( 0xffffffffu, met.n > 0 ) && !__any_sync( 0xffffffffu, wait.n == 8 ) )
                                if ( met.n > 0 )
                                {
                                    const uint32_t k = met.pop();
                                    uint2          ij;
                                    f3             q;
                                    float          ec;
                                    if ( geometry( k, ij, q, ec ) )
                                        wait.push( k );
                                }
                            const bool done = k0 >= held && !__any_sync( 0xffffffffu, met.n > 0 );
                            // and is accessible
                            if ( done || __any_sync( 0xffffffffu, wait.n == 8 ) )
                                while ( __any_sync( 0xffffffffu, wait.n > 0 ) )
                                {
                                    uint2 ij;
                                    f3    q;
                                    float ec;
                                    if ( wait.n == 0 || !geometry( wait.pop(), ij, q, ec ) )
                                        continue;
                                    const int h = ec < inf ? tile_hidden( sm, query, na, q, ec, ij.x, ij.y ) : -1;
                                    if ( h > 0 )
                                        continue;
                                    const float4 ci = b.atoms[ ij.x ], cj = b.atoms[ ij.y ];
                                    float        dm = inf;
                                    bool         axis = false;
#pragma unroll 1
                                    for ( int e = 0; e < 2; e++ )
                                    {
                                        const float4 u = e ? cj : ci, o = e ? ci : cj;
                                        float        d, turn;
                                        float3       t;
                                        const int    at = sdf_circle_point( x, u, u.w + b.rp, make_float4( o.x, o.y, o.z, o.w + b.rp ), d, t, turn );
                                        if ( at >= 0 )
                                            dm = fminf( dm, d );
                                        axis |= at == 0;
                                    }
                                    if ( !( dm <= best.c0.d + tol ) )
                                        continue;
                                    if ( axis )
                                        exact = true;
                                    else if ( h == 0 || !near_point_hidden_d( b, sm, query, na, x, (int)ij.x, (int)ij.y, q, ec ) )
                                        best.insert( { dm, kSdfCircle, (int)ij.x, (int)ij.y }, tol );
                                }
                            if ( done )
                                break;
                        }
                    }
                    best.combine( G, tol );
                    for ( uint32_t o = 1; o < G; o <<= 1 )
                        exact |= __shfl_xor_sync( 0xffffffffu, exact ? 1 : 0, o ) != 0;
                }
                if ( inside )
                {
                    if ( best.c0.kind != kSdfCircle && !( best.c1.d <= best.c0.d + tol ) && !( best.dropped <= best.c0.d + tol ) )
                    {
                        hit.kind  = best.c0.kind;
                        hit.value = b.rp - best.c0.d;
                        if ( best.c0.kind == kSdfSphere )
                            hit.a = best.c0.a;
                        else if ( best.c0.kind == kSdfProbe )
                        {
                            const float4 p  = b.probePos[ best.c0.a ];
                            const int4   id = b.probeIds[ best.c0.a ];
                            hit.a           = id.x;
                            hit.b           = id.y;
                            hit.c           = id.z;
                            hit.q           = make_float3( p.x, p.y, p.z );
                        }
                    }
                    else
                    {
                        const SdfCand c[ 3 ] = { best.c0, best.c1, best.c2 };
                        const int     count  = best.c2.d <= best.c0.d + tol ? 3 : ( best.c1.d <= best.c0.d + tol ? 2 : 1 );
                        if ( best.dropped <= best.c0.d + tol || !sdf_decide( b, x, c, count, T, depth, hit ) )
                            exact = true;
                    }
                }
                edge = kTileEdge;
                __syncwarp();
            }
        }

        struct TileHit
        {
            SdfHit   h;
            float3   x;
            uint32_t query;
        };
        static_assert( 32 * sizeof( TileHit ) <= sizeof( TileSmem ), "a warp's hits in its tile's memory" );

        // Queries in cell order, G lanes each (32 / G to a warp's tile); a query left to the general
        // search goes to the list (one in 100,000). Issue- and latency-bound: 15,000 warp instructions a
        // tile of 16 (G = 2) at 22 of 32 lanes, where the general search takes 33,000 a query at 15. 1M queries around a
        // 20,000-atom globule: 38.7 ms with the general search alone, 2.3 ms with this (1.96 ms here, 0.17 the
        // arcs); 4,999 around 2,000 atoms: 489 and 115 us.
        template<bool kBackward>
        __global__ void __launch_bounds__( 32 * kSdfWarps ) k_sdf_tile( Build b, SdfIndex ix, const float * queries, uint32_t m, float band,
                                                                        uint32_t G, float * sdf, const float * gradSdf, float * gradSorted,
                                                                        int * kind, uint32_t * list, uint32_t * listCount )
        {
            __shared__ TileSmem smem[ kSdfWarps ];
            const uint32_t      warp = threadIdx.x >> 5, lane = lane_id();
            const uint32_t      at   = ( blockIdx.x * kSdfWarps + warp ) * ( 32u / G ) + lane / G;
            // (the adjoint's warps meet at the end)
            const bool any = ( blockIdx.x * kSdfWarps + warp ) * ( 32u / G ) < m;
            if ( !kBackward && !any )
                return;
            const bool     want = at < m;
            uint32_t       qi   = 0;
            float3         x    = make_float3( 0.f, 0.f, 0.f );
            if ( want )
            {
                qi = ix.id[ ix.start[ ix.items * ix.grid.cells ] + at ];
                x  = make_float3( queries[ 3 * (size_t)qi ], queries[ 3 * (size_t)qi + 1 ], queries[ 3 * (size_t)qi + 2 ] );
            }
            SdfHit h;
            bool   exact = want;
            if ( any && ix.flags[ 2 ] == 0u )
                sdf_tile_search( b, ix, x, want, G, smem[ warp ], band, h, exact );
            const bool     first = want && ( lane & ( G - 1u ) ) == 0u;
            const uint32_t mk    = __ballot_sync( 0xffffffffu, first && exact );
            uint32_t       base  = 0;
            if ( lane == 0 && mk )
                base = atomicAdd( listCount, (uint32_t)__popc( mk ) );
            base = __shfl_sync( 0xffffffffu, base, 0 );
            if ( first && exact )
                list[ base + __popc( mk & lanemask_lt() ) ] = qi;
            if constexpr ( kBackward )
            {
                // The gradients of the block's queries by as few warps as hold them: a query's terms are ~150 FP64
                // instructions of 64 cycles whatever the lanes hold (200,000 queries at G = 4: 1079 us with 8 lanes of
                // every warp, 935 now). Few queries, whose latency is the time, don't wait for one another (500 atoms, 1000
                // queries: 104 us, 107 with the block's wait).
                bool         mine = first && !exact;
                TileHit      t;
                t.h     = h;
                t.x     = x;
                t.query = qi;
                if ( G <= 8u )
                {
                    __syncwarp();
                    if ( !mine )
                        t.query = 0xffffffffu;
                    if ( ( lane & ( G - 1u ) ) == 0u )
                        reinterpret_cast<TileHit *>( &smem[ warp ] )[ lane / G ] = t;
                    __syncthreads();
                    const uint32_t each = 32u / G;
                    mine                = threadIdx.x < kSdfWarps * each;
                    if ( mine )
                        t = reinterpret_cast<const TileHit *>( &smem[ threadIdx.x / each ] )[ threadIdx.x % each ];
                    mine = mine && t.query != 0xffffffffu;
                }
                if ( mine )
                    sdf_gradient( b, t.h, t.x, gradSdf[ t.query ], gradSorted );
            }
            else if ( first && !exact )
            {
                sdf[ qi ] = h.value;
                if ( kind )
                    kind[ qi ] = h.kind;
            }
        }

        // All m queries by the general search, a warp each, in cell order: the float32 pass; what it leaves open goes
        // to the list. Nothing here calls a function with the build (but for a gradient), and the pass fits 64 registers: eight blocks
        // a SM. Issue-bound (51 % at 15 of 32 lanes). 200,000 queries of 20,001 atoms one of which lies outside the box: 17.7 ms
        // with both passes in one function at six blocks, 10.1 now; 1M atoms, 40,000 queries 3.75 and 2.9 ms.
        template<bool kBackward>
        __global__ void __launch_bounds__( 32 * kSdfWarps, 8 ) k_sdf_general( const __grid_constant__ Build b, const __grid_constant__ SdfIndex ix,
                                                                              const float * queries, uint32_t m, float band, float * sdf,
                                                                              const float * gradSdf, float * gradSorted, int * kind, uint32_t * list,
                                                                              uint32_t * listCount )
        {
            __shared__ SdfSmem smem[ kSdfWarps ];
            const uint32_t     warp = threadIdx.x >> 5, lane = lane_id();
            uint32_t           overflow = 0;
            for ( uint32_t e = blockIdx.x * kSdfWarps + warp; e < m; e += gridDim.x * kSdfWarps )
            {
                const uint32_t qi = ix.id[ ix.start[ ix.items * ix.grid.cells ] + e ];
                const float3   x  = make_float3( queries[ 3 * (size_t)qi ], queries[ 3 * (size_t)qi + 1 ], queries[ 3 * (size_t)qi + 2 ] );
                bool           exact;
                const SdfHit   h = sdf_query_float( b, ix, x, smem[ warp ], band, overflow, exact );
                if ( lane == 0 )
                {
                    if ( exact )
                        list[ atomicAdd( listCount, 1u ) ] = qi;
                    else if ( kBackward )
                        sdf_gradient( b, h, x, gradSdf[ qi ], gradSorted );
                    else
                    {
                        sdf[ qi ] = h.value;
                        if ( kind )
                            kind[ qi ] = h.kind;
                    }
                }
                __syncwarp();
            }
            if ( lane == 0 && overflow )
                atomicOr( &b.counts->overflow, (uint32_t)kOverflowSdfList );
        }

        // The listed queries by the general search in double precision where it takes that, a warp each: the few that the
        // tile search or the float32 pass left open, whose latency counts (1M atoms, 50,000 queries: 46 us less with five blocks
        // a SM, which need no spills, than with eight); and every query where the arcs did not fit, those through float32 first.
        template<bool kBackward>
        __global__ void __launch_bounds__( 32 * kSdfWarps, 5 ) k_sdf_exact( const __grid_constant__ Build b, const __grid_constant__ SdfIndex ix,
                                                                            const float * queries, float band, float * sdf, const float * gradSdf,
                                                                            float * gradSorted, int * kind, const uint32_t * list,
                                                                            const uint32_t * listCount )
        {
            __shared__ SdfSmem smem[ kSdfWarps ];
            const uint32_t     warp = threadIdx.x >> 5, lane = lane_id();
            const uint32_t     count = *listCount;
            const bool         all   = ix.flags[ 2 ] != 0u;
            uint32_t           overflow = 0;
            for ( uint32_t e = blockIdx.x * kSdfWarps + warp; e < count; e += gridDim.x * kSdfWarps )
            {
                const uint32_t qi = list[ e ];
                const float3 x = make_float3( queries[ 3 * (size_t)qi ], queries[ 3 * (size_t)qi + 1 ], queries[ 3 * (size_t)qi + 2 ] );
                SdfHit       h;
                bool         exact = true;
                if ( all )
                {
                    h = sdf_query_float( b, ix, x, smem[ warp ], band, overflow, exact );
                    __syncwarp();
                }
                if ( exact )
                    h = sdf_query_exact( b, ix, x, smem[ warp ], band, overflow );
                if ( lane == 0 )
                {
                    if ( kBackward )
                        sdf_gradient( b, h, x, gradSdf[ qi ], gradSorted );
                    else
                    {
                        sdf[ qi ] = h.value;
                        if ( kind )
                            kind[ qi ] = h.kind;
                    }
                }
                __syncwarp();
            }
            if ( lane == 0 && overflow )
                atomicOr( &b.counts->overflow, (uint32_t)kOverflowSdfList );
        }

        __global__ void k_sdf_unsort( Build b, const float * gradSorted, float * gradInput )
        {
            for ( uint32_t s = blockIdx.x * blockDim.x + threadIdx.x; s < b.n; s += gridDim.x * blockDim.x )
            {
                const uint32_t i = b.perm[ s ];
                for ( int k = 0; k < 4; k++ )
                    gradInput[ 4 * (size_t)i + k ] = gradSorted[ 4 * (size_t)s + k ];
            }
        }

        // ---- headless image: sphere tracing of the signed distance ------------------
        // Every pixel's ray x(t) = eye + t d advances by a step that never crosses the SES:
        // inside the SAS (kinds 3-5) the value rp - dist(x, E) bounds the distance to the SES
        // (every SES point lies at rp from E); outside (kinds 1, 2) value - rp bounds the distance
        // to the SAS, which holds the SES. A ray stops when an inside value falls below eps (a hit
        // at t), when it reaches a point deeper than the band (kind 0, taken as a hit), or when t
        // passes tFar; it advances by at least eps / 4. The ray setup, the march (points eye + t d,
        // steps, t) and the normals are in float32 with every operation rounded on its own, in the
        // order the host tracer writes them, so that the image does not depend on contraction
        // choices. The normal of a hit is the normalised central difference of the signed distance
        // (step normalStep) at the hit point.
        // A warp takes 8 x 4 pixels or fewer (rays_per_warp), a lane each: their rays run close together, so that one tile
        // search serves the warp's points; the few points it leaves go through the general search one
        // after another. Bound by the longest rays: up to maxSteps searches one after another (512 x 512
        // pixels of a 20,000-atom globule: 27.9 ms with a warp and a general search a ray, 12.9 ms).
        // kTiles false: the general search alone, a warp per ray.
        template<bool kTiles>
        __global__ void __launch_bounds__( 32 * kSdfWarps, kTiles ? 4 : 6 ) k_trace( const __grid_constant__ Build b, const __grid_constant__ SdfIndex ix,
                                                                                     const __grid_constant__ TraceParams p, float band,
                                                                                     uint32_t logX, uint32_t logY, float * depth, float * normals )
        {
            __shared__ std::conditional_t<kTiles, SdfScratch, SdfSmem> smem[ kSdfWarps ];
            const uint32_t     warp = threadIdx.x >> 5, lane = lane_id();
            uint32_t           overflow = 0;
            const uint32_t     tilesX   = ( ( p.width - 1u ) >> logX ) + 1u, tiles = tilesX * ( ( ( p.height - 1u ) >> logY ) + 1u );
            // with arcs both kernels are launched: where the pieces fitted, the tiles' takes the image
            if ( ix.open && kTiles == ( ix.flags[ 2 ] != 0u ) )
                return;
            const float3       f        = make_float3( (float)p.forward[ 0 ], (float)p.forward[ 1 ], (float)p.forward[ 2 ] );
            const float3       r        = make_float3( (float)p.right[ 0 ], (float)p.right[ 1 ], (float)p.right[ 2 ] );
            const float3       u        = make_float3( (float)p.up[ 0 ], (float)p.up[ 1 ], (float)p.up[ 2 ] );
            const float3       ef       = make_float3( (float)p.eye[ 0 ], (float)p.eye[ 1 ], (float)p.eye[ 2 ] );
            const float        th       = (float)p.tanHalfFov, W = (float)p.width, H = (float)p.height;
            const float        eps      = (float)p.eps, tFar = (float)p.tFar, hn = (float)p.normalStep;
            const float        minStep  = __fmul_rn( 0.25f, eps );
            for ( uint32_t tile = blockIdx.x * kSdfWarps + warp; tile < tiles; tile += gridDim.x * kSdfWarps )
            {
                const uint32_t at0 = kTiles ? lane : 0u; // pixel of the tile (without tiles all lanes march the one ray)
                const uint32_t px = ( ( tile % tilesX ) << logX ) + ( at0 & ( ( 1u << logX ) - 1u ) ), py = ( ( tile / tilesX ) << logY ) + ( at0 >> logX );
                const bool     mine = at0 < 1u << ( logX + logY ) && px < p.width && py < p.height;
                // pinhole ray through the pixel centre, row-major from the top left
                const float xs  = __fdiv_rn( __fmul_rn( __fmul_rn( __fsub_rn( __fdiv_rn( __fmul_rn( 2.f, __fadd_rn( (float)px, 0.5f ) ), W ), 1.f ),
                                                                  th ),
                                                        W ),
                                             H );
                const float ys  = __fmul_rn( __fsub_rn( 1.f, __fdiv_rn( __fmul_rn( 2.f, __fadd_rn( (float)py, 0.5f ) ), H ) ), th );
                const float dx  = __fadd_rn( __fadd_rn( f.x, __fmul_rn( r.x, xs ) ), __fmul_rn( u.x, ys ) );
                const float dy  = __fadd_rn( __fadd_rn( f.y, __fmul_rn( r.y, xs ) ), __fmul_rn( u.y, ys ) );
                const float dz  = __fadd_rn( __fadd_rn( f.z, __fmul_rn( r.z, xs ) ), __fmul_rn( u.z, ys ) );
                const float len = __fsqrt_rn( __fadd_rn( __fadd_rn( __fmul_rn( dx, dx ), __fmul_rn( dy, dy ) ), __fmul_rn( dz, dz ) ) );
                const float3 df = make_float3( __fdiv_rn( dx, len ), __fdiv_rn( dy, len ), __fdiv_rn( dz, len ) );
                float        t   = (float)p.tNear;
                float        hit = __int_as_float( 0x7f800000 ); // +inf: background
                // Evaluation k of the normal moves the hit point by +hn (k even) or -hn (k odd) along
                // axis k / 2.
                float3   xh = make_float3( 0.f, 0.f, 0.f ), g = make_float3( 0.f, 0.f, 0.f );
                float    vp = 0.f;
                uint32_t step = 0;
                int      k    = mine ? -1 : 6; // -1: marching, 6: done
                while ( true )
                {
                    if ( k < 0 && !( step < p.maxSteps && t <= tFar ) )
                        k = 6;
                    const bool live = k < 6;
                    if ( !__any_sync( 0xffffffffu, live ) )
                        break;
                    float3 q = xh;
                    if ( k < 0 )
                        q = make_float3( __fadd_rn( ef.x, __fmul_rn( t, df.x ) ), __fadd_rn( ef.y, __fmul_rn( t, df.y ) ),
                                         __fadd_rn( ef.z, __fmul_rn( t, df.z ) ) );
                    else
                    {
                        const float e = ( k & 1 ) ? -hn : hn;
                        if ( k < 2 )
                            q.x = __fadd_rn( xh.x, e );
                        else if ( k < 4 )
                            q.y = __fadd_rn( xh.y, e );
                        else
                            q.z = __fadd_rn( xh.z, e );
                    }
                    SdfHit h;
                    if constexpr ( !kTiles )
                    {
                        bool exact;
                        __syncwarp();
                        h = sdf_query_float( b, ix, q, smem[ warp ], band, overflow, exact );
                        __syncwarp();
                        if ( exact )
                            h = sdf_query_exact( b, ix, q, smem[ warp ], band, overflow );
                    }
                    else
                    {
                        bool exact = live;
                        // the rays still live, side by side, with all lanes shared among them (the last rays of a
                        // tile, up to maxSteps steps long, decide when the image is done)
                        const uint32_t rays = __ballot_sync( 0xffffffffu, live ), count = (uint32_t)__popc( rays );
                        uint32_t       G    = 1;
                        while ( count * G * 2u <= 32u )
                            G *= 2u;
                        const uint32_t rank = (uint32_t)__popc( rays & lanemask_lt() );
                        __syncwarp();
                        if ( live )
                            smem[ warp ].tile.rowStart[ rank ] = lane;
                        __syncwarp();
                        const bool     want = lane / G < count;
                        const uint32_t src  = want ? smem[ warp ].tile.rowStart[ lane / G ] : 0u;
                        __syncwarp();
                        const float3 x = make_float3( __shfl_sync( 0xffffffffu, q.x, (int)src ), __shfl_sync( 0xffffffffu, q.y, (int)src ),
                                                      __shfl_sync( 0xffffffffu, q.z, (int)src ) );
                        bool         ex;
                        sdf_tile_search( b, ix, x, want, G, smem[ warp ].tile, band, h, ex );
                        const int from = (int)min( rank * G, 31u );
                        h.kind         = __shfl_sync( 0xffffffffu, h.kind, from );
                        h.value        = __shfl_sync( 0xffffffffu, h.value, from );
                        exact          = __shfl_sync( 0xffffffffu, ex ? 1 : 0, from ) != 0;
                        for ( uint32_t left = __ballot_sync( 0xffffffffu, live && exact ); left; left &= left - 1u )
                        {
                            const int    src = __ffs( (int)left ) - 1;
                            const float3 xs  = make_float3( __shfl_sync( 0xffffffffu, q.x, src ), __shfl_sync( 0xffffffffu, q.y, src ),
                                                            __shfl_sync( 0xffffffffu, q.z, src ) );
                            __syncwarp();
                            const SdfHit hs = sdf_query_exact( b, ix, xs, smem[ warp ].query, band, overflow );
                            __syncwarp();
                            if ( (int)lane == src )
                            {
                                h.kind  = hs.kind;
                                h.value = hs.value;
                            }
                        }
                    }
                    if ( !live )
                        continue;
                    if ( k < 0 )
                    {
                        step++;
                        const bool inside = h.kind == kSdfSphere || h.kind == kSdfCircle || h.kind == kSdfProbe;
                        if ( ( inside && h.value < eps ) || h.kind == kSdfClampInside )
                        {
                            hit = t;
                            // the hit point as the march computed it
                            xh = q;
                            k  = normals ? 0 : 6;
                            continue;
                        }
                        const float st = inside ? h.value : __fsub_rn( h.value, b.rp );
                        t              = __fadd_rn( t, fmaxf( st, minStep ) );
                        continue;
                    }
                    if ( ( k & 1 ) == 0 )
                        vp = h.value;
                    else
                    {
                        const float ga = __fdiv_rn( __fsub_rn( vp, h.value ), __fmul_rn( 2.f, hn ) );
                        if ( k == 1 )
                            g.x = ga;
                        else if ( k == 3 )
                            g.y = ga;
                        else
                            g.z = ga;
                    }
                    k++;
                }
                float3 nrm = make_float3( 0.f, 0.f, 0.f );
                if ( normals && hit < 3.4e38f )
                {
                    const float gl  = __fsqrt_rn( __fadd_rn( __fadd_rn( __fmul_rn( g.x, g.x ), __fmul_rn( g.y, g.y ) ), __fmul_rn( g.z, g.z ) ) );
                    const float inv = gl > 0.f ? gl : 1.f;
                    nrm = make_float3( __fdiv_rn( g.x, inv ), __fdiv_rn( g.y, inv ), __fdiv_rn( g.z, inv ) );
                }
                if ( mine && ( kTiles || lane == 0u ) )
                {
                    const size_t at = (size_t)py * p.width + px;
                    depth[ at ]     = hit;
                    if ( normals )
                    {
                        normals[ 3 * at ]     = nrm.x;
                        normals[ 3 * at + 1 ] = nrm.y;
                        normals[ 3 * at + 2 ] = nrm.z;
                    }
                }
            }
            if ( lane == 0 && overflow )
                atomicOr( &b.counts->overflow, (uint32_t)kOverflowSdfList );
        }
    } // namespace

    namespace
    {
        inline uint32_t blocks_of( uint64_t n, uint32_t threads ) { return (uint32_t)( ( n + threads - 1 ) / threads ); }
        inline size_t   rounded( size_t bytes ) { return ( bytes + 255 ) & ~(size_t)255; }

        // arc pieces held: a protein has ~5 an atom; where more exist every query takes the general search
        uint32_t arc_capacity( uint32_t n ) { return 16u * n + 4096u; }

        // Builds whose queries all take the general search: truncated neighbour lists, atoms outside the box, and
        // SAS spheres or coordinates so large that the ball of an arc piece can pass kArcBall (k_sdf_arcs: half a piece is at most
        // kArcHalf long, or half a bin of the largest circle).
        bool general_build( const Build & b, const SdfState & st )
        {
            const float R    = st.rmax + b.rp;
            const float half = std::max( kArcHalf + 1.1e-3f * R, R * std::sin( 0.5f * kArcStep + 1e-3f ) );
            float       far  = 0.f;
            for ( int a = 0; a < 3; a++ )
            {
                const float lo = ( &b.grid.origin.x )[ a ], hi = lo + ( &b.grid.cell.x )[ a ] * (float)b.grid.size;
                far            = std::max( far, std::max( std::fabs( lo ), std::fabs( hi ) ) );
            }
            return st.truncated || st.outside || !( half + 1e-3f + 1e-6f * far < kArcBall );
        }

        // Cells of half a query's reach over the reference grid's box, coarsened until they fit
        // (a sparse molecule). For few queries of a large molecule, which take the general search, 0.7 of it: fewer cells to zero
        // and to scan (1,000 queries of 1M atoms 729 us with a half, 678 with 0.7, 716 with 1.0); where all of a build's queries take it
        // the half is faster (100,000 of 20,001 atoms 5458 us, 5618 with 0.7).
        void index_grid( const Build & b, const SdfState & st, float band, uint32_t m, uint32_t items, FineGrid & g, uint32_t & sub )
        {
            const double   size = b.grid.size;
            const double   e[ 3 ] = { b.grid.cell.x * size, b.grid.cell.y * size, b.grid.cell.z * size };
            const uint64_t most = std::min<uint64_t>( std::max<uint64_t>( 1u << 18, 24ull * b.n + 4ull * m ), 1u << 28 );
            sub                 = m ? 8u : 0u;
            double h            = ( items == 1u && !general_build( b, st ) ? 0.7 : 0.5 ) * ( st.rmax + 2.0 * b.rp + band );
            int    d[ 3 ]       = { 1, 1, 1 };
            for ( int it = 0; it < 400; it++ )
            {
                for ( int a = 0; a < 3; a++ )
                    d[ a ] = b.n && e[ a ] >= 0.0 && std::isfinite( e[ a ] ) ? (int)std::min( std::max( 1.0, std::ceil( e[ a ] / h ) ), 1e6 ) : 1;
                if ( (uint64_t)d[ 0 ] * d[ 1 ] * d[ 2 ] * ( items + sub ) <= most )
                    break;
                if ( sub == 8u )
                    sub = 1u;
                else
                    h *= 1.1;
            }
            g.origin = b.grid.origin;
            g.h      = (float)h;
            g.dims   = make_int3( d[ 0 ], d[ 1 ], d[ 2 ] );
            g.cells  = (uint32_t)d[ 0 ] * (uint32_t)d[ 1 ] * (uint32_t)d[ 2 ];
            g.span   = 2;
        }

        struct SdfLayout
        {
            size_t flags, balls, arcs, open, count, start, rank, pos, id, list, scan, total;
        };
        SdfLayout layout_of( const Build & b, const FineGrid & g, uint32_t sub, uint32_t kinds, uint32_t m )
        {
            const bool     arcs  = kinds == 3u;
            const uint64_t items = b.n + ( arcs ? (uint64_t)b.capProbes + arc_capacity( b.n ) : 0ull );
            const uint64_t cells = (uint64_t)g.cells * ( kinds + sub );
            SdfLayout      L;
            size_t         p = 0;
            auto           take = [ & ]( size_t bytes ) {
                const size_t at = p;
                p += rounded( bytes );
                return at;
            };
            L.flags = take( 16 );
            L.count = take( cells * 4 ); // zeroed together with the flags
            L.start = take( ( cells + 1 ) * 4 );
            L.balls = take( arcs ? (size_t)arc_capacity( b.n ) * 16 : 0 );
            L.arcs  = take( arcs ? (size_t)arc_capacity( b.n ) * 8 : 0 );
            L.open  = take( arcs ? (size_t)b.n * 32 : 0 );
            L.rank  = take( ( items + m ) * 4 );
            L.pos   = take( items * 16 );
            L.id    = take( ( items + m ) * 4 );
            L.list  = take( (size_t)m * 4 );
            L.scan  = take( scan_scratch_bytes( cells ) );
            L.total = p;
            return L;
        }

        // Builds the index in scratch (arcs: for the tile search): 5 launches for any number of atoms and queries (the grid and the query
        // order were 17, with a radix sort of the queries)
        SdfIndex build_index( const Build & b, const SdfState & st, const float * queries, uint32_t m, bool arcs, bool quarters, float band,
                              void * scratch, uint32_t *& list, uint32_t *& flags, cudaStream_t s )
        {
            SdfIndex ix;
            ix.items = arcs ? 3u : 1u;
            index_grid( b, st, band, m, ix.items, ix.grid, ix.sub );
            const SdfLayout L = layout_of( b, ix.grid, ix.sub, ix.items, m );
            char *          p = static_cast<char *>( scratch );
            flags             = reinterpret_cast<uint32_t *>( p + L.flags );
            list              = reinterpret_cast<uint32_t *>( p + L.list );
            SdfItems it;
            it.balls   = reinterpret_cast<float4 *>( p + L.balls );
            it.queries = queries;
            it.m       = m;
            it.capArcs = arc_capacity( b.n );
            it.count   = reinterpret_cast<uint32_t *>( p + L.count );
            it.rank    = reinterpret_cast<uint32_t *>( p + L.rank );
            it.pos     = reinterpret_cast<float4 *>( p + L.pos );
            it.id      = reinterpret_cast<uint32_t *>( p + L.id );
            uint32_t * start = reinterpret_cast<uint32_t *>( p + L.start );
            ix.outside = st.outside ? 1u : 0u;
            ix.rmax    = st.rmax;
            ix.start   = start;
            ix.pos     = it.pos;
            ix.id      = it.id;
            ix.arcs    = reinterpret_cast<uint2 *>( p + L.arcs );
            ix.flags   = flags;
            ix.open    = arcs ? reinterpret_cast<uint32_t *>( p + L.open ) : nullptr;
            cudaMemsetAsync( p + L.flags, 0, L.start - L.flags, s );
            if ( b.n && arcs )
                k_sdf_arcs<<<blocks_of( b.n, kArcWarps ), 32 * kArcWarps, 0, s>>>( b, reinterpret_cast<float4 *>( p + L.balls ),
                                                                                  reinterpret_cast<uint2 *>( p + L.arcs ), it.capArcs,
                                                                                  reinterpret_cast<uint32_t *>( p + L.open ), quarters, flags );
            const uint32_t blocks = (uint32_t)std::min<uint64_t>( 152u * 8u, blocks_of( 8ull * b.n + m + 1, 256 ) );
            k_sdf_bin<false><<<blocks, 256, 0, s>>>( b, ix, it );
            exclusive_scan( it.count, start, (uint64_t)ix.grid.cells * ( ix.items + ix.sub ), nullptr, nullptr, p + L.scan, s );
            k_sdf_bin<true><<<blocks, 256, 0, s>>>( b, ix, it );
            count_launches( arcs ? 3 : 2 );
            return ix;
        }

        // Lanes per query. Few queries per atom make the tile of a warp wide, so that its lists are long, and few queries
        // leave the GPU idle; more lanes per query make the tile smaller and the walk over its lists shorter, and cost
        // the tile's own work again. Measured over 2,000 to 100,000 atoms and 1,000 to 4,000,000 queries in the molecule's
        // box, the best G falls with m^(2/3) and grows with n^(1/3): 20,000 atoms with 20,000 queries 349 us at G = 16 (377
        // at 8, 353 at 32), with 200,000 queries 850 us at G = 4 (890 at 2, 939 at 8, 1123 at 1); 100,000 atoms with 200,000 queries
        // 1867 us at 8 (2009 at 4, 1952 at 16). One lane and two (values / gradients, us): 2,000 atoms, 250,000 queries 531/573 and
        // 525/633, 500,000 713/822 and 876/1063; 20,000 atoms, 1,000,000 queries 2536/2697 and 2280/2662, 1,500,000
        // 3126/3376 and 3032/3603, 2,000,000 3563/3899 and 3818/4570; 100,000 atoms, 1,500,000 queries 5482/5767 and 5239/5938, 2,000,000
        // 6199/6567 and 6119/7003.
        uint32_t lanes_per_query( uint32_t m, uint32_t n )
        {
            uint32_t G = m < std::min( 150000ull + 60ull * n, 1800000ull ) ? 2u : 1u;
            while ( G < 32u && (double)m * m * G * G * G < 3.2e7 * (double)n )
                G *= 2u;
            return G;
        }
        // the arcs' bins in quarters: worth their pass from about four queries per atom on (20,000 atoms: 60,000 queries 522 us
        // without and 528 with them, 200,000 queries 913 and 850)
        bool quarters_pay( uint32_t m, uint32_t n ) { return m >= 4u * (uint64_t)n; }
        // Pixels of a warp. A warp's time is that of its longest ray, up to maxSteps searches one after another, each
        // of which takes 76k cycles for 8 x 4 rays and 23k for 2 x 2; in all 2 x 2 take more work. 20,000 atoms, 512 x 512 pixels:
        // 12.9 ms with 8 x 4, 13.0 with 8 x 2, 14.0 with 4 x 2, 18.1 with 2 x 2; 384 x 384: 11.7, 8.9, 9.4, 11.2;
        // 256 x 256: 11.5, 8.1, 7.0, 6.7 (2,000 atoms: 7.4, 5.6, 5.8, 5.8); 128 x 128: 10.4, 5.9, 4.2, 3.5
        // (one ray 4.0); 64 x 64: 11.1, 5.5, 4.0, 3.2 (3.0).
        void rays_per_warp( uint64_t pixels, uint32_t & logX, uint32_t & logY )
        {
            logX = pixels >= 3u << 15 ? 3u : pixels >= 3u << 14 ? 2u : pixels >= 3u << 11 ? 1u : 0u;
            logY = pixels >= 3u << 16 ? 2u : pixels >= 3u << 11 ? 1u : 0u;
        }

        // Whether the general search alone, without arcs and tiles, is the faster one. Before its first query the tile
        // search finds the arcs of all atoms and bins these and the probes, 5.6 us per 1000 atoms; of the general
        // search, the latency and the time per query grow with the atoms within reach and their neighbours, that is with a
        // high power of the SAS radius R (of the largest atom; 3.2 A for a protein and a 1.4 A probe). In atoms' worth of arcs the latency is
        // `lat`, a query `per`; a molecule of a few atoms is cheap to search at any radius. Measured over 1 to 1,000,000 atoms, probes of 0.4 to 2.8 A
        // and 1 to 300,000 queries near the surface (general search and tiles, us):
        //   1.4 A:  20,000 atoms, 1 query 311 and 186 (78 and 178 in the molecule's box), 2 queries 349 and 183; 100,000 atoms, 5000 queries
        //           634 and 705, 7000 746 and 725; 300,000 atoms, 20,000 queries 1522 and 2071, 26,000 2136 and 2146;
        //           1,000,000 atoms, 100,000 queries 5579 and 7478, 150,000 8438 and 8131
        //   0.4 A:  tiles / general 1.07 and 0.81 for 5000 and 20,000 queries of 1000 atoms, 1.29 and 0.68 for 80,000 and 300,000 of 20,000
        //   0.7 A:  1.06 and 0.79 for 20,000 and 80,000 queries of 20,000 atoms, 1.19 and 0.79 for 80,000 and 300,000 of 60,000
        //   1.0 A:  1.27 and 0.96 for 64 and 300 queries of 20,000 atoms, 1.25 and 0.95 for 5000 and 20,000 of 60,000
        //   2.0 A:  1.25 and 0.51 for 5000 and 20,000 queries of 200,000 atoms; 2.8 A: 1.05 and 0.80 for 1200 and 5000
        //   10 atoms (any probe): 1.0 to 1.5 and 0.6 to 0.8 for 1200 and 20,000 queries; 1 atom 1.1 to 1.2 and 0.8 for 20,000 and 80,000
        struct SearchCost
        {
            double per, lat;
            bool   cheap; // few atoms within reach of anything
        };
        SearchCost search_cost( float R, uint32_t n )
        {
            const double e = std::pow( std::max( 0.0, (double)R - 2.2 ), 1.5 );
            return { std::pow( (double)R / 3.2, R < 3.2f ? 10.8 : 4.2 ), e, n <= 10u || n * e <= 25.0 };
        }
        bool general_only( uint32_t m, uint32_t n, float R )
        {
            const SearchCost c = search_cost( R, n );
            return 12500ull * m <= n || 8.0 * c.per * m + 55000.0 * c.lat < n || ( c.cheap && m * std::pow( (double)n, 0.6 ) <= 20000.0 );
        }
        // Images of few pixels likewise: by the general search, a warp per ray, and by tiles (1.4 A) 363 and 426 us for one pixel of 20,000
        // atoms (1154 and 1026 for 8 x 8); 100,000 atoms, 64 x 64 pixels 2.79 and 3.12 ms, 128 x 128 7.0 and 5.2; 300,000 atoms,
        // 128 x 128 6.5 and 7.8, 256 x 256 22.6 and 12.5; 1,000,000 atoms, 128 x 128 9.5 and 14.8, 256 x 256 34.0 and 23.9. Cheap searches:
        // tiles / general with a 0.4 A probe 1.1 to 1.5 at 256 x 256 pixels and 0.7 to 0.9 at 512 x 512 (300 to 20,000 atoms), with 0.7 A 1.0 to 1.2
        // and 0.6 to 0.9; 1 atom 1.1 to 2.2 and 0.5 to 0.7.
        bool general_image( uint64_t pixels, uint32_t n, float R )
        {
            const SearchCost c = search_cost( R, n );
            const double     per = R < 3.2f ? c.per : c.per * c.per;
            return 12500ull * pixels <= n || ( 12.0 * per * pixels + 50000.0 * c.lat < n && pixels < 33000u )
                   || ( ( c.cheap || ( R < 2.55f && n <= 30000u ) ) && pixels <= 70000u );
        }
        bool general_search( const Build & b, const SdfState & st, uint32_t m )
        {
            const float R = st.rmax + b.rp;
            return general_build( b, st ) || ( st.pixels ? general_image( st.pixels, b.n, R ) : general_only( m, b.n, R ) );
        }

        template<bool kBackward>
        void launch_search( const Build & b, const SdfState & st, const float * queries, uint32_t m, float band, float * sdf, int * kind,
                            const float * gradSdf, float * gradSorted, void * scratch, cudaStream_t s )
        {
            const uint32_t exactBlocks = std::min( blocks_of( m, kSdfWarps ), 152u * 8u );
            uint32_t *     list, *flags;
            if ( general_search( b, st, m ) )
            {
                const SdfIndex ix = build_index( b, st, queries, m, false, false, band, scratch, list, flags, s );
                // Few queries of a large molecule by warps that go on by themselves (1M atoms, 100,000 queries 5838 us with blocks of four
                // that each wait for the longest, 5579 so); other builds by the blocks (20,000 atoms, 2.9 A probe, 100,000 queries 61.0 and 57.2 ms).
                const uint32_t most = general_build( b, st ) ? 0xffffffffu : 152u * 32u;
                k_sdf_general<kBackward><<<std::min( blocks_of( m, kSdfWarps ), most ), 32 * kSdfWarps, 0, s>>>( b, ix, queries, m, band, sdf, gradSdf, gradSorted, kind,
                                                                                              list, flags + 1 );
                k_sdf_exact<kBackward><<<exactBlocks, 32 * kSdfWarps, 0, s>>>( b, ix, queries, band, sdf, gradSdf, gradSorted, kind, list, flags + 1 );
                count_launches( 2 );
                return;
            }
            const SdfIndex ix = build_index( b, st, queries, m, true, quarters_pay( m, b.n ), band, scratch, list, flags, s );
            const uint32_t G  = lanes_per_query( m, b.n );
            k_sdf_tile<kBackward><<<blocks_of( (uint64_t)m * G, 32 * kSdfWarps ), 32 * kSdfWarps, 0, s>>>( b, ix, queries, m, band, G, sdf, gradSdf,
                                                                                                          gradSorted, kind, list, flags + 1 );
            k_sdf_exact<kBackward><<<exactBlocks, 32 * kSdfWarps, 0, s>>>( b, ix, queries, band, sdf, gradSdf, gradSorted, kind, list, flags + 1 );
            count_launches( 2 );
        }
    } // namespace

    size_t sdf_scratch_bytes( const Build & b, const SdfState & st, uint32_t m )
    {
        FineGrid g;
        uint32_t sub;
        const uint32_t items = general_search( b, st, m ) ? 1u : 3u;
        index_grid( b, st, SESGB_SDF_BAND, m, items, g, sub );
        return layout_of( b, g, sub, items, m ).total;
    }

    void launch_sdf( const Build & b, const SdfState & st, const float * queries, uint32_t m, float band, float * sdf, int * kind,
                     void * scratch, cudaStream_t s )
    {
        if ( m )
            launch_search<false>( b, st, queries, m, band, sdf, kind, nullptr, nullptr, scratch, s );
    }

    void launch_trace( const Build & b, const SdfState & st, const TraceParams & p, float band, float * depth, float * normals,
                       void * scratch, cudaStream_t s )
    {
        if ( !p.width || !p.height )
            return;
        const uint64_t pixels  = st.pixels;
        const bool     general = general_search( b, st, 0 );
        uint32_t *     list, *flags;
        const SdfIndex ix = build_index( b, st, nullptr, 0, !general, pixels >= b.n, band, scratch, list, flags, s );
        if ( !general )
        {
            uint32_t logX, logY;
            rays_per_warp( pixels, logX, logY );
            const uint64_t tiles = (uint64_t)( ( ( p.width - 1u ) >> logX ) + 1u ) * ( ( ( p.height - 1u ) >> logY ) + 1u );
            k_trace<true><<<(uint32_t)std::min<uint64_t>( blocks_of( tiles, kSdfWarps ), 152u * 64u ), 32 * kSdfWarps, 0, s>>>( b, ix, p, band, logX,
                                                                                                                             logY, depth, normals );
            count_launches( 1 );
        }
        k_trace<false><<<(uint32_t)std::min<uint64_t>( blocks_of( pixels, kSdfWarps ), 152u * 32u ), 32 * kSdfWarps, 0, s>>>( b, ix, p, band, 0, 0, depth,
                                                                                                                           normals );
        count_launches( 1 );
    }

    void launch_sdf_backward( const Build & b, const SdfState & st, const float * queries, uint32_t m, float band, const float * gradSdf,
                              float * gradSorted, float * gradInput, void * scratch, cudaStream_t s )
    {
        cudaMemsetAsync( gradSorted, 0, sizeof( float ) * 4 * (size_t)b.n, s );
        if ( m )
            launch_search<true>( b, st, queries, m, band, nullptr, nullptr, gradSdf, gradSorted, scratch, s );
        if ( b.n )
        {
            k_sdf_unsort<<<blocks_of( b.n, 256 ), 256, 0, s>>>( b, gradSorted, gradInput );
            count_launches( 1 );
        }
    }
} // namespace sesgb
