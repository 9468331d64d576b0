// sesgb_area.cu -- solvent-excluded surface area of the primitives of a
// full-surface build, and its adjoint with respect to the atoms.
//
// The reference renders its primitives and computes no area; the area here is
// the area of those primitives: the convex patch of every atom (the directions
// of its SAS sphere outside every other SAS sphere of N(i), scaled to the vdW
// sphere: the sectors of buildConvexPatchesSectors, operations.inl:175-228),
// the torus swept over the accessible arcs of every circle (the segments and
// full circles, operations.inl:552-668), trimmed at its axis when it
// self-intersects, and the concave triangle of every probe (operations.inl:
// 230-486) outside the spheres of its listed neighbour probes
// (findIntersectionsNeighbors, operations.cu:271-338).
//
// Every patch is a region R = {y : |y| = 1, y . w_m <= c_m} of a sphere. By
// Gauss-Bonnet its area is 2 pi chi + sum_m c_m dphi_m - sum_v theta_v, with
// dphi_m the angle of circle m on the boundary of R and theta_v the turning
// angle at a corner. Cut into three lunes of 120 degrees around z, every piece
// has area < 2 pi, so the sum reduced mod 2 pi is the area and the Euler
// characteristic is never needed. The corner terms are written per arc, as the
// change of the boundary tangent's angle against a fixed frame field between the
// arc's ends, so that no corner has to be matched with the arc on its other side
// (several circles through one point, as at the axis points of a self-intersecting
// torus, need no special case, and float32 rounding moves the sum only by as much
// as it moves the arcs). Adjoint: dA/dc_m = dphi_m,
// dA/dw_m = -integral of y over the boundary arcs of m; an arc's angle moves with
// the circles that bound its ends; probe positions follow their atoms by the
// implicit function of |p - c_a|^2 = R_a^2.
//
// Work split: a warp per region (an atom's sphere, a probe with neighbour probes). Its lanes
// first look over the circles, one each, and keep the few whose arcs the others do not hide
// together (6 of ~37 for an atom of a globule); then, circle by circle, over the cuts of the
// kept ones and over their ends; the arcs found wait in shared memory until a warp's worth of
// them is there for their angle terms. A probe without neighbour probes is a plain
// triangle, a thread each.
#include "sesgb_device.cuh"
#include "sesgb_stages.cuh"

namespace sesgb
{
    namespace
    {
        constexpr float    kPiF       = 3.14159265358979f;
        constexpr float    k2PiF      = 6.28318530717959f;
        constexpr int      kAreaWarps = 2;
        constexpr int      kAreaNbr   = 128;             // neighbour constraints of one atom region
        constexpr int      kAreaIv    = 64;              // cuts of one constraint circle
        constexpr int      kLuneIv    = kAreaNbr + 2;    // cuts of one lune-plane circle
        constexpr int      kAreaArcs  = 232;             // arcs that wait for their terms: 32 a pass, and one circle's most (3 x 66)
        constexpr int      kProbeCons = 3 + (int)kMaxProbeNbr;
        // |tw| below which a torus arc end's angle terms are taken in double precision: its float32
        // position carries rounding ~1e-7 / |tw|, and the terms go as 1 / tw
        constexpr float kShallowCrossing = 0.1f;
        static_assert( kMaxProbeNbr <= 32, "one neighbour cap per lane" );

        struct Circ
        {
            f3    w, e1, e2;
            float c, s;
        };

        // reduces an angle in (-4 pi, 6 pi) to [0, 2 pi)
        __device__ __forceinline__ float wrapf( float a )
        {
            if ( a < 0.f )
                a += k2PiF;
            if ( a < 0.f )
                a += k2PiF;
            if ( a >= k2PiF )
                a -= k2PiF;
            if ( a >= k2PiF )
                a -= k2PiF;
            return a;
        }

        __device__ __forceinline__ Circ circ_of( float4 k )
        {
            Circ         C;
            C.w            = F3( k.x, k.y, k.z );
            C.c            = k.w;
            C.s            = sqrtf( fmaxf( 0.f, ( 1.f - k.w ) * ( 1.f + k.w ) ) );
            const float ax = fabsf( k.x ), ay = fabsf( k.y ), az = fabsf( k.z );
            const f3    t  = ( ax <= ay && ax <= az ) ? F3( 1.f, 0.f, 0.f ) : ( ay <= az ? F3( 0.f, 1.f, 0.f ) : F3( 0.f, 0.f, 1.f ) );
            C.e1           = normalize( cross( C.w, t ) );
            C.e2           = cross( C.w, C.e1 );
            return C;
        }

        // y . w <= 0 bounding lune L (side 0: the plane at 2 pi L / 3, side 1: the next one)
        __device__ __forceinline__ float4 lune_cons( int L, int side )
        {
            float sn, cs;
            sincosf( ( k2PiF / 3.f ) * (float)( L + side ), &sn, &cs );
            return side == 0 ? make_float4( sn, -cs, 0.f, 0.f ) : make_float4( -sn, cs, 0.f, 0.f );
        }

        // Circle C against constraint k (k.w < 1): 0 no cut, 1 a cut (p1, p2, B, rhs: its ends), 2 all of it cut
        __device__ __forceinline__ int cut_test( const Circ & C, float4 k, float & p1, float & p2, float & B, float & rhs )
        {
            const f3 wn = F3( k.x, k.y, k.z );
            p1          = dot( C.e1, wn );
            p2          = dot( C.e2, wn );
            B           = C.s * sqrtf( p1 * p1 + p2 * p2 );
            rhs         = k.w - C.c * dot( C.w, wn );
            if ( !( B > fabsf( rhs ) ) )
                return rhs < 0.f ? 2 : 0;
            return 1;
        }

        // Forbidden arc of circle C under constraint k: 0 none, 1 [start, start + len), 2 all of it.
        __device__ __forceinline__ int cut_of( const Circ & C, float4 k, float & start, float & len )
        {
            if ( !( k.w < 1.f ) )
                return 0;
            float     p1, p2, B, rhs;
            const int r = cut_test( C, k, p1, p2, B, rhs );
            if ( r == 1 )
            {
                const float delta = atan2f( sqrtf( ( B - rhs ) * ( B + rhs ) ), rhs );
                start             = wrapf( atan2f( p2, p1 ) - delta );
                len               = 2.f * delta;
            }
            return r;
        }

        __device__ __forceinline__ f3 point_at( const Circ & C, float phi )
        {
            float sn, cs;
            sincosf( phi, &sn, &cs );
            return C.w * C.c + ( C.e1 * cs + C.e2 * sn ) * C.s;
        }

        // frame field xi(y) = a - (a . y) y, singular only at +-a (a generic direction)
        __device__ __forceinline__ float frame_angle( f3 y, f3 t )
        {
            const f3    a  = F3( 0.32140077f, 0.55410134f, 0.76790185f );
            const float ay = dot( a, y );
            const f3    xi = a - y * ay;
            return atan2f( dot( cross( xi, t ), y ), dot( xi, t ) );
        }

        // tangent-angle change against the frame field along the arc [st, st + ln] of C,
        // traversed with the region on its left (decreasing phi: the cap lies towards w)
        __device__ __forceinline__ float arc_turn( const Circ & C, float st, float ln )
        {
            float s0, c0, s1, c1;
            sincosf( st + ln, &s0, &c0 );
            sincosf( st, &s1, &c1 );
            const f3 y0 = C.w * C.c + ( C.e1 * c0 + C.e2 * s0 ) * C.s, t0 = C.e1 * s0 - C.e2 * c0;
            const f3 y1 = C.w * C.c + ( C.e1 * c1 + C.e2 * s1 ) * C.s, t1 = C.e1 * s1 - C.e2 * c1;
            return frame_angle( y1, t1 ) - frame_angle( y0, t0 );
        }

        // A warp's work area for one region.
        struct RegionSmem
        {
            // cuts of the circle at hand (and of its three lunes at kLuneIv + 2 lune + side): start, length,
            // rounded end, re-measured length, constraint
            float    s[ kLuneIv + 6 ], l[ kLuneIv + 6 ], ev[ kLuneIv + 6 ], el[ kLuneIv + 6 ];
            uint16_t n[ kLuneIv + 6 ];
            int      lune[ 6 ]; // cut_of each lune plane
            // arcs that wait: start, length, circle (M + 2 lune + side: a lune plane's), bounding constraints, lune
            float    st[ kAreaArcs ], ln[ kAreaArcs ];
            uint32_t who[ kAreaArcs ]; // m, na + 1, nb + 1, lune: a byte each
            uint8_t  live[ kAreaNbr ];
        };

        // The circles of region cons[0, M) that may have allowed arcs, in order, to live; returns how many, -1
        // where one cap holds the whole sphere. A lane per circle: it is gone when another cap holds all of it
        // (or an equal constraint comes first), and hidden when the others' cuts, each less a margin far
        // above the float32 error of its ends, cover every one of 64 bins of its angle: then every end
        // of a cut lies inside another one and the walk over them would find no arc.
        __device__ int live_circles( const float4 * cons, int M, uint8_t * live, uint32_t & overflow )
        {
            constexpr float kBins = 64.f / k2PiF;
            const int       lane  = (int)lane_id();
            bool            empty = false;
            for ( int m = lane; m < M; m += 32 )
                if ( !( cons[ m ].w > -1.f ) )
                    empty = true;
            if ( __any_sync( 0xffffffffu, empty ) )
                return -1;
            int count = 0;
            for ( int m0 = 0; m0 < M; m0 += 32 )
            {
                const int m    = m0 + lane;
                bool      keep = false;
                if ( m < M && cons[ m ].w < 1.f )
                {
                    const float4 km     = cons[ m ];
                    const Circ   C      = circ_of( km );
                    uint64_t     hidden = 0;
                    int          cuts   = 0;
                    keep                = true;
                    for ( int n = 0; n < M; n++ )
                    {
                        const float4 k = cons[ n ];
                        if ( n == m || !( k.w < 1.f ) )
                            continue;
                        if ( k.x == km.x && k.y == km.y && k.z == km.z && k.w == km.w )
                        {
                            keep = keep && n > m; // the same constraint twice: the first keeps the circle
                            if ( !keep )
                                break;
                            continue;
                        }
                        float     p1, p2, B, rhs;
                        const int r = cut_test( C, k, p1, p2, B, rhs );
                        if ( r == 2 )
                        {
                            keep = false;
                            break;
                        }
                        if ( r == 0 )
                            continue;
                        if ( cuts++ >= kAreaIv )
                            overflow = 1;
                        const float half = bin_atan2( sqrtf( ( B - rhs ) * ( B + rhs ) ), rhs ) - 1e-3f, mid = bin_atan2( p2, p1 );
                        const int   b0   = (int)ceilf( ( mid - half ) * kBins );
                        const int   len  = (int)floorf( ( mid + half ) * kBins ) - b0;
                        if ( len >= 64 )
                            hidden = ~0ull;
                        else if ( len > 0 )
                        {
                            const uint64_t w  = ( 1ull << len ) - 1ull;
                            const uint32_t sh = (uint32_t)b0 & 63u;
                            hidden |= ( w << sh ) | ( sh ? w >> ( 64u - sh ) : 0ull );
                        }
                        if ( !~hidden && M <= kAreaIv )
                            break; // (a longer list goes on to its count of cuts)
                    }
                    keep = keep && ~hidden;
                }
                const uint32_t mk = __ballot_sync( 0xffffffffu, keep );
                if ( keep )
                    live[ count + __popc( mk & lanemask_lt() ) ] = (uint8_t)m;
                count += __popc( mk );
            }
            __syncwarp();
            return count;
        }

        static_assert( 31 + 3 * ( kAreaIv + 2 ) <= kAreaArcs, "a circle's arcs fit behind those that wait" );

        // One region of the unit sphere, held by a warp: constraints cons[0, M) in shared memory.
        // per_arc(m, C, start, len, na, nb) is called for every allowed arc of an original circle, in
        // the lane that has the circle (na, nb: the constraints whose cuts bound it, M and M + 1 a lune's planes, -1 for a whole circle).
        // The circles are cut into the three lunes; with kArea the lune planes' own circles join them and the area is
        // returned (all lanes), without, 0 is returned.
        // Corners need no partner: the arcs that meet at a corner share its point, so their frame
        // angles add up to its turning angle. An end strictly inside another cut is covered (lengths re-measured
        // from the rounded ends, so that equal ends compare equal); of equal uncovered ends the first one counts.
        template<bool kArea, class PerArc>
        __device__ float region_area_warp( const float4 * cons, int M, RegionSmem & W, uint32_t & overflow, PerArc per_arc )
        {
            const int lane = (int)lane_id();
            const int live = live_circles( cons, M, W.live, overflow );
            if ( live < 0 )
                return 0.f;
            float tot[ 3 ] = { 0.f, 0.f, 0.f };
            int   arcs     = 0;
            auto  circle   = [ & ]( int m ) { return circ_of( m < M ? cons[ m ] : lune_cons( ( m - M ) >> 1, ( m - M ) & 1 ) ); };
            const int circles = live + ( kArea ? 6 : 0 );
            for ( int t = 0; t <= circles; t++ )
            {
                if ( t == circles || arcs >= 32 )
                {
                    // the terms of the waiting arcs, a circle's in one lane and in order: its sums round alike
                    // every time
                    __syncwarp();
                    for ( int q0 = lane; q0 < arcs; q0 += 32 )
                    {
                        const int m = (int)( W.who[ q0 ] & 255u );
                        if ( q0 > 0 && (int)( W.who[ q0 - 1 ] & 255u ) == m )
                            continue;
                        const Circ C = circle( m );
                        for ( int q = q0; q < arcs && (int)( W.who[ q ] & 255u ) == m; q++ )
                        {
                            const uint32_t who = W.who[ q ];
                            const int      na = (int)( who >> 8 & 255u ) - 1, lune = (int)( who >> 24 );
                            const float    st = W.st[ q ], ln = W.ln[ q ];
                            if ( kArea )
                            {
                                const float add = na < 0 ? C.c * k2PiF : C.c * ln + arc_turn( C, st, ln );
                                tot[ 0 ] += lune == 0 ? add : 0.f;
                                tot[ 1 ] += lune == 1 ? add : 0.f;
                                tot[ 2 ] += lune == 2 ? add : 0.f;
                            }
                            if ( m < M )
                                per_arc( m, C, st, ln, na, (int)( who >> 16 & 255u ) - 1 );
                        }
                    }
                    arcs = 0;
                    __syncwarp();
                    if ( t == circles )
                        break;
                }
                const bool plane = t >= live;
                const int  m     = plane ? M + ( t - live ) : (int)W.live[ t ];
                const Circ C     = circle( m );
                // its cuts by the other constraints (a lune plane's: and by the lune's other plane)
                const int    most = plane ? kLuneIv : kAreaIv;
                const float4 km   = plane ? make_float4( 0.f, 0.f, 0.f, 2.f ) : cons[ m ];
                int          nIv  = 0;
                bool         gone = false;
                for ( int n0 = 0; n0 < M + ( plane ? 1 : 0 ); n0 += 32 )
                {
                    const int n  = n0 + lane;
                    float     st = 0.f, ln = 0.f;
                    int       r  = 0;
                    if ( n < M + ( plane ? 1 : 0 ) && ( plane || n != m ) )
                    {
                        const float4 k = n < M ? cons[ n ] : lune_cons( ( m - M ) >> 1, 1 - ( ( m - M ) & 1 ) );
                        if ( !( k.x == km.x && k.y == km.y && k.z == km.z && k.w == km.w ) )
                            r = cut_of( C, k, st, ln );
                    }
                    gone |= r == 2;
                    const uint32_t mk = __ballot_sync( 0xffffffffu, r == 1 );
                    const int      at = nIv + __popc( mk & lanemask_lt() );
                    if ( r == 1 && at < most )
                    {
                        W.s[ at ]  = st;
                        W.l[ at ]  = ln;
                        W.ev[ at ] = wrapf( st + ln );
                        const float len2 = wrapf( W.ev[ at ] - st );
                        W.el[ at ] = len2 >= 0.5f * ln ? len2 : ln;
                        W.n[ at ]  = (uint16_t)n;
                    }
                    nIv += __popc( mk );
                }
                if ( nIv > most )
                {
                    overflow = 1;
                    nIv      = most;
                }
                if ( __any_sync( 0xffffffffu, gone ) )
                    continue;
                // and, for an original circle, by the planes of every lune
                const bool split = !plane;
                if ( split && lane < 6 )
                {
                    float     st = 0.f, ln = 0.f;
                    const int at   = kLuneIv + lane;
                    W.lune[ lane ] = cut_of( C, lune_cons( lane >> 1, lane & 1 ), st, ln );
                    W.s[ at ]      = st;
                    W.l[ at ]      = ln;
                    W.ev[ at ]     = wrapf( st + ln );
                    const float len2 = wrapf( W.ev[ at ] - st );
                    W.el[ at ]     = len2 >= 0.5f * ln ? len2 : ln;
                    W.n[ at ]      = (uint16_t)( M + ( lane & 1 ) );
                }
                __syncwarp();
                // the ends of all cuts, lune after lune, a lane each
                int first[ 4 ];
                first[ 0 ] = 0;
                bool whole[ 3 ];
                for ( int L = 0; L < 3; L++ )
                {
                    const bool use = split ? W.lune[ 2 * L ] != 2 && W.lune[ 2 * L + 1 ] != 2 : L == 0;
                    const int  cnt = !use ? 0 : nIv + ( split ? ( W.lune[ 2 * L ] == 1 ) + ( W.lune[ 2 * L + 1 ] == 1 ) : 0 );
                    whole[ L ]     = use && cnt == 0;
                    first[ L + 1 ] = first[ L ] + cnt;
                }
                const int own = plane ? ( m - M ) >> 1 : 0; // the lune of a plane's arcs
                for ( int i0 = 0; i0 < max( first[ 3 ], 1 ); i0 += 32 )
                {
                    const int it   = i0 + lane;
                    bool      arc  = false;
                    float     end = 0.f, gap = k2PiF;
                    int       na = -1, nb = -1, L = 0;
                    if ( it < first[ 3 ] )
                    {
                        L            = it < first[ 1 ] ? 0 : ( it < first[ 2 ] ? 1 : 2 );
                        const int cnt = first[ L + 1 ] - first[ L ], a = it - first[ L ];
                        // entry k of the lune's cuts: the circle's, then those of its planes
                        auto at = [ & ]( int k ) {
                            return k < nIv ? k : kLuneIv + 2 * L + ( k > nIv || W.lune[ 2 * L ] != 1 ? 1 : 0 );
                        };
                        auto covered = [ & ]( float e, int self ) {
                            for ( int k = 0; k < cnt; k++ )
                            {
                                const int x = at( k );
                                if ( k != self && wrapf( e - W.s[ x ] ) < W.el[ x ] )
                                    return true;
                            }
                            return false;
                        };
                        end = W.ev[ at( a ) ];
                        arc = !covered( end, a );
                        // an equal end of an earlier uncovered cut already walks this gap
                        for ( int k = 0; k < a && arc; k++ )
                            if ( W.ev[ at( k ) ] == end )
                                arc = covered( end, k );
                        if ( arc )
                        {
                            na = W.n[ at( a ) ];
                            for ( int k = 0; k < cnt; k++ )
                            {
                                const int   x = at( k );
                                const float g = wrapf( W.s[ x ] - end );
                                if ( g > 0.f && ( nb < 0 || g < gap ) )
                                {
                                    gap = g;
                                    nb  = W.n[ x ];
                                }
                            }
                            arc = nb >= 0;
                        }
                    }
                    // a circle without cuts in a lune is one arc
                    if ( i0 == 0 && lane >= 29 && it >= first[ 3 ] && whole[ lane - 29 ] )
                    {
                        arc = true;
                        L   = lane - 29;
                    }
                    const uint32_t mk = __ballot_sync( 0xffffffffu, arc );
                    const int      to = arcs + __popc( mk & lanemask_lt() );
                    if ( arc )
                    {
                        W.st[ to ] = end;
                        W.ln[ to ] = gap;
                        W.who[ to ] = (uint32_t)m | (uint32_t)( na + 1 ) << 8 | (uint32_t)( nb + 1 ) << 16 | (uint32_t)( plane ? own : L ) << 24;
                    }
                    arcs += __popc( mk );
                }
                __syncwarp();
            }
            if ( !kArea )
                return 0.f;
            float area = 0.f;
            for ( int L = 0; L < 3; L++ )
            {
                float t = tot[ L ];
                for ( int o = 16; o > 0; o >>= 1 )
                    t += __shfl_xor_sync( 0xffffffffu, t, o );
                // the sum spans many turns: reduce it with a full modulo
                float r = fmodf( t, k2PiF );
                if ( r < 0.f )
                    r += k2PiF;
                if ( r > 5.f * kPiF / 3.f )
                    r -= k2PiF; // a piece of (nearly) zero area
                area += fmaxf( r, 0.f );
            }
            return area;
        }

        // integral of y over the arc [st, st + ln] of C
        __device__ __forceinline__ f3 arc_integral( const Circ & C, float st, float ln )
        {
            float s0, c0, s1, c1;
            sincosf( st, &s0, &c0 );
            sincosf( st + ln, &s1, &c1 );
            return C.w * ( C.c * ln ) + ( C.e1 * ( s1 - s0 ) - C.e2 * ( c1 - c0 ) ) * C.s;
        }

        // Pair constraint of atom i and neighbour j: w = D / d, c = (R_i^2 - R_j^2 + d^2) / (2 d R_i).
        struct PairGeo
        {
            f3    D;
            float d, Ri, Rj;
        };
        __device__ __forceinline__ float4 pair_cons( const PairGeo & p )
        {
            if ( !( p.d > 0.f ) )
                return make_float4( 0.f, 0.f, 1.f, 2.f ); // coincident centres: ignored
            const f3 w = p.D * ( 1.f / p.d );
            return make_float4( w.x, w.y, w.z, ( p.Ri * p.Ri - p.Rj * p.Rj + p.d * p.d ) / ( 2.f * p.d * p.Ri ) );
        }

        // toroidal patch per unit angle (rp times the integral of max(0, rho - rp cos beta)
        // over [beta_i, beta_j]) and its derivatives by (d, R_i, R_j)
        __device__ __forceinline__ float torus_F( float d, float Ri, float Rj, float rp, float dF[ 3 ] )
        {
            const float hi = ( Ri * Ri - Rj * Rj + d * d ) / ( 2.f * d ), hj = d - hi;
            const float rr = Ri * Ri - hi * hi;
            dF[ 0 ] = dF[ 1 ] = dF[ 2 ] = 0.f;
            if ( !( rr > 0.f ) )
                return 0.f;
            const float rho = sqrtf( rr );
            const float bi = -atan2f( hi, rho ), bj = atan2f( hj, rho );
            float       F  = rho * ( bj - bi ) - rp * ( hj / Rj + hi / Ri );
            float       Fr = ( bj - bi ) - rho * ( hj / ( Rj * Rj ) + hi / ( Ri * Ri ) )
                       + rp * rho * ( hj / ( Rj * Rj * Rj ) + hi / ( Ri * Ri * Ri ) );
            const float Fhi = ( rho * rho / ( Ri * Ri ) ) * ( 1.f - rp / Ri );
            const float Fhj = ( rho * rho / ( Rj * Rj ) ) * ( 1.f - rp / Rj );
            if ( rho < rp && hi > 0.f && hj > 0.f )
            {
                const float b0 = acosf( rho / rp );
                F -= 2.f * rho * b0 - 2.f * rp * sqrtf( ( 1.f - rho / rp ) * ( 1.f + rho / rp ) );
                Fr -= 2.f * b0;
            }
            const float rd = -hi * hj / ( d * rho ), rRi = Ri * hj / ( d * rho ), rRj = Rj * hi / ( d * rho );
            dF[ 0 ] = rp * ( Fr * rd + Fhi * ( hj / d ) + Fhj * ( hi / d ) );
            dF[ 1 ] = rp * ( Fr * rRi + Fhi * ( Ri / d ) - Fhj * ( Ri / d ) );
            dF[ 2 ] = rp * ( Fr * rRj - Fhi * ( Rj / d ) + Fhj * ( Rj / d ) );
            return rp * F;
        }

        __device__ __forceinline__ void add4( float * g, uint32_t a, f3 v, float r )
        {
            atomicAdd( g + 4 * (size_t)a + 0, v.x );
            atomicAdd( g + 4 * (size_t)a + 1, v.y );
            atomicAdd( g + 4 * (size_t)a + 2, v.z );
            if ( r != 0.f )
                atomicAdd( g + 4 * (size_t)a + 3, r );
        }

        // Pair constraint (w, c) of atom i and neighbour atom j in double precision, from the float32 atoms.
        __device__ __forceinline__ void pair_cons_d( float4 ai, float4 aj, double rp, d3 & w, double & c )
        {
            const d3     D  = D3( (double)aj.x - (double)ai.x, (double)aj.y - (double)ai.y, (double)aj.z - (double)ai.z );
            const double d  = sqrt( ddot( D, D ) );
            const double Ri = (double)ai.w + rp, Rj = (double)aj.w + rp;
            w               = dmul( D, 1.0 / d );
            c               = ( Ri * Ri - Rj * Rj + d * d ) / ( 2.0 * d * Ri );
        }

        // Angle part of the torus of circle m at one arc end where circle m crosses the plane of
        // constraint nn at a small angle (|tw| small): there the end's float32 position, and so tw
        // and 1 / tw, carry rounding magnified by the shallow crossing. The end is taken again in
        // double precision as the point of circle m on that plane (the one on the side of the
        // float32 end), with both constraints recomputed from the atoms, and its terms are formed
        // in double precision (coef = Gs / tw; Gs = -G or G by the end): out = gc[nn], gw[nn],
        // gc[m], gw[m].
        __device__ __noinline__ void arc_end_terms_d( const Build & b, uint32_t i, uint32_t jm, uint32_t jn, f3 yf, float Gs,
                                                      double out[ 8 ] )
        {
            const float4 ai = b.atoms[ i ];
            d3           wm, wn;
            double       cm, cn;
            pair_cons_d( ai, b.atoms[ jm ], (double)b.rp, wm, cm );
            pair_cons_d( ai, b.atoms[ jn ], (double)b.rp, wn, cn );
            const double g   = ddot( wm, wn );
            const double den = 1.0 - g * g;
            for ( int k = 0; k < 8; k++ )
                out[ k ] = 0.0;
            if ( !( den > 0.0 ) )
                return;
            const double al = ( cm - g * cn ) / den, be = ( cn - g * cm ) / den;
            const d3     nv = dcross( wm, wn );
            double       g2 = ( 1.0 - ( al * al + be * be + 2.0 * al * be * g ) ) / den;
            g2              = g2 > 0.0 ? g2 : 0.0;
            const double ga = ( (double)yf.x * nv.x + (double)yf.y * nv.y + (double)yf.z * nv.z ) < 0.0 ? -sqrt( g2 ) : sqrt( g2 );
            const d3     y  = dadd( dadd( dmul( wm, al ), dmul( wn, be ) ), dmul( nv, ga ) );
            const d3     yc = dsub( y, dmul( wm, cm ) );
            const double tw = ddot( dcross( wm, yc ), wn );
            if ( !( fabs( tw ) > 0.0 ) )
                return;
            const double coef = (double)Gs / tw;
            const double sm2  = 1.0 - cm * cm;
            out[ 0 ]          = coef;
            out[ 1 ] = -coef * y.x, out[ 2 ] = -coef * y.y, out[ 3 ] = -coef * y.z;
            out[ 4 ]          = -coef * ( g - ( cm / sm2 ) * ddot( yc, wn ) );
            const d3 gwm      = dmul( dsub( dmul( wn, cm ), dmul( yc, g ) ), -coef );
            out[ 5 ] = gwm.x, out[ 6 ] = gwm.y, out[ 7 ] = gwm.z;
        }

        struct AreaSums // of the adjoint: per constraint, integral of y, and the terms of (c, w) from arc ends
        {
            float4 iy[ kAreaNbr ];
            float  gc[ kAreaNbr ];
            float4 gw[ kAreaNbr ];
        };
        struct AreaSmem
        {
            float4 cons[ kAreaNbr ];
            float  dphi[ kAreaNbr ];
            float  dist[ kAreaNbr ];
            float  Rn[ kAreaNbr ];
            RegionSmem region;
        };

        // Warp per atom: convex patch and the tori of its circles (i, j), i < j. Latency- and issue-bound (12 of
        // 32 lanes, 26,000 warp instructions an atom); with the cuts of a lane's own circle in local memory and
        // every circle walked it was 3.44 ms for 20,000 atoms (4.84 with the adjoint) and is 0.75 (1.28).
        // parts (double[3]) accumulate convex, toroidal (and concave in k_area_probes);
        // atomArea (input order) receives convex + half of each torus. With kGrad,
        // gradSorted (float4 per sorted atom) accumulates gConvex d convex + gTorus d tori.
        template<bool kGrad>
        __global__ void __launch_bounds__( 32 * kAreaWarps ) k_area_atoms( Build b, double * parts, float * atomArea,
                                                                             float gConvex, float gTorus, float * gradSorted )
        {
            __shared__ AreaSmem sm[ kAreaWarps ];
            __shared__ AreaSums sums[ kGrad ? kAreaWarps : 1 ];
            const uint32_t      warp = threadIdx.x >> 5, lane = lane_id();
            AreaSmem &          S    = sm[ warp ];
            AreaSums &          A    = sums[ kGrad ? warp : 0 ];
            double              convexSum = 0.0, torusSum = 0.0;
            uint32_t            overflow = 0;
            for ( uint32_t i = blockIdx.x * kAreaWarps + warp; i < b.n; i += gridDim.x * kAreaWarps )
            {
                const float4   ai = b.atoms[ i ];
                const float    Ri = ai.w + b.rp, ri = ai.w;
                const uint32_t ni = b.nbrCount[ i ];
                const size_t   row = (size_t)i * b.cap;
                // an atom whose circles are all buried has no accessible patch
                bool open = false;
                for ( uint32_t s = lane; s < ni; s += 32 )
                    open |= b.status[ row + s ] != 0;
                if ( ni > 0 && !__any_sync( 0xffffffffu, open ) )
                    continue;
                if ( ni > (uint32_t)kAreaNbr )
                {
                    overflow = 1;
                    continue;
                }
                const int M = (int)ni;
                for ( int m = (int)lane; m < M; m += 32 )
                {
                    const float4 aj = b.atoms[ b.nbr[ row + m ] ];
                    PairGeo      p;
                    p.D          = F3( aj.x - ai.x, aj.y - ai.y, aj.z - ai.z );
                    p.d          = sqrtf( dot( p.D, p.D ) );
                    p.Ri         = Ri;
                    p.Rj         = aj.w + b.rp;
                    S.cons[ m ]  = pair_cons( p );
                    S.dist[ m ]  = p.d;
                    S.Rn[ m ]    = p.Rj;
                    S.dphi[ m ]  = 0.f;
                    if ( kGrad )
                    {
                        A.iy[ m ] = make_float4( 0.f, 0.f, 0.f, 0.f );
                        A.gc[ m ] = 0.f;
                        A.gw[ m ] = make_float4( 0.f, 0.f, 0.f, 0.f );
                    }
                }
                __syncwarp();
                const float U = region_area_warp<true>( S.cons, M, S.region, overflow, [ & ]( int m, const Circ & C, float st, float ln, int na, int nb ) {
                    S.dphi[ m ] += ln;
                    if ( !kGrad )
                        return;
                    const f3 I = arc_integral( C, st, ln );
                    A.iy[ m ].x += I.x, A.iy[ m ].y += I.y, A.iy[ m ].z += I.z;
                    const uint32_t j = b.nbr[ row + m ];
                    if ( !( j > i ) || !( S.dist[ m ] > 0.f ) )
                        return;
                    // angle part of the torus of (i, j): its arc ends move with the circles
                    float       dF[ 3 ];
                    const float G = gTorus * torus_F( S.dist[ m ], Ri, S.Rn[ m ], b.rp, dF );
                    for ( int e = 0; e < 2; e++ )
                    {
                        const int nn = e == 0 ? na : nb;
                        if ( nn < 0 || nn >= M )
                            continue; // whole circle, or a cut between lunes
                        const float  phi = e == 0 ? st : st + ln;
                        const f3     y   = point_at( C, phi );
                        const f3     yc  = y - C.w * C.c;
                        const float4 kn  = S.cons[ nn ];
                        const f3     wn  = F3( kn.x, kn.y, kn.z );
                        const float  tw  = dot( cross( C.w, yc ), wn );
                        if ( fabsf( tw ) < kShallowCrossing )
                        {
                            double t[ 8 ];
                            arc_end_terms_d( b, i, j, b.nbr[ row + nn ], y, e == 0 ? -G : G, t );
                            atomicAdd( &A.gc[ nn ], (float)t[ 0 ] );
                            atomicAdd( &A.gw[ nn ].x, (float)t[ 1 ] );
                            atomicAdd( &A.gw[ nn ].y, (float)t[ 2 ] );
                            atomicAdd( &A.gw[ nn ].z, (float)t[ 3 ] );
                            atomicAdd( &A.gc[ m ], (float)t[ 4 ] );
                            atomicAdd( &A.gw[ m ].x, (float)t[ 5 ] );
                            atomicAdd( &A.gw[ m ].y, (float)t[ 6 ] );
                            atomicAdd( &A.gw[ m ].z, (float)t[ 7 ] );
                            continue;
                        }
                        const float coef = ( e == 0 ? -G : G ) / tw;
                        const float wwn  = dot( C.w, wn );
                        atomicAdd( &A.gc[ nn ], coef );
                        atomicAdd( &A.gw[ nn ].x, -coef * y.x );
                        atomicAdd( &A.gw[ nn ].y, -coef * y.y );
                        atomicAdd( &A.gw[ nn ].z, -coef * y.z );
                        const f3 gwm = ( wn * C.c - yc * wwn ) * ( -coef );
                        atomicAdd( &A.gc[ m ], -coef * ( wwn - ( C.c / ( C.s * C.s ) ) * dot( yc, wn ) ) );
                        atomicAdd( &A.gw[ m ].x, gwm.x );
                        atomicAdd( &A.gw[ m ].y, gwm.y );
                        atomicAdd( &A.gw[ m ].z, gwm.z );
                    }
                } );
                __syncwarp();
                float mine = 0.f, tori = 0.f;
                f3    gi   = F3( 0.f, 0.f, 0.f );
                float gRi  = 0.f;
                for ( int m = (int)lane; m < M; m += 32 )
                {
                    const uint32_t j = b.nbr[ row + m ];
                    if ( j > i && S.dphi[ m ] > 0.f && S.dist[ m ] > 0.f )
                    {
                        float       dF[ 3 ];
                        const float F = torus_F( S.dist[ m ], Ri, S.Rn[ m ], b.rp, dF );
                        const float T = F * S.dphi[ m ];
                        tori += T;
                        mine += 0.5f * T;
                        if ( atomArea )
                            atomicAdd( atomArea + b.perm[ j ], 0.5f * T );
                        if ( kGrad )
                        {
                            const float4 k  = S.cons[ m ];
                            const f3     w  = F3( k.x, k.y, k.z );
                            const float  gs = gTorus * S.dphi[ m ];
                            add4( gradSorted, j, w * ( gs * dF[ 0 ] ), gs * dF[ 2 ] );
                            gi  = gi - w * ( gs * dF[ 0 ] );
                            gRi += gs * dF[ 1 ];
                        }
                    }
                    if ( kGrad && S.dist[ m ] > 0.f )
                    {
                        // convex part and the angle parts gathered above, through (w, c) of the pair
                        const float4 k   = S.cons[ m ];
                        const f3     w   = F3( k.x, k.y, k.z );
                        const float  d   = S.dist[ m ], Rj = S.Rn[ m ];
                        const float  gc  = A.gc[ m ] + gConvex * ri * ri * S.dphi[ m ];
                        const f3     gw  = F3( A.gw[ m ].x, A.gw[ m ].y, A.gw[ m ].z ) - F3( A.iy[ m ].x, A.iy[ m ].y, A.iy[ m ].z ) * ( gConvex * ri * ri );
                        const float  dcd = 1.f / ( 2.f * Ri ) - ( Ri * Ri - Rj * Rj ) / ( 2.f * d * d * Ri );
                        const float  dcRi = ( Ri * Ri + Rj * Rj - d * d ) / ( 2.f * d * Ri * Ri );
                        const float  dcRj = -Rj / ( d * Ri );
                        const f3     gD   = ( gw - w * dot( gw, w ) ) * ( 1.f / d ) + w * ( gc * dcd );
                        add4( gradSorted, j, gD, gc * dcRj );
                        gi  = gi - gD;
                        gRi += gc * dcRi;
                    }
                }
                for ( int o = 16; o > 0; o >>= 1 )
                {
                    mine += __shfl_xor_sync( 0xffffffffu, mine, o );
                    tori += __shfl_xor_sync( 0xffffffffu, tori, o );
                    if ( kGrad )
                    {
                        gi.x += __shfl_xor_sync( 0xffffffffu, gi.x, o );
                        gi.y += __shfl_xor_sync( 0xffffffffu, gi.y, o );
                        gi.z += __shfl_xor_sync( 0xffffffffu, gi.z, o );
                        gRi += __shfl_xor_sync( 0xffffffffu, gRi, o );
                    }
                }
                const float cA = ri * ri * U;
                if ( lane == 0 )
                {
                    convexSum += cA;
                    torusSum += tori;
                    if ( atomArea )
                        atomicAdd( atomArea + b.perm[ i ], cA + mine );
                    if ( kGrad )
                        add4( gradSorted, i, gi, gRi + gConvex * 2.f * ri * U );
                }
                __syncwarp();
            }
            if ( lane == 0 )
            {
                if ( parts && convexSum != 0.0 )
                    atomicAdd( parts + 0, convexSum );
                if ( parts && torusSum != 0.0 )
                    atomicAdd( parts + 1, torusSum );
            }
            overflow = __any_sync( 0xffffffffu, overflow != 0 );
            if ( lane == 0 && overflow )
                atomicOr( &b.counts->overflow, (uint32_t)kOverflowArea );
        }

        // ---- double-precision twin of a probe region's adjoint ------------------------------
        // A neighbour probe closer than kCloseProbe makes a cap of nearly a hemisphere whose terms
        // go as 1 / L (L the distance of the two probes): the float32 arc integrals' rounding shows
        // there. Such a region's adjoint is taken again in double precision: the same constraints
        // from the float32 probe positions and atoms, every constraint's allowed arcs (the gaps
        // between its cuts by the others; the lune split of the area does not change their sums),
        // and the same terms as the float32 path.
        constexpr float kCloseProbe = 0.5f;

        struct dcons
        {
            double x, y, z, w;
        };
        __device__ __forceinline__ dcons dcons_of( double x, double y, double z, double w ) { return { x, y, z, w }; }

        constexpr int kPairsD = 160; // cuts held at a time, of whole circles (at most 34 each)
        struct RegionSmemD
        {
            dcons    kd[ kProbeCons ];   // constraints
            dcons    sums[ kProbeCons ]; // allowed-arc integrals of y, and lengths
            dcons    e1[ kProbeCons ], e2[ kProbeCons ]; // frame and radius (e1.w) of the kept circles
            double   s[ kPairsD ], l[ kPairsD ], ev[ kPairsD ], el[ kPairsD ];
            uint8_t  pm[ kPairsD ], pn[ kPairsD ];
            uint8_t  from[ kProbeCons + 1 ]; // first cut of the circles at hand
            uint32_t gone[ 2 ];              // circles at hand that another cap holds
        };

        // angle in (-2 pi, 4 pi) to [0, 2 pi)
        __device__ __forceinline__ double wrap2pi_d( double a )
        {
            const double k2Pi = 2.0 * 3.14159265358979323846;
            a                 = a < 0.0 ? a + k2Pi : a;
            return a >= k2Pi ? a - k2Pi : a;
        }

        // Allowed-arc lengths and integrals of y over the kept circles (live, of live_circles) of the region
        // D.kd[0, M), to D.sums. The cuts of several circles share the lanes: the trigonometry in double
        // precision is what this costs, and a circle has ~8 cuts among ~12 constraints. Which pairs may cut
        // is screened in float32 with a margin.
        __device__ void region_arcs_d( const float4 * cons, int M, const uint8_t * live, int count, RegionSmemD & D )
        {
            const int    lane = (int)lane_id();
            const double k2Pi = 2.0 * 3.14159265358979323846;
            for ( int t = lane; t < count; t += 32 )
            {
                const dcons  k  = D.kd[ live[ t ] ];
                const d3     wm = D3( k.x, k.y, k.z );
                const double ax = fabs( wm.x ), ay = fabs( wm.y ), az = fabs( wm.z );
                const d3     u  = ( ax <= ay && ax <= az ) ? D3( 1.0, 0.0, 0.0 ) : ( ay <= az ? D3( 0.0, 1.0, 0.0 ) : D3( 0.0, 0.0, 1.0 ) );
                d3           e1 = dcross( wm, u );
                e1              = dmul( e1, 1.0 / sqrt( ddot( e1, e1 ) ) );
                const d3 e2     = dcross( wm, e1 );
                D.e1[ t ]       = dcons_of( e1.x, e1.y, e1.z, sqrt( ( 1.0 - k.w ) * ( 1.0 + k.w ) ) );
                D.e2[ t ]       = dcons_of( e2.x, e2.y, e2.z, 0.0 );
            }
            __syncwarp();
            for ( int t0 = 0; t0 < count; )
            {
                // circles t0 .. t1 - 1 with their cuts
                int pairs = 0, t1 = t0;
                if ( lane < 2 )
                    D.gone[ lane ] = 0u;
                for ( ; t1 < count && pairs + 34 <= kPairsD; t1++ )
                {
                    const int    m  = live[ t1 ];
                    const float4 km = cons[ m ];
                    const Circ   C  = circ_of( km );
                    if ( lane == 0 )
                        D.from[ t1 - t0 ] = (uint8_t)pairs;
                    for ( int n0 = 0; n0 < M; n0 += 32 )
                    {
                        const int n    = n0 + lane;
                        bool      near = false;
                        if ( n < M && n != m && cons[ n ].w < 1.f )
                        {
                            float p1, p2, B, rhs;
                            cut_test( C, cons[ n ], p1, p2, B, rhs );
                            near = rhs < B + 1e-4f; // cuts, or holds the circle
                        }
                        const uint32_t mk = __ballot_sync( 0xffffffffu, near );
                        const int      at = pairs + __popc( mk & lanemask_lt() );
                        if ( near )
                        {
                            D.pm[ at ] = (uint8_t)t1;
                            D.pn[ at ] = (uint8_t)n;
                        }
                        pairs += __popc( mk );
                    }
                }
                if ( lane == 0 )
                    D.from[ t1 - t0 ] = (uint8_t)pairs;
                __syncwarp();
                for ( int q = lane; q < pairs; q += 32 )
                {
                    const int    t = D.pm[ q ], m = live[ t ], n = D.pn[ q ];
                    const dcons  a = D.kd[ m ], c = D.kd[ n ], f1 = D.e1[ t ], f2 = D.e2[ t ];
                    const d3     wm = D3( a.x, a.y, a.z ), wn = D3( c.x, c.y, c.z );
                    double       len = -1.0, st = 0.0; // no cut
                    if ( wn.x == wm.x && wn.y == wm.y && wn.z == wm.z && c.w == a.w )
                    {
                        if ( n < m ) // the same constraint twice: the first one keeps the circle
                            atomicOr( &D.gone[ ( t - t0 ) >> 5 ], 1u << ( ( t - t0 ) & 31 ) );
                    }
                    else
                    {
                        const double p1 = ddot( D3( f1.x, f1.y, f1.z ), wn ), p2 = ddot( D3( f2.x, f2.y, f2.z ), wn );
                        const double B = f1.w * sqrt( p1 * p1 + p2 * p2 ), rhs = c.w - a.w * ddot( wm, wn );
                        if ( B > fabs( rhs ) )
                        {
                            const double delta = atan2( sqrt( ( B - rhs ) * ( B + rhs ) ), rhs );
                            st                 = wrap2pi_d( atan2( p2, p1 ) - delta );
                            len                = 2.0 * delta;
                        }
                        else if ( rhs < 0.0 ) // the whole circle lies inside cap n
                            atomicOr( &D.gone[ ( t - t0 ) >> 5 ], 1u << ( ( t - t0 ) & 31 ) );
                    }
                    D.s[ q ]  = st;
                    D.l[ q ]  = len;
                    D.ev[ q ] = wrap2pi_d( st + len );
                    const double len2 = wrap2pi_d( D.ev[ q ] - st );
                    D.el[ q ] = len2 >= 0.5 * len ? len2 : len;
                }
                __syncwarp();
                // the ends, a lane each, and the circles without a cut
                for ( int q = lane; q < pairs + ( t1 - t0 ); q += 32 )
                {
                    const int t  = q < pairs ? (int)D.pm[ q ] : t0 + ( q - pairs );
                    const int q0 = D.from[ t - t0 ], q1 = D.from[ t - t0 + 1 ], m = live[ t ];
                    if ( D.gone[ ( t - t0 ) >> 5 ] >> ( ( t - t0 ) & 31 ) & 1u )
                        continue;
                    const dcons k   = D.kd[ m ], f1 = D.e1[ t ], f2 = D.e2[ t ];
                    const d3    wm  = D3( k.x, k.y, k.z );
                    double      gap = k2Pi;
                    d3          iy;
                    if ( q < pairs )
                    {
                        if ( D.l[ q ] < 0.0 )
                            continue;
                        const double end     = D.ev[ q ];
                        auto         covered = [ & ]( int self ) {
                            for ( int c = q0; c < q1; c++ )
                                if ( c != self && D.l[ c ] >= 0.0 && wrap2pi_d( end - D.s[ c ] ) < D.el[ c ] )
                                    return true;
                            return false;
                        };
                        bool skip = covered( q );
                        for ( int c = q0; c < q && !skip; c++ )
                            skip = D.l[ c ] >= 0.0 && D.ev[ c ] == end && !covered( c );
                        if ( skip )
                            continue;
                        bool any = false;
                        for ( int c = q0; c < q1; c++ )
                        {
                            const double g = wrap2pi_d( D.s[ c ] - end );
                            if ( D.l[ c ] >= 0.0 && g > 0.0 && ( !any || g < gap ) )
                            {
                                gap = g;
                                any = true;
                            }
                        }
                        if ( !any )
                            continue;
                        double s0, c0, s1, c1;
                        sincos( end, &s0, &c0 );
                        sincos( end + gap, &s1, &c1 );
                        iy = dadd( dmul( wm, k.w * gap ), dmul( dsub( dmul( D3( f1.x, f1.y, f1.z ), s1 - s0 ), dmul( D3( f2.x, f2.y, f2.z ), c1 - c0 ) ), f1.w ) );
                    }
                    else
                    {
                        bool cut = false;
                        for ( int c = q0; c < q1; c++ )
                            cut |= D.l[ c ] >= 0.0;
                        if ( cut )
                            continue;
                        iy = dmul( wm, k.w * k2Pi );
                    }
                    atomicAdd( &D.sums[ m ].x, iy.x );
                    atomicAdd( &D.sums[ m ].y, iy.y );
                    atomicAdd( &D.sums[ m ].z, iy.z );
                    atomicAdd( &D.sums[ m ].w, gap );
                }
                __syncwarp();
                t0 = t1;
            }
        }

        // The warp's probe p (a region with a nearly coincident neighbour): its adjoint terms in
        // double precision into gradSorted (contact directions) and probeGrad (probe positions).
        // cons: the region's constraints in float32.
        __device__ __noinline__ void probe_region_grad_d( const Build & b, uint32_t p, float gConcave, float * gradSorted,
                                                          float4 * probeGrad, const float4 * cons, uint8_t * live,
                                                          uint32_t & overflow, RegionSmemD & D )
        {
            dcons * kd = D.kd, * sums = D.sums;
            const uint32_t lane = lane_id();
            const double   rp   = (double)b.rp;
            const int4     id   = b.probeIds[ p ];
            const float4   pf   = b.probePos[ p ];
            const d3       P    = D3( (double)pf.x, (double)pf.y, (double)pf.z );
            const int      ia[ 3 ] = { id.x, id.y, id.z };
            d3             v[ 3 ];
            double         Lv[ 3 ];
            for ( int a = 0; a < 3; a++ )
            {
                const float4 c = b.atoms[ ia[ a ] ];
                const d3     D = D3( (double)c.x - P.x, (double)c.y - P.y, (double)c.z - P.z );
                Lv[ a ]        = sqrt( ddot( D, D ) );
                v[ a ]         = dmul( D, 1.0 / Lv[ a ] );
            }
            d3     u[ 3 ];
            double ul[ 3 ], sg[ 3 ];
            bool   flat = false;
            for ( int e = 0; e < 3; e++ )
            {
                u[ e ]            = dcross( v[ e ], v[ ( e + 1 ) % 3 ] );
                ul[ e ]           = sqrt( ddot( u[ e ], u[ e ] ) );
                const double side = ddot( u[ e ], v[ ( e + 2 ) % 3 ] );
                flat |= !( ul[ e ] > 0.0 ) || side == 0.0;
                sg[ e ] = side > 0.0 ? 1.0 : -1.0;
            }
            if ( flat )
                return; // a flat triangle has no area
            const uint32_t Q   = min( b.counts->Q, b.capProbes );
            const uint32_t cnt = p < Q ? min( (uint32_t)id.w, kMaxProbeNbr ) : 0u;
            const int      M   = 3 + (int)cnt;
            if ( lane < 3 )
            {
                const d3 w  = dmul( u[ lane ], -sg[ lane ] / ul[ lane ] );
                kd[ lane ] = dcons_of( w.x, w.y, w.z, 0.0 );
            }
            uint32_t q = 0;
            double   L = 0.0;
            if ( lane < cnt )
            {
                q               = b.probeNbrIdx[ (size_t)p * kMaxProbeNbr + lane ];
                const float4 pq = b.probePos[ q ];
                const d3     D  = D3( (double)pq.x - P.x, (double)pq.y - P.y, (double)pq.z - P.z );
                L               = sqrt( ddot( D, D ) );
                kd[ 3 + lane ]  = L > 0.0 && L < 2.0 * rp ? dcons_of( D.x / L, D.y / L, D.z / L, L / ( 2.0 * rp ) )
                                                          : dcons_of( 0.0, 0.0, 1.0, 2.0 ); // vacuous
            }
            for ( int m = (int)lane; m < M; m += 32 )
                sums[ m ] = dcons_of( 0.0, 0.0, 0.0, 0.0 );
            __syncwarp();
            const int count = live_circles( cons, M, live, overflow );
            if ( count > 0 )
                region_arcs_d( cons, M, live, count, D );
            const double k2 = (double)gConcave * rp * rp;
            d3           gP = D3( 0.0, 0.0, 0.0 );
            if ( lane == 0 )
            {
                d3 gv[ 3 ] = { D3( 0.0, 0.0, 0.0 ), D3( 0.0, 0.0, 0.0 ), D3( 0.0, 0.0, 0.0 ) };
                for ( int e = 0; e < 3; e++ )
                {
                    const d3  gw = dmul( D3( sums[ e ].x, sums[ e ].y, sums[ e ].z ), -k2 );
                    const d3  wh = dmul( u[ e ], 1.0 / ul[ e ] );
                    const d3  gu = dmul( dsub( gw, dmul( wh, ddot( gw, wh ) ) ), -sg[ e ] / ul[ e ] );
                    const int a = e, c2 = ( e + 1 ) % 3;
                    gv[ a ]     = dadd( gv[ a ], dcross( v[ c2 ], gu ) );
                    gv[ c2 ]    = dadd( gv[ c2 ], dcross( gu, v[ a ] ) );
                }
                for ( int a = 0; a < 3; a++ )
                {
                    const d3 gD = dmul( dsub( gv[ a ], dmul( v[ a ], ddot( gv[ a ], v[ a ] ) ) ), 1.0 / Lv[ a ] );
                    add4( gradSorted, (uint32_t)ia[ a ], F3( (float)gD.x, (float)gD.y, (float)gD.z ), 0.f );
                    gP = dsub( gP, gD );
                }
            }
            if ( lane < cnt && L > 0.0 && L < 2.0 * rp )
            {
                const int    m  = 3 + (int)lane;
                const d3     w  = D3( kd[ m ].x, kd[ m ].y, kd[ m ].z );
                const d3     gw = dmul( D3( sums[ m ].x, sums[ m ].y, sums[ m ].z ), -k2 );
                const double gc = k2 * sums[ m ].w;
                const d3     gD = dadd( dmul( dsub( gw, dmul( w, ddot( gw, w ) ) ), 1.0 / L ), dmul( w, gc / ( 2.0 * rp ) ) );
                gP              = dsub( gP, gD );
                atomicAdd( &probeGrad[ q ].x, (float)gD.x );
                atomicAdd( &probeGrad[ q ].y, (float)gD.y );
                atomicAdd( &probeGrad[ q ].z, (float)gD.z );
            }
            for ( int o = 16; o > 0; o >>= 1 )
            {
                gP.x += __shfl_xor_sync( 0xffffffffu, gP.x, o );
                gP.y += __shfl_xor_sync( 0xffffffffu, gP.y, o );
                gP.z += __shfl_xor_sync( 0xffffffffu, gP.z, o );
            }
            if ( lane == 0 )
            {
                atomicAdd( &probeGrad[ p ].x, (float)gP.x );
                atomicAdd( &probeGrad[ p ].y, (float)gP.y );
                atomicAdd( &probeGrad[ p ].z, (float)gP.z );
            }
            __syncwarp();
        }

        struct ProbeAreaSmem
        {
            float4 cons[ kProbeCons ];
            float  dphi[ kProbeCons ];
            float4 iy[ kProbeCons ];
            float  dist[ kProbeCons ];
            uint32_t nq[ kProbeCons ];
            RegionSmem region;
        };
        template<bool kGrad> struct ProbeSmemD
        {
        };
        template<> struct ProbeSmemD<true>
        {
            RegionSmemD d;
        };

        // Contact directions v of a probe (L: distances), the normals u = v_a x v_b of its edges with their lengths
        // ul and the side sg of the third contact; false for a flat triangle, which has no area.
        __device__ __forceinline__ bool probe_triangle( const Build & b, const int ia[ 3 ], f3 P, f3 v[ 3 ], float L[ 3 ], f3 u[ 3 ], float ul[ 3 ],
                                                        float sg[ 3 ] )
        {
            for ( int a = 0; a < 3; a++ )
            {
                const float4 c = b.atoms[ ia[ a ] ];
                const f3     D = F3( c.x - P.x, c.y - P.y, c.z - P.z );
                L[ a ]         = sqrtf( dot( D, D ) );
                v[ a ]         = D * ( 1.f / L[ a ] );
            }
            bool flat = false;
            for ( int e = 0; e < 3; e++ )
            {
                u[ e ]           = cross( v[ e ], v[ ( e + 1 ) % 3 ] );
                ul[ e ]          = sqrtf( dot( u[ e ], u[ e ] ) );
                const float side = dot( u[ e ], v[ ( e + 2 ) % 3 ] );
                flat |= !( ul[ e ] > 0.f ) || side == 0.f;
                sg[ e ] = side > 0.f ? 1.f : -1.f;
            }
            return !flat;
        }

        // The contact directions' part of a probe's adjoint, from the integrals of y over the edges' arcs; returns the
        // gradient of its position.
        __device__ __forceinline__ f3 probe_edges_back( const int ia[ 3 ], const f3 v[ 3 ], const float L[ 3 ], const f3 u[ 3 ], const float ul[ 3 ],
                                                        const float sg[ 3 ], const f3 iy[ 3 ], float k2, float * gradSorted )
        {
            f3 gP      = F3( 0.f, 0.f, 0.f );
            f3 gv[ 3 ] = { gP, gP, gP };
            for ( int e = 0; e < 3; e++ )
            {
                const f3  gw = iy[ e ] * ( -k2 );
                const f3  wh = u[ e ] * ( 1.f / ul[ e ] );
                const f3  gu = ( gw - wh * dot( gw, wh ) ) * ( -sg[ e ] / ul[ e ] );
                const int a = e, c = ( e + 1 ) % 3;
                gv[ a ]     = gv[ a ] + cross( v[ c ], gu );
                gv[ c ]     = gv[ c ] + cross( gu, v[ a ] );
            }
            for ( int a = 0; a < 3; a++ )
            {
                const f3 gD = ( gv[ a ] - v[ a ] * dot( gv[ a ], v[ a ] ) ) * ( 1.f / L[ a ] );
                add4( gradSorted, (uint32_t)ia[ a ], gD, 0.f );
                gP = gP - gD;
            }
            return gP;
        }

        // Probes without listed neighbours, a thread each: the whole triangle. Its area from the solid angle of the
        // three directions (Van Oosterom and Strackee 1983), the integral of y over an edge's arc
        // (v_a + v_b) tan(angle / 2).
        template<bool kGrad>
        __global__ void __launch_bounds__( 128 ) k_area_triangles( Build b, double * parts, float * atomArea, float gConcave, float * gradSorted,
                                                                   float4 * probeGrad )
        {
            const uint32_t I   = min( b.counts->I, b.capProbes ), Q = min( b.counts->Q, b.capProbes );
            double         sum = 0.0;
            for ( uint32_t p = Q + blockIdx.x * blockDim.x + threadIdx.x; p < I; p += gridDim.x * blockDim.x )
            {
                const int4   id      = b.probeIds[ p ];
                const float4 pp      = b.probePos[ p ];
                const int    ia[ 3 ] = { id.x, id.y, id.z };
                f3           v[ 3 ], u[ 3 ];
                float        L[ 3 ], ul[ 3 ], sg[ 3 ];
                if ( !probe_triangle( b, ia, F3( pp.x, pp.y, pp.z ), v, L, u, ul, sg ) )
                    continue;
                const float d[ 3 ] = { dot( v[ 0 ], v[ 1 ] ), dot( v[ 1 ], v[ 2 ] ), dot( v[ 2 ], v[ 0 ] ) };
                if ( !kGrad )
                {
                    const float U  = 2.f * atan2f( fabsf( dot( u[ 0 ], v[ 2 ] ) ), 1.f + d[ 0 ] + d[ 1 ] + d[ 2 ] );
                    const float cA = b.rp * b.rp * U;
                    sum += cA;
                    if ( atomArea )
                        for ( int a = 0; a < 3; a++ )
                            atomicAdd( atomArea + b.perm[ ia[ a ] ], cA * ( 1.f / 3.f ) );
                }
                else
                {
                    f3 iy[ 3 ];
                    for ( int e = 0; e < 3; e++ )
                        iy[ e ] = ( v[ e ] + v[ ( e + 1 ) % 3 ] ) * ( ul[ e ] / ( 1.f + d[ e ] ) );
                    const f3 gP = probe_edges_back( ia, v, L, u, ul, sg, iy, gConcave * b.rp * b.rp, gradSorted );
                    atomicAdd( &probeGrad[ p ].x, gP.x );
                    atomicAdd( &probeGrad[ p ].y, gP.y );
                    atomicAdd( &probeGrad[ p ].z, gP.z );
                }
            }
            if constexpr ( !kGrad )
            {
                for ( int o = 16; o > 0; o >>= 1 )
                    sum += __shfl_xor_sync( 0xffffffffu, sum, o );
                if ( lane_id() == 0 && parts && sum != 0.0 )
                    atomicAdd( parts + 2, sum );
            }
        }

        // Warp per singular probe: its concave triangle outside the listed neighbour probes. 29,500 probes of a
        // 20,000-atom globule, the plain triangles (a thread each, 7 us) included: 0.80 ms before, 0.31 now; adjoint
        // 3.51 and 0.88, most of it the double-precision regions.
        // With kGrad, probeGrad (float4 per probe) accumulates d/d(position) of every
        // probe involved and gradSorted the direct terms of the contact directions; the lune planes
        // are not needed then.
        template<bool kGrad>
        __global__ void __launch_bounds__( 32 * kAreaWarps ) k_area_probes( Build b, double * parts, float * atomArea, float gConcave,
                                                                             float * gradSorted, float4 * probeGrad )
        {
            __shared__ ProbeAreaSmem     sm[ kAreaWarps ];
            __shared__ ProbeSmemD<kGrad> smD[ kAreaWarps ];
            const uint32_t               warp = threadIdx.x >> 5, lane = lane_id();
            ProbeAreaSmem &              S    = sm[ warp ];
            const uint32_t               Q    = min( b.counts->Q, b.capProbes );
            const float                  rp   = b.rp;
            double                       concaveSum = 0.0;
            uint32_t                     overflow   = 0;
            for ( uint32_t p = blockIdx.x * kAreaWarps + warp; p < Q; p += gridDim.x * kAreaWarps )
            {
                const int4   id = b.probeIds[ p ];
                const float4 pp = b.probePos[ p ];
                const f3     P  = F3( pp.x, pp.y, pp.z );
                const int    ia[ 3 ] = { id.x, id.y, id.z };
                f3           v[ 3 ], u[ 3 ];
                float        Lv[ 3 ], ul[ 3 ], sg[ 3 ];
                if ( !probe_triangle( b, ia, P, v, Lv, u, ul, sg ) )
                    continue; // a flat triangle has no area
                const uint32_t cnt = min( (uint32_t)id.w, kMaxProbeNbr );
                const int      M   = 3 + (int)cnt;
                if ( lane < 3 )
                {
                    const f3 w     = u[ lane ] * ( -sg[ lane ] / ul[ lane ] );
                    S.cons[ lane ] = make_float4( w.x, w.y, w.z, 0.f );
                }
                // neighbour caps at 3 .. M - 1 (up to 35 constraints: lane + 3 covers them in one pass)
                if ( lane < cnt )
                {
                    const int      m  = 3 + (int)lane;
                    const uint32_t q  = b.probeNbrIdx[ (size_t)p * kMaxProbeNbr + lane ];
                    const float4   pq = b.probePos[ q ];
                    const f3       D  = F3( pq.x - P.x, pq.y - P.y, pq.z - P.z );
                    const float    L  = sqrtf( dot( D, D ) );
                    S.dist[ m ]       = L;
                    S.nq[ m ]         = q;
                    if ( L > 0.f && L < 2.f * rp )
                    {
                        const f3 w  = D * ( 1.f / L );
                        S.cons[ m ] = make_float4( w.x, w.y, w.z, L / ( 2.f * rp ) );
                    }
                    else
                        S.cons[ m ] = make_float4( 0.f, 0.f, 1.f, 2.f ); // vacuous
                }
                for ( int m = (int)lane; m < M; m += 32 )
                {
                    S.dphi[ m ] = 0.f;
                    S.iy[ m ]   = make_float4( 0.f, 0.f, 0.f, 0.f );
                }
                __syncwarp();
                if constexpr ( !kGrad )
                {
                    const float U  = region_area_warp<true>( S.cons, M, S.region, overflow, []( int, const Circ &, float, float, int, int ) {} );
                    const float cA = rp * rp * U;
                    if ( lane == 0 )
                    {
                        concaveSum += cA;
                        if ( atomArea )
                            for ( int a = 0; a < 3; a++ )
                                atomicAdd( atomArea + b.perm[ ia[ a ] ], cA * ( 1.f / 3.f ) );
                    }
                }
                else if ( __any_sync( 0xffffffffu, lane < cnt && S.dist[ 3 + lane ] < kCloseProbe ) )
                    // a nearly coincident neighbour probe: the region's adjoint in double precision
                    probe_region_grad_d( b, p, gConcave, gradSorted, probeGrad, S.cons, S.region.live, overflow, smD[ warp ].d );
                else
                {
                    region_area_warp<false>( S.cons, M, S.region, overflow, [ & ]( int m, const Circ & C, float st, float ln, int, int ) {
                        const f3 Iy = arc_integral( C, st, ln );
                        S.dphi[ m ] += ln;
                        S.iy[ m ].x += Iy.x, S.iy[ m ].y += Iy.y, S.iy[ m ].z += Iy.z;
                    } );
                    __syncwarp();
                    const float k2 = gConcave * rp * rp;
                    f3          gP = F3( 0.f, 0.f, 0.f );
                    if ( lane == 0 )
                    {
                        const f3 iy[ 3 ] = { F3( S.iy[ 0 ] ), F3( S.iy[ 1 ] ), F3( S.iy[ 2 ] ) };
                        gP               = probe_edges_back( ia, v, Lv, u, ul, sg, iy, k2, gradSorted );
                    }
                    if ( lane < cnt )
                    {
                        const int   m = 3 + (int)lane;
                        const float L = S.dist[ m ];
                        if ( L > 0.f && L < 2.f * rp )
                        {
                            const float4 k  = S.cons[ m ];
                            const f3     w  = F3( k.x, k.y, k.z );
                            const f3     gw = F3( S.iy[ m ].x, S.iy[ m ].y, S.iy[ m ].z ) * ( -k2 );
                            const float  gc = k2 * S.dphi[ m ];
                            const f3     gD = ( gw - w * dot( gw, w ) ) * ( 1.f / L ) + w * ( gc / ( 2.f * rp ) );
                            gP              = gP - gD;
                            atomicAdd( &probeGrad[ S.nq[ m ] ].x, gD.x );
                            atomicAdd( &probeGrad[ S.nq[ m ] ].y, gD.y );
                            atomicAdd( &probeGrad[ S.nq[ m ] ].z, gD.z );
                        }
                    }
                    for ( int o = 16; o > 0; o >>= 1 )
                    {
                        gP.x += __shfl_xor_sync( 0xffffffffu, gP.x, o );
                        gP.y += __shfl_xor_sync( 0xffffffffu, gP.y, o );
                        gP.z += __shfl_xor_sync( 0xffffffffu, gP.z, o );
                    }
                    if ( lane == 0 )
                    {
                        atomicAdd( &probeGrad[ p ].x, gP.x );
                        atomicAdd( &probeGrad[ p ].y, gP.y );
                        atomicAdd( &probeGrad[ p ].z, gP.z );
                    }
                }
                __syncwarp();
            }
            if ( lane == 0 && parts && concaveSum != 0.0 )
                atomicAdd( parts + 2, concaveSum );
            overflow = __any_sync( 0xffffffffu, overflow != 0 );
            if ( lane == 0 && overflow )
                atomicOr( &b.counts->overflow, (uint32_t)kOverflowArea );
        }

        // probe positions follow their atoms: M^T lambda = g with rows p - c_a;
        // d/dc_a = lambda_a (p - c_a), d/dR_a = lambda_a R_a. The 3x3 solve is in double
        // precision: for a probe near the plane of its three centres (its mirror probe about to
        // merge with it) M is nearly singular and lambda grows as 1 / det, so float32 rounding of
        // the rows and of det would show in the atoms' gradients. One solve per probe: the FP64
        // pipe's rate does not matter here.
        __global__ void k_area_probe_back( Build b, const float4 * probeGrad, float * gradSorted )
        {
            const uint32_t I = min( b.counts->I, b.capProbes );
            for ( uint32_t p = blockIdx.x * blockDim.x + threadIdx.x; p < I; p += gridDim.x * blockDim.x )
            {
                const float4 g4 = probeGrad[ p ];
                if ( g4.x == 0.f && g4.y == 0.f && g4.z == 0.f )
                    continue;
                const d3     g  = D3( (double)g4.x, (double)g4.y, (double)g4.z );
                const int4   id = b.probeIds[ p ];
                const float4 pp = b.probePos[ p ];
                const int    ia[ 3 ] = { id.x, id.y, id.z };
                d3           r[ 3 ];
                double       R[ 3 ];
                for ( int k = 0; k < 3; k++ )
                {
                    const float4 c = b.atoms[ ia[ k ] ];
                    // differences of float32 values: exact in double
                    r[ k ] = D3( (double)pp.x - (double)c.x, (double)pp.y - (double)c.y, (double)pp.z - (double)c.z );
                    R[ k ] = (double)c.w + (double)b.rp;
                }
                const double det = ddot( r[ 0 ], dcross( r[ 1 ], r[ 2 ] ) );
                if ( !( fabs( det ) > 0.0 ) )
                    continue;
                const double lam[ 3 ] = { ddot( g, dcross( r[ 1 ], r[ 2 ] ) ) / det, ddot( r[ 0 ], dcross( g, r[ 2 ] ) ) / det,
                                          ddot( r[ 0 ], dcross( r[ 1 ], g ) ) / det };
                for ( int k = 0; k < 3; k++ )
                    add4( gradSorted, (uint32_t)ia[ k ],
                          F3( (float)( r[ k ].x * lam[ k ] ), (float)( r[ k ].y * lam[ k ] ), (float)( r[ k ].z * lam[ k ] ) ),
                          (float)( lam[ k ] * R[ k ] ) );
            }
        }

        __global__ void k_area_unsort( Build b, const float * gradSorted, float * gradInput )
        {
            for ( uint32_t s = blockIdx.x * blockDim.x + threadIdx.x; s < b.n; s += gridDim.x * blockDim.x )
            {
                const uint32_t i = b.perm[ s ];
                for ( int k = 0; k < 4; k++ )
                    gradInput[ 4 * (size_t)i + k ] = gradSorted[ 4 * (size_t)s + k ];
            }
        }

        // A warp per item: regions differ several times in their work, and 152 x 16 blocks that took every n-th item
        // were 1.3 waves of unequal blocks (20,000 atoms: 1.01 ms, 0.75 now; with the adjoint 1.56 and 1.28)
        inline uint32_t area_blocks( uint64_t items )
        {
            const uint64_t want = ( items + kAreaWarps - 1 ) / kAreaWarps;
            const uint64_t cap  = 152ull * 8192ull;
            return (uint32_t)( want < 1 ? 1 : ( want < cap ? want : cap ) );
        }
    } // namespace

    size_t area_scratch_bytes( const Build & b ) { return sizeof( float4 ) * (size_t)b.capProbes + 256; }

    void launch_area( const Build & b, double * parts, float * atomArea, cudaStream_t s )
    {
        cudaMemsetAsync( parts, 0, 3 * sizeof( double ), s );
        if ( atomArea )
            cudaMemsetAsync( atomArea, 0, sizeof( float ) * (size_t)b.n, s );
        if ( !b.n )
            return;
        k_area_atoms<false><<<area_blocks( b.n ), 32 * kAreaWarps, 0, s>>>( b, parts, atomArea, 0.f, 0.f, nullptr );
        k_area_probes<false><<<area_blocks( b.capProbes ), 32 * kAreaWarps, 0, s>>>( b, parts, atomArea, 0.f, nullptr, nullptr );
        k_area_triangles<false><<<152 * 8, 128, 0, s>>>( b, parts, atomArea, 0.f, nullptr, nullptr );
        count_launches( 3 );
    }

    void launch_area_backward( const Build & b, const float gParts[ 3 ], float * gradSorted, float * gradInput, void * scratch,
                               cudaStream_t s )
    {
        cudaMemsetAsync( gradSorted, 0, sizeof( float ) * 4 * (size_t)b.n, s );
        if ( !b.n )
        {
            return;
        }
        float4 * probeGrad = static_cast<float4 *>( scratch );
        cudaMemsetAsync( probeGrad, 0, sizeof( float4 ) * (size_t)b.capProbes, s );
        k_area_atoms<true><<<area_blocks( b.n ), 32 * kAreaWarps, 0, s>>>( b, nullptr, nullptr, gParts[ 0 ], gParts[ 1 ], gradSorted );
        k_area_probes<true><<<area_blocks( b.capProbes ), 32 * kAreaWarps, 0, s>>>( b, nullptr, nullptr, gParts[ 2 ], gradSorted, probeGrad );
        k_area_triangles<true><<<152 * 8, 128, 0, s>>>( b, nullptr, nullptr, gParts[ 2 ], gradSorted, probeGrad );
        k_area_probe_back<<<min( 152u * 8u, ( b.capProbes + 255 ) / 256 + 1 ), 256, 0, s>>>( b, probeGrad, gradSorted );
        k_area_unsort<<<( b.n + 255 ) / 256, 256, 0, s>>>( b, gradSorted, gradInput );
        count_launches( 5 );
    }
} // namespace sesgb
