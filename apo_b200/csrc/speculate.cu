// Edge validation as an edge-parallel search with an exact fallback per cell.
//
// The reference validates the edges of a cell 32 at a time with one warp, and every
// candidate site met by any lane's BVH walk costs the whole warp a collective "is it a
// known neighbour" scan and a collective emptiness predicate over all edges
// (apo/include/apo/gpu/algorithm.inl:478-857). Almost no edge finds a contributor (a few
// per 100,000 edges on uniform clouds), and while none is found the cell does not change,
// so every edge's search sees the same cell and the searches are independent.
//
// Here each edge is one work item of a persistent kernel whose lanes fetch items one at a
// time: the walk, the neighbour test (binary search in the cell's sorted neighbour list)
// and the emptiness test (over that list) run lane-locally, with the reference's
// arithmetic and walk order. A cell none of whose edges found a contributor ends exactly
// as the reference leaves it (every edge validated, the cell validated); a cell where one
// did, or whose neighbour list is too long, is re-run from its stored state by the exact
// warp algorithm (k_edge_validation), so the result is the reference's in every case.
#include "cells.cuh"

namespace apo2
{
    constexpr uint32_t kNbrBlock      = 128; // 4 warps, one cell each
    constexpr uint32_t kSpecBlock     = 128;
    constexpr uint32_t kFlagFound     = 1;
    constexpr uint32_t kFlagOverflow  = 2;
#ifndef APO2_SPEC_LANE_BUDGET
#define APO2_SPEC_LANE_BUDGET 160
#endif
#ifndef APO2_SPEC_SPLIT_AT
#define APO2_SPEC_SPLIT_AT 192
#endif
#ifndef APO2_SPEC_MIN_BLOCKS
#define APO2_SPEC_MIN_BLOCKS 4
#endif
    // Nodes one lane may visit before the search goes to a warp. The lane kernel lasts as long as its
    // longest walk, some 1.9 us a node, which is what counts for few sites; many are better off with longer
    // walks. All edge-search kernels, of 128 / 160 / 256 nodes: 1,000 uniform sites 1.55 / 1.61 / 1.87 ms,
    // 10,000 2.8 / 2.9 / 3.3, 61k protein 14.5 / 14.4 / 14.9, 1M protein 127 / 121 / 119, 1M log-normal 198 / 185 / 176.
    constexpr uint32_t kLaneBudget    = APO2_SPEC_LANE_BUDGET;
    constexpr uint32_t kHeavyBlock    = 128;
    constexpr uint32_t kHeavyStack    = 3072; // shared node stack per warp of the cooperative walk
    constexpr uint32_t kSplitAt       = APO2_SPEC_SPLIT_AT; // pending subtrees at which a long walk is handed out
    constexpr uint32_t kSplitSlot     = 0x80000000u; // marks a subtree whose search set-up is cached
#ifndef APO2_SPEC_REFILL_AT
#define APO2_SPEC_REFILL_AT 28
#endif
    // Idle lanes of a speculation warp fetch and set up new edges together, once at least
    // this many are idle (or none is walking): the set-up (bounding sphere, certificate test)
    // is long FP64 code, and run by one or two lanes at a time it held the warp for most
    // of its time.
    constexpr uint32_t kRefillAt = APO2_SPEC_REFILL_AT;
    constexpr uint32_t kSpecSteps = 16; // nodes of every walk between two votes
    // the same for the bisectors, whose set-up is short, and the nodes a walk takes between two votes
    // (nodes / idle lanes, 1M protein packing: 4 / 16 5.5 ms, 8 / 8 5.7, 8 / 16 5.4, 8 / 24 5.0, 16 / 16 5.2)
    constexpr uint32_t kBisectorRefillAt = 24;
    constexpr uint32_t kBisectorSteps    = 8;

    __device__ __forceinline__ uint32_t lane_of() { return threadIdx.x & 31; }

    // Sorted unique ids of a task cell's edge sites (the set the reference's known-neighbour
    // and emptiness tests range over), and the cell's items for the item scan: its edges, or
    // with Bisectors its neighbours of larger id (the tasks are then all cells of the handle).
    template<bool Bisectors>
    __global__ void __launch_bounds__( kNbrBlock ) k_neighbor_lists( CellContext c, const uint32_t * __restrict__ tasks,
                                                                     const uint32_t * __restrict__ task_count,
                                                                     SpecBuffers b )
    {
        __shared__ uint32_t buf[ kNbrBlock / 32 ][ 1024 ];
        const uint32_t      warp  = threadIdx.x >> 5, lane = lane_of();
        const uint32_t      gwarp = blockIdx.x * ( kNbrBlock / 32 ) + warp;
        const uint32_t      nwarp = gridDim.x * ( kNbrBlock / 32 );
        const uint32_t      count = Bisectors ? c.hi - c.lo : *task_count;
        uint32_t *          ids   = buf[ warp ];
        for ( uint32_t t = gwarp; t < c.n; t += nwarp )
        {
            if ( t >= count )
            {
                if ( lane == 0 )
                    b.item_count[ t ] = 0;
                continue;
            }
            const uint32_t i  = Bisectors ? c.lo + t : tasks[ t ];
            const uint32_t en = c.edge_nb[ i ];
            const uint8_t  st = c.status[ i ];
            if ( !Bisectors && lane < kMaybeWords )
                b.maybe_bits[ size_t( t ) * kMaybeWords + lane ] = 0;
            if ( ( !Bisectors && st == kFullyValidated ) || st == kBuried )
            {
                if ( lane == 0 )
                {
                    b.item_count[ t ] = 0;
                    b.cell_flag[ t ]  = 0;
                    b.nbr_count[ t ]  = 0;
                }
                continue;
            }
            const uint32_t total = 2 * en;
            uint32_t       size  = 64;
            while ( size < total )
                size <<= 1;
            for ( uint32_t x = lane; x < size; x += 32 )
            {
                uint32_t v = kNone;
                if ( x < total )
                {
                    const uint4 r = c.edges[ store_row( c, i ) * kMaxEdges + ( x >> 1 ) ];
                    v             = ( x & 1 ) ? r.y : r.x;
                }
                ids[ x ] = v;
            }
            __syncwarp();
            for ( uint32_t s2 = 2; s2 <= size; s2 <<= 1 )
                for ( uint32_t stride = s2 >> 1; stride > 0; stride >>= 1 )
                {
                    for ( uint32_t x = lane; x < size; x += 32 )
                    {
                        const uint32_t y = x ^ stride;
                        if ( y > x )
                        {
                            const uint32_t a = ids[ x ], bb = ids[ y ];
                            if ( ( a > bb ) == ( ( x & s2 ) == 0 ) )
                            {
                                ids[ x ] = bb;
                                ids[ y ] = a;
                            }
                        }
                    }
                    __syncwarp();
                }
            uint32_t kept = 0, above = 0, carried = kNone;
            for ( uint32_t base = 0; base < size; base += 32 )
            {
                const uint32_t x    = base + lane;
                const uint32_t v    = ids[ x ];
                uint32_t       prev = __shfl_up_sync( 0xffffffffu, v, 1 );
                if ( lane == 0 )
                    prev = carried;
                const bool     keep = v != kNone && ( x == 0 || v != prev );
                const uint32_t bal  = __ballot_sync( 0xffffffffu, keep );
                carried             = __shfl_sync( 0xffffffffu, v, 31 );
                const uint32_t dst  = kept + __popc( bal & ( ( 1u << lane ) - 1u ) );
                if ( keep && dst < kNbrCap )
                    b.nbr[ size_t( t ) * kNbrCap + dst ] = v;
                kept += __popc( bal );
                if ( Bisectors )
                    above += __popc( __ballot_sync( 0xffffffffu, keep && v > i && v < c.n ) );
            }
            __syncwarp();
            if ( !Bisectors && kept > kNbrCap && lane < kMaybeWords )
                b.maybe_bits[ size_t( t ) * kMaybeWords + lane ] = 0xffffffffu; // nothing decided: full exact pass
            if ( lane == 0 )
            {
                b.nbr_count[ t ]  = min( kept, kNbrCap );
                b.cell_flag[ t ]  = kept > kNbrCap ? kFlagOverflow : 0u;
                b.item_count[ t ] = kept > kNbrCap ? 0u : ( Bisectors ? above : en );
            }
        }
    }

    __device__ __forceinline__ bool in_sorted( const uint32_t * __restrict__ list, uint32_t count, uint32_t v )
    {
        uint32_t lo = 0, hi = count;
        while ( lo < hi )
        {
            const uint32_t mid = ( lo + hi ) >> 1;
            const uint32_t x   = list[ mid ];
            if ( x == v )
                return true;
            if ( x < v )
                lo = mid + 1;
            else
                hi = mid;
        }
        return false;
    }

    // Per-lane state of one edge search.
    struct EdgeSearch
    {
        uint32_t t, e, i, k, l;
        double4  si, sk, sl;
        float4   bsph;
        EdgeReach reach; // where every possible contributor is
        bool     closed;
        TangentPlanes planes;
        bool     hyperbola;
        const uint32_t * nbr;
        uint32_t nbr_count;
        // the third sites of the edge's vertices: the neighbours bounding its arc, which a
        // candidate root outside the arc almost always lies inside (tested first)
        uint32_t hint[ 2 ];
        uint32_t from; // node the walk starts at
        bool     covered; // the reach lies in what the cell's vertex spheres can touch
    };

    // Bounding volume of edge (k, l) of cell i (algorithm.inl:555-600); the trisector's roots are
    // left in ev0 and ev1. Returns whether it is an ellipse.
    __device__ __forceinline__ bool bound_edge( EdgeSearch & s, double4 & ev0, double4 & ev1 )
    {
        ev0 = ev1 = make_double4( 0, 0, 0, 0 );
        const uint32_t type = trisector( s.si, s.sk, s.sl, ev0, ev1 );
        s.hyperbola         = type == 1;
        const bool   ellipse = type == 2;
        const float4 v1 = to_float( ev0 ), v2 = to_float( ev1 );
        s.planes.n1 = s.planes.n2 = s.planes.p1 = s.planes.p2 = make_float3( 0, 0, 0 );
        if ( ellipse )
        {
            const float3 center = ( f3( v1 ) + f3( v2 ) ) * .5f;
            const float  radius = flength( center - f3( v1 ) ) + v1.w;
            s.bsph              = make_float4( center.x, center.y, center.z, radius );
        }
        else
        {
            double3 nn1, nn2;
            tangent_planes( s.si, s.sk, s.sl, nn1, nn2 );
            s.planes.n1      = to_float( nn1 );
            s.planes.n2      = to_float( nn2 );
            const double3 p1 = d3( s.si ) + nn1 * s.si.w;
            const double3 p2 = d3( s.sk ) + nn1 * s.sk.w;
            const double3 p3 = d3( s.sl ) + nn1 * s.sl.w;
            const double3 p4 = d3( s.si ) + nn2 * s.si.w;
            const double3 p5 = d3( s.sk ) + nn2 * s.sk.w;
            s.bsph           = to_float( sphere_from_points( p1, p2, p3, p5 ) );
            s.planes.p1      = to_float( p1 );
            s.planes.p2      = to_float( p4 );
        }
        return ellipse;
    }

    // Does the security radius cover the edge (algorithm.inl:601-614)? Then it needs no search.
    __device__ __forceinline__ bool covers_edge( const EdgeSearch & s, float known )
    {
        return lt_eps( flength( f3( to_float( s.si ) ) - f3( s.bsph ) ), known - s.bsph.w );
    }

    // Reach of the search of a bounded edge, from the arc's ends and its largest radius. To be settled.
    __device__ __forceinline__ void reach_edge( const CellContext & c, EdgeSearch & s, bool ellipse, double4 ev0, double4 ev1, ArcEnds & ends,
                                                OpenEnds & open )
    {
        double wmax = stored_ends( c, s.i, s.si, s.k, s.l, ends, s.hint );
        if ( ellipse || s.closed )
        {
#pragma unroll 1
            for ( uint32_t a = 0; a < 2; a++ )
            {
                const double4 apex = a ? ev1 : ev0;
                bool          out  = false;
                for ( uint32_t q = 0; q < s.nbr_count && !out; q++ )
                {
                    const uint32_t u = s.nbr[ q ];
                    if ( u != s.k && u != s.l )
                        out = clearly_outside( c.sites[ u ], apex );
                }
                if ( !out )
                    wmax = fmax( wmax, apex.w );
            }
        }
        // only neighbours bound the arc, are tested first, and skipped by the walk
        for ( uint32_t h = 0; h < 2; h++ )
            if ( s.hint[ h ] != kNone && !in_sorted( s.nbr, s.nbr_count, s.hint[ h ] ) )
                s.hint[ h ] = kNone;
        const auto known = [ & ]( uint32_t m ) { return m == s.hint[ 0 ] || m == s.hint[ 1 ]; };
        s.reach = edge_reach( c, s.si, s.sk, s.sl, s.hyperbola, ends, ends.count == 2 && known( ends.m[ 0 ] ) && known( ends.m[ 1 ] ), wmax,
                              s.bsph, open );
        s.covered = wmax <= 1.001 * double( c.largest[ s.i ] );
        s.from    = s.covered ? c.around[ s.i ] : 0u;
    }

    // The reach once its open ends have been looked at, and the planes that need not be.
    __device__ __forceinline__ void settle_edge( const CellContext & c, EdgeSearch & s, const OpenEnds & open )
    {
        const float4 fsi = to_float( s.si );
        settle( c, s.reach, open );
        if ( s.reach.kind == kReachArcPlanes )
        {
            bool open1 = true, open2 = true;
            for ( uint32_t q = 0; q < s.nbr_count && ( open1 || open2 ); q++ )
            {
                const uint32_t u = s.nbr[ q ];
                if ( u == s.k || u == s.l || u >= c.n )
                    continue;
                const float4 m = c.sites_f[ u ];
                open1          = open1 && !far_roots_blocked( s.planes.n1, fsi, m, s.reach.far );
                open2          = open2 && !far_roots_blocked( s.planes.n2, fsi, m, s.reach.far );
            }
            if ( !open1 )
                s.reach.slab[ 0 ] = -FLT_MAX;
            if ( !open2 )
                s.reach.slab[ 1 ] = -FLT_MAX;
            if ( !open1 && !open2 )
                s.reach.kind = kReachArc;
        }
    }
    __device__ __forceinline__ SiteSequence neighbours( const EdgeSearch & s ) { return { s.nbr, s.nbr_count, 0u }; }
    __device__ __forceinline__ void set_reach( const CellContext & c, EdgeSearch & s, bool ellipse, double4 ev0, double4 ev1 )
    {
        ArcEnds  ends;
        OpenEnds open;
        reach_edge( c, s, ellipse, ev0, ev1, ends, open );
        close_ends( c, s.si, s.k, s.l, ends, neighbours( s ), open, s.reach );
        settle_edge( c, s, open );
    }

    // The walk is bound by the node steps (two boxes against three balls and three planes, some hundred
    // nodes an edge); the balls of the arc and the planes replaced the ball around c_i, most of whose
    // leaves went through a quadrisector solve each.
    //
    // May the box hold a contributor? Without an arc, also the reference's own test for entering it
    // (algorithm.inl:642-667: the box meets the bounding sphere and, for a hyperbolic edge, the
    // closest point of the box lies below both tangent planes).
    __device__ __forceinline__ bool enter_child( const EdgeSearch & s, const Box & b, bool leaf )
    {
        if ( !within( s.reach, s.planes, b ) )
            return false;
        if ( leaf && s.reach.kind != kReachBall )
            return within( s.reach, s.planes, sphere_in( b ) );
        if ( s.reach.kind != kReachBall )
            return true;
        bool enter = b.distance( s.bsph ) < 0.f;
        if ( s.hyperbola && enter )
        {
            const float3 p = b.closest( s.bsph );
            enter          = fdot( s.planes.n1, p - s.planes.p1 ) < 0.f && fdot( s.planes.n2, p - s.planes.p2 ) < 0.f;
        }
        return enter;
    }

    // Does site j give the edge two vertices, one of them empty of every other neighbour?
    // (algorithm.inl:683-774, with the known-neighbour and emptiness tests lane-local.)
    __device__ __forceinline__ bool contributes( const CellContext & c, const EdgeSearch & s, uint32_t j )
    {
        if ( j == s.i || j == s.k || j == s.l || c.status[ j ] == kBuried )
            return false;
        const double4 sj = c.sites[ j ];
        const float4  fj = to_float( sj );
        if ( !intersects( fj, s.bsph ) )
            return false;
        if ( !within( s.reach, s.planes, fj ) )
            return false;
        if ( s.hyperbola
             && !( double( fdot( s.planes.n1, f3( fj ) - s.planes.p1 ) ) < -sj.w
                   && double( fdot( s.planes.n2, f3( fj ) - s.planes.p2 ) ) < -sj.w ) )
            return false;
        if ( in_sorted( s.nbr, s.nbr_count, j ) )
            return false;
        double4        x[ 2 ] = { make_double4( 0, 0, 0, 0 ), make_double4( 0, 0, 0, 0 ) };
        const uint32_t mask   = quadrisector( s.si, sj, s.sk, s.sl, x[ 0 ], x[ 1 ] );
        if ( mask != 3 )
            return false;
        // the FP32 filter decides here too; its counts are kept for the cell kernels only
        FilterTally untallied;
        // A root is empty when no neighbour other than k, l conflicts with it: the neighbours
        // bounding the edge's arc go first (a root outside the arc is nearly always inside one of
        // them), then the whole sorted list. The conjunction is the same.
        const auto conflicts = [ & ]( uint32_t u, double4 root ) {
            return c.fp32 ? site_conflict<true>( c, u, root, untallied ) : site_conflict<false>( c, u, root, untallied );
        };
#pragma unroll 1
        for ( uint32_t r = 0; r < 2; r++ )
        {
            const double4 root = r ? x[ 1 ] : x[ 0 ];
            bool          ok   = true;
#pragma unroll 1
            for ( uint32_t h = 0; h < 2 && ok; h++ )
            {
                const uint32_t u = h ? s.hint[ 1 ] : s.hint[ 0 ];
                ok               = u == kNone || !conflicts( u, root );
            }
            for ( uint32_t q = 0; q < s.nbr_count && ok; q++ )
            {
                const uint32_t u = s.nbr[ q ];
                if ( u != s.k && u != s.l )
                    ok = !conflicts( u, root );
            }
            if ( ok )
                return true;
        }
        return false;
    }

    __device__ __forceinline__ void send_to_exact( const SpecBuffers & b, uint32_t t, uint32_t e )
    {
        // the exact path decides, searching this edge again
        atomicOr( &b.maybe_bits[ size_t( t ) * kMaybeWords + ( e >> 5 ) ], 1u << ( e & 31 ) );
        atomicOr( &b.cell_flag[ t ], kFlagFound );
    }

    // Edge e of task t, bounded; false if it needs no search.
    __device__ __forceinline__ bool load_edge( const CellContext & c, const uint32_t * tasks, const SpecBuffers & b, uint32_t t,
                                               uint32_t e, EdgeSearch & s, bool & ellipse, double4 & ev0, double4 & ev1 )
    {
        s.t           = t;
        s.e           = e;
        s.i           = tasks[ t ];
        const uint4 r = c.edges[ store_row( c, s.i ) * kMaxEdges + e ];
        s.k           = r.x;
        s.l           = r.y;
        s.closed      = r.z == kNone;
        s.si          = c.sites[ s.i ];
        s.nbr         = b.nbr + size_t( t ) * kNbrCap;
        s.nbr_count   = b.nbr_count[ t ];
        // an edge validated before is not searched (algorithm.inl:522-526, 552)
        if ( ( r.w & 0xffu ) == 1u )
            return false;
        s.sk = c.sites[ s.k ];
        s.sl = c.sites[ s.l ];
        ellipse = bound_edge( s, ev0, ev1 );
        return !covers_edge( s, c.known_radii[ s.i ] );
    }

    // Edges of cells with few surroundings, nearly all: a warp per cell collects the sites, other than
    // the neighbours, within the bound of the cell's edges (some hundred), and its lanes, an edge
    // each, go through that list together. Per edge that is some hundred tests of a sphere against
    // three balls, read by all lanes at once, where a walk of its own took 50 to 90 nodes of two boxes
    // each, on lanes that part at every node. Cells with more surroundings than the list holds (hull
    // cells) keep their items for k_edge_speculate, edges that reach past the list go to a warp of
    // their own (k_edge_heavy). The set-up of an edge is straight double-precision code, run by 16 warps at 16
    // places of it: the kernel's size decides whether it stays in the instruction cache (per issue of a warp, 2.9
    // cycles of waiting for instructions at 93 KB of code, 8.4 at 104; it is 96 now). All edge-search kernels of a build, against searches bounded by one ball and
    // a walk per edge: 1M log-normal cloud 387 -> 185 ms, 1M-site protein packing 146 -> 121, 100k uniform
    // 27 -> 16, 46^3 lattice 6.7 -> 6.8.
    __global__ void __launch_bounds__( kCellBlock, 4 ) k_edge_cells( CellContext c, const uint32_t * __restrict__ tasks,
                                                                     const uint32_t * __restrict__ task_count, SpecBuffers b )
    {
        const uint32_t warp  = threadIdx.x >> 5, lane = lane_of();
        const uint32_t gwarp = blockIdx.x * ( kCellBlock / 32 ) + warp;
        const uint32_t count = *task_count;
        float4 *       list  = reinterpret_cast<float4 *>( c.walk_scratch + size_t( gwarp ) * kWalkScratchWords );
        uint32_t *     ids   = reinterpret_cast<uint32_t *>( list + kListCap );
        const Scene &  scene = *c.scene;
        const float    density = float( c.n ) / float( ( scene.hi[ 0 ] - scene.lo[ 0 ] ) * ( scene.hi[ 1 ] - scene.lo[ 1 ] ) * ( scene.hi[ 2 ] - scene.lo[ 2 ] ) );
        while ( true )
        {
            uint32_t t = 0;
            if ( lane == 0 )
                t = atomicAdd( c.work_counter, 1u );
            t = __shfl_sync( 0xffffffffu, t, 0 );
            if ( t >= count )
                break;
            const uint32_t i = tasks[ t ], edges = b.item_count[ t ]; // none where the cell needs no search
            if ( edges == 0 )
                continue;
            const uint32_t * nbr   = b.nbr + size_t( t ) * kNbrCap;
            const uint32_t   known = b.nbr_count[ t ];
            const double4    si    = c.sites[ i ];
            float4           ball  = touch_ball( c, si, c.largest[ i ] );
            ball.w += 1.001f * float( c.scene->rmax - c.scene->rmin );
            // far more than the list holds, at the scene's mean density: not worth collecting
            if ( 4.2f * ball.w * ball.w * ball.w * density > 4.f * float( kListCap ) )
                continue;
            const uint32_t listed = collect_sites( c, i, ball, c.around[ i ], list, ids, ids + kListCap,
                                                   [ & ]( uint32_t j ) { return in_sorted( nbr, known, j ); } );
            if ( listed == kNone )
                continue; // its items stay
            for ( uint32_t base = 0; base < edges; base += 32 )
            {
                EdgeSearch s;
                ArcEnds    ends;
                OpenEnds   loose;
                bool       ellipse;
                double4    ev0, ev1;
                bool       open = base + lane < edges && load_edge( c, tasks, b, t, base + lane, s, ellipse, ev0, ev1 );
                if ( open )
                    reach_edge( c, s, ellipse, ev0, ev1, ends, loose );
                __syncwarp();
                close_ends_together( c, si, s.k, s.l, ends, SiteSequence { nbr, known, 0u }, loose, s.reach );
                if ( open )
                    settle( c, s.reach, loose );
                if ( open && !s.covered )
                {
                    const uint32_t slot = atomicAdd( b.heavy_count, 1u );
                    if ( slot < b.heavy_cap )
                        b.heavy[ slot ] = make_uint2( s.t, s.e );
                    else
                        send_to_exact( b, s.t, s.e );
                    open = false;
                }
                // 32 sites at a time: first which of them are near, a bit each, then every lane its own
                for ( uint32_t first = 0; first < listed; first += 32 )
                {
                    const uint32_t block = min( listed - first, 32u );
                    uint32_t       near  = 0;
                    for ( uint32_t q = 0; q < block; q++ )
                        near |= uint32_t( within<false>( s.reach, s.planes, list[ first + q ] ) ) << q;
                    near = open ? near : 0u;
                    while ( __any_sync( 0xffffffffu, near != 0 ) )
                    {
                        if ( near == 0 )
                            continue;
                        const uint32_t q = __ffs( near ) - 1;
                        near &= near - 1;
                        if ( contributes( c, s, ids[ first + q ] ) )
                        {
                            send_to_exact( b, s.t, s.e );
                            open = false;
                            near = 0;
                        }
                    }
                }
            }
            if ( lane == 0 )
                b.item_count[ t ] = 0;
            __syncwarp();
        }
    }

    __global__ void __launch_bounds__( kSpecBlock, APO2_SPEC_MIN_BLOCKS ) k_edge_speculate( CellContext c, const uint32_t * __restrict__ tasks,
                                                                      const uint32_t * __restrict__ task_count,
                                                                      SpecBuffers b, uint32_t * error )
    {
        const uint32_t count = *task_count;
        if ( count == 0 )
            return;
        const uint64_t total = *b.item_total;
        const uint32_t n     = c.n;
        uint32_t       err   = 0;

        EdgeSearch s;
        bool       active    = false;
        bool       exhausted = false; // the queue is empty for this lane
        uint32_t   stack[ kStack ];
        int        sp    = 0;
        uint32_t   node  = 0;
        uint32_t   steps = 0;
        while ( true )
        {
            // warp-uniform choice between a refill round and a walk step
            const uint32_t idle = __ballot_sync( 0xffffffffu, !active && !exhausted );
            const uint32_t busy = __ballot_sync( 0xffffffffu, active );
            if ( idle == 0 && busy == 0 )
                break;
            if ( idle != 0 && ( busy == 0 || uint32_t( __popc( idle ) ) >= kRefillAt ) )
            {
                if ( !active && !exhausted )
                {
                    // warp-aggregated fetch of the next item by the idle lanes
                    const uint32_t leader = __ffs( idle ) - 1;
                    uint64_t       base   = 0;
                    if ( lane_of() == leader )
                        base = atomicAdd( reinterpret_cast<unsigned long long *>( b.item_counter ), __popc( idle ) );
                    base                = __shfl_sync( idle, base, leader );
                    const uint64_t item = base + __popc( idle & ( ( 1u << lane_of() ) - 1u ) );
                    if ( item >= total )
                        exhausted = true;
                    else
                    {
                        // task holding this item: last t with offset[t] <= item
                        uint32_t lo = 0, hi = count;
                        while ( hi - lo > 1 )
                        {
                            const uint32_t mid = ( lo + hi ) >> 1;
                            if ( b.item_offset[ mid ] <= item )
                                lo = mid;
                            else
                                hi = mid;
                        }
                        bool             ellipse;
                        double4          ev0, ev1;
                        s.t              = lo;
                        const uint32_t e = uint32_t( item - b.item_offset[ s.t ] );
                        s.e              = e;
                        if ( b.cell_flag[ s.t ] & kFlagOverflow )
                        {
                            // no neighbour list for this cell: the exact path searches this edge
                            atomicOr( &b.maybe_bits[ size_t( s.t ) * kMaybeWords + ( e >> 5 ) ], 1u << ( e & 31 ) );
                        }
                        else if ( load_edge( c, tasks, b, lo, e, s, ellipse, ev0, ev1 ) )
                        {
                            set_reach( c, s, ellipse, ev0, ev1 );
                            active = true;
                            sp     = 0;
                            node   = s.from;
                            steps  = 0;
                        }
                    }
                }
                continue;
            }
            // some nodes of every walk between two votes. A lane that meets sites to be tested (the leaf
            // children of its node) waits for the others: the test is long FP64 code.
            uint32_t found[ 2 ] = { kNone, kNone };
#pragma unroll 1
            for ( uint32_t turn = 0; turn < kSpecSteps && active && ( found[ 0 ] & found[ 1 ] ) == kNone; turn++ )
            {
                if ( ++steps > kLaneBudget )
                {
                    // a long search: restart it on a whole warp (k_edge_heavy)
                    const uint32_t slot = atomicAdd( b.heavy_count, 1u );
                    if ( slot < b.heavy_cap )
                        b.heavy[ slot ] = make_uint2( s.t, s.e );
                    else
                        send_to_exact( b, s.t, s.e ); // with a full search of this edge
                    active = false;
                    break;
                }
                Box      lb, rb;
                uint32_t lc, rc;
                load_node( c.nodes, node, lb, rb, lc, rc );
                uint32_t   next = kNone;
                const bool eL = enter_child( s, lb, lc >= n - 1 ), eR = enter_child( s, rb, rc >= n - 1 );
                if ( eL )
                {
                    if ( lc >= n - 1 )
                        found[ 0 ] = lc - ( n - 1 );
                    else
                        next = lc;
                }
                if ( eR )
                {
                    if ( rc >= n - 1 )
                        found[ 1 ] = rc - ( n - 1 );
                    else if ( next == kNone )
                        next = rc;
                    else if ( sp < int( kStack ) )
                        stack[ sp++ ] = rc;
                    else
                        err |= kErrStack;
                }
                // the edge's own sites and the neighbours that bound it touch every ball
#pragma unroll
                for ( uint32_t q = 0; q < 2; q++ )
                    if ( found[ q ] == s.i || found[ q ] == s.k || found[ q ] == s.l || found[ q ] == s.hint[ 0 ] || found[ q ] == s.hint[ 1 ] )
                        found[ q ] = kNone;
                if ( next != kNone )
                    node = next;
                else if ( sp > 0 )
                    node = stack[ --sp ];
                else
                    active = false; // once the sites found are tested
            }
            // the sites found, of all lanes together
#pragma unroll 1
            for ( uint32_t q = 0; q < 2; q++ )
            {
                const uint32_t j = q ? found[ 1 ] : found[ 0 ];
                if ( j != kNone && contributes( c, s, j ) )
                {
                    send_to_exact( b, s.t, s.e );
                    active = false;
                    break;
                }
            }
        }
        if ( err )
            atomicOr( error, err );
    }

    // Searches that outgrew one lane: the warp walks the tree together, 32 nodes per step
    // from a shared stack. Only whether a contributor exists matters here, which does not
    // depend on the visit order, so a long walk can also be cut into subtrees that other
    // warps finish (k_edge_heavy spills its stack once it holds kSplitAt nodes; k_edge_heavy_sub
    // walks each spilled subtree).
    enum WalkEnd : uint32_t
    {
        kWalkDone,
        kWalkFound,
        kWalkOverflow,
        kWalkSplit
    };

    __device__ uint32_t cooperative_walk( const CellContext & c, const EdgeSearch & s, uint32_t * st, uint32_t & size,
                                          uint32_t split_at )
    {
        const uint32_t lane = lane_of();
        const uint32_t n    = c.n;
        while ( size > 0 )
        {
            if ( size >= split_at )
                return kWalkSplit;
            const uint32_t take = min( size, 32u );
            uint32_t       node = kNone;
            if ( lane < take )
                node = st[ size - take + lane ];
            size -= take;
            __syncwarp();
            bool     hit = false, eL = false, eR = false;
            uint32_t lc = 0, rc = 0;
            if ( node != kNone )
            {
                if ( node >= n - 1 )
                    hit = node < 2 * n - 1 && contributes( c, s, node - ( n - 1 ) );
                else
                {
                    Box lb, rb;
                    load_node( c.nodes, node, lb, rb, lc, rc );
                    eL = enter_child( s, lb, lc >= n - 1 );
                    eR = enter_child( s, rb, rc >= n - 1 );
                }
            }
            if ( __any_sync( 0xffffffffu, hit ) )
                return kWalkFound;
            const uint32_t pushes = uint32_t( eL ) + uint32_t( eR );
            uint32_t       x      = pushes;
#pragma unroll
            for ( int o = 1; o < 32; o <<= 1 )
            {
                const uint32_t y = __shfl_up_sync( 0xffffffffu, x, o );
                if ( lane >= uint32_t( o ) )
                    x += y;
            }
            const uint32_t total = __shfl_sync( 0xffffffffu, x, 31 );
            uint32_t       off   = x - pushes;
            if ( size + total > kHeavyStack )
                return kWalkOverflow;
            if ( eL )
                st[ size + off++ ] = lc;
            if ( eR )
                st[ size + off ] = rc;
            size += total;
            __syncwarp();
        }
        return kWalkDone;
    }

    // The search of a listed edge. Whether the security radius covers it was decided where it was
    // listed and is not asked again: that compares floats near a threshold, and another copy of the
    // code may round them the other way.
    __device__ __forceinline__ void search_of_heavy( const CellContext & c, const uint32_t * tasks, const SpecBuffers & b,
                                                     uint2 h, EdgeSearch & s )
    {
        s.t           = h.x;
        s.e           = h.y;
        s.i           = tasks[ s.t ];
        const uint4 r = c.edges[ store_row( c, s.i ) * kMaxEdges + s.e ];
        s.k           = r.x;
        s.l           = r.y;
        s.closed      = r.z == kNone;
        s.si          = c.sites[ s.i ];
        s.sk          = c.sites[ s.k ];
        s.sl          = c.sites[ s.l ];
        s.nbr         = b.nbr + size_t( s.t ) * kNbrCap;
        s.nbr_count   = b.nbr_count[ s.t ];
        double4    ev0, ev1;
        const bool ellipse = bound_edge( s, ev0, ev1 );
        set_reach( c, s, ellipse, ev0, ev1 );
    }

    __global__ void __launch_bounds__( kHeavyBlock, 4 ) k_edge_heavy( CellContext c, const uint32_t * __restrict__ tasks,
                                                                      SpecBuffers b, uint32_t * error )
    {
        __shared__ uint32_t stacks[ kHeavyBlock / 32 ][ kHeavyStack ];
        const uint32_t      warp  = threadIdx.x >> 5, lane = lane_of();
        uint32_t *          st    = stacks[ warp ];
        const uint32_t      count = min( *b.heavy_count, b.heavy_cap );
        while ( true )
        {
            uint32_t item = 0;
            if ( lane == 0 )
                item = atomicAdd( b.heavy_next, 1u );
            item = __shfl_sync( 0xffffffffu, item, 0 );
            if ( item >= count )
                break;
            const uint2 h = b.heavy[ item ];
            // Edges of a cell that already goes to the exact path are still searched: every
            // edge proven empty here is one the exact pass skips.
            if ( b.cell_flag[ h.x ] & kFlagOverflow )
            {
                if ( lane == 0 )
                    atomicOr( &b.maybe_bits[ size_t( h.x ) * kMaybeWords + ( h.y >> 5 ) ], 1u << ( h.y & 31 ) );
                continue;
            }
            EdgeSearch s;
            search_of_heavy( c, tasks, b, h, s );
            uint32_t size = 1;
            if ( lane == 0 )
                st[ 0 ] = s.from;
            __syncwarp();
            const uint32_t end = cooperative_walk( c, s, st, size, kSplitAt );
            if ( end == kWalkSplit )
            {
                // hand the pending subtrees to other warps, with the search's set-up computed once
                // for all of them (a full slot table leaves them to recompute it)
                uint32_t base = 0, slot = 0;
                if ( lane == 0 )
                {
                    base = atomicAdd( b.sub_count, size );
                    slot = atomicAdd( b.split_count, 1u );
                    if ( slot < b.split_cap )
                        static_cast<EdgeSearch *>( b.splits )[ slot ] = s;
                }
                base = __shfl_sync( 0xffffffffu, base, 0 );
                slot = __shfl_sync( 0xffffffffu, slot, 0 );
                const uint32_t search = slot < b.split_cap ? ( slot | kSplitSlot ) : item;
                if ( base + size <= b.sub_cap )
                {
                    for ( uint32_t q = lane; q < size; q += 32 )
                        b.sub[ base + q ] = make_uint2( search, st[ q ] );
                }
                else if ( lane == 0 )
                    send_to_exact( b, s.t, s.e );
            }
            else if ( ( end == kWalkFound || end == kWalkOverflow ) && lane == 0 )
                send_to_exact( b, s.t, s.e );
            __syncwarp();
        }
    }

    __global__ void __launch_bounds__( kHeavyBlock, 4 ) k_edge_heavy_sub( CellContext c, const uint32_t * __restrict__ tasks,
                                                                          SpecBuffers b, uint32_t * error )
    {
        __shared__ uint32_t stacks[ kHeavyBlock / 32 ][ kHeavyStack ];
        const uint32_t      warp  = threadIdx.x >> 5, lane = lane_of();
        uint32_t *          st    = stacks[ warp ];
        const uint32_t      count = min( *b.sub_count, b.sub_cap );
        while ( true )
        {
            uint32_t q = 0;
            if ( lane == 0 )
                q = atomicAdd( b.sub_next, 1u );
            q = __shfl_sync( 0xffffffffu, q, 0 );
            if ( q >= count )
                break;
            const uint2 sub    = b.sub[ q ];
            const bool  cached = ( sub.x & kSplitSlot ) != 0;
            EdgeSearch  s;
            uint2       h;
            if ( cached )
            {
                s = static_cast<const EdgeSearch *>( b.splits )[ sub.x & ~kSplitSlot ];
                h = make_uint2( s.t, s.e );
            }
            else
                h = b.heavy[ sub.x ];
            // another part of this edge's search already found a contributor
            if ( ( b.cell_flag[ h.x ] & kFlagOverflow )
                 || ( ( b.maybe_bits[ size_t( h.x ) * kMaybeWords + ( h.y >> 5 ) ] >> ( h.y & 31 ) ) & 1u ) )
            {
                if ( lane == 0 )
                    atomicOr( &b.maybe_bits[ size_t( h.x ) * kMaybeWords + ( h.y >> 5 ) ], 1u << ( h.y & 31 ) );
                continue;
            }
            if ( !cached )
                search_of_heavy( c, tasks, b, h, s );
            uint32_t size = 1;
            if ( lane == 0 )
                st[ 0 ] = sub.y;
            __syncwarp();
            const uint32_t end = cooperative_walk( c, s, st, size, kHeavyStack + 1 );
            if ( ( end == kWalkFound || end == kWalkOverflow ) && lane == 0 )
                send_to_exact( b, s.t, s.e );
            __syncwarp();
        }
    }

    // Cells with no contributor are final: every edge validated, the cell validated
    // (what the reference's pass leaves when no update happens). The others are listed for
    // the exact pass.
    __global__ void k_edge_commit( CellContext c, const uint32_t * __restrict__ tasks, const uint32_t * __restrict__ task_count,
                                   SpecBuffers b )
    {
        const uint32_t gwarp = ( blockIdx.x * blockDim.x + threadIdx.x ) >> 5;
        const uint32_t nwarp = ( gridDim.x * blockDim.x ) >> 5;
        const uint32_t lane  = lane_of();
        const uint32_t count = *task_count;
        for ( uint32_t t = gwarp; t < count; t += nwarp )
        {
            const uint32_t i  = tasks[ t ];
            const uint8_t  st = c.status[ i ];
            if ( st == kFullyValidated || st == kBuried )
                continue;
            if ( b.cell_flag[ t ] )
            {
                if ( lane == 0 )
                {
                    const uint32_t q  = atomicAdd( b.exact_count, 1u );
                    b.exact_tasks[ q ] = i;
                    b.exact_slot[ q ]  = t;
                }
                continue;
            }
            const uint32_t en = c.edge_nb[ i ];
            for ( uint32_t e = lane; e < en; e += 32 )
            {
                uint32_t * w = &c.edges[ store_row( c, i ) * kMaxEdges + e ].w;
                *w           = ( *w & 0xffffff00u ) | 1u;
            }
            if ( lane == 0 )
                c.status[ i ] = kFullyValidated;
        }
    }

    // -----------------------------------------------------------------------------------
    // Bisector validation as a search over all (cell, neighbour) pairs, with the warp-per-cell pass
    // (k_bisector_validation) for the cells where one found a site
    // -----------------------------------------------------------------------------------
    // A bisector (i, k) is searched for a site inside the cylinder between its two spheres that would
    // close a trisector on it (algorithm.inl:859-1233). Hardly any is found, and while none is the
    // cell stays as it is, so as for the edges only existence matters and the pairs of all cells are
    // independent: each is one lane's item. The warp-per-cell pass had a cell's 7 or so neighbours of
    // larger id on 32 lanes, 150 registers and its cell in shared memory for each such walk; bound by
    // the latency of dependent node loads, which 64 registers and full warps hide far better. With
    // the pruned entry below: 1M-site protein packing 67.6 -> 7.5 ms (2.5 of it the neighbour
    // lists), 1M log-normal cloud 97 -> 30 ms (5.9 in the exact pass), 61k protein 13.1 -> 0.6 ms
    // (one cell's walk), 46^3 lattice 4.7 -> 0.5 ms.
    struct BisectorSearch
    {
        uint32_t t, i, k;
        float3   fci, fck;
        float4   bsph;     // the ball that must hold the site
        float    cylinder; // and the radius of the cylinder around the axis
        // entering a box: the site's sphere lies in the ball, so a box at a distance has to reach at
        // least a smallest sphere's diameter (`shrink`, less a rounding margin) into it; and it
        // lies in the cylinder, so the box has to come within `tube` of the axis
        float3   axis;
        float    shrink, tube, slack;
    };

    // Sets up the search of pair (i, k); false when the security radius covers it.
    __device__ __forceinline__ bool setup_bisector( const CellContext & c, BisectorSearch & s, float known )
    {
        const float4 si = c.sites_f[ s.i ], sk = c.sites_f[ s.k ];
        s.fci = f3( si );
        s.fck = f3( sk );
        if ( lt_eps( flength( s.fci - s.fck ) + si.w + sk.w, known ) )
            return false;
        const float3 center = ( s.fci + s.fck ) * .5f;
        const float  radius = flength( center - s.fci ) + fmaxf( si.w, sk.w );
        s.bsph              = make_float4( center.x, center.y, center.z, radius );
        s.cylinder          = fmaxf( si.w, sk.w );
        // Margins: the leaf's containment test rounds within 4e-7 of the radius, boxes and centre
        // within 2e-7 of the coordinates; the distance from the axis is a root of a difference
        // of squares that are off by 1.1e-6 of the squared distance from c_i, at most twice the
        // radius. Each is taken several times over.
        const float diameter = 2.f * fmaxf( 0.f, float( c.scene->rmin ) );
        const float reach    = 4e-6f * ( fabsf( center.x ) + fabsf( center.y ) + fabsf( center.z ) + radius );
        s.shrink             = fmaxf( 0.f, diameter - reach );
        s.slack              = 5e-6f;
        s.tube               = s.cylinder - s.shrink + fmaxf( 0.f, -float( c.scene->rmin ) ) + 6e-3f * radius + reach;
        s.axis               = fnormalize( s.fck - s.fci );
        return true;
    }

    __device__ __forceinline__ bool enter_child( const BisectorSearch & s, const Box & b )
    {
        const float d = b.distance( s.bsph );
        // -radius: the centre is inside the box
        if ( !( d < 0.f ) || !( d < -s.shrink || d == -s.bsph.w ) )
            return false;
        const float3 half = ( b.hi - b.lo ) * .5f;
        const float3 from = ( b.lo + b.hi ) * .5f - s.fci;
        const float  v    = fdot( from, s.axis ), ff = fdot( from, from );
        const float  r    = s.tube + flength( half ) * 1.0001f;
        return !( ff - v * v - s.slack * ff > r * r ); // r > 0; NaN enters
    }

    __device__ __forceinline__ bool closes_trisector( const CellContext & c, const SpecBuffers & b, const BisectorSearch & s, uint32_t j )
    {
        if ( j == s.i || j == s.k )
            return false;
        const float4 fj = c.sites_f[ j ];
        const float3 cj = f3( fj );
        if ( !( s.bsph.w >= fj.w && ( flength( f3( s.bsph ) - cj ) <= ( s.bsph.w - fj.w ) ) ) )
            return false;
        const float3 itoj = cj - s.fci;
        const float  v    = fdot( itoj, s.axis );
        const float  d    = sqrtf( fdot( itoj, itoj ) - v * v );
        if ( !( ( d + fj.w ) < s.cylinder ) )
            return false;
        const uint32_t * nbr   = b.nbr + size_t( s.t ) * kNbrCap;
        const uint32_t   count = b.nbr_count[ s.t ];
        if ( in_sorted( nbr, count, j ) )
            return false;
        double4 x0 = make_double4( 0, 0, 0, 0 ), x1 = make_double4( 0, 0, 0, 0 );
        if ( trisector( c.sites[ s.i ], c.sites[ j ], c.sites[ s.k ], x0, x1 ) != 2 )
            return false;
        FilterTally untallied;
        for ( uint32_t q = 0; q < count; q++ )
            if ( nbr[ q ] != s.k
                 && ( c.fp32 ? site_conflict<true>( c, nbr[ q ], x1, untallied ) : site_conflict<false>( c, nbr[ q ], x1, untallied ) ) )
                return false;
        return true;
    }

    __global__ void __launch_bounds__( kSpecBlock, 8 ) k_bisector_speculate( CellContext c, SpecBuffers b )
    {
        const uint32_t count = c.hi - c.lo;
        const uint64_t total = *b.item_total;
        const uint32_t n     = c.n;
        uint32_t       err   = 0;

        BisectorSearch s;
        bool           active = false, exhausted = false;
        uint32_t       stack[ kStack ];
        int            sp   = 0;
        uint32_t       node = 0;
        while ( true )
        {
            const uint32_t idle = __ballot_sync( 0xffffffffu, !active && !exhausted );
            const uint32_t busy = __ballot_sync( 0xffffffffu, active );
            if ( idle == 0 && busy == 0 )
                break;
            if ( idle != 0 && ( busy == 0 || uint32_t( __popc( idle ) ) >= kBisectorRefillAt ) )
            {
                if ( !active && !exhausted )
                {
                    const uint32_t leader = __ffs( idle ) - 1;
                    uint64_t       base   = 0;
                    if ( lane_of() == leader )
                        base = atomicAdd( reinterpret_cast<unsigned long long *>( b.item_counter ), __popc( idle ) );
                    base                = __shfl_sync( idle, base, leader );
                    const uint64_t item = base + __popc( idle & ( ( 1u << lane_of() ) - 1u ) );
                    if ( item >= total )
                        exhausted = true;
                    else
                    {
                        uint32_t lo = 0, hi = count;
                        while ( hi - lo > 1 )
                        {
                            const uint32_t mid = ( lo + hi ) >> 1;
                            if ( b.item_offset[ mid ] <= item )
                                lo = mid;
                            else
                                hi = mid;
                        }
                        s.t = lo;
                        s.i = c.lo + lo;
                        // the item's place among the sorted neighbours, counted from the first above i
                        const uint32_t * nbr   = b.nbr + size_t( s.t ) * kNbrCap;
                        uint32_t         first = 0, last = b.nbr_count[ s.t ];
                        while ( first < last )
                        {
                            const uint32_t mid = ( first + last ) >> 1;
                            if ( nbr[ mid ] <= s.i )
                                first = mid + 1;
                            else
                                last = mid;
                        }
                        s.k = nbr[ first + uint32_t( item - b.item_offset[ s.t ] ) ];
                        if ( setup_bisector( c, s, c.known_radii[ s.i ] ) )
                        {
                            active = true;
                            sp     = 0;
                            node   = 0;
                        }
                    }
                }
                continue;
            }
            // some nodes of every walk between two votes; the leaf children of a node are tested with it
#pragma unroll 1
            for ( uint32_t step = 0; step < kBisectorSteps && active; step++ )
            {
                Box      lb, rb;
                uint32_t lc, rc;
                load_node( c.nodes, node, lb, rb, lc, rc );
                const bool eL = enter_child( s, lb ), eR = enter_child( s, rb );
                uint32_t   next = kNone;
                bool       hit  = false;
                if ( eL )
                {
                    if ( lc >= n - 1 )
                        hit = closes_trisector( c, b, s, lc - ( n - 1 ) );
                    else
                        next = lc;
                }
                if ( eR && !hit )
                {
                    if ( rc >= n - 1 )
                        hit = closes_trisector( c, b, s, rc - ( n - 1 ) );
                    else if ( next == kNone )
                        next = rc;
                    else if ( sp < int( kStack ) )
                        stack[ sp++ ] = rc;
                    else
                        err |= kErrStack;
                }
                if ( hit )
                {
                    atomicOr( &b.cell_flag[ s.t ], kFlagFound );
                    active = false;
                }
                else if ( next != kNone )
                    node = next;
                else if ( sp > 0 )
                    node = stack[ --sp ];
                else
                    active = false;
            }
        }
        if ( err )
            atomicOr( c.error, err );
    }

    // Cells where no bisector found a site are validated; the others are listed for the exact pass.
    __global__ void k_bisector_commit( CellContext c, SpecBuffers b )
    {
        const uint32_t t = blockIdx.x * blockDim.x + threadIdx.x;
        if ( t >= c.hi - c.lo || c.status[ c.lo + t ] == kBuried )
            return;
        if ( b.cell_flag[ t ] )
            b.exact_tasks[ atomicAdd( b.exact_count, 1u ) ] = c.lo + t;
        else
            c.status[ c.lo + t ] = kFullyValidated;
    }

    // long lane searches per round: log-normal radii reach 1.5 per site
    static size_t heavy_capacity( uint32_t n ) { return 6 * size_t( n ) + 65536; }
    static size_t sub_capacity( uint32_t n ) { return 4 * size_t( n ) + 65536; }
    // searches split into subtrees per round (each hands out up to kSplitAt subtrees)
    static size_t split_capacity( uint32_t n ) { return size_t( n ) / 8 + 4096; }

    size_t spec_bytes( uint32_t n )
    {
        auto a = []( size_t x ) { return ( x + 255 ) & ~size_t( 255 ); };
        return a( 4 * size_t( n ) * kNbrCap ) + a( 4 * size_t( n ) ) * 5 + a( 16 )
               + a( 4 * output_scan_scratch_words( n ) ) + a( sizeof( uint2 ) * heavy_capacity( n ) )
               + a( 4 * size_t( n ) * kMaybeWords ) + a( sizeof( uint2 ) * sub_capacity( n ) )
               + a( sizeof( EdgeSearch ) * split_capacity( n ) );
    }

    void spec_carve( SpecBuffers & b, void * base, uint32_t n )
    {
        auto   a = []( size_t x ) { return ( x + 255 ) & ~size_t( 255 ); };
        char * p = static_cast<char *>( base );
        b.nbr    = reinterpret_cast<uint32_t *>( p );
        p += a( 4 * size_t( n ) * kNbrCap );
        b.nbr_count = reinterpret_cast<uint32_t *>( p );
        p += a( 4 * size_t( n ) );
        b.item_count = reinterpret_cast<uint32_t *>( p ); // becomes the offsets after the scan
        b.item_offset = b.item_count;
        p += a( 4 * size_t( n ) );
        b.cell_flag = reinterpret_cast<uint32_t *>( p );
        p += a( 4 * size_t( n ) );
        b.exact_tasks = reinterpret_cast<uint32_t *>( p );
        p += a( 4 * size_t( n ) );
        b.exact_slot = reinterpret_cast<uint32_t *>( p );
        p += a( 4 * size_t( n ) );
        b.item_total = reinterpret_cast<uint64_t *>( p );
        p += a( 16 );
        b.scan_sums = reinterpret_cast<uint32_t *>( p );
        p += a( 4 * output_scan_scratch_words( n ) );
        b.heavy = reinterpret_cast<uint2 *>( p );
        p += a( sizeof( uint2 ) * heavy_capacity( n ) );
        b.maybe_bits = reinterpret_cast<uint32_t *>( p );
        p += a( 4 * size_t( n ) * kMaybeWords );
        b.sub = reinterpret_cast<uint2 *>( p );
        p += a( sizeof( uint2 ) * sub_capacity( n ) );
        b.splits      = p;
        b.split_cap   = uint32_t( split_capacity( n ) );
        b.sub_cap   = uint32_t( sub_capacity( n ) );
        b.heavy_cap = uint32_t( heavy_capacity( n ) );
    }

    // Persistent grid sizes per device (148 SMs x resident blocks of each kernel on B200).
    constexpr int        kSpecDevices = 64;
    static int           g_spec_grid[ kSpecDevices ], g_heavy_grid[ kSpecDevices ], g_bisector_grid[ kSpecDevices ];
    static PerDeviceOnce g_spec_config;

    static int spec_device()
    {
        int dev = 0;
        cudaGetDevice( &dev );
        return ( dev >= 0 && dev < kSpecDevices ) ? dev : -1;
    }

    void configure_spec_kernels()
    {
        g_spec_config.run( [] {
            const int dev = spec_device();
            if ( dev < 0 )
                return;
            int sms = 148, per_sm = 0;
            cudaDeviceGetAttribute( &sms, cudaDevAttrMultiProcessorCount, dev );
            cudaOccupancyMaxActiveBlocksPerMultiprocessor( &per_sm, k_edge_speculate, kSpecBlock, 0 );
            g_spec_grid[ dev ] = sms * std::max( 1, per_sm );
            cudaOccupancyMaxActiveBlocksPerMultiprocessor( &per_sm, k_edge_heavy, kHeavyBlock, 0 );
            g_heavy_grid[ dev ] = sms * std::max( 1, per_sm );
            cudaOccupancyMaxActiveBlocksPerMultiprocessor( &per_sm, k_bisector_speculate, kSpecBlock, 0 );
            g_bisector_grid[ dev ] = sms * std::max( 1, per_sm );
        } );
    }

    void launch_edge_validation_speculative( const CellContext & context, const uint32_t * tasks, const uint32_t * task_count,
                                             const SpecBuffers & buffers, ZeroWords & z, cudaStream_t s )
    {
        CellContext c  = context;
        SpecBuffers b  = buffers;
        c.work_counter = z.take();
        b.item_counter = z.take64();
        b.exact_count  = z.take();
        b.heavy_count  = z.take();
        b.heavy_next   = z.take();
        b.sub_count    = z.take();
        b.sub_next     = z.take();
        b.split_count  = z.take();
        configure_spec_kernels();
        const int dev        = spec_device();
        const int spec_grid  = dev >= 0 ? g_spec_grid[ dev ] : 148 * 4; // an ordinal outside the table
        const int heavy_grid = dev >= 0 ? g_heavy_grid[ dev ] : 148 * 4;
        const uint32_t nbr_blocks = std::max( 1u, std::min<uint32_t>( ( c.n + 3 ) / 4, 148 * 32 ) );
        APO2_LAUNCH( "k_neighbor_lists", s, k_neighbor_lists<false><<<nbr_blocks, kNbrBlock, 0, s>>>( c, tasks, task_count, b ) );
        APO2_LAUNCH( "k_edge_cells", s, k_edge_cells<<<cell_grid_blocks( c.n ), kCellBlock, 0, s>>>( c, tasks, task_count, b ) );
        scan_exclusive( b.item_count, c.n, b.scan_sums, b.item_total, s );
        APO2_LAUNCH( "k_edge_speculate", s, k_edge_speculate<<<spec_grid, kSpecBlock, 0, s>>>( c, tasks, task_count, b, c.error ) );
        APO2_LAUNCH( "k_edge_heavy", s, k_edge_heavy<<<heavy_grid, kHeavyBlock, 0, s>>>( c, tasks, b, c.error ) );
        APO2_LAUNCH( "k_edge_heavy_sub", s, k_edge_heavy_sub<<<heavy_grid, kHeavyBlock, 0, s>>>( c, tasks, b, c.error ) );
        APO2_LAUNCH( "k_edge_commit", s, k_edge_commit<<<std::max( 1u, std::min<uint32_t>( ( c.n + 7 ) / 8, 148 * 16 ) ), 256, 0, s>>>( c, tasks, task_count, b ) );
        SearchProof proof;
        proof.slots      = b.exact_slot;
        proof.maybe_bits = b.maybe_bits;
        proof.nbr        = b.nbr;
        proof.nbr_count  = b.nbr_count;
        launch_edge_validation( c, b.exact_tasks, b.exact_count, z, s, proof );
    }

    void launch_bisector_validation_speculative( const CellContext & c, const SpecBuffers & buffers, ZeroWords & z, cudaStream_t s )
    {
        SpecBuffers b  = buffers;
        b.item_counter = z.take64();
        b.exact_count  = z.take();
        configure_spec_kernels();
        const int      dev        = spec_device();
        const int      grid       = dev >= 0 ? g_bisector_grid[ dev ] : 148 * 8; // an ordinal outside the table
        const uint32_t cells      = c.hi - c.lo;
        const uint32_t nbr_blocks = std::max( 1u, std::min<uint32_t>( ( c.n + 3 ) / 4, 148 * 32 ) );
        APO2_LAUNCH( "k_neighbor_lists", s, k_neighbor_lists<true><<<nbr_blocks, kNbrBlock, 0, s>>>( c, nullptr, nullptr, b ) );
        scan_exclusive( b.item_count, c.n, b.scan_sums, b.item_total, s );
        APO2_LAUNCH( "k_bisector_speculate", s, k_bisector_speculate<<<grid, kSpecBlock, 0, s>>>( c, b ) );
        APO2_LAUNCH( "k_bisector_commit", s, k_bisector_commit<<<std::max( 1u, ( cells + 255 ) / 256 ), 256, 0, s>>>( c, b ) );
        launch_bisector_validation( c, b.exact_tasks, b.exact_count, z, s );
    }
} // namespace apo2
