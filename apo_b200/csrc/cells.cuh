// Cell-construction kernels: shared constants, the device context and launch helpers.
#pragma once

#include "internal.cuh"
#include "proposal.cuh"

namespace apo2
{
    constexpr uint32_t kCellBlock = 128; // 4 warps, one cell per warp at a time
    constexpr uint32_t kKnnBlock  = 256; // one site per thread
    constexpr uint32_t kMaxK      = 16;  // kNN heap slots per thread (the reference's K)
    constexpr uint32_t kStack     = 64;  // traversal stack entries (the tree height bound)

    // Shared-memory slots per warp: the reference capacities plus room for the records an
    // update appends before it compacts; writes past the slots are dropped and flagged.
    //
    // Sites of the neighbour list: what the 57,344 bytes a block may have at four blocks per SM leave
    // over. A cell of simple vertices with E edges has E / 3 + 2 neighbours, so only cells above
    // 230 edges (of 264) can outgrow it; their edges are scanned instead.
    //
    // Small cells, nearly all (20 to 27 vertices, 31 to 40 edges on average), take part of that, which
    // leaves the rest of the SM's 256 KB to the L1 cache: the walks' nodes, sites and stacks hit it.
    // A cell that outgrows the small slots is done again from its start by a second launch. (64 / 96
    // and 128 / 208 slots: vertex validation of the 1M log-normal cloud 122 and 105.5 ms, of the 1M
    // protein packing 168 and 172 ms, against 104.9 and 165.9 ms.)
    template<bool Small>
    struct CellSlots
    {
        static constexpr uint32_t kVertices = Small ? 96 : 192;
        static constexpr uint32_t kEdges    = Small ? 160 : 296;
        static constexpr uint32_t kSites    = Small ? 64 : 80;
        static constexpr size_t   kBytes    = ( sizeof( double4 ) + sizeof( uint4 ) ) * kVertices + sizeof( uint4 ) * kEdges
                                         + sizeof( uint32_t ) * kSites;
        static_assert( kBytes % 32 == 0, "warp cell must keep double4 alignment" );
    };
    constexpr size_t   kBisectorBytes = sizeof( uint32_t ) * 2 * kMaxBisectors;

    inline size_t cell_smem_bytes( bool bisector )
    {
        return ( CellSlots<false>::kBytes + ( bisector ? kBisectorBytes : 0 ) ) * ( kCellBlock / 32 );
    }
    inline size_t small_cell_smem_bytes() { return CellSlots<true>::kBytes * ( kCellBlock / 32 ); }

    // Words that one memset at the start of a build clears: every counter of its launches is a fresh one,
    // so that no launch has to wait for a memset of its own (they were half of a round's operations).
    class ZeroWords
    {
      public:
        static constexpr uint32_t kPerRound = 24, kOther = 64;
        explicit ZeroWords( uint32_t * base ) : next_( base ) {}
        uint32_t * take() { return next_++; }
        uint64_t * take64() // base is 8-byte aligned
        {
            next_ += ( reinterpret_cast<uintptr_t>( next_ ) >> 2 ) & 1u;
            uint64_t * p = reinterpret_cast<uint64_t *>( next_ );
            next_ += 2;
            return p;
        }

      private:
        uint32_t * next_;
    };

    struct CellContext
    {
        uint32_t         n = 0, k = 16;
        uint32_t         lo = 0, hi = 0; // cells built: sorted ids [lo, hi) (a shard of the diagram)
        const double4 *  sites   = nullptr; // n + 6, Morton order then the artificial sites
        const float4 *   sites_f = nullptr; // n
        const WideNode * nodes   = nullptr;
        const uint32_t * indices = nullptr; // sorted -> original
        uint8_t *        status  = nullptr;
        uint32_t *       knn     = nullptr; // n * k
        float *          known_radii = nullptr;
        uint32_t *       vertex_nb   = nullptr;
        uint32_t *       edge_nb     = nullptr;
        uint4 *          vertices    = nullptr; // n * 152 records (j, k, l, type | status << 8)
        uint4 *          edges       = nullptr; // n * 264 records (j, k, vertex count, status)
        uint32_t *       error       = nullptr;
        const Scene *    scene       = nullptr; // bounds and radius range of the sites
        uint32_t *       walk_scratch = nullptr; // kWalkScratchWords per warp of the exact edge pass
        uint32_t *       work_counter = nullptr; // next cell of the dynamically scheduled passes
        uint32_t *       deferred       = nullptr; // cells that outgrew the small slots, and their number
        uint32_t *       deferred_count = nullptr;
        // left by the vertex validation for the edge searches of the same round: the largest vertex
        // radius of each cell, and the node around everything within the general bound of its edges
        float * largest = nullptr;
        uint32_t * around = nullptr;
        // learned k-proposal (null: the plain form): the network, the Morton codes its features
        // read, and the proposed rank of every site (written by the first kNN step)
        const ProposalNet * proposal   = nullptr;
        const uint64_t *    codes      = nullptr;
        uint8_t *           proposed_k = nullptr;
        uint32_t            proposal_max = 0; // largest proposed rank (k .. 2k)
        uint32_t            scheduled    = 0; // 1: cells proposed beyond k get a second kNN step
        // build counters: kNN insertions, cells checked at a proposed rank, fallbacks, skipped
        // neighbours, conflict predicates decided by the FP32 filter, those it left to FP64
        unsigned long long * counters = nullptr;
        // FP32-filtered form: conflict predicates against sites first in single precision
        uint32_t fp32 = 0;
    };
    constexpr uint32_t kCountInsertions = 0, kCountChecked = 1, kCountFallbacks = 2, kCountSkipped = 3, kCountFiltered = 4,
                       kCountEscalated = 5, kCountSecondStep = 6, kCounters = 7;

    // Learned form with a second kNN step: is cell i one of those proposed beyond k?
    __device__ __forceinline__ bool second_step_cell( const CellContext & c, uint32_t i )
    {
        return c.scheduled && c.proposed_k[ i ] > c.k;
    }

    // Lane-local tallies of the FP32 filter, added to the build's counters when a kernel ends.
    struct FilterTally
    {
        uint32_t tests = 0, escalated = 0;
    };

    // The reference's conflict test of site `id` against the sphere x (gpu/math.cuh:374-388),
    // decided by the FP32 filter where it can in the filtered form (Fp32: a kernel instantiation of
    // its own, so that neither form carries the other's code through the instruction cache).
    template<bool Fp32>
    __device__ __forceinline__ bool site_conflict( const CellContext & c, uint32_t id, double4 x, FilterTally & t )
    {
        if constexpr ( Fp32 )
        {
            t.tests++;
            // the float copy holds the n input sites; the six bounding sites are rounded here
            const float4 s = id < c.n ? c.sites_f[ id ] : to_float( c.sites[ id ] );
            const int    f = conflict_filter( s, x );
            if ( f != 2 )
                return f == 1;
            t.escalated++;
        }
        return intersects_wide( c.sites[ id ], x );
    }
    // The same for a site given by value (its float copy is exact for float input and bounded otherwise).
    template<bool Fp32>
    __device__ __forceinline__ bool sphere_conflict( double4 site, double4 x, FilterTally & t )
    {
        if constexpr ( Fp32 )
        {
            t.tests++;
            const int f = conflict_filter( to_float( site ), x );
            if ( f != 2 )
                return f == 1;
            t.escalated++;
        }
        return intersects_wide( site, x );
    }

    // Row of cell i in the per-cell stores (vertices, edges), which hold only the cells
    // [lo, hi) a handle builds: a shard of the diagram needs stores for its own cells alone.
    __host__ __device__ __forceinline__ size_t store_row( const CellContext & c, uint32_t i ) { return size_t( i - c.lo ); }

    // Exact edge validation: a lane walks its edge's search alone for kLaneWalk steps; a
    // search still running then is finished by the whole warp, in the same order, from a
    // frontier of at most kCoopCap nodes kept in global scratch (plus each lane's saved stack),
    // kCoopWidth x 32 frontier nodes per step.
#ifndef APO2_EXACT_LANE_WALK
#define APO2_EXACT_LANE_WALK 256
#endif
    constexpr uint32_t kLaneWalk         = APO2_EXACT_LANE_WALK;
    // After the edge-parallel search a cell has few edges left to search, and a warp whose few walking
    // lanes go one node per step, each candidate stopping them all, takes longer than the same searches
    // one after another by the whole warp: they go there after 4 steps (longest launches of the pass
    // summed over the rounds, 256 -> 32 -> 4 steps: 100,000 uniform sites 5.4 -> 2.6 -> 1.8 ms, 10,000 0.42 ->
    // 0.29 -> 0.26, 300,000 log-normal 3.9 -> 3.7 -> 3.6, 800,000 8.2 -> 8.6 -> 8.2, 1M protein-like 1.1 ->
    // 0.6 -> 0.6). Without that search, and once a neighbour has left the cell and its proofs lapse, every edge
    // walks, 32 at a time, and lanes keep kLaneWalk (4 steps there too: the longest launch of 5M log-normal
    // sites 766 and 777 ms, all of the 126^3 lattice 1648 and 1645).
    constexpr uint32_t kLaneWalkLeft     = 4;
#ifndef APO2_COOP_WIDTH
#define APO2_COOP_WIDTH 4
#endif
    constexpr uint32_t kCoopWidth        = APO2_COOP_WIDTH; // frontier nodes per lane per step
    constexpr uint32_t kCoopCap          = 8192;
    constexpr uint32_t kWalkScratchWords = kCoopCap + 32 * ( kStack + 1 );
    // The edge search keeps a cell's surroundings in the same scratch: up to kListCap sites
    // (float4, then ids) and the stack of the walk that collects them. An edge's walk is 50 to 90
    // nodes whatever the density, its share of the list grows with it. Edge search of all kernels, with
    // lists of up to 64 / 128 / 256 / 384 / 1024 sites (0: 75.5, 105.9 and 7.7 ms): 1M protein packing
    // 76.9 / 73.8 / 72.7 / 74.6 / 88.6 ms, 1M log-normal cloud 112 / 107 / 86 / 83 / 75 ms, 46^3
    // lattice 6.0 / 5.9 / 6.0 / 5.8 / 5.9 ms.
    constexpr uint32_t kListCap   = 384;
    constexpr uint32_t kListStack = 4096;
    static_assert( 5 * kListCap + kListStack <= kWalkScratchWords && kWalkScratchWords % 4 == 0, "the list fits the scratch" );

    // Position of a stored vertex: root `type` of quadrisector(si, sj, sk, sl) with the
    // sorted ids (topology_update.inl:104-111).
    __device__ __forceinline__ double4 solve_vertex( const CellContext & c, double4 si, uint4 r )
    {
        double4 x[ 2 ] = { make_double4( 0, 0, 0, 0 ), make_double4( 0, 0, 0, 0 ) };
        quadrisector( si, c.sites[ r.x ], c.sites[ r.y ], c.sites[ r.z ], x[ 0 ], x[ 1 ] );
        return ( r.w & 0xffu ) ? x[ 1 ] : x[ 0 ];
    }

    // The sites the emptiness and known-neighbour tests range over, those of the cell's edges, as a
    // sequence. The neighbour list holds each once (an edge list names every neighbour about six
    // times); a cell with more neighbours than slots goes by its edges.
    struct SiteSequence
    {
        const uint32_t * words;
        uint32_t         count, shift; // shift 0: a list of ids; 1: two ids at the front of 16-byte records
        __device__ __forceinline__ uint32_t operator[]( uint32_t q ) const
        {
            return words[ ( ( q >> shift ) << ( 2 * shift ) ) + ( q & shift ) ];
        }
    };
    // ---------------------------------------------------------------------------------
    // Reach of an edge search. A site j contributes to edge (k, l) of cell i only through a
    // root x that passes the emptiness test against the cell's neighbours, i.e. a point of
    // the edge's arc inside the current cell, whose empty-sphere radius w(x) is at most the
    // largest radius over the arc: its vertices and, on an elliptic trisector, an apex that
    // may lie on the arc (the cell certificate of the reference rests on the same bound,
    // algorithm.inl:186-190, topology_update.inl:595-653). Sphere j touches the sphere of radius
    // w(x) around x, so the search may skip every BVH node and leaf away from all such spheres: the
    // leaves it visits are a subsequence of the reference's, in the same order, and every site
    // that could contribute is among them, so the first contributor found is the same.
    //
    // That bound is kReachBall: one ball around c_i, |c_j - c_i| <= 2 w + r_i + r_max, or the
    // reference's own bounding sphere where that is smaller. Between two vertices the spheres along
    // the arc lie in three far smaller balls, and arc_reach shows for each edge that the rest of the
    // trisector is closed by neighbours of the cell, whichever vertices the cell has or lacks: with
    // duplicate sites, and where roots went lost to rounding, a cell lacks some, and an arc between two
    // of the others is not all that is open.
    //
    // Two kinds of contributor lie outside the balls all the same.
    //
    // A root so far away that the single-precision lengths of the emptiness test cannot tell the
    // neighbours apart (its radius was 7e7 and more where it happened, once in some ten builds, on edges
    // of hull cells). The reference takes such a root, so it has to be found. A neighbour that stands out by h
    // beyond the tangent plane conflicts by about as much with every root there, which rounding hides
    // from a radius of h / 4e-7 on: `far`, at most kFarRoot. From there on a site of such a root touches the
    // plane, so on a hyperbolic trisector the boxes that reach one of the two planes within the general
    // bound are entered too (kReachArcPlanes); an elliptic one has no point further than its apex. Most
    // planes are out, though (far_roots_blocked).
    //
    // A root of four sites whose centres lie in a plane, but for rounding: its height over the plane is a quotient
    // of two small numbers, and it can come out anywhere. Of relative errors of 1.1e-16 in coordinates of
    // size L and a height h of c_j over the plane of the other three, the root's height is off by up to
    // 1e-8 L sqrt(w d) / h, d the difference of the radii, which is inside the balls' margin from h = 1.7e-6 L
    // sqrt(d) on; centres nearer than kFlat L_1 (L_1 the sum over the axes, and 1 / sin of the triangle's angle
    // more) are tested within the general bound.
    // ---------------------------------------------------------------------------------
    constexpr uint32_t kReachBall = 0, kReachArc = 1, kReachArcPlanes = 2;
    constexpr double   kFarRoot   = 2.5e5; // radius from which a root counts as far: single precision is off by 0.1 there
    constexpr float    kFarOut    = 2.5e6f; // ... by 4e-7 of the radius: least radius, by the depth of the conflict
    constexpr float    kFlat      = 2e-6f; // of the coordinates: centres so near to a plane count as in it

    struct EdgeReach
    {
        float4   ball[ 3 ]; // kReachBall: the same one three times
        float4   limit;     // ball holding every site that the planes let in
        float    slab[ 2 ]; // kReachArcPlanes: how near to each tangent plane it has to come
        float4   flat;      // the plane of the three centres (normal, offset), and how near a centre
        float    near;      // has to come to it
        // hyperbolic trisectors: a contributor lies wholly below both planes (algorithm.inl:695-700), so
        // a box has to go below them by a smallest sphere's diameter; less this rounding margin
        float    diameter, margin;
        float    far; // kReachArcPlanes: least radius of a far root
        bool     below;
        uint32_t kind;
    };
    struct TangentPlanes
    {
        float3 n1, n2, p1, p2;
    };

    __device__ __forceinline__ bool meets( float4 ball, const Box & b )
    {
        const float3 d = f3( ball ) - b.closest( ball );
        return fdot( d, d ) <= ball.w * ball.w;
    }
    __device__ __forceinline__ bool meets( float4 ball, float4 site )
    {
        const float3 d = f3( ball ) - f3( site );
        const float  r = ball.w + site.w;
        return ( r >= 0.f ) & ( fdot( d, d ) <= r * r );
    }
    // Heights over a plane: .x, negative if something of the box or the sphere can be wholly below,
    // and .y of its highest point.
    __device__ __forceinline__ float2 heights( float3 n, float3 p, float diameter, const Box & b )
    {
        const float3 m = ( b.lo + b.hi ) * .5f - p, h = ( b.hi - b.lo ) * .5f;
        const float  s = fdot( n, m ), e = fabsf( n.x ) * h.x + fabsf( n.y ) * h.y + fabsf( n.z ) * h.z;
        return make_float2( s - e + diameter, s + e );
    }
    __device__ __forceinline__ float2 heights( float3 n, float3 p, float, float4 site )
    {
        const float top = fdot( n, f3( site ) - p ) + site.w;
        return make_float2( top, top );
    }
    // The sphere of a leaf from its box, which was made from it: the rounding of the box's corners
    // is in the radius.
    __device__ __forceinline__ float4 sphere_in( const Box & b )
    {
        const float3 m = ( b.lo + b.hi ) * .5f;
        const float  r = fmaxf( fmaxf( b.hi.x - b.lo.x, b.hi.y - b.lo.y ), b.hi.z - b.lo.z ) * .5f;
        return make_float4( m.x, m.y, m.z, r + 1e-6f * ( fabsf( m.x ) + fabsf( m.y ) + fabsf( m.z ) + fabsf( r ) ) );
    }
    // Distance of a centre from the plane (at least so much for the centres in a box).
    __device__ __forceinline__ float off_plane( float4 p, const Box & b )
    {
        const float3 n = f3( p ), m = ( b.lo + b.hi ) * .5f, h = ( b.hi - b.lo ) * .5f;
        return fabsf( fdot( n, m ) - p.w ) - ( fabsf( n.x ) * h.x + fabsf( n.y ) * h.y + fabsf( n.z ) * h.z );
    }
    __device__ __forceinline__ float off_plane( float4 p, float4 site ) { return fabsf( fdot( f3( p ), f3( site ) ) - p.w ); }
    // May box or site `x` be, or hold, a contributor? The balls are tested without branches: a walk's
    // lanes would take them all the same.
    template<bool Limited = true, class X>
    __device__ __forceinline__ bool within( const EdgeReach & a, const TangentPlanes & t, const X & x )
    {
        bool in   = meets( a.ball[ 0 ], x ) | meets( a.ball[ 1 ], x ) | meets( a.ball[ 2 ], x );
        bool more = off_plane( a.flat, x ) <= a.near;
        if ( a.below )
        {
            const float2 h1 = heights( t.n1, t.p1, a.diameter, x ), h2 = heights( t.n2, t.p2, a.diameter, x );
            if ( a.kind == kReachArcPlanes )
                more = more | ( h1.y >= -a.slab[ 0 ] ) | ( h2.y >= -a.slab[ 1 ] );
            if ( Limited )
                more = more & meets( a.limit, x );
            return ( in | more ) & ( h1.x < a.margin ) & ( h2.x < a.margin );
        }
        if ( Limited )
            more = more & meets( a.limit, x );
        return in | more;
    }

    // Does neighbour m conflict with every far root beyond the plane of outward normal n? Its
    // distance to the root and that of c_i, taken from the same far point, are rounded to single
    // precision alike: where m is the nearer one it does not come out farther, and the test of m
    // against the root's radius, re-measured from c_i, is decided by the larger radius of m. (The
    // approximate root falls between neighbouring floats at 508 of the 2^31 positive ones.)
    __device__ __forceinline__ bool far_roots_blocked( float3 n, float4 fi, float4 m, float far )
    {
        const float3 e  = f3( m ) - f3( fi );
        const float  ee = fdot( e, e );
        return m.w >= fi.w + 1e-3f && fdot( n, e ) >= 5e-3f * sqrtf( ee ) + ee / far;
    }

    // The ball with its margins: 1 % and 1e-3 as the reach always had, and the rounding of a far
    // centre to float.
    __device__ __forceinline__ float4 reach_ball( double3 x, double r )
    {
        r = fmax( r, 0.0 );
        r = r * 1.01 + 1e-3 * ( 1.0 + r ) + 1e-6 * ( fabs( x.x ) + fabs( x.y ) + fabs( x.z ) );
        return make_float4( float( x.x ), float( x.y ), float( x.z ), float( r ) );
    }

    __device__ __forceinline__ bool vertex_on_edge( uint4 r, uint32_t k, uint32_t l )
    {
        return ( r.x == k || r.y == k || r.z == k ) && ( r.x == l || r.y == l || r.z == l );
    }

    // Ends of an edge's arc: its two vertices and the third site of each.
    struct ArcEnds
    {
        double4  v[ 2 ];
        uint32_t m[ 2 ];
        uint32_t count = 0; // stored vertices on the edge
        __device__ __forceinline__ void add( double4 x, uint32_t site )
        {
            if ( count < 2 )
            {
                ( count ? v[ 1 ] : v[ 0 ] ) = x;
                ( count ? m[ 1 ] : m[ 0 ] ) = site;
            }
            count++;
        }
    };
    __device__ __forceinline__ uint32_t third_site( uint4 r, uint32_t k, uint32_t l )
    {
        return ( r.x != k && r.x != l ) ? r.x : ( ( r.y != k && r.y != l ) ? r.y : r.z );
    }

    // The stored vertices of cell i on its edge (k, l): the ends, the largest radius (at least 0) and
    // up to two distinct third sites. The records are scanned first and the vertices solved after, so that
    // the lanes of a warp, whose vertices stand at different places of the store, solve them together.
    __device__ __forceinline__ double stored_ends( const CellContext & c, uint32_t i, double4 si, uint32_t k, uint32_t l, ArcEnds & ends,
                                                   uint32_t ( &hint )[ 2 ] )
    {
        const uint4 *  store = c.vertices + store_row( c, i ) * kMaxVertices;
        const uint32_t vn    = c.vertex_nb[ i ];
        uint32_t       at[ 2 ] = { vn, vn }, more = vn, count = 0;
        hint[ 0 ] = hint[ 1 ] = kNone;
        for ( uint32_t v = 0; v < vn; v++ )
        {
            const uint4 r = store[ v ];
            if ( vertex_on_edge( r, k, l ) )
            {
                const uint32_t m = third_site( r, k, l );
                if ( hint[ 0 ] == kNone )
                    hint[ 0 ] = m;
                else if ( hint[ 1 ] == kNone && m != hint[ 0 ] )
                    hint[ 1 ] = m;
                if ( count == 0 )
                    at[ 0 ] = v;
                else if ( count == 1 )
                    at[ 1 ] = v;
                else if ( count == 2 )
                    more = v;
                count++;
            }
        }
        double   wmax = 0.0;
        uint32_t v    = at[ 0 ];
#pragma unroll 1
        while ( v < vn ) // hardly ever more than two
        {
            const uint4   r = store[ v ];
            const double4 x = solve_vertex( c, si, r );
            wmax            = fmax( wmax, x.w );
            ends.add( x, third_site( r, k, l ) );
            if ( v == at[ 0 ] )
                v = at[ 1 ];
            else
            {
                v = v == at[ 1 ] ? more : v + 1;
                while ( v < vn && !vertex_on_edge( store[ v ], k, l ) )
                    v++;
            }
        }
        return wmax;
    }

    __device__ __forceinline__ float4 neighbour( const CellContext & c, uint32_t u ) { return u < c.n ? c.sites_f[ u ] : to_float( c.sites[ u ] ); }

    // Shortly before the conflict of an end's third site ends again, further out: the point and its radius, what the
    // curve goes on to (a hyperbola to infinity, in a direction; an ellipse to a point half-way round to
    // the other end, with its radius), and the least radius on the way.
    struct OpenEnds
    {
        float4   at[ 2 ], away[ 2 ];
        float    low[ 2 ];
        uint32_t mask = 0;
        __device__ __forceinline__ void add( int a, float3 x, float w, float3 on, float on_w, float least )
        {
            ( a ? at[ 1 ] : at[ 0 ] )     = make_float4( x.x, x.y, x.z, w );
            ( a ? away[ 1 ] : away[ 0 ] ) = make_float4( on.x, on.y, on.z, on_w );
            ( a ? low[ 1 ] : low[ 0 ] )   = least;
            mask |= 1u << a;
        }
    };

    // The balls of the arc of trisector (i, k, l) between its two vertices. With c_i as the origin,
    // e_k = c_k - c_i, d_k = r_k - r_i and rho = w + r_i = |x|, the trisector's points are
    // x = A + rho B + s n, n the normal of the plane of the centres, A and B in it from
    // e.x = (|e|^2 - d^2) / 2 - rho d for e_k and e_l; and |x| = rho makes (rho, s) a conic,
    // s^2 = alpha rho^2 - 2 beta rho - gamma. Whether site j conflicts with the sphere at x is the
    // sign of |x - e_j|^2 - (rho + d_j)^2, on the conic equal to |e_j|^2 - d_j^2 - 2 (e_j.x + rho d_j):
    // linear in (rho, s). The arc lies in the triangle of its ends and the meeting point T of their
    // tangents, so a site that conflicts at none of these three conflicts nowhere on the arc. At
    // the ends that is a ball each. T lies off the conic by D = |x|^2 - rho^2, and for a sphere of
    // radius r_j >= 0 the linear form there is at least delta^2 - w^2 - D, delta the distance of
    // the sphere (or of a box around it) from x: a ball of radius sqrt(w^2 + D). (With equal radii
    // it passes through the three centres, in the union of the other two: only unequal radii
    // leave anything to find.) On a hyperbola (of which the points with rho > 0 are one branch) the
    // arc is the piece between the ends, on an ellipse the smaller one, if at both ends the third
    // site's conflict fades that way. (It does not in a cell that has one of two equal sites twice:
    // both its vertices on an edge may be the same point, and the rest of the arc is open.) False
    // where the points do not determine this safely.
    __device__ __forceinline__ bool arc_reach( const CellContext & c, double4 si, double4 sk, double4 sl,
                                               const ArcEnds & ends, OpenEnds & open, EdgeReach & reach )
    {
        const double3 o   = d3( si );
        const double3 ek  = d3( sk ) - o, el = d3( sl ) - o;
        const double  dk  = sk.w - si.w, dl = sl.w - si.w;
        const double  gkk = ddot( ek, ek ), gll = ddot( el, el ), gkl = ddot( ek, el );
        const double  det = gkk * gll - gkl * gkl;
        if ( !( det > 1e-9 * gkk * gll ) )
            return false; // centres nearly in line
        const double  inv = 1.0 / det;
        const double  ak = .5 * ( gkk - dk * dk ), al = .5 * ( gll - dl * dl );
        const double3 A = ek * ( ( ak * gll - al * gkl ) * inv ) + el * ( ( al * gkk - ak * gkl ) * inv );
        const double3 B = ek * ( ( dl * gkl - dk * gll ) * inv ) + el * ( ( dk * gkl - dl * gkk ) * inv );
        const double3 n = dcross( ek, el ) * rsqrt( det );
        const double  alpha = 1.0 - ddot( B, B ), beta = ddot( A, B ), gamma = ddot( A, A );
        const double3 u0 = d3( ends.v[ 0 ] ) - o, u1 = d3( ends.v[ 1 ] ) - o;
        const double  rho0 = sqrt( ddot( u0, u0 ) ), rho1 = sqrt( ddot( u1, u1 ) );
        const double  s0 = ddot( u0, n ), s1 = ddot( u1, n );
        // the vertices lie on the curve (they are solved in another order, and may be badly conditioned)
        const double3 off0 = A + B * rho0 + n * s0 - u0, off1 = A + B * rho1 + n * s1 - u1;
        if ( !( ddot( off0, off0 ) <= 1e-8 * ( 1.0 + rho0 ) * ( 1.0 + rho0 )
                && ddot( off1, off1 ) <= 1e-8 * ( 1.0 + rho1 ) * ( 1.0 + rho1 ) && fmax( rho0, rho1 ) < 1e9 ) )
            return false;
        // the curve at the ends, in one direction along it, and how far the second end lies ahead of the first
        double2 along0, along1;
        double  ahead, near; // ends less than `near` apart coincide
        double  sT = s0, rhoT = rho0;
        double  rc = 0.0, ar = 0.0, as = 0.0; // ellipse: centre and axes, and the ends on its unit circle
        double2 c0 = make_double2( 0, 0 ), c1 = make_double2( 0, 0 );
        if ( alpha > 1e-6 )
        {
            // s_a s + (beta - alpha rho_a) rho = -(beta rho_a + gamma) is the tangent at end a
            const double m0 = beta - alpha * rho0, m1 = beta - alpha * rho1;
            const double h0 = -( beta * rho0 + gamma ), h1 = -( beta * rho1 + gamma );
            const double meet  = s0 * m1 - s1 * m0;
            const double slack = 1e-3 * ( 1.0 + fabs( s0 ) + fabs( s1 ) );
            near               = 1e-3 * slack;
            if ( fabs( s0 - s1 ) >= near )
            {
                sT   = ( h0 * m1 - h1 * m0 ) / meet;
                rhoT = ( s0 * h1 - s1 * h0 ) / meet;
            }
            if ( !( m0 < 0.0 && m1 < 0.0 && sT >= fmin( s0, s1 ) - slack && sT <= fmax( s0, s1 ) + slack && rhoT >= -1e-3
                    && rhoT <= 1.001 * fmax( rho0, rho1 ) + 1e-3 ) )
                return false;
            along0     = make_double2( s0, -m0 );
            along1     = make_double2( s1, -m1 );
            ahead      = s1 - s0;
            reach.kind = kReachArcPlanes;
        }
        else if ( alpha < -1e-6 && beta * beta + alpha * gamma > 0.0 )
        {
            // (rho, s) = (rc + ar cos, as sin)
            const double disc = beta * beta + alpha * gamma;
            rc                = beta / alpha;
            ar                = sqrt( disc ) / -alpha;
            as                = sqrt( disc / -alpha );
            if ( !( rc + ar < kFarRoot ) )
                return false;
            c0                  = make_double2( ( rho0 - rc ) / ar, s0 / as );
            c1                  = make_double2( ( rho1 - rc ) / ar, s1 / as );
            const double  cosine = ddot( c0, c1 );
            if ( !( cosine > -.5 && fabs( ddot( c0, c0 ) - 1.0 ) < 1e-3 && fabs( ddot( c1, c1 ) - 1.0 ) < 1e-3 ) )
                return false; // more than a third of the ellipse apart
            along0     = make_double2( -ar * c0.y, as * c0.x );
            along1     = make_double2( -ar * c1.y, as * c1.x );
            ahead      = c0.x * c1.y - c0.y * c1.x;
            near       = 1e-6;
            rhoT       = rc + ar * ( c0.x + c1.x ) / ( 1.0 + cosine );
            sT         = as * ( c0.y + c1.y ) / ( 1.0 + cosine );
            reach.kind = kReachArc;
        }
        else
            return false;
        // Is every root of the cell in the piece between the ends? Each end's third site, a neighbour, has to
        // conflict from its end on outward, and the two have to cover the rest of the curve: then no root
        // outside is empty, whatever other vertices the cell has or lacks. (Half the form over rho is the
        // depth of a conflict, which the rounding of lengths hides up to 4e-7 of rho: it has to be above
        // that half the balls' margin away, where x and w have moved by 1 + |B| of rho's change and by s's.)
        // Single precision does, by margins far above its rounding.
        const float4 fi = to_float( si );
        const float3 fB = to_float( B ), fn = to_float( n ), fA = f3( fi ) + to_float( A );
        const float  fal = float( alpha ), fbe = float( beta ), wide = fmaxf( 2.f, 2.f - fal );
        const float  frc = float( rc ), arf = float( ar ), fas = float( as );
        float2       g[ 2 ]; // gradient of the third site's form, times -1/2
        float        r[ 2 ]; // and its radius
        bool         ahead0 = false, ahead1 = false;
        float        far = FLT_MAX;
        const float  root = sqrtf( fmaxf( fal, 0.f ) );
#pragma unroll 1
        for ( int a = 0; a < 2; a++ )
        {
            const float4 m    = neighbour( c, a ? ends.m[ 1 ] : ends.m[ 0 ] );
            const float3 em   = f3( m ) - f3( fi );
            const float2 t    = a ? make_float2( float( along1.x ), float( along1.y ) ) : make_float2( float( along0.x ), float( along0.y ) );
            const float2 x    = a ? make_float2( float( rho1 ), float( s1 ) ) : make_float2( float( rho0 ), float( s0 ) );
            const float2 f    = make_float2( fdot( em, fB ) + ( m.w - fi.w ), fdot( em, fn ) );
            const float  rise = f.x * t.x + f.y * t.y; // the conflict's, along the curve
            const float  hide = 4e-7f * x.x * x.x * ( wide * fabsf( t.x ) + fabsf( t.y ) ), reach_w = 5e-3f * fmaxf( x.x - fi.w, 0.f ) + 5e-4f;
            const float  blur = 1e-6f * ( fabsf( fi.x ) + fabsf( fi.y ) + fabsf( fi.z ) + fabsf( m.x ) + fabsf( m.y ) + fabsf( m.z ) );
            if ( !( fabsf( rise ) > 1e-3f * ( fabsf( f.x * t.x ) + fabsf( f.y * t.y ) ) + blur * ( wide * fabsf( t.x ) + fabsf( t.y ) )
                    && fabsf( rise ) * reach_w > hide ) )
                return false;
            ( a ? ahead1 : ahead0 ) = rise > 0.f;
            ( a ? g[ 1 ] : g[ 0 ] ) = f;
            ( a ? r[ 1 ] : r[ 0 ] ) = m.w;
            if ( fal <= 0.f )
                continue;
            // Along s the form is concave where it falls with rho, and then falls on as at the end; else it is
            // convex, and falls less and less, down to its asymptote's slope. By `slope` or more either way:
            // a root that passes all the same has a rho of slope sqrt(alpha) / 4e-7 and more.
            // (The form is that of a conflict only where w is not below -r; w is least where s is 0.)
            const float out   = rise > 0.f ? 1.f : -1.f;
            const float least = out * x.y >= 0.f ? x.x - fi.w : ( fbe + sqrtf( fmaxf( fbe * fbe + fal * float( gamma ), 0.f ) ) ) / fal - fi.w;
            if ( !( least + m.w >= blur ) )
                return false;
            const float slope = f.x > 0.f ? out * ( f.x * t.x / t.y + f.y ) : f.x / root + out * f.y;
            if ( slope > 1e-3f * ( fabsf( f.x ) + fabsf( f.y ) ) + blur * wide && slope * t.y * reach_w > hide )
            {
                far = fminf( far, slope * root );
                continue;
            }
            // it ends at the site's other root: another neighbour has to take over before, a fiftieth of the way,
            // which is more than the rounding of that root's place
            const float q = f.y / f.x, w = 1.f - fal * q * q;
            const float last = -2.f * q * ( fal * ( x.x + q * x.y ) - fbe ) / w - x.y;
            const float s    = last - .02f * ( last - x.y ), rho = ( fbe + sqrtf( fmaxf( fbe * fbe + fal * ( float( gamma ) + s * s ), 0.f ) ) ) / fal;
            if ( !( f.x < 0.f && w > 1e-3f && out * ( last - x.y ) > 0.f && fal * ( x.x + q * ( x.y - last ) ) > fbe && rho < float( kFarRoot ) ) )
                return false;
            open.add( a, fA + fB * rho + fn * s, rho - fi.w, fB + fn * ( out * root ), 0.f, least );
        }
        // outward of one end is inward of the other
        if ( ahead0 == ahead1 || !( fabs( ahead ) < near || ahead > 0.0 == ahead1 ) )
            return false;
        if ( fal > 0.f )
            reach.far = fminf( kFarOut * far, float( kFarRoot ) );
        else
        {
            // Half-way round, opposite the piece, each of the two has to hold, or another neighbour has to take
            // over before it ends, at its other root: the end's mirror image in the gradient (all in the
            // ellipse's unit circle)
            const float  low = frc - arf - fi.w;
            const float2 e0 = make_float2( float( c0.x ), float( c0.y ) ), e1 = make_float2( float( c1.x ), float( c1.y ) );
            const float  scale = -rsqrtf( 2.f + 2.f * ( e0.x * e1.x + e0.y * e1.y ) );
            const float2 half  = make_float2( scale * ( e0.x + e1.x ), scale * ( e0.y + e1.y ) );
            const float  deep  = 8e-7f * ( frc + arf ) * ( frc + arf ) + 2e-6f * ( fabsf( fi.x ) + fabsf( fi.y ) + fabsf( fi.z ) + frc + arf ) * ( arf + fas );
            if ( !( low + fminf( r[ 0 ], r[ 1 ] ) >= 1e-5f * ( frc + arf ) ) )
                return false;
#pragma unroll 1
            for ( int a = 0; a < 2; a++ )
            {
                const float2 f = a ? g[ 1 ] : g[ 0 ], x = a ? e1 : e0;
                const float2 v = make_float2( f.x * arf, f.y * fas );
                if ( v.x * ( half.x - x.x ) + v.y * ( half.y - x.y ) > deep )
                    continue;
                const float  vv = v.x * v.x + v.y * v.y, m = 2.f * ( v.x * x.x + v.y * x.y ) / vv + .02f * rsqrtf( vv );
                const float2 z  = make_float2( m * v.x - x.x, m * v.y - x.y );
                const float  iz = rsqrtf( z.x * z.x + z.y * z.y );
                const float2 y  = make_float2( iz * z.x, iz * z.y );
                open.add( a, fA + fB * ( frc + arf * y.x ) + fn * ( fas * y.y ), frc + arf * y.x - fi.w,
                          fA + fB * ( frc + arf * half.x ) + fn * ( fas * half.y ), frc + arf * half.x - fi.w, low );
            }
        }
        // how near to the plane of the centres a root is not to be trusted
        const float size = float( fmax( fabs( c.scene->lo[ 0 ] ), fabs( c.scene->hi[ 0 ] ) ) + fmax( fabs( c.scene->lo[ 1 ] ), fabs( c.scene->hi[ 1 ] ) )
                                  + fmax( fabs( c.scene->lo[ 2 ] ), fabs( c.scene->hi[ 2 ] ) ) );
        reach.flat       = make_float4( float( n.x ), float( n.y ), float( n.z ), float( ddot( n, o ) ) );
        reach.near       = kFlat * size * sqrtf( float( gkk * gll * inv ) );
        const double3 uT = A + B * rhoT + n * sT;
        const double  wT = rhoT - si.w;
        reach.ball[ 0 ]  = reach_ball( d3( ends.v[ 0 ] ), fabs( rho0 - si.w ) );
        reach.ball[ 1 ]  = reach_ball( d3( ends.v[ 1 ] ), fabs( rho1 - si.w ) );
        reach.ball[ 2 ]  = reach_ball( o + uT, sqrt( wT * wT + fmax( 0.0, ddot( uT, uT ) - rhoT * rhoT ) ) );
        return true;
    }

    __device__ __forceinline__ float3 shfl3( float3 v, uint32_t src )
    {
        return make_float3( __shfl_sync( 0xffffffffu, v.x, src ), __shfl_sync( 0xffffffffu, v.y, src ), __shfl_sync( 0xffffffffu, v.z, src ) );
    }
    __device__ __forceinline__ float4 shfl4f( float4 v, uint32_t src )
    {
        return make_float4( __shfl_sync( 0xffffffffu, v.x, src ), __shfl_sync( 0xffffffffu, v.y, src ), __shfl_sync( 0xffffffffu, v.z, src ),
                            __shfl_sync( 0xffffffffu, v.w, src ) );
    }

    // Does neighbour m close an open end? It conflicts at the point, not at the end, and where the curve goes on to
    // (at infinity it stands out by `out`): then all the way. (On a hyperbola its form, see arc_reach, is
    // concave, and lower at the point than at the end, or convex; on an ellipse it is below 0 on one piece,
    // which is not the one with the end.) In single precision, by margins of a hundred times its rounding.
    __device__ __forceinline__ bool closes( float4 at, float4 end, float4 away, float low, bool ellipse, float4 fi, float4 m, float & out )
    {
        const float  size = fabsf( fi.x ) + fabsf( fi.y ) + fabsf( fi.z ) + fabsf( m.x ) + fabsf( m.y ) + fabsf( m.z ) + 4.f * fabsf( m.w );
        const float3 da = f3( m ) - f3( at ), de = f3( m ) - f3( end ), dy = f3( m ) - f3( away );
        const float  ra = at.w + m.w - 1e-5f * ( size + fabsf( at.w ) ), re = end.w + m.w, ry = away.w + m.w - 1e-5f * ( size + fabsf( away.w ) );
        out             = fdot( f3( m ) - f3( fi ), f3( away ) ) + m.w - fi.w;
        return ra > 0.f && fdot( da, da ) < ra * ra && fdot( de, de ) >= re * re && low + m.w >= 0.f
               && ( ellipse ? ry > 0.f && fdot( dy, dy ) < ry * ry : out > 1e-5f * size );
    }

    // The open ends that other neighbours close. One lane's edge.
    __device__ __forceinline__ void close_ends( const CellContext & c, double4 si, uint32_t k, uint32_t l, const ArcEnds & ends,
                                                const SiteSequence & sites, OpenEnds & open, EdgeReach & reach )
    {
        const float4 fi      = to_float( si );
        const bool   ellipse = reach.kind == kReachArc;
        for ( uint32_t q = 0; q < sites.count && open.mask; q++ )
        {
            const uint32_t u = sites[ q ];
            if ( u == k || u == l )
                continue;
            const float4 m = neighbour( c, u );
#pragma unroll 1
            for ( int a = 0; a < 2; a++ )
            {
                float out;
                if ( ( ( open.mask >> a ) & 1u )
                     && closes( a ? open.at[ 1 ] : open.at[ 0 ], to_float( a ? ends.v[ 1 ] : ends.v[ 0 ] ), a ? open.away[ 1 ] : open.away[ 0 ],
                                a ? open.low[ 1 ] : open.low[ 0 ], ellipse, fi, m, out ) )
                {
                    open.mask &= ~( 1u << a );
                    reach.far = ellipse ? 0.f : fminf( reach.far, kFarOut * out );
                }
            }
        }
    }

    // The same for the edges of one cell, one per lane, by the warp: a neighbour per lane.
    __device__ __forceinline__ void close_ends_together( const CellContext & c, double4 si, uint32_t k, uint32_t l, const ArcEnds & ends,
                                                         const SiteSequence & sites, OpenEnds & open, EdgeReach & reach )
    {
        constexpr uint32_t all = 0xffffffffu;
        const uint32_t lane = threadIdx.x & 31;
        const float4   fi   = to_float( si );
        for ( uint32_t base = 0; base < sites.count; base += 32 )
        {
            uint32_t todo = __ballot_sync( all, open.mask != 0 );
            if ( todo == 0 )
                break;
            const bool     has = base + lane < sites.count;
            const uint32_t u   = has ? sites[ base + lane ] : kNone;
            const float4   m   = has ? neighbour( c, u ) : make_float4( 0, 0, 0, 0 );
            while ( todo )
            {
                const uint32_t src = __ffs( todo ) - 1;
                todo &= todo - 1;
                const uint32_t mask    = __shfl_sync( all, open.mask, src );
                const uint32_t sk      = __shfl_sync( all, k, src ), sl = __shfl_sync( all, l, src );
                const bool     ellipse = __shfl_sync( all, reach.kind, src ) == kReachArc;
#pragma unroll 1
                for ( int a = 0; a < 2; a++ )
                {
                    if ( !( ( mask >> a ) & 1u ) )
                        continue;
                    const float4   at   = shfl4f( a ? open.at[ 1 ] : open.at[ 0 ], src ), away = shfl4f( a ? open.away[ 1 ] : open.away[ 0 ], src );
                    const float4   end  = shfl4f( to_float( a ? ends.v[ 1 ] : ends.v[ 0 ] ), src );
                    const float    low  = __shfl_sync( all, a ? open.low[ 1 ] : open.low[ 0 ], src );
                    float          out  = 0.f;
                    const uint32_t hits = __ballot_sync( all, closes( at, end, away, low, ellipse, fi, m, out ) && has && u != sk && u != sl );
                    out                 = __shfl_sync( all, out, hits ? __ffs( hits ) - 1 : 0 );
                    if ( lane == src && hits )
                    {
                        open.mask &= ~( 1u << a );
                        reach.far = ellipse ? 0.f : fminf( reach.far, kFarOut * out );
                    }
                }
            }
        }
    }

    // Reach of edge (k, l) of cell i: wmax is the largest radius on its arc, `around` the reference's
    // bounding sphere of the trisector (`known`: the third sites of the ends are neighbours). To be settled.
    __device__ __forceinline__ EdgeReach edge_reach( const CellContext & c, double4 si, double4 sk, double4 sl, bool hyperbola,
                                                     const ArcEnds & ends, bool known, double wmax, float4 around, OpenEnds & open )
    {
        EdgeReach    reach;
        const double rmin = c.scene->rmin;
        // spheres of negative radius reach out of their boxes by less than four radii
        const float low = fmaxf( 0.f, float( -4.0 * rmin ) );
        reach.limit     = reach_ball( d3( si ), 2.0 * wmax + si.w );
        const float margin = 1e-5f * ( around.w + fabsf( around.x ) + fabsf( around.y ) + fabsf( around.z ) );
        if ( around.w + margin < reach.limit.w )
            reach.limit = make_float4( around.x, around.y, around.z, around.w + margin );
        else
            reach.limit.w += float( c.scene->rmax - rmin );
        reach.limit.w += low;
        reach.margin    = 1e-5f * ( reach.limit.w + fabsf( reach.limit.x ) + fabsf( reach.limit.y ) + fabsf( reach.limit.z ) );
        reach.diameter  = 2.f * fmaxf( 0.f, float( rmin ) );
        reach.below     = hyperbola && rmin >= 0.0;
        if ( !( ends.count == 2 && known && rmin >= 0.0 && arc_reach( c, si, sk, sl, ends, open, reach )
                && ( hyperbola || reach.kind == kReachArc ) ) )
        {
            reach.kind = kReachBall;
            open.mask  = 0;
        }
        return reach;
    }
    // Once its open ends have been looked at: an arc with one left is searched in the ball.
    __device__ __forceinline__ void settle( const CellContext & c, EdgeReach & reach, const OpenEnds & open )
    {
        if ( reach.kind == kReachBall || open.mask )
        {
            reach.kind      = kReachBall;
            reach.ball[ 0 ] = reach.ball[ 1 ] = reach.ball[ 2 ] = reach.limit;
            reach.flat      = make_float4( 0.f, 0.f, 0.f, 0.f );
            reach.near      = -1.f;
            reach.far       = 1.f;
        }
        // a root of radius w touches the plane to L^2 / 2w at a distance of L, at most 2.5 times the
        // limit's radius and that of a site
        const float span = reach.limit.w + fmaxf( 0.f, float( c.scene->rmax ) );
        reach.slab[ 0 ]  = reach.slab[ 1 ] = 3.2f / reach.far * span * span + reach.margin;
    }

    // An apex (trisector root in the plane of the centres) counts unless a neighbour other
    // than k, l clearly intersects its sphere (IEEE double distance, relative margin 1e-4).
    __device__ __forceinline__ bool clearly_outside( double4 site, double4 apex )
    {
        const double dx = site.x - apex.x, dy = site.y - apex.y, dz = site.z - apex.z;
        const double d  = __dsqrt_rn( __dadd_rn( __dadd_rn( __dmul_rn( dx, dx ), __dmul_rn( dy, dy ) ), __dmul_rn( dz, dz ) ) );
        const double pen = ( site.w + apex.w ) - d;
        return pen > 1e-4 * ( site.w + fabs( apex.w ) ) + 1e-6;
    }

    // The node every walk inside a ball may start from: from the root down to where both children
    // meet the ball. The walk would go the same way, one box after another, without meeting a leaf.
    __device__ __forceinline__ uint32_t node_around( const WideNode * nodes, uint32_t n, float4 ball )
    {
        uint32_t node = 0;
        while ( true )
        {
            Box      lb, rb;
            uint32_t lc, rc;
            load_node( nodes, node, lb, rb, lc, rc );
            const bool l = meets( ball, lb ), r = meets( ball, rb );
            const uint32_t next = l ? lc : rc;
            if ( l == r || next >= n - 1 )
                return node;
            node = next;
        }
    }
    // Ball holding every site that a sphere of radius up to w touching sphere i can touch.
    __device__ __forceinline__ float4 touch_ball( const CellContext & c, double4 si, double w )
    {
        return reach_ball( d3( si ), 2.002 * w + si.w + fmax( 0.0, -4.0 * c.scene->rmin ) );
    }
    // The sites that reach into the ball, other than i, the buried ones and those that `skip` names,
    // collected by the warp from `node` down. Returns their number, or kNone if there are more than
    // kListCap.
    template<class Skip>
    __device__ __forceinline__ uint32_t collect_sites( const CellContext & c, uint32_t i, float4 ball, uint32_t node, float4 * sites,
                                                       uint32_t * ids, uint32_t * stack, Skip && skip )
    {
        constexpr uint32_t all   = 0xffffffffu;
        const uint32_t     lane  = threadIdx.x & 31, n = c.n;
        const uint32_t below = ( 1u << lane ) - 1u;
        uint32_t       size = 1, found = 0;
        if ( lane == 0 )
            stack[ 0 ] = node;
        __syncwarp();
        while ( size > 0 )
        {
            const uint32_t take = min( size, 32u );
            size -= take;
            uint32_t child[ 2 ] = { 0, 0 };
            bool     in[ 2 ]    = { false, false };
            if ( lane < take )
            {
                Box lb, rb;
                load_node( c.nodes, stack[ size + lane ], lb, rb, child[ 0 ], child[ 1 ] );
                in[ 0 ] = meets( ball, lb );
                in[ 1 ] = meets( ball, rb );
            }
            __syncwarp();
#pragma unroll 1
            for ( uint32_t q = 0; q < 2; q++ )
            {
                const uint32_t x    = q ? child[ 1 ] : child[ 0 ];
                const bool     here = q ? in[ 1 ] : in[ 0 ];
                const uint32_t j    = x - ( n - 1 );
                bool           site = here && x >= n - 1 && j != i;
                float4         s    = make_float4( 0, 0, 0, 0 );
                if ( site )
                {
                    s    = c.sites_f[ j ];
                    site = meets( ball, s ) && c.status[ j ] != kBuried && !skip( j );
                }
                const uint32_t leaves = __ballot_sync( all, site ), nodes = __ballot_sync( all, here && x < n - 1 );
                if ( found + __popc( leaves ) > kListCap || size + __popc( nodes ) > kListStack )
                    return kNone;
                if ( site )
                {
                    sites[ found + __popc( leaves & below ) ] = s;
                    ids[ found + __popc( leaves & below ) ]   = j;
                }
                if ( here && x < n - 1 )
                    stack[ size + __popc( nodes & below ) ] = x;
                found += __popc( leaves );
                size += __popc( nodes );
            }
            __syncwarp();
        }
        return found;
    }

    void configure_cell_kernels();
    // blocks of kCellBlock threads that the cell kernels are launched with, one walk-scratch region per warp
    int cell_grid_blocks( uint32_t cells );
    // bytes of CellContext::walk_scratch: one region per warp the cell kernels launch
    size_t walk_scratch_bytes( uint32_t cells );
    // k_cells modes: first kNN step, a later kNN step, initial cells only (no kNN step)
    constexpr uint32_t kCellsFirst    = 0;
    constexpr uint32_t kCellsNext     = 1;
    constexpr uint32_t kCellsInitOnly = 2;
    void launch_knn( const CellContext & c, uint32_t step, cudaStream_t s );
    // kNN cells with per-rank labels (contribution, certificate), rows of `row` bytes per cell
    void launch_cells_profile( const CellContext & c, uint32_t step, uint32_t row, uint8_t * contributed, uint8_t * certified,
                               cudaStream_t s );
    void launch_cells( const CellContext & c, uint32_t mode, ZeroWords & z, cudaStream_t s );
    // *count must be 0
    void launch_tasks( const CellContext & c, uint32_t * tasks, uint32_t * count, cudaStream_t s );
    void launch_vertex_validation( const CellContext & c, const uint32_t * tasks, const uint32_t * count, ZeroWords & z, cudaStream_t s );
    constexpr uint32_t kMaybeWords = ( kMaxEdges + 31 ) / 32; // 9 words of edge bits per task
    constexpr uint32_t kNbrCap     = 272;                     // neighbour slots per task cell (>= the 265 a full cell can have)

    // What the edge-parallel search proved, handed to the exact pass of the same cells.
    struct SearchProof
    {
        const uint32_t * slots      = nullptr; // task index of each listed cell
        const uint32_t * maybe_bits = nullptr; // per task, bit e: edge e may have a contributor
        const uint32_t * nbr        = nullptr; // per task, the sorted neighbour ids searched against
        const uint32_t * nbr_count  = nullptr;
    };
    void launch_edge_validation( const CellContext & c, const uint32_t * tasks, const uint32_t * count, ZeroWords & z, cudaStream_t s,
                                 SearchProof proof = SearchProof {} );
    // warp per cell, over the listed cells or (null) all of the handle's
    void launch_bisector_validation( const CellContext & c, const uint32_t * tasks, const uint32_t * count, ZeroWords & z, cudaStream_t s );

    // Output extraction: per-cell owned counts, exclusive scans (totals[0] vertices,
    // totals[1] closed edges), then the writes bounded by the capacities.
    struct OutputBuffers
    {
        uint32_t * vcount = nullptr; // n, then offsets
        uint32_t * ccount = nullptr;
        uint32_t * tile_sums = nullptr; // scan scratch
        uint64_t * totals    = nullptr; // [2]
        double4 *  vpos      = nullptr;
        uint4 *    vids      = nullptr;
        double4 *  cpos      = nullptr;
        uint4 *    cids      = nullptr;
        uint64_t   vcap = 0, ccap = 0;
    };
    size_t output_scan_scratch_words( uint32_t n );
    void   launch_output( const CellContext & c, const OutputBuffers & o, cudaStream_t s );

    // Exclusive scan of n u32 values in place; the total goes to *total. `sums` holds
    // output_scan_scratch_words(n) words.
    void scan_exclusive( uint32_t * data, uint32_t n, uint32_t * sums, uint64_t * total, cudaStream_t s );

    // Edge-parallel edge validation with an exact per-cell fallback (speculate.cu).
    struct SpecBuffers
    {
        // the counters (item_counter and every *_count and *_next) are null until a launch takes its own
        uint32_t * nbr          = nullptr; // per task: sorted unique neighbour ids (kNbrCap slots)
        uint32_t * nbr_count    = nullptr;
        uint32_t * item_count   = nullptr; // per task: edges to search; scanned into item_offset
        uint32_t * item_offset  = nullptr;
        uint32_t * cell_flag    = nullptr; // 1: a contributor was found, 2: neighbour list too long
        uint32_t * exact_tasks  = nullptr; // cells re-run by the exact warp algorithm
        uint32_t * exact_slot   = nullptr; // their task index (row of maybe_bits)
        uint32_t * exact_count  = nullptr;
        uint32_t * maybe_bits   = nullptr; // per task, bit e: edge e may have a contributor
        uint64_t * item_total   = nullptr;
        uint64_t * item_counter = nullptr;
        uint32_t * scan_sums    = nullptr;
        uint2 *    heavy        = nullptr; // (task, edge) searches handed to whole warps
        uint32_t * heavy_count  = nullptr;
        uint32_t * heavy_next   = nullptr;
        uint32_t   heavy_cap    = 0;
        uint2 *    sub          = nullptr; // (search, BVH node) subtrees of long searches; the search is a
                                           // split set-up slot (high bit set) or a heavy item
        uint32_t * sub_count    = nullptr;
        uint32_t * sub_next     = nullptr;
        uint32_t   sub_cap      = 0;
        void *     splits       = nullptr; // set-up of each split search, computed once for its subtrees
        uint32_t * split_count  = nullptr;
        uint32_t   split_cap    = 0;
    };
    size_t spec_bytes( uint32_t n );
    // interval certificate of output points (certify.cu): flags (optional) and a count of the
    // points some other site is certainly closer to than their defining sites
    void launch_certify( const double4 * by_id, const double4 * sorted, const uint32_t * indices, const WideNode * nodes,
                         uint32_t n, const double4 * points, const uint4 * ids, uint32_t arity, uint64_t count, float rmax,
                         uint8_t * flags, unsigned long long * bad, uint32_t * error, cudaStream_t s );
    // relative error of output vertices against Newton-refined IEEE double solves (certify.cu):
    // per-vertex errors (optional), the largest (as the bits of a non-negative double), the
    // count above `threshold` and the count of singular systems
    void launch_vertex_error( const double4 * by_id, uint32_t n, const double4 * points, const uint4 * ids, uint64_t count,
                              double threshold, float * errors, unsigned long long * max_bits, unsigned long long * above,
                              unsigned long long * singular, cudaStream_t s );
    // grid sizes of the speculation kernels (once per process; call before concurrent builds)
    void configure_spec_kernels();
    void   spec_carve( SpecBuffers & b, void * base, uint32_t n );
    void   launch_edge_validation_speculative( const CellContext & c, const uint32_t * tasks, const uint32_t * task_count,
                                               const SpecBuffers & b, ZeroWords & z, cudaStream_t s );
    void   launch_bisector_validation_speculative( const CellContext & c, const SpecBuffers & b, ZeroWords & z, cudaStream_t s );
} // namespace apo2
