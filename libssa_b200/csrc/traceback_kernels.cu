// traceback_kernels.cu -- CIGAR traceback of the top hits on the GPU.
//
// For every hit the CPU library runs three scalar O(q*d) passes and a walk
// (reference: src/algo/align.c:39-182, src/algo/cigar.c:48-346):
//
//   1. SW only: a forward local-alignment pass that finds the end cell, the
//      first cell (database-row major) holding the maximum;
//   2. SW only: a reverse pass from the end cell that finds the begin cell,
//      the first cell (scanning rows and columns downwards) whose value
//      reaches the score.  The reference resets its work rows only up to the
//      database end index, so when the query end lies beyond it the reverse
//      pass reads the forward pass's last-row values there; that is
//      reproduced exactly;
//   3. a direction pass over the matrix whose 4 flag bits collapse to the
//      three observable traceback moves, stored here as 2 bits per cell in HBM;
//   4. the walk from the end cell with the priority I > D > M.
//
// Each pass is a wavefront on warps: lane k owns R query rows of a stripe of
// 32 x R, database columns stream through the warp, the bottom row of a lane
// goes to the next lane by shuffle, and the stripes of a hit follow one
// another on different warps through the hit's boundary row
// (stream_stripes.cuh).  All arithmetic is exact (int32, with the host
// guaranteeing the range), matching the reference's int64 code.
//
// What bounds it: the integer ALU pipe (16 lanes per clock per SM
// sub-partition) when many hits fill the GPU, the latency of one warp's steps
// (columns + 64 x stripes of them per hit) when few do.  So R is 4 while all
// stripes of 128 rows of a call can be resident at once (half the work per
// step of R = 8, twice the warps), and 8 past that, where the fixed cost of a
// step is spread over more cells.  Measured on a B200 against groups of 1, 2 or
// 4 warps of one CTA per hit, whose stripes waited at a group barrier every 32
// steps (one call each): 48 pairs of 5,000-30,000 residues, SW 780 -> 53 ms and
// NW 470 -> 35 ms; 10 hits of 300 x 33,000 20.5 -> 9.3 ms; 320 hits of 30-1,355
// rows 4.7 -> 1.3 ms; 4,096 long pairs, SW and NW, 6.4 -> 3.9 s.  A lane's scores of a column are one (two at
// R = 8) shared-memory word of int8 entries, added to the diagonal by dp4a
// (off the ALU pipe); tables past int8 are read entry by entry.
#include "device_common.cuh"
#include "stream_stripes.cuh"

#include <climits>

namespace ssa {

constexpr int TB_THREADS = 128;
constexpr int TB_WARPS = TB_THREADS / 32;

// What the stripe bodies share: the lane's rows and their scores.
template <int R, bool P8>
struct TbLane {
    static constexpr int WORDS = R / 4;
    uint32_t * table;              // P8: the warp's scores, [code][lane][WORDS] words of four int8 entries
    const int32_t * smat;          // the score table, [database code][query code]
    int lane;
    int32_t gO, gE, gOE;
    int qa[P8 ? 1 : R];            // !P8: query codes of the rows (0 past the end)
    int32_t H[R], E[R];
    int32_t diag, out_h, out_f, row0;
    int nvalid;                    // rows of this lane inside the query

    // rows first, first + step, ... of the codes `a`
    __device__ void load_rows( const uint8_t * a, int64_t first, int64_t step ) {
        int code[R];
#pragma unroll
        for( int r = 0; r < R; r++ )
            code[r] = (r < nvalid) ? a[first + step * r] : 0;
        if constexpr( P8 ) {
            // every lane reads back its own entries only
            for( int d = 0; d < 32; d++ ) {
#pragma unroll
                for( int w = 0; w < WORDS; w++ ) {
                    uint32_t v = 0;
#pragma unroll
                    for( int b = 0; b < 4; b++ ) {
                        const int r = 4 * w + b;
                        const int32_t m = (r < nvalid) ? smat[(d << 5) + code[r]] : -128;
                        v |= ((uint32_t) m & 0xffu) << (8 * b);
                    }
                    table[(d * 32 + lane) * WORDS + w] = v;
                }
            }
        }
        else {
#pragma unroll
            for( int r = 0; r < R; r++ )
                qa[r] = code[r];
        }
    }
    struct Column {
        uint32_t w[WORDS];
        const int32_t * m;
    };
    __device__ __forceinline__ Column scores( int d ) const {
        Column c;
        if constexpr( P8 ) {
            if constexpr( WORDS == 2 ) {
                const uint2 v = *reinterpret_cast<const uint2 *>( table + (d * 32 + lane) * 2 );
                c.w[0] = v.x;
                c.w[1] = v.y;
            }
            else {
                c.w[0] = table[d * 32 + lane];
            }
            c.m = nullptr;
        }
        else {
            c.m = smat + (d << 5);
        }
        return c;
    }
    // hd + score of row r in column c
    __device__ __forceinline__ int32_t add_score( const Column & c, int r, int32_t hd ) const {
        if constexpr( P8 )
            return __dp4a( (int) c.w[r / 4], 1 << (8 * (r % 4)), hd );
        else
            return hd + c.m[qa[r]];
    }
};

// Largest of the lane's new cells.
template <int R>
__device__ __forceinline__ int32_t column_max( const int32_t (&x)[R] ) {
    int32_t m = x[0];
#pragma unroll
    for( int r = 1; r + 1 < R; r += 2 )
        m = __vimax3_s32( m, x[r], x[r + 1] );
    return max( m, x[R - 1] );
}

// One wavefront step's direction flags of a lane: 2 bits per row, bit 1 =
// insertion (LEFT | EXT_LEFT, takes priority), bit 0 = deletion (UP | EXT_UP).
// A step's 32 lanes are contiguous: one transaction of 32 (R = 4) or 64 bytes.
template <int R>
__device__ __forceinline__ void store_flags( uint8_t * dir, uint32_t s, int lane, uint32_t flags ) {
    if constexpr( R == 8 )
        reinterpret_cast<uint16_t *>( dir )[(uint64_t) s * 32 + lane] = (uint16_t) flags;
    else
        dir[(uint64_t) s * 32 + lane] = (uint8_t) flags;
}

// The best end cell (value desc, database index asc, query index asc) or
// begin cell (column asc, row asc) so far, as it goes down the stripes.
struct Cell {
    int32_t v, i, j;
};

__device__ __forceinline__ bool end_before( const Cell & x, const Cell & y ) {
    return x.v > y.v || (x.v == y.v && (x.i < y.i || (x.i == y.i && x.j < y.j)));
}

__device__ __forceinline__ Cell warp_best( Cell c ) {
    for( int o = 16; o > 0; o >>= 1 ) {
        const Cell t{ __shfl_xor_sync( 0xffffffffu, c.v, o ), __shfl_xor_sync( 0xffffffffu, c.i, o ),
            __shfl_xor_sync( 0xffffffffu, c.j, o ) };
        if( end_before( t, c ) )
            c = t;
    }
    return c;
}

// The reverse pass's limit: the first column that holds a candidate so far.
template <bool REVERSE>
struct ColumnLimit {
    static constexpr bool NONE = !REVERSE;
    const int32_t * p;
    __device__ int32_t operator()() const { return *(volatile const int32_t *) p; }
};

enum TbPhase { TB_FORWARD, TB_REVERSE, TB_DIRECTIONS, TB_FWDDIR };

// ---------------------------------------------------------------------------
// The stripes of one pass over the hits.
//
// TB_FORWARD, the SW forward region pass (reference: src/algo/align.c:39-82).
//    The reference iterates database rows outer and query columns inner,
//    scoring matrix[query][db]; the recurrence is symmetric, so the warp
//    streams the database and keeps the query on lanes.
//
// TB_REVERSE, the SW reverse pass (reference: src/algo/align.c:84-131).  Both
//    sequences are read backwards from the end cell: row j' = a_end - j,
//    column i' = b_end - i.  The boundary row before column 0 is the
//    reference's work row: -1 for query indices <= b_end, the forward pass's
//    last row above that.  The begin cell is the first cell in (i' asc, j'
//    asc) order whose value reaches the forward score; columns past the first
//    column holding a candidate cannot change it, so that column is the hit's
//    limit.
//
// TB_DIRECTIONS, the direction pass (reference: src/algo/cigar.c:48-198).
//    Query rows on lanes, database columns streamed, exactly the reference
//    orientation, rows 0 .. a_end and columns 0 .. b_end.
//
// TB_FWDDIR, both in one sweep of the whole matrix (Smith-Waterman, symmetric
//    score table).  The direction pass's recurrence (reference:
//    src/algo/cigar.c:125-200) and the forward pass's (src/algo/align.c:39-82)
//    give every cell the same H: they differ only in the E and F values that
//    enter the first column and row, which are never above zero and so never
//    reach a Smith-Waterman cell.  With a symmetric table the two orientations
//    score alike.  So this pass computes the directions with the direction
//    pass's values, the end cell (first maximum, database index then query
//    index) from H, and the last column's H and E for the reverse pass.  That
//    E is the forward pass's: at the last column the E chain from earlier
//    cells is at least gapO + gapE (H >= 0), and the host runs this pass only
//    where (B - 1) x gapE < gapO + gapE, so neither pass's initial term can be
//    the maximum there.
// ---------------------------------------------------------------------------
template <int PHASE, int R, bool P8>
__global__ void __launch_bounds__( TB_THREADS ) tb_stripes_kernel( TbParams p ) {
    constexpr int ROWS = 32 * R;
    constexpr bool DIRS = PHASE == TB_DIRECTIONS || PHASE == TB_FWDDIR;
    constexpr bool ENDS = PHASE == TB_FORWARD || PHASE == TB_FWDDIR;       // looks for the end cell
    __shared__ StreamStage<int2> stages[TB_WARPS];
    __shared__ uint8_t residues[TB_WARPS][64];
    __shared__ int32_t smat[1024];
    __shared__ __align__( 16 ) uint32_t tables[P8 ? TB_WARPS : 1][P8 ? 32 * 32 * (R / 4) : 1];
    const int lane = threadIdx.x & 31;
    const int warp = threadIdx.x >> 5;
    // laid out [database code][query code], so that the lanes of a warp (other
    // query rows, same column) read other banks; the region passes score
    // matrix[query][db]
    for( int i = threadIdx.x; i < 1024; i += TB_THREADS ) {
        const int d = i >> 5, q = i & 31;
        smat[i] = (int32_t) (DIRS ? p.matrix[(d << 5) + q] : p.matrix[(q << 5) + d]);
    }
    __syncthreads();
    StreamStage<int2> & st = stages[warp];

    for( ;; ) {
        const uint32_t ticket = next_hit( p.counter, lane );
        if( ticket >= p.n_tickets )
            break;
        const uint32_t stripe = ticket_stripe( p.cum, p.levels, ticket );
        const uint32_t h = ticket - p.cum[stripe];
        const uint32_t pred = stripe ? p.cum[stripe - 1] + h : 0u;
        const TbHit hit = p.hits[h];
        const TbRegion rg = p.regions[h];
        if( PHASE != TB_FORWARD && PHASE != TB_FWDDIR && rg.status != 0 )
            continue;                                   // every stripe of the hit
        const bool nw = hit.algo == 1;
        uint32_t A, B;
        if constexpr( ENDS ) {
            A = p.qlen[hit.qslot];
            B = p.db.lens[hit.id];
        }
        else {
            A = (uint32_t) rg.a_end + 1u;
            B = (uint32_t) rg.b_end + 1u;
        }
        if( stripe * (uint32_t) ROWS >= A )
            continue;                                   // the reverse pass may need fewer rows than the query has
        const uint8_t * a = p.qcodes + p.qoff[hit.qslot];

        StreamStripe<int2> sp;
        sp.cols = B;
        sp.row = p.boundary + p.bnd_off[h];
        sp.above = stripe ? p.progress + pred : nullptr;
        sp.mine = p.progress + ticket;
        sp.last = (stripe + 1u) * (uint32_t) ROWS >= A;
        sp.error_flags = p.error_flags;
        ResidueRing rr{ residues[warp], 0, p.db.codes + p.db.offsets[hit.id], (int32_t) B,
            PHASE == TB_REVERSE ? rg.b_end : -1 };

        TbLane<R, P8> t;
        t.table = tables[P8 ? warp : 0];
        t.smat = smat;
        t.lane = lane;
        t.gO = p.gap_open;
        t.gE = p.gap_extend;
        t.gOE = p.gap_open + p.gap_extend;
        t.row0 = (int32_t) (stripe * (uint32_t) ROWS) + lane * R;
        t.nvalid = max( 0, min( R, (int) A - t.row0 ) );
        t.out_h = 0;
        t.out_f = 0;
        t.diag = 0;
        const int32_t gO = t.gO, gE = t.gE, gOE = t.gOE, row0 = t.row0;
        int32_t * lh = nullptr;
        int32_t * le = nullptr;
        if( ENDS || PHASE == TB_REVERSE ) {
            lh = p.last_h + p.last_off[h];
            le = p.last_e + p.last_off[h];
        }
        if constexpr( PHASE == TB_REVERSE )
            t.load_rows( a, (int64_t) rg.a_end - row0, -1 );
        else
            t.load_rows( a, row0, 1 );
#pragma unroll
        for( int r = 0; r < R; r++ ) {
            if constexpr( PHASE == TB_FORWARD ) {
                t.H[r] = 0;                             // HH[j] = 0
                t.E[r] = gO + gE;                       // max(EE = gapO, HH + gapO) + gapE at row 0
            }
            else if constexpr( PHASE == TB_REVERSE ) {
                const int32_t j = rg.a_end - (row0 + r);    // query index
                int32_t hh = -1, ee = -1;
                if( r < t.nvalid && j > rg.b_end ) {
                    hh = lh[j];
                    ee = le[j];
                }
                t.H[r] = hh;                            // HH(b_end + 1, j)
                t.E[r] = max( ee, hh + gO ) + gE;       // EE(b_end, j)
            }
            else {
                const int32_t i = row0 + r;
                t.H[r] = nw ? gO + (i + 1) * gE : 0;
                t.E[r] = nw ? 2 * gO + (i + 2) * gE : 0;
            }
        }
        // the diagonal of the lane's first row at column 0
        if constexpr( PHASE == TB_REVERSE ) {
            // HH(b_end + 1, j + 1), or 0 for the end cell itself
            const int32_t jprev = rg.a_end - (row0 - 1);
            t.diag = (row0 == 0) ? 0 : ((jprev > rg.b_end && t.nvalid > 0) ? lh[jprev] : -1);
        }
        else if constexpr( PHASE == TB_DIRECTIONS ) {
            t.diag = (nw && row0 > 0) ? gO + row0 * gE : 0;
        }
        // end cell: this lane's first maximum; begin cell: its first candidate (i = column, j = row)
        Cell best{ 0, INT_MAX, INT_MAX };
        uint8_t * dir = nullptr;
        if constexpr( DIRS )
            dir = p.dirs + p.dir_off[h] + (uint64_t) stripe * ((uint64_t) B + 31) * (32 * R / 4);

        auto column = [&]( const uint32_t s, const bool edge, const uint32_t cols ) {
            int32_t up_h = __shfl_up_sync( 0xffffffffu, t.out_h, 1 );
            int32_t up_f = __shfl_up_sync( 0xffffffffu, t.out_f, 1 );
            const int32_t c = (int32_t) s - lane;
            if( edge && (c < 0 || c >= (int32_t) cols) )
                return;
            if( lane == 0 ) {
                if( stripe == 0 ) {
                    if constexpr( PHASE == TB_FORWARD ) {
                        up_h = 0;
                        up_f = gO + gE;                 // f starts at gapO: max(gapO, 0 + gapO) + gapE
                    }
                    else if constexpr( PHASE == TB_REVERSE ) {
                        up_h = -1;                      // h starts at -1 per row; f = max(-1, h + gapO) + gapE
                        up_f = max( -1, -1 + gO ) + gE;
                    }
                    else {
                        // H(-1, c) is the next column's row-0 diagonal
                        up_h = nw ? gO + (c + 1) * gE : 0;
                        up_f = nw ? 2 * gO + (c + 2) * gE : 0;
                    }
                }
                else {
                    const int2 v = st.in[s & 31u];
                    up_h = v.x;
                    up_f = v.y;
                }
            }
            const auto sc = t.scores( rr.get( s, lane ) );
            int32_t f = up_f, hd = t.diag;
            int32_t x[R];
            uint32_t flags = 0;
            const bool last_col = ENDS && edge && c == (int32_t) B - 1;
#pragma unroll
            for( int r = 0; r < R; r++ ) {
                const int32_t e = t.E[r];
                const int32_t x0 = t.add_score( sc, r, hd );
                hd = t.H[r];
                if constexpr( DIRS ) {
                    // flags as in the reference (strict compares in its
                    // order): each max also yields the negation of one
                    bool no_up, no_left, no_ext_up, no_ext_left;
                    const int32_t m1 = __vibmax_s32( x0, f, &no_up );       // UP: f > x0
                    const int32_t xr = __vibmax_s32( m1, e, &no_left );     // LEFT: e > max(x0, f)
                    x[r] = (PHASE == TB_DIRECTIONS && nw) ? xr : max( xr, 0 );
                    const int32_t y = x[r] + gOE;
                    f = __vibmax_s32( y, f + gE, &no_ext_up );               // EXT_UP: f + gapE > y
                    t.E[r] = __vibmax_s32( y, e + gE, &no_ext_left );        // EXT_LEFT: e + gapE > y
                    // rows past the query's end get flags too; the walk never reads them
                    if( !(no_left && no_ext_left) )
                        flags |= 2u << (2 * r);
                    if( !(no_up && no_ext_up) )
                        flags |= 1u << (2 * r);
                }
                else {
                    x[r] = PHASE == TB_FORWARD ? __vimax3_s32( max( x0, 0 ), f, e ) : __vimax3_s32( x0, f, e );
                    const int32_t y = x[r] + gOE;
                    f = __viaddmax_s32( f, gE, y );
                    t.E[r] = __viaddmax_s32( e, gE, y );
                }
                t.H[r] = x[r];
                if( last_col && r < t.nvalid ) {
                    lh[row0 + r] = x[r];
                    le[row0 + r] = e;
                }
            }
            if constexpr( DIRS )
                store_flags<R>( dir, s, lane, flags );
            if constexpr( ENDS ) {
                // the lane visits its cells in (column, row) order: its first
                // maximum wins with a strict compare, and rarely is there one
                if( column_max<R>( x ) > best.v ) {
#pragma unroll
                    for( int r = 0; r < R; r++ )
                        if( r < t.nvalid && x[r] > best.v )
                            best = Cell{ x[r], c, row0 + r };
                }
            }
            if constexpr( PHASE == TB_REVERSE ) {
                if( column_max<R>( x ) >= rg.fwd_score && best.i == INT_MAX ) {
#pragma unroll
                    for( int r = R - 1; r >= 0; r-- )
                        if( r < t.nvalid && x[r] >= rg.fwd_score )
                            best = Cell{ 0, c, row0 + r };
                    if( best.i != INT_MAX )
                        atomicMin( p.limit + h, c );
                }
            }
            if constexpr( PHASE == TB_DIRECTIONS ) {
                if( nw && edge && c == (int32_t) B - 1 ) {
                    // the global score: the last cell of the full matrix
#pragma unroll
                    for( int r = 0; r < R; r++ )
                        if( row0 + r == (int32_t) A - 1 )
                            p.regions[h].fwd_score = x[r];
                }
            }
            t.diag = up_h;
            t.out_h = x[R - 1];
            t.out_f = f;
            if( lane == 31 )
                st.out[s & 31u] = make_int2( t.out_h, t.out_f );
        };
        rr.start( lane );
        const ColumnLimit<PHASE == TB_REVERSE> limit{ p.limit + h };
        const uint32_t swept = stream_columns<32>( sp, st, lane, limit, [&]( uint32_t s0 ) { rr.step( s0, lane ); },
                column );
        if constexpr( PHASE != TB_DIRECTIONS ) {
            // this stripe's cell against that of the stripes above (theirs is
            // final once the stripe above has ended)
            best = warp_best( best );
            if( sp.above ) {
                stream_wait( sp.above, STREAM_DONE, lane, sp.error_flags );
                const int4 o = __ldcg( p.result + pred );
                const Cell other{ o.x, o.y, o.z };
                if( !end_before( best, other ) )
                    best = other;
            }
            if( lane == 0 ) {
                if( !sp.last ) {
                    __stcg( p.result + ticket, make_int4( best.v, best.i, best.j, 0 ) );
                }
                else if constexpr( ENDS ) {
                    TbRegion out = rg;                  // the host set the rest of the region; keep it
                    out.fwd_score = best.v;
                    out.a_end = best.j;
                    out.b_end = best.i;
                    out.a_begin = 0;
                    out.b_begin = 0;
                    out.status = (best.v > 0) ? 0 : 1;
                    p.regions[h] = out;
                }
                else {
                    TbRegion out = rg;
                    if( best.i == INT_MAX ) {
                        out.status = 2;
                    }
                    else {
                        out.b_begin = rg.b_end - best.i;
                        out.a_begin = rg.a_end - best.j;
                    }
                    p.regions[h] = out;
                }
            }
        }
        stream_end( sp, swept, lane );
    }
}

// ---------------------------------------------------------------------------
// 4. Walk (reference: src/algo/cigar.c:300-334): one warp per hit writes the
//    moves in traceback order (end to begin); the host run-length encodes.
//    Each step reads the direction word of the current cell, which the
//    previous step chose, so a walk that reads HBM or L2 word by word waits a
//    memory round trip per move.  In 32 moves the path stays within 32 rows
//    and 32 columns of its current cell (every move leaves the row or the
//    column or both by one), so the warp loads that window (32 columns, at
//    most 9 bytes of 4 rows each) into shared memory with one load round,
//    lane 0 walks up to 32 moves from it, and the warp loads the next window.
// ---------------------------------------------------------------------------
constexpr int TB_WALK_WARPS = 4;                 // hits per CTA
constexpr int TB_WALK_GROUPS = 32 / 4 + 1;       // bytes of four rows that a 32-row window spans

__global__ void __launch_bounds__( 32 * TB_WALK_WARPS ) tb_walk_kernel( TbParams p, int R ) {
    __shared__ uint8_t win[TB_WALK_WARPS][32][TB_WALK_GROUPS + 3];
    const int lane = threadIdx.x & 31;
    const int wib = threadIdx.x >> 5;
    const uint32_t h = blockIdx.x * TB_WALK_WARPS + (uint32_t) wib;
    if( h >= p.n_hits )
        return;                                  // the whole warp
    const TbRegion rg = p.regions[h];
    if( rg.status != 0 ) {
        if( lane == 0 )
            p.ops_len[h] = 0;
        return;
    }
    const uint8_t * dir = p.dirs + p.dir_off[h];
    char * out = p.ops + p.ops_off[h];
    const uint64_t cap = p.ops_off[h + 1] - p.ops_off[h];
    const int32_t a_begin = rg.a_begin, b_begin = rg.b_begin;
    const int stripe_rows = 32 * R, lane_bytes = R / 4;
    const uint64_t stripe_bytes = (uint64_t) rg.dir_steps * 32 * lane_bytes;
    int32_t i = rg.a_end, j = rg.b_end;
    uint64_t n = 0;
    while( i >= a_begin && j >= b_begin && i >= 0 && j >= 0 ) {
        // the window: columns j - 31 .. j, groups of four rows that hold i - 31 .. i
        const int32_t g0 = max( i - 31, 0 ) / 4;
        const int32_t jc = j - lane;
#pragma unroll
        for( int k = 0; k < TB_WALK_GROUPS; k++ ) {
            const int32_t row = 4 * (g0 + k);
            uint8_t v = 0;
            if( jc >= b_begin && row <= i ) {
                const int32_t in_stripe = row % stripe_rows;
                const int32_t owner = in_stripe / R;           // the row's lane, at step jc + owner
                v = dir[(uint64_t) (row / stripe_rows) * stripe_bytes +
                        ((uint64_t) (jc + owner) * 32 + owner) * lane_bytes + (in_stripe % R) / 4];
            }
            win[wib][lane][k] = v;
        }
        __syncwarp();
        if( lane == 0 ) {
            const int32_t j0 = j;
            for( int m = 0; m < 32 && i >= a_begin && j >= b_begin && i >= 0 && j >= 0; m++ ) {
                const uint32_t op = ((uint32_t) win[wib][j0 - j][i / 4 - g0] >> (2 * (i % 4))) & 3u;
                char ch;
                if( op & 2u ) {
                    j--;
                    ch = 'I';
                }
                else if( op == 1u ) {
                    i--;
                    ch = 'D';
                }
                else {
                    i--;
                    j--;
                    ch = 'M';
                }
                if( n < cap )
                    out[n] = ch;
                n++;
            }
        }
        i = __shfl_sync( 0xffffffffu, i, 0 );
        j = __shfl_sync( 0xffffffffu, j, 0 );
        n = __shfl_sync( 0xffffffffu, n, 0 );
        __syncwarp();
    }
    if( lane == 0 )
        p.ops_len[h] = (uint32_t) n;
}

cudaError_t launch_tb_walk( const TbParams & p, int R, cudaStream_t st ) {
    if( p.n_hits )
        tb_walk_kernel<<<(p.n_hits + TB_WALK_WARPS - 1) / TB_WALK_WARPS, 32 * TB_WALK_WARPS, 0, st>>>( p, R );
    return cudaGetLastError();
}

template <int PHASE, int R, bool P8>
static cudaError_t launch_stripes( const TbParams & p, int sms, cudaStream_t st ) {
    static LaunchShape shape;
    const cudaError_t e = shape.set( tb_stripes_kernel<PHASE, R, P8>, TB_THREADS, 0 );
    if( e != cudaSuccess )
        return e;
    const uint32_t want = (p.n_tickets + TB_WARPS - 1) / TB_WARPS;
    const uint32_t grid = min( want, (uint32_t) (sms * max( 1, shape.blocks )) );
    if( grid )
        tb_stripes_kernel<PHASE, R, P8><<<grid, TB_THREADS, 0, st>>>( p );
    return cudaGetLastError();
}

template <int PHASE>
static cudaError_t launch_phase( const TbParams & p, int R, bool p8, int sms, cudaStream_t st ) {
    if( R == 4 )
        return p8 ? launch_stripes<PHASE, 4, true>( p, sms, st ) : launch_stripes<PHASE, 4, false>( p, sms, st );
    return p8 ? launch_stripes<PHASE, 8, true>( p, sms, st ) : launch_stripes<PHASE, 8, false>( p, sms, st );
}

cudaError_t launch_tb_forward( const TbParams & p, int R, bool p8, int sms, cudaStream_t st ) {
    return launch_phase<TB_FORWARD>( p, R, p8, sms, st );
}

cudaError_t launch_tb_reverse( const TbParams & p, int R, bool p8, int sms, cudaStream_t st ) {
    return launch_phase<TB_REVERSE>( p, R, p8, sms, st );
}

cudaError_t launch_tb_directions( const TbParams & p, int R, bool p8, int sms, cudaStream_t st ) {
    return launch_phase<TB_DIRECTIONS>( p, R, p8, sms, st );
}

cudaError_t launch_tb_fwddir( const TbParams & p, int R, bool p8, int sms, cudaStream_t st ) {
    return launch_phase<TB_FWDDIR>( p, R, p8, sms, st );
}

}  // namespace ssa
