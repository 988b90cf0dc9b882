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
// 32 x R, database columns stream through the warp in blocks of four, the bottom
// row of a lane goes to the next lane by shuffle, and the stripes of a hit
// follow one another on different warps through the hit's boundary row
// (stream_stripes.cuh).  All arithmetic is exact (int32, with the host
// guaranteeing the range), matching the reference's int64 code.  The same sweep
// without directions scores pairs of a query and one chosen sequence
// (ssa_align_pairs): for a database of one sequence every entry width of the
// reference reports the exact score.
//
// What bounds it: the integer ALU pipe (16 lanes per clock per SM
// sub-partition) when many hits fill the GPU, the latency of one warp's steps
// (blocks + STREAM_LAG x stripes of them per hit) when few do.  A step interleaves the
// four columns of a block row by row (cell (it - j, j) in iteration `it`): four
// independent dependency chains where one column at a time has one, and the
// step's fixed work (shuffles, residues, boundary, stores) once per 4 R cells.
// R is 4: 8 rows per lane measured the same where hits fill the GPU (48 long
// pairs 32 and 30 ms) and up to 1.7 times longer where they do not (half the
// warps, twice the work per step); the host takes 2 for a few Smith-Waterman
// hits much longer than high (10 of 300 x 33,000: 3.8 -> 2.9 ms).  A lane's scores of a column are one
// shared-memory word of int8 entries, added to the diagonal by dp4a (off the ALU
// pipe); tables past int8 are read entry by entry.
//
// The flags of a cell are two minimum-of-three and two signs (8 ALU instructions
// per cell with the recurrence); maxima that also return a predicate, with the
// predicates combined into flags, took 24 (counters: 647 -> 365 instructions per
// warp and step of 16 cells).
//
// Measured on a B200 (one call each): groups of 1, 2 or 4 warps of one CTA per
// hit with a group barrier every 32 steps / streamed stripes, one column per
// step / four columns per step / signs as flags and three CTAs per SM and
// the walk by runs: 48 pairs of 5,000-30,000 residues, SW 780 / 53 / 42 / 28 ms
// and NW 470 / 35 / 24 / 16 ms; 10 hits of 300 x 33,000 20.5 / 9.3 / 4.3 / 4.0 ms (3.1 with R = 2); 320 hits
// of 30-1,355 rows 4.7 / 1.3 / 1.1 / 1.0 ms.
#include "device_common.cuh"
#include "stream_stripes.cuh"

#include <climits>

namespace ssa {

constexpr int TB_THREADS = 128;
constexpr int TB_WARPS = TB_THREADS / 32;
// CTAs per SM.  Five fit, but where many long hits are aligned at once the call
// takes as long as the stripes of the longest do, one after the other, and those
// run slower the more other warps share their sub-partition; three keep the ALU as
// busy.  48 pairs of 5,000-30,000 residues with five / three / two: SW 24.7 /
// 20.2 / 20.0 ms and the reverse pass 9.0 / 7.3 / 7.2, NW 18.1 / 15.7 / 15.6 ms;
// 320 hits of 30-1,355 rows 0.60 / 0.60 / 0.60, 1,600 hits 0.58 / 0.58 / 0.62 ms.
constexpr int TB_BLOCKS = 3;

// What the stripe bodies share: the lane's rows and their scores.
template <int R, bool P8>
struct TbLane {
    uint32_t * table;              // P8: the warp's scores, a word of four int8 entries per code and lane
    const int32_t * smat;          // the score table, [database code][query code]
    int lane;
    int32_t gO, gE, gOE;
    int qa[P8 ? 1 : R];            // !P8: query codes of the rows (0 past the end)
    int32_t H[R], E[R];
    int32_t diag, row0;
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
                uint32_t v = 0;
#pragma unroll
                for( int r = 0; r < R; r++ ) {
                    const int32_t m = (r < nvalid) ? smat[(d << 5) + code[r]] : -128;
                    v |= ((uint32_t) m & 0xffu) << (8 * r);
                }
                table[d * 32 + lane] = v;
            }
        }
        else {
#pragma unroll
            for( int r = 0; r < R; r++ )
                qa[r] = code[r];
        }
    }
    struct Column {
        uint32_t w;
        const int32_t * m;
    };
    __device__ __forceinline__ Column scores( int d ) const {
        if constexpr( P8 )
            return Column{ table[d * 32 + lane], nullptr };
        else
            return Column{ 0, smat + (d << 5) };
    }
    // hd + score of row r in column c
    __device__ __forceinline__ int32_t add_score( const Column & c, int r, int32_t hd ) const {
        if constexpr( P8 )
            return __dp4a( (int) c.w, 1 << (8 * r), hd );
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

// The reverse pass's limit: the first block that holds a candidate so far.
template <bool REVERSE>
struct ColumnLimit {
    static constexpr bool NONE = !REVERSE;
    const int32_t * p;
    __device__ int32_t operator()() const { return *(volatile const int32_t *) p; }
};

enum TbPhase { TB_FORWARD, TB_REVERSE, TB_DIRECTIONS, TB_FWDDIR, TB_NW_DIRECTIONS, TB_SCORE, TB_NW_SCORE };

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
// TB_DIRECTIONS and TB_NW_DIRECTIONS, the direction pass (reference:
//    src/algo/cigar.c:48-198).  Query rows on lanes, database columns streamed,
//    exactly the reference orientation, rows 0 .. a_end and columns 0 .. b_end.
//
// TB_SCORE and TB_NW_SCORE, the same recurrence without directions: the
//    largest cell, or H of the last row and column
//    (src/algo/64/smith_waterman_63.c:32-98, needleman_wunsch_64.c:32-98).
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
    constexpr int C = 4;
    constexpr bool NW = PHASE == TB_NW_DIRECTIONS || PHASE == TB_NW_SCORE;
    constexpr bool DIRS = PHASE == TB_DIRECTIONS || PHASE == TB_FWDDIR || PHASE == TB_NW_DIRECTIONS;
    constexpr bool ENDS = PHASE == TB_FORWARD || PHASE == TB_FWDDIR;       // looks for the end cell
    constexpr bool MATRIX = ENDS || PHASE == TB_SCORE || PHASE == TB_NW_SCORE;     // every row and column
    constexpr bool MAXIMUM = ENDS || PHASE == TB_SCORE;
    constexpr bool REVERSE = PHASE == TB_REVERSE;
    __shared__ StreamStage stages[TB_WARPS];
    __shared__ uint32_t rings[TB_WARPS][64];
    __shared__ int32_t smat[1024];
    __shared__ uint32_t tables[P8 ? TB_WARPS : 1][P8 ? 32 * 32 : 1];
    const int lane = threadIdx.x & 31;
    const int warp = threadIdx.x >> 5;
    // laid out [database code][query code], so that the lanes of a warp (other
    // query rows, same column) read other banks; the region passes score
    // matrix[query][db]
    for( int i = threadIdx.x; i < 1024; i += TB_THREADS ) {
        const int d = i >> 5, q = i & 31;
        smat[i] = (int32_t) (PHASE == TB_FORWARD || REVERSE ? p.matrix[(q << 5) + d] : p.matrix[(d << 5) + q]);
    }
    __syncthreads();
    StreamStage & st = stages[warp];

    for( ;; ) {
        const uint32_t ticket = next_ticket( p.counter, lane );
        if( ticket >= p.n_tickets )
            break;
        const uint32_t stripe = ticket_stripe( p.cum, p.levels, ticket );
        const uint32_t h = ticket - p.cum[stripe];
        const uint32_t pred = stripe ? p.cum[stripe - 1] + h : 0u;
        const TbHit hit = p.hits[h];
        const TbRegion rg = p.regions[h];
        if( !MATRIX && rg.status != 0 )
            continue;                                   // every stripe of the hit
        uint32_t A, B;
        if constexpr( MATRIX ) {
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
        const uint32_t nb = (B + 3u) >> 2;              // blocks of four columns

        StreamStripe sp;
        sp.cols = nb;
        sp.row = p.boundary + p.bnd_off[h];
        sp.above = stripe ? p.progress + pred : nullptr;
        sp.mine = p.progress + ticket;
        sp.last = (stripe + 1u) * (uint32_t) ROWS >= A;
        sp.error_flags = p.error_flags;

        TbLane<R, P8> t;
        t.table = tables[P8 ? warp : 0];
        t.smat = smat;
        t.lane = lane;
        t.gO = p.gap_open;
        t.gE = p.gap_extend;
        t.gOE = p.gap_open + p.gap_extend;
        t.row0 = (int32_t) (stripe * (uint32_t) ROWS) + lane * R;
        t.nvalid = max( 0, min( R, (int) A - t.row0 ) );
        const int32_t gO = t.gO, gE = t.gE, gOE = t.gOE, row0 = t.row0;
        int32_t * lh = nullptr;
        int32_t * le = nullptr;
        if( ENDS || REVERSE ) {
            lh = p.last_h + p.last_off[h];
            le = p.last_e + p.last_off[h];
        }
        if constexpr( REVERSE )
            t.load_rows( a, (int64_t) rg.a_end - row0, -1 );
        else
            t.load_rows( a, row0, 1 );
#pragma unroll
        for( int r = 0; r < R; r++ ) {
            if constexpr( PHASE == TB_FORWARD ) {
                t.H[r] = 0;                             // HH[j] = 0
                t.E[r] = gO + gE;                       // max(EE = gapO, HH + gapO) + gapE at row 0
            }
            else if constexpr( REVERSE ) {
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
                // the reference's column before the first: H(i, -1), E(i, -1)
                const int32_t i = row0 + r;
                t.H[r] = NW ? gO + (i + 1) * gE : 0;
                t.E[r] = NW ? 2 * gO + (i + 2) * gE : 0;
            }
        }
        // the diagonal of the lane's first row at column 0
        t.diag = 0;
        if constexpr( REVERSE ) {
            // HH(b_end + 1, j + 1), or 0 for the end cell itself
            const int32_t jprev = rg.a_end - (row0 - 1);
            t.diag = (row0 == 0) ? 0 : ((jprev > rg.b_end && t.nvalid > 0) ? lh[jprev] : -1);
        }
        else if constexpr( NW ) {
            t.diag = row0 > 0 ? gO + row0 * gE : 0;
        }
        // end cell: this lane's first maximum; begin cell: its first candidate (i = column, j = row)
        Cell best{ 0, INT_MAX, INT_MAX };
        uint32_t * dir = nullptr;
        if constexpr( DIRS )
            dir = p.dirs + p.dir_off[h] + (uint64_t) stripe * ((uint64_t) nb + 31) * 32;
        int32_t out_h[C] = {}, out_f[C] = {};

        // Residue words, read a step ahead of use: block b of the forward
        // direction is word b.  The reverse pass reads columns b_end - 4b down
        // to b_end - 4b - 3, which lie in the word of the last of them and the
        // word after it (the previous block's).
        const uint32_t * res = reinterpret_cast<const uint32_t *>( p.db.codes + p.db.offsets[hit.id] );
        auto fetch = [&]( int32_t b ) -> uint32_t {
            const int32_t w = REVERSE ? (rg.b_end - 4 * b - 3) >> 2 : b;
            return (uint32_t) w < nb ? __ldg( res + w ) : 0u;
        };
        StreamResidues<uint32_t> residues{ rings[warp], 0u };
        residues.start( lane, fetch );
        uint32_t before = REVERSE ? residues.at( -lane - 1 ) : 0u, w0 = residues.at( -lane );
        const int32_t last_block = (int32_t) nb - 1, last_chain = (int32_t) (B - 1u) & 3;

        auto block = [&]( const uint32_t s, const bool edge, const uint32_t blocks ) {
            int32_t up_h[C], up_f[C];
#pragma unroll
            for( int j = 0; j < C; j++ ) {
                up_h[j] = __shfl_up_sync( 0xffffffffu, out_h[j], 1 );
                up_f[j] = __shfl_up_sync( 0xffffffffu, out_f[j], 1 );
            }
            const int32_t b = (int32_t) s - lane;
            uint32_t word = w0;
            if constexpr( REVERSE ) {
                word = __byte_perm( __funnelshift_r( w0, before, 8u * ((uint32_t) (rg.b_end - 3) & 3u) ), 0, 0x0123 );
                before = w0;
            }
            w0 = residues.at( b + 1 );
            if( edge && (b < 0 || b >= (int32_t) blocks) )
                return;
            if( lane == 0 ) {
                const int4 x = st.in[2 * (s % STREAM_CHUNK)], y = st.in[2 * (s % STREAM_CHUNK) + 1];
                up_h[0] = x.x;
                up_f[0] = x.y;
                up_h[1] = x.z;
                up_f[1] = x.w;
                up_h[2] = y.x;
                up_f[2] = y.y;
                up_h[3] = y.z;
                up_f[3] = y.w;
            }
            typename TbLane<R, P8>::Column sc[C];
            int32_t f[C], hv[C][R];
            // 2 bits per cell (bit 1 = insertion, LEFT | EXT_LEFT, takes priority;
            // bit 0 = deletion, UP | EXT_UP), a byte per column, the first row in its top bits
            uint32_t flags[C] = {};
#pragma unroll
            for( int j = 0; j < C; j++ ) {
                sc[j] = t.scores( (int) ((word >> (8 * j)) & 0xffu) );
                f[j] = up_f[j];
            }
            const bool last_col = ENDS && edge && b == last_block;
            // chain j is column j of the block; H[r] keeps the column before the
            // block until chain 3 overwrites it, E[r] passes from chain to chain
#pragma unroll
            for( int it = 0; it < R + C - 1; it++ ) {
#pragma unroll
                for( int j = 0; j < C; j++ ) {
                    const int r = it - j;
                    if( r < 0 || r >= R )
                        continue;
                    const int32_t e = t.E[r];
                    const int32_t hd = r == 0 ? (j == 0 ? t.diag : up_h[j - 1]) : (j == 0 ? t.H[r - 1] : hv[j - 1][r - 1]);
                    const int32_t x0 = t.add_score( sc[j], r, hd );
                    int32_t x;
                    if constexpr( DIRS ) {
                        // The reference's flags with its strict compares: UP, f > x0;
                        // LEFT, e > max(x0, f); EXT_UP, f + gapE > y; EXT_LEFT,
                        // e + gapE > y, where y = x + gapO + gapE.  So UP or EXT_UP is
                        // f > min(x0, x + gapO), and LEFT or EXT_LEFT the same with
                        // e and max(x0, f); each sign goes in from the right.  Rows past
                        // the query's end get flags too; the walk never reads them.
                        const int32_t m1 = max( x0, f[j] );
                        x = NW ? max( m1, e ) : __vimax3_s32( m1, e, 0 );
                        const int32_t y = x + gOE;
                        flags[j] = __funnelshift_l( (uint32_t) (__viaddmin_s32( x, gO, m1 ) - e), flags[j], 1 );
                        flags[j] = __funnelshift_l( (uint32_t) (__viaddmin_s32( x, gO, x0 ) - f[j]), flags[j], 1 );
                        f[j] = __viaddmax_s32( f[j], gE, y );
                        t.E[r] = __viaddmax_s32( e, gE, y );
                    }
                    else {
                        x = PHASE == TB_FORWARD || PHASE == TB_SCORE ? __vimax3_s32( max( x0, 0 ), f[j], e )
                                                                     : __vimax3_s32( x0, f[j], e );
                        const int32_t y = x + gOE;
                        f[j] = __viaddmax_s32( f[j], gE, y );
                        t.E[r] = __viaddmax_s32( e, gE, y );
                    }
                    hv[j][r] = x;
                    if( last_col && j == last_chain && r < t.nvalid ) {
                        lh[row0 + r] = x;
                        le[row0 + r] = e;
                    }
                    if( j == C - 1 )
                        t.H[r] = x;
                }
            }
            if constexpr( DIRS ) {
                const uint32_t lo = __byte_perm( flags[0], flags[1], 0x0040 ), hi = __byte_perm( flags[2], flags[3], 0x0040 );
                dir[(uint64_t) s * 32 + lane] = __byte_perm( lo, hi, 0x5410 );     // one transaction of 128 bytes per step
            }
            if constexpr( MAXIMUM || REVERSE ) {
                // the lane visits its cells in (column, row) order: its first
                // maximum (its first candidate) counts, and rarely is there one
                int32_t most = column_max( hv[0] );
#pragma unroll
                for( int j = 1; j < C; j++ )
                    most = max( most, column_max( hv[j] ) );
                if( MAXIMUM && most > best.v ) {
#pragma unroll
                    for( int j = 0; j < C; j++ )
#pragma unroll
                        for( int r = 0; r < R; r++ )
                            if( r < t.nvalid && 4 * b + j < (int32_t) B && hv[j][r] > best.v )
                                best = Cell{ hv[j][r], 4 * b + j, row0 + r };
                }
                if( REVERSE && most >= rg.fwd_score && best.i == INT_MAX ) {
#pragma unroll
                    for( int j = 0; j < C; j++ )
#pragma unroll
                        for( int r = 0; r < R; r++ )
                            if( r < t.nvalid && 4 * b + j < (int32_t) B && hv[j][r] >= rg.fwd_score &&
                                    best.i == INT_MAX )
                                best = Cell{ 0, 4 * b + j, row0 + r };
                    if( best.i != INT_MAX )
                        atomicMin( p.limit + h, b );
                }
            }
            if constexpr( NW ) {
                if( edge && sp.last && b == last_block ) {
                    // the global score: the last cell of the full matrix
#pragma unroll
                    for( int j = 0; j < C; j++ )
#pragma unroll
                        for( int r = 0; r < R; r++ )
                            if( j == last_chain && row0 + r == (int32_t) A - 1 )
                                p.regions[h].fwd_score = hv[j][r];
                }
            }
            t.diag = up_h[C - 1];
#pragma unroll
            for( int j = 0; j < C; j++ ) {
                out_h[j] = hv[j][R - 1];
                out_f[j] = f[j];
            }
            if( lane == 31 ) {
                st.out[2 * (s % STREAM_CHUNK)] = make_int4( out_h[0], out_f[0], out_h[1], out_f[1] );
                st.out[2 * (s % STREAM_CHUNK) + 1] = make_int4( out_h[2], out_f[2], out_h[3], out_f[3] );
            }
        };
        // the row above the first stripe, columns c and c + 1: H(-1, c) (the next
        // column's diagonal) and F entering row 0
        auto top = [&]( int32_t c ) -> int4 {
            if constexpr( PHASE == TB_FORWARD )         // f starts at gapO: max(gapO, 0 + gapO) + gapE
                return make_int4( 0, gO + gE, 0, gO + gE );
            else if constexpr( REVERSE )                // h starts at -1 per row; f = max(-1, h + gapO) + gapE
                return make_int4( -1, max( -1, -1 + gO ) + gE, -1, max( -1, -1 + gO ) + gE );
            else if constexpr( NW )
                return make_int4( gO + (c + 1) * gE, 2 * gO + (c + 2) * gE, gO + (c + 2) * gE, 2 * gO + (c + 3) * gE );
            else
                return make_int4( 0, 0, 0, 0 );
        };
        auto refill = [&]( uint32_t s0 ) {
            if( stripe == 0 && lane < (int) (2 * STREAM_CHUNK) )
                st.in[lane] = top( 4 * (int32_t) s0 + 2 * lane );
            residues.refill( s0, lane, fetch );
        };
        const ColumnLimit<REVERSE> limit{ p.limit + h };
        const uint32_t swept = stream_columns( sp, st, lane, limit, refill, block );
        if constexpr( MAXIMUM || REVERSE ) {
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
                else if constexpr( MAXIMUM ) {
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
//    Each step reads the direction bits of the current cell, which the
//    previous step chose.  So that no move waits a memory round trip, the warp
//    loads a band of words of 4 x 4 cells along the diagonal from its current
//    cell (33 words down, 8 to either side; 18 loads per lane in flight
//    together) into shared memory and walks until it leaves the band; and so
//    that few moves wait for the one before, the lanes read the next 32 cells of
//    the diagonal, the row or the column, and the moves of one kind up to the
//    first other one are written together.  Bound by the latency of the loads
//    and of a shared-memory read and a vote per run.  Paths of 5,500-33,000 moves,
//    48 hits: lane 0 alone in windows of 32 and of 64 moves 4.6 and 2.3 ms, this
//    0.64 ms.
// ---------------------------------------------------------------------------
constexpr int TB_WALK_ROWS = 33;                 // words of the band down the diagonal
constexpr int TB_WALK_SIDE = 8;                  // words to either side of it
constexpr int TB_WALK_WIDTH = 2 * TB_WALK_SIDE + 1;

template <int R>
__global__ void __launch_bounds__( 32 ) tb_walk_kernel( TbParams p ) {
    constexpr int ROWS = 32 * R, WORDS = TB_WALK_ROWS * TB_WALK_WIDTH, LOADS = (WORDS + 31) / 32;
    __shared__ uint32_t band[WORDS];
    const int lane = threadIdx.x;
    const uint32_t h = blockIdx.x;
    const TbRegion rg = p.regions[h];
    if( rg.status != 0 ) {
        if( lane == 0 )
            p.ops_len[h] = 0;
        return;
    }
    const uint32_t * dir = p.dirs + p.dir_off[h];
    char * out = p.ops + p.ops_off[h];
    const uint64_t cap = p.ops_off[h + 1] - p.ops_off[h];
    const int32_t a_begin = max( rg.a_begin, 0 ), b_begin = max( rg.b_begin, 0 );
    const uint64_t stripe_words = (uint64_t) rg.dir_steps * 32;
    int32_t i = rg.a_end, j = rg.b_end;          // the same in every lane, like n
    uint64_t n = 0;
    while( i >= a_begin && j >= b_begin ) {
        // word (y, x): rows 4 (i4 - y) .. + 3 of columns 4 (j4 - x) .. + 3, at [y][x - y + SIDE]
        const int32_t i4 = i / 4, j4 = j / 4;
        uint32_t v[LOADS];
#pragma unroll
        for( int k = 0; k < LOADS; k++ ) {
            const int t = lane + 32 * k;
            const int32_t y = t / TB_WALK_WIDTH, x = y + t % TB_WALK_WIDTH - TB_WALK_SIDE;
            const int32_t row = 4 * (i4 - y), blk = j4 - x;
            v[k] = 0;
            if( t < WORDS && row >= 0 && x >= 0 && blk >= 0 ) {
                const int32_t owner = (row % ROWS) / R;        // the rows' lane, at step blk + owner
                const uint32_t * w = dir + (uint64_t) (row / ROWS) * stripe_words + (uint64_t) (blk + owner) * 32 + owner;
                v[k] = R == 4 ? w[0] : w[0] << 4 | w[33];       // two rows: the next lane has the others a step later
            }
        }
        __syncwarp();
#pragma unroll
        for( int k = 0; k < LOADS; k++ )
            if( lane + 32 * k < WORDS )
                band[lane + 32 * k] = v[k];
        __syncwarp();
        // the move at a cell (2, 3: I; 1: D; 0: M), or 4: not in the band or past the begin cell
        auto move = [&]( int32_t r, int32_t c ) -> uint32_t {
            if( r < a_begin || c < b_begin )
                return 4u;
            const int32_t y = i4 - r / 4, d = j4 - c / 4 - y + TB_WALK_SIDE;
            if( y >= TB_WALK_ROWS || d < 0 || d >= TB_WALK_WIDTH )
                return 4u;
            return (band[y * TB_WALK_WIDTH + d] >> (8 * (c % 4) + 6 - 2 * (r % 4))) & 3u;
        };
        // `all`: which lanes' cells continue the run from lane 0's
        auto run = [&]( unsigned all, char ch ) -> int32_t {
            const int32_t len = all == 0xffffffffu ? 32 : __ffs( (int) ~all ) - 1;
            if( lane < len && n + (uint64_t) lane < cap )
                out[n + lane] = ch;
            n += (uint64_t) len;
            return len;
        };
        for( ;; ) {
            const uint32_t m = move( i - lane, j - lane );
            const int32_t diagonal = run( __ballot_sync( 0xffffffffu, m == 0u ), 'M' );
            i -= diagonal;
            j -= diagonal;
            if( diagonal == 32 )
                continue;
            const uint32_t op = __shfl_sync( 0xffffffffu, m, diagonal );
            if( op == 4u )
                break;                           // the end, or the next band
            if( op & 2u )
                j -= run( __ballot_sync( 0xffffffffu, (move( i, j - lane ) & 6u) == 2u ), 'I' );
            else
                i -= run( __ballot_sync( 0xffffffffu, move( i - lane, j ) == 1u ), 'D' );
        }
    }
    if( lane == 0 )
        p.ops_len[h] = (uint32_t) n;
}

cudaError_t launch_tb_walk( const TbParams & p, cudaStream_t st ) {
    if( p.n_hits )
        (p.rows_per_lane == 2 ? tb_walk_kernel<2> : tb_walk_kernel<4>)<<<p.n_hits, 32, 0, st>>>( p );
    return cudaGetLastError();
}

template <int PHASE, int R, bool P8>
static cudaError_t launch_stripes( const TbParams & p, int sms, cudaStream_t st ) {
    static LaunchShape shape;
    const cudaError_t e = shape.set( tb_stripes_kernel<PHASE, R, P8>, TB_THREADS, 0 );
    if( e != cudaSuccess )
        return e;
    const uint32_t want = (p.n_tickets + TB_WARPS - 1) / TB_WARPS;
    const uint32_t grid = min( want, (uint32_t) (sms * min( TB_BLOCKS, max( 1, shape.blocks ) )) );
    if( grid )
        tb_stripes_kernel<PHASE, R, P8><<<grid, TB_THREADS, 0, st>>>( p );
    return cudaGetLastError();
}

template <int PHASE>
static cudaError_t launch_phase( const TbParams & p, bool p8, int sms, cudaStream_t st ) {
    if constexpr( PHASE == TB_FWDDIR || PHASE == TB_REVERSE )
        if( p8 && p.rows_per_lane == 2 )
            return launch_stripes<PHASE, 2, true>( p, sms, st );
    return p8 ? launch_stripes<PHASE, 4, true>( p, sms, st ) : launch_stripes<PHASE, 4, false>( p, sms, st );
}

cudaError_t launch_tb_forward( const TbParams & p, bool p8, int sms, cudaStream_t st ) {
    return launch_phase<TB_FORWARD>( p, p8, sms, st );
}

cudaError_t launch_tb_reverse( const TbParams & p, bool p8, int sms, cudaStream_t st ) {
    return launch_phase<TB_REVERSE>( p, p8, sms, st );
}

cudaError_t launch_tb_directions( const TbParams & p, bool nw, bool p8, int sms, cudaStream_t st ) {
    return nw ? launch_phase<TB_NW_DIRECTIONS>( p, p8, sms, st ) : launch_phase<TB_DIRECTIONS>( p, p8, sms, st );
}

cudaError_t launch_tb_fwddir( const TbParams & p, bool p8, int sms, cudaStream_t st ) {
    return launch_phase<TB_FWDDIR>( p, p8, sms, st );
}

cudaError_t launch_tb_scores( const TbParams & p, bool nw, bool p8, int sms, cudaStream_t st ) {
    return nw ? launch_phase<TB_NW_SCORE>( p, p8, sms, st ) : launch_phase<TB_SCORE>( p, p8, sms, st );
}

}  // namespace ssa
