// sw_stream_kernel.cu -- scores of chosen (query, sequence) pairs, two sequences
// of one query per register, on streamed stripes.
//
// For the pairs that would outlast everything else in a call.  The kernels of
// the entry pass give a sequence to 4 to 32 threads, which pass over it once
// per 80 to 500 query rows, one pass after the other: (a) the longest sequences
// of a database against long queries, in a call without enough other work to
// hide them; (b) the pairs that the 8-bit entry re-queued (255 and more), a few
// per query, often the longest of both.  Here lane k of a warp owns R rows of a
// stripe of 32 x R rows, and the stripes of a pair follow one another on as many
// warps as the pair has stripes (stream_stripes.cuh).
//
// Arithmetic and range are those of sw_fast4_kernel (exact 16x2 scores with a
// bias of 1024; a sequence whose running maximum reaches the limit goes to
// sink.redo, for the lane emulation): one 4-column block per step, four
// skewed dependency chains, 5.5 ALU instructions and one IADD per cell pair.
// Bound by the ALU pipe when many pairs are re-queued (78 % of its cycles; what
// is left is padding of the last stripe and 20 instructions a step besides the
// cells), by the latency of one warp's steps (blocks + STREAM_LAG x stripes) when few
// are.  The host picks R (4 to 6) and the CTAs per SM (2 to 4) for each launch.
// Measured on a B200 against the lane emulation (one warp per pair, int32): 102
// pairs of 375 rows x 380 columns 0.50 -> 0.12 ms; 1,927 of 300 x 21,000 38.7 ->
// 3.9 ms; 2,014 of 30-1,803 x 21,000 94 -> 7.1 ms.
#include "device_common.cuh"
#include "stream_stripes.cuh"

namespace ssa {

constexpr uint32_t STREAM_BIAS = 1024u;
constexpr uint32_t STREAM_BIAS2 = (STREAM_BIAS << 16) | STREAM_BIAS;
constexpr int STREAM_THREADS = 128;
constexpr int STREAM_WARPS = STREAM_THREADS / 32;
constexpr int STREAM_BLOCKS = 4;                     // most CTAs per SM
constexpr uint32_t STREAM_PAD = FAST_PAD_CODE * 0x01010101u;   // past a sequence's last block: scores -128

// byte j of a and of b, sign-extended to 16 bits each
template <int J>
__device__ __forceinline__ uint32_t pair_score( uint32_t a, uint32_t b ) {
    constexpr uint32_t sel = (uint32_t) J | ((uint32_t) (J | 8) << 4) | ((uint32_t) (4 + J) << 8) |
            ((uint32_t) (12 + J) << 12);
    uint32_t d;
    asm( "prmt.b32 %0, %1, %2, %3;" : "=r"( d ) : "r"( a ), "r"( b ), "n"( sel ) );
    return d;
}

// BLOCKS: also find the first 4-column block in which each sequence reaches the
// limit (the 8-bit entry: the lane's overflow block), and end a pair when both
// of its sequences have.
template <bool BLOCKS>
struct CrossLimit {
    static constexpr bool NONE = !BLOCKS;
    const int32_t * p;
    bool two;
    __device__ int32_t operator()() const {
        const volatile int32_t * c = p;
        return two ? max( c[0], c[1] ) : c[0];
    }
};

// NW: Needleman-Wunsch as in nw_qpair4_kernel (exact unsigned 16x2 values with a
// bias of 32768, for sequences up to the host's length limit; the score is H of
// the query's last row in the sequence's last column).
constexpr uint32_t STREAM_NW_BIAS = 32768u;

__device__ __forceinline__ uint32_t stream_nw_pack( int32_t v ) {
    return ((uint32_t) (v + (int32_t) STREAM_NW_BIAS) & 0xffffu) * 0x10001u;
}

template <int R, bool BLOCKS, bool NW>
__global__ void __launch_bounds__( STREAM_THREADS, STREAM_BLOCKS ) sw_stream_kernel( SwStreamParams p ) {
    constexpr int C = 4;
    constexpr int WORDS = (R + 3) / 4;
    constexpr int ROWS = 32 * R;
    __shared__ StreamStage stages[STREAM_WARPS];
    __shared__ uint2 rings[STREAM_WARPS][64];
    __shared__ __align__( 16 ) uint32_t tables[STREAM_WARPS][32 * 32 * WORDS];
    __shared__ int8_t smat[1024];
    const int lane = threadIdx.x & 31;
    const int warp = threadIdx.x >> 5;
    for( int i = threadIdx.x; i < 1024; i += STREAM_THREADS )
        smat[i] = (int8_t) p.matrix[i];              // [database code][query code]
    __syncthreads();
    StreamStage & st = stages[warp];
    uint32_t * table = tables[warp] + lane * WORDS;  // the lane's scores of code d at [d * 32 * WORDS]
    const uint32_t GOE32 = (uint32_t) (p.gap_oe * 65536 + p.gap_oe);
    const uint32_t GE2 = ((uint32_t) (uint16_t) (int16_t) p.gap_e << 16) | (uint16_t) (int16_t) p.gap_e;
    // sets bit 15 of a half exactly when the half is >= STREAM_BIAS + limit
    const int gO = p.gap_open, gE = p.gap_e;
    const uint32_t CROSS_ADD = (0x8000u - (STREAM_BIAS + (uint32_t) p.limit)) * 0x10001u;

    uint64_t loaded_key = ~0ull;
    for( ;; ) {
        const uint32_t ticket = next_ticket( p.counter, lane );
        if( ticket >= p.n_tickets )
            break;
        const uint32_t stripe = ticket_stripe( p.cum, p.levels, ticket );
        const uint32_t it = ticket - p.cum[stripe];
        const uint32_t pred = stripe ? p.cum[stripe - 1] + it : 0u;
        const SwStreamItem item = p.items[it];
        const uint32_t Q = p.qlen[item.slot];
        const uint8_t * q = p.qcodes + p.qoff[item.slot];
        const bool two = item.id_b != 0xffffffffu;
        const uint32_t nba = (p.db.lens[item.id_a] + 3u) >> 2;              // 4-column blocks
        const uint32_t nbb = two ? (p.db.lens[item.id_b] + 3u) >> 2 : 0u;
        const uint32_t * ra = reinterpret_cast<const uint32_t *>( p.db.codes + p.db.offsets[item.id_a] );
        const uint32_t * rb = two ? reinterpret_cast<const uint32_t *>( p.db.codes + p.db.offsets[item.id_b] ) : ra;

        StreamStripe sp;
        sp.cols = max( nba, nbb );
        sp.row = p.boundary + p.bnd_off[it];
        sp.above = stripe ? p.progress + pred : nullptr;
        sp.mine = p.progress + ticket;
        sp.last = (stripe + 1u) * (uint32_t) ROWS >= Q;
        sp.error_flags = p.sink.error_flags;

        // the lane's rows: int8 scores of every code; past the query and for the
        // pad code -128 (never raises a maximum), or 0 (Needleman-Wunsch: never
        // reaches the score, and keeps every value in range)
        constexpr int PAST = NW ? 0 : -128;
        const int32_t row0 = (int32_t) (stripe * (uint32_t) ROWS) + lane * R;
        const uint64_t key = ((uint64_t) item.slot << 32) | stripe;
        if( key != loaded_key ) {                   // the same for the next ticket of this stripe of the query
            loaded_key = key;
            int code[R];
#pragma unroll
            for( int r = 0; r < R; r++ )
                code[r] = row0 + r < (int32_t) Q ? q[row0 + r] : -1;
            for( int d = 0; d < 32; d++ ) {
#pragma unroll
                for( int w = 0; w < WORDS; w++ ) {
                    uint32_t v = 0;
#pragma unroll
                    for( int b = 0; b < 4; b++ ) {
                        const int c = 4 * w + b < R ? code[4 * w + b < R ? 4 * w + b : 0] : -1;
                        const int m = (c >= 0 && d != (int) FAST_PAD_CODE) ? smat[(d << 5) + c] : PAST;
                        v |= ((uint32_t) m & 0xffu) << (8 * b);
                    }
                    table[d * 32 * WORDS + w] = v;
                }
            }
        }
        uint32_t H[R], E[R];
#pragma unroll
        for( int r = 0; r < R; r++ ) {
            // the reference's column before the first: H(i, -1), E(i, -1)
            H[r] = NW ? stream_nw_pack( gO + (row0 + r + 1) * gE ) : STREAM_BIAS2;
            E[r] = NW ? stream_nw_pack( 2 * gO + (row0 + r + 2) * gE ) : STREAM_BIAS2;
        }
        uint32_t diag = NW ? stream_nw_pack( row0 ? gO + row0 * gE : 0 ) : STREAM_BIAS2, smax = STREAM_BIAS2, seen = 0;
        // Needleman-Wunsch: the lane of the query's last row, where it is in the
        // lane, and the last column of each sequence
        const int q_last = (int) Q - 1 - row0;
        const bool owner = NW && sp.last && q_last >= 0 && q_last < R;
        const int32_t la = (int32_t) p.db.lens[item.id_a] - 1, lb = two ? (int32_t) p.db.lens[item.id_b] - 1 : -1;
        uint32_t cap_a = 0, cap_b = 0;
        int32_t * cross = BLOCKS ? p.cross + 2 * it : nullptr;
        uint32_t out_h[C], out_f[C];
#pragma unroll
        for( int j = 0; j < C; j++ ) {
            out_h[j] = STREAM_BIAS2;
            out_f[j] = STREAM_BIAS2;
        }
        // the blocks' residues, read a step ahead
        auto fetch = [&]( const uint32_t * res, uint32_t nb, int32_t b ) -> uint32_t {
            return (b >= 0 && (uint32_t) b < nb) ? __ldg( res + b ) : STREAM_PAD;
        };
        auto fetch2 = [&]( int32_t b ) -> uint2 { return make_uint2( fetch( ra, nba, b ), fetch( rb, nbb, b ) ); };
        StreamResidues<uint2> residues{ rings[warp], {} };
        residues.start( lane, fetch2 );
        uint2 next = residues.at( -lane );

        auto column = [&]( const uint32_t s, const bool edge, const uint32_t cols ) {
            uint32_t up_h[C], up_f[C];
#pragma unroll
            for( int j = 0; j < C; j++ ) {
                up_h[j] = __shfl_up_sync( 0xffffffffu, out_h[j], 1 );
                up_f[j] = __shfl_up_sync( 0xffffffffu, out_f[j], 1 );
            }
            const int32_t b = (int32_t) s - lane;
            const uint32_t wa = next.x, wb = next.y;
            next = residues.at( b + 1 );
            if( edge && (b < 0 || b >= (int32_t) cols) )
                return;
            if( lane == 0 ) {
                const int4 x = st.in[2 * (s % STREAM_CHUNK)], y = st.in[2 * (s % STREAM_CHUNK) + 1];
                up_h[0] = (uint32_t) x.x;
                up_f[0] = (uint32_t) x.y;
                up_h[1] = (uint32_t) x.z;
                up_f[1] = (uint32_t) x.w;
                up_h[2] = (uint32_t) y.x;
                up_f[2] = (uint32_t) y.y;
                up_h[3] = (uint32_t) y.z;
                up_f[3] = (uint32_t) y.w;
            }
            uint32_t pa[C][WORDS], pb[C][WORDS], f[C];
#pragma unroll
            for( int j = 0; j < C; j++ ) {
                const uint32_t * ta = table + ((wa >> (8 * j)) & 0xffu) * (32 * WORDS);
                const uint32_t * tb = table + ((wb >> (8 * j)) & 0xffu) * (32 * WORDS);
#pragma unroll
                for( int w = 0; w < WORDS; w++ ) {
                    pa[j][w] = ta[w];
                    pb[j][w] = tb[w];
                }
                f[j] = up_f[j];
            }
            // chain j computes column j of the block, cell (it - j, j) in
            // iteration `it` (as in sw_fast4_kernel)
            uint32_t hv[C][R];
#pragma unroll
            for( int it2 = 0; it2 < R + C - 1; it2++ ) {
#pragma unroll
                for( int j = 0; j < C; j++ ) {
                    const int r = it2 - j;
                    if( r < 0 || r >= R )
                        continue;
                    const uint32_t x = pa[j][r / 4], y = pb[j][r / 4];
                    const uint32_t v = (r & 3) == 0 ? pair_score<0>( x, y ) : (r & 3) == 1 ? pair_score<1>( x, y )
                            : (r & 3) == 2 ? pair_score<2>( x, y ) : pair_score<3>( x, y );
                    const uint32_t hd = r == 0 ? (j == 0 ? diag : up_h[j - 1]) : (j == 0 ? H[r - 1] : hv[j - 1][r - 1]);
                    uint32_t h;
                    if constexpr( NW ) {
                        h = __viaddmax_u16x2( hd, v, __vmaxu2( E[r], f[j] ) );
                        const uint32_t hg = h + GOE32;                  // one carry out of the low half
                        f[j] = __viaddmax_u16x2( f[j], GE2, hg );
                        E[r] = __viaddmax_u16x2( E[r], GE2, hg );
                    }
                    else {
                        const uint32_t t = __vimax3_s16x2( E[r], f[j], STREAM_BIAS2 );
                        h = __viaddmax_s16x2( hd, v, t );
                        const uint32_t hg = h + GOE32;                  // no borrow: h >= bias
                        f[j] = __viaddmax_s16x2( f[j], GE2, hg );
                        E[r] = __viaddmax_s16x2( E[r], GE2, hg );
                    }
                    hv[j][r] = h;
                    if( !NW && (j & 1) )
                        smax = __vimax3_s16x2( smax, hv[j - 1][r], h );
                    if( j == C - 1 )
                        H[r] = h;
                }
            }
            diag = up_h[C - 1];
#pragma unroll
            for( int j = 0; j < C; j++ ) {
                out_h[j] = hv[j][R - 1];
                out_f[j] = f[j];
            }
            if constexpr( NW ) {
                if( owner && (b == la >> 2 || b == lb >> 2) ) {
#pragma unroll
                    for( int j = 0; j < C; j++ )
#pragma unroll
                        for( int r = 0; r < R; r++ ) {
                            if( r == q_last && 4 * b + j == la )
                                cap_a = hv[j][r];
                            if( r == q_last && 4 * b + j == lb )
                                cap_b = hv[j][r];
                        }
                }
            }
            if constexpr( BLOCKS ) {
                // first block in which this lane's maximum reached the limit
                const uint32_t ge = (smax + CROSS_ADD) & 0x80008000u;
                if( ge != seen ) {
                    if( (ge ^ seen) & 0x8000u )
                        atomicMin( cross, b );
                    if( (ge ^ seen) & 0x80000000u )
                        atomicMin( cross + 1, b );
                    __threadfence();
                    seen = ge;
                }
            }
            if( lane == 31 ) {
                st.out[2 * (s % STREAM_CHUNK)] = make_int4( (int) out_h[0], (int) out_f[0], (int) out_h[1], (int) out_f[1] );
                st.out[2 * (s % STREAM_CHUNK) + 1] = make_int4( (int) out_h[2], (int) out_f[2], (int) out_h[3], (int) out_f[3] );
            }
        };
        // the row above the first stripe, columns c and c + 1: H(-1, c) and F entering row 0
        auto top = [&]( int32_t c ) -> int4 {
            if constexpr( NW )
                return make_int4( (int) stream_nw_pack( gO + (c + 1) * gE ), (int) stream_nw_pack( 2 * gO + (c + 2) * gE ),
                        (int) stream_nw_pack( gO + (c + 2) * gE ), (int) stream_nw_pack( 2 * gO + (c + 3) * gE ) );
            else
                return make_int4( (int) STREAM_BIAS2, (int) STREAM_BIAS2, (int) STREAM_BIAS2, (int) STREAM_BIAS2 );
        };
        auto refill = [&]( uint32_t s0 ) {
            if( stripe == 0 && lane < (int) (2 * STREAM_CHUNK) )
                st.in[lane] = top( 4 * (int32_t) s0 + 2 * lane );
            residues.refill( s0, lane, fetch2 );
        };
        const CrossLimit<BLOCKS> limit{ cross, two };
        const uint32_t swept = stream_columns( sp, st, lane, limit, refill, column );
        if constexpr( NW ) {
            if( owner ) {
                const uint64_t row = (uint64_t) item.slot * p.sink.score_stride;
                if( pair_wanted( p.sink, p.marked_only, item.slot, item.id_a ) )
                    p.sink.score[row + item.id_a] = (int32_t) (cap_a & 0xffffu) - (int32_t) STREAM_NW_BIAS;
                if( two && pair_wanted( p.sink, p.marked_only, item.slot, item.id_b ) )
                    p.sink.score[row + item.id_b] = (int32_t) (cap_b >> 16) - (int32_t) STREAM_NW_BIAS;
            }
            stream_end( sp, swept, lane );
            continue;
        }
        // the pair's maximum goes down the stripes; a half that reached the
        // limit anywhere holds a value at or above it
#pragma unroll
        for( int o = 16; o > 0; o >>= 1 )
            smax = __vmaxs2( smax, __shfl_xor_sync( 0xffffffffu, smax, o ) );
        __syncwarp();
        if( sp.above ) {
            stream_wait( sp.above, STREAM_DONE, lane, sp.error_flags );
            smax = __vmaxs2( smax, __ldcg( p.result + pred ) );
        }
        if( lane == 0 ) {
            if( !sp.last ) {
                __stcg( p.result + ticket, smax );
            }
            else {
                const uint32_t ids[2] = { item.id_a, item.id_b };
                const uint32_t crossed = smax + CROSS_ADD;
#pragma unroll
                for( int h = 0; h < 2; h++ ) {
                    if( h == 1 && !two )
                        continue;
                    if( (crossed >> (16 * h)) & 0x8000u )
                        report_crossing( p.sink, item.slot, ids[h],
                                BLOCKS ? *(volatile const int32_t *) (cross + h) + 1 : 0 );
                    else
                        p.sink.score[(uint64_t) item.slot * p.sink.score_stride + ids[h]] =
                                (int32_t) ((smax >> (16 * h)) & 0xffffu) - (int32_t) STREAM_BIAS;
                }
            }
        }
        stream_end( sp, swept, lane );
    }
}

template <int R, bool BLOCKS, bool NW>
static cudaError_t launch_stream( const SwStreamParams & p, int sms, cudaStream_t st ) {
    static LaunchShape shape;
    const cudaError_t e = shape.set( sw_stream_kernel<R, BLOCKS, NW>, STREAM_THREADS, 0 );
    if( e != cudaSuccess )
        return e;
    const uint32_t grid = min( (p.n_tickets + STREAM_WARPS - 1) / STREAM_WARPS,
            (uint32_t) (sms * max( 1, min( p.ctas_per_sm, shape.blocks ) )) );
    if( grid )
        sw_stream_kernel<R, BLOCKS, NW><<<grid, STREAM_THREADS, 0, st>>>( p );
    return cudaGetLastError();
}

template <bool BLOCKS>
static cudaError_t launch_rows( int R, const SwStreamParams & p, int sms, cudaStream_t st ) {
    switch( R ) {
        case 4: return launch_stream<4, BLOCKS, false>( p, sms, st );
        case 5: return launch_stream<5, BLOCKS, false>( p, sms, st );
        case 6: return launch_stream<6, BLOCKS, false>( p, sms, st );
        default: return cudaErrorInvalidValue;
    }
}

cudaError_t launch_sw_stream( int R, const SwStreamParams & p, int sms, cudaStream_t st ) {
    return p.cross ? launch_rows<true>( R, p, sms, st ) : launch_rows<false>( R, p, sms, st );
}

cudaError_t launch_nw_stream( const SwStreamParams & p, int sms, cudaStream_t st ) {
    return launch_stream<4, false, true>( p, sms, st );
}

}  // namespace ssa
