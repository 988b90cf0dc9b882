// stream_stripes.cuh -- one alignment on many warps of the whole GPU.
//
// A wavefront kernel cuts the query into stripes of 32 x R rows; a warp sweeps
// a stripe over the database columns (lane k on column s - k at step s), and
// the stripe's bottom row (H, F per column) is the next stripe's top row.
// Stripe i can follow stripe i - 1 at a distance of a few dozen columns, so the
// stripes of one alignment run at the same time on as many warps as there are,
// on any SM: the row travels through the alignment's boundary row in global
// memory (which stays in L2), and each stripe publishes, every 32 columns, how
// many columns of it are written.
//
//   * Work items ("tickets") are (stripe, alignment), handed out from a global
//     counter stripe by stripe: first stripe 0 of every alignment, then stripe
//     1 of every alignment that has one, and so on.  A warp finishes its ticket
//     before it takes another, and a ticket only waits for the ticket of the
//     stripe above, which has a smaller number: a running warp holds it or has
//     finished it, down to stripe 0, which waits for nothing.  So the launch
//     needs no co-residency of its blocks and cannot deadlock.  Stripe-major
//     order also keeps few stripes of many alignments in flight rather than all
//     of one, whose last ones would wait for the whole pipeline to fill.
//   * The boundary row is updated in place: stripe i reads column c before it
//     writes it (it writes 31 columns behind its own reads); stripe i + 1 reads
//     it after stripe i published it.
//   * A wait has an iteration limit, after which it sets ERR_PIPELINE, and every
//     other wait sees the flag and gives up too; the stripe below takes what
//     was published as the alignment's width, so all warps run to their end.
//   * A stripe may end early (the reverse region pass: columns past the first
//     begin-cell candidate cannot change the result).  Its final count says how
//     many columns it wrote, and the stripe below ends there as well.
#pragma once

#include "device_common.cuh"

namespace ssa {

constexpr uint32_t STREAM_DONE = 0x80000000u;         // progress word: the stripe has ended
constexpr uint32_t STREAM_WAIT_LIMIT = 1u << 24;      // polls of 100 ns and more each

// Shared memory of one warp: the rows entering and leaving the stripe in the
// current chunk of steps, one word per lane.  A column of a row is 32 / CHUNK
// words: CHUNK = 32 with int2 words (H and F of one column), CHUNK = 16 with
// int4 words (two per block of four columns).
template <class Word>
struct StreamStage {
    Word in[32], out[32];
};

__device__ __forceinline__ uint32_t load_acquire( const uint32_t * p ) {
    uint32_t v;
    asm volatile( "ld.acquire.gpu.global.u32 %0, [%1];" : "=r"( v ) : "l"( p ) : "memory" );
    return v;
}

__device__ __forceinline__ void store_release( uint32_t * p, uint32_t v ) {
    asm volatile( "st.release.gpu.global.u32 [%0], %1;" ::"l"( p ), "r"( v ) : "memory" );
}

// Lane 0 polls until `need` columns are written or the stripe has ended; every
// lane gets the progress word, and reads what it covers afterwards.
__device__ __forceinline__ uint32_t stream_wait( const uint32_t * progress, uint32_t need, int lane,
        unsigned * error_flags ) {
    uint32_t v = 0;
    if( lane == 0 ) {
        for( uint32_t n = 1;; n++ ) {
            v = load_acquire( progress );
            if( (v & STREAM_DONE) || v >= need )
                break;
            __nanosleep( 100 );
            if( n >= STREAM_WAIT_LIMIT ||
                    ((n & 1023u) == 0 && (*(volatile unsigned *) error_flags & ERR_PIPELINE)) ) {
                atomicOr( error_flags, ERR_PIPELINE );
                v |= STREAM_DONE;
                break;
            }
        }
    }
    v = __shfl_sync( 0xffffffffu, v, 0 );
    __syncwarp();
    return v;
}

// One stripe's place among the alignment's.  "Columns" are whatever one
// wavefront step advances by (the 16x2 kernels: blocks of four columns).
template <class Word>
struct StreamStripe {
    uint32_t cols;                 // database columns
    Word * row;                    // the alignment's boundary row
    const uint32_t * above;        // progress of the stripe above, nullptr: the first stripe
    uint32_t * mine;               // this stripe's progress
    bool last;                     // no stripe below
    unsigned * error_flags;
};

// The database residues of a stripe on their way through the warp: lane k needs
// word s - k at step s.  The warp loads 16 words at a time, a chunk of steps
// ahead, into 64 words of shared memory, and every lane reads its word from
// there.  (Loads by each lane from global memory, two steps ahead, miss the L1
// cache most of the time: every acquire of a progress word on the SM empties it.)
template <class T>
struct StreamResidues {
    T * ring;                      // 64 words, the warp's
    T next;                        // lanes 0 .. 15: the words of the next refill

    // fetch( b ): word b, any value outside the sequence
    template <class Fetch>
    __device__ __forceinline__ void start( int lane, const Fetch & fetch ) {
        __syncwarp();                                   // the last ticket's readers
        ring[lane] = fetch( lane );
        ring[32 + lane] = fetch( lane - 32 );
        next = fetch( 32 + lane );
        __syncwarp();
    }
    // before the steps s0 .. s0 + 15: afterwards words s0 - 32 .. s0 + 31 are there
    template <class Fetch>
    __device__ __forceinline__ void refill( uint32_t s0, int lane, const Fetch & fetch ) {
        if( s0 == 0 )
            return;
        __syncwarp();
        if( lane < 16 ) {
            ring[(s0 + 16u + (uint32_t) lane) & 63u] = next;
            next = fetch( (int32_t) s0 + 32 + lane );
        }
        __syncwarp();
    }
    __device__ __forceinline__ T at( int32_t b ) const { return ring[b & 63]; }
};

__device__ __forceinline__ int2 zero_word( const int2 * ) { return make_int2( 0, 0 ); }
__device__ __forceinline__ int4 zero_word( const int4 * ) { return make_int4( 0, 0, 0, 0 ); }

// No column limit.
struct StreamAll {
    static constexpr bool NONE = true;
    __device__ int32_t operator()() const { return 0; }
};

// Sweeps one stripe.  limit() reads the last column worth computing, which may
// shrink while the stripes run (lane 0's value counts).  refill( s0 ) runs before the steps s0 .. s0 + CHUNK - 1,
// column( s, edge, cols ) computes wavefront step s: edge says that some lane
// may be on a column outside 0 .. cols - 1, or on the last one.  Lane 0 finds
// the row above column s in st.in (word s % CHUNK, or the words from there),
// lane 31 leaves the row below column s - 31 in the same place of st.out.
// Returns the columns swept; the caller publishes the end with stream_end().
template <int CHUNK, class Word, class Limit, class Refill, class Column>
__device__ __forceinline__ uint32_t stream_columns( const StreamStripe<Word> & sp, StreamStage<Word> & st, int lane,
        const Limit & limit, Refill && refill, Column && column ) {
    constexpr uint32_t WPC = 32 / CHUNK;       // words per column
    uint32_t cols = sp.cols;
    uint32_t avail = 0;            // columns of the row above known to be written
    bool have = false;             // pf holds the next chunk of it
    Word pf = zero_word( (const Word *) nullptr );
    int32_t last = 0;              // the limit as it was a chunk ago, so that its load is not waited for
    if constexpr( !Limit::NONE )
        last = limit();
    for( uint32_t s0 = 0;; s0 += CHUNK ) {
        if constexpr( !Limit::NONE ) {
            cols = min( cols, (uint32_t) __shfl_sync( 0xffffffffu, last, 0 ) + 1u );
            last = limit();
        }
        if( sp.above && s0 < cols ) {
            if( !have ) {
                const uint32_t need = min( s0 + (uint32_t) CHUNK, cols );
                if( avail < need ) {
                    const uint32_t v = stream_wait( sp.above, need, lane, sp.error_flags );
                    avail = v & ~STREAM_DONE;
                    if( avail < need )             // the stripe above has ended there
                        cols = min( cols, avail );
                }
                if( s0 * WPC + (uint32_t) lane < cols * WPC )
                    pf = __ldcg( sp.row + (uint64_t) s0 * WPC + lane );
            }
            __syncwarp();
            st.in[lane] = pf;
            __syncwarp();
            // the next chunk now if it is there, so that its load is not on
            // the critical path; else after a wait at the next turn
            have = false;
            const uint32_t s2 = s0 + (uint32_t) CHUNK;
            if( s2 < cols ) {
                const uint32_t need = min( s2 + (uint32_t) CHUNK, cols );
                if( avail < need ) {
                    uint32_t v = 0;
                    if( lane == 0 )
                        v = load_acquire( sp.above );
                    v = __shfl_sync( 0xffffffffu, v, 0 );
                    __syncwarp();
                    avail = max( avail, v & ~STREAM_DONE );
                }
                if( avail >= need ) {
                    if( s2 * WPC + (uint32_t) lane < cols * WPC )
                        pf = __ldcg( sp.row + (uint64_t) s2 * WPC + lane );
                    have = true;
                }
            }
        }
        const uint32_t steps = cols + 31u;
        if( cols == 0 || s0 >= steps )
            break;
        refill( s0 );
        const uint32_t s1 = min( s0 + (uint32_t) CHUNK, steps );
        if( s0 >= 31u && s1 < cols ) {
            for( uint32_t s = s0; s < s1; s++ )
                column( s, false, cols );
        }
        else {
            for( uint32_t s = s0; s < s1; s++ )
                column( s, true, cols );
        }
        if( !sp.last ) {
            __syncwarp();
            const int32_t c = (int32_t) s0 - 31 + lane / (int) WPC;
            if( c >= 0 && c < (int32_t) s1 - 31 )
                __stcg( sp.row + (uint64_t) c * WPC + lane % WPC, st.out[lane] );
            __syncwarp();
            if( lane == 0 && s1 > 31u )
                store_release( sp.mine, s1 - 31u );
        }
        if( s1 == steps )
            break;
    }
    return cols;
}

// The stripe has ended after `cols` columns; whatever the warp wrote before is
// visible to a warp that sees this.
template <class Word>
__device__ __forceinline__ void stream_end( const StreamStripe<Word> & sp, uint32_t cols, int lane ) {
    __syncwarp();
    if( lane == 0 && !sp.last )
        store_release( sp.mine, STREAM_DONE | cols );
}

// Tickets are handed out one per warp from a global counter.
__device__ __forceinline__ uint32_t next_ticket( unsigned long long * counter, int lane ) {
    unsigned long long v = 0;
    if( lane == 0 )
        v = atomicAdd( counter, 1ull );
    return (uint32_t) __shfl_sync( 0xffffffffu, v, 0 );
}

// The ticket's stripe and alignment: cum[i] is the first ticket of stripe i,
// cum[levels] the number of tickets.
__device__ __forceinline__ uint32_t ticket_stripe( const uint32_t * cum, uint32_t levels, uint32_t ticket ) {
    uint32_t lo = 0, hi = levels;              // cum[lo] <= ticket < cum[hi]
    while( hi - lo > 1 ) {
        const uint32_t mid = (lo + hi) / 2;
        if( cum[mid] <= ticket )
            lo = mid;
        else
            hi = mid;
    }
    return lo;
}

}  // namespace ssa
