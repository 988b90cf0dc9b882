// stream_stripes.cuh -- one alignment on many warps of the whole GPU.
//
// A wavefront kernel cuts the query into stripes of 32 x R rows; a warp sweeps
// a stripe over the database columns (lane k on column s - k at step s), and
// the stripe's bottom row (H, F per column) is the next stripe's top row.
// Stripe i can follow stripe i - 1 at a distance of a few dozen columns, so the
// stripes of one alignment run at the same time on as many warps as there are,
// on any SM: the row travels through the alignment's boundary row in global
// memory (which stays in L2), and each stripe publishes, every 16 steps, how
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

// Wavefront steps between two publications: 8 shorten the way from stripe to
// stripe but cost a fence every 8 steps (10 hits of 300 x 33,000: 3.8 ms against
// 4.2, 48 long pairs 20.2 against 21.1).
constexpr uint32_t STREAM_CHUNK = 16;
// Steps from a stripe to the next at the same speed: a chunk starts when the chunk
// above that holds its last block, 31 steps further on, has ended.
constexpr uint32_t STREAM_LAG = 48;
constexpr uint32_t STREAM_DONE = 0x80000000u;         // progress word: the stripe has ended
constexpr uint32_t STREAM_WAIT_LIMIT = 1u << 24;      // polls of 100 ns and more each

// Shared memory of one warp: the rows entering and leaving the stripe in the
// current chunk of 16 steps.
struct StreamStage {
    int4 in[2 * STREAM_CHUNK], out[2 * STREAM_CHUNK];
};

__device__ __forceinline__ uint32_t load_acquire( const uint32_t * p ) {
    uint32_t v;
    asm volatile( "ld.acquire.gpu.global.u32 %0, [%1];" : "=r"( v ) : "l"( p ) : "memory" );
    return v;
}

__device__ __forceinline__ void store_release( uint32_t * p, uint32_t v ) {
    asm volatile( "st.release.gpu.global.u32 [%0], %1;" ::"l"( p ), "r"( v ) : "memory" );
}

__device__ __forceinline__ uint32_t load_relaxed( const uint32_t * p ) {
    uint32_t v;
    asm volatile( "ld.relaxed.gpu.global.u32 %0, [%1];" : "=r"( v ) : "l"( p ) : "memory" );
    return v;
}

__device__ __forceinline__ void store_relaxed( uint32_t * p, uint32_t v ) {
    asm volatile( "st.relaxed.gpu.global.u32 [%0], %1;" ::"l"( p ), "r"( v ) : "memory" );
}

__device__ __forceinline__ void fence_acq_rel() { asm volatile( "fence.acq_rel.gpu;" ::: "memory" ); }

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
    // before the steps s0 .. s0 + 15, between two __syncwarp(): afterwards words
    // s0 - 32 .. s0 + 31 are there
    template <class Fetch>
    __device__ __forceinline__ void refill( uint32_t s0, int lane, const Fetch & fetch ) {
        if( s0 && lane < (int) STREAM_CHUNK ) {
            ring[(s0 + 32u - STREAM_CHUNK + (uint32_t) lane) & 63u] = next;
            next = fetch( (int32_t) s0 + 32 + lane );
        }
    }
    __device__ __forceinline__ T at( int32_t b ) const { return ring[b & 63]; }
};

// One stripe's place among the alignment's.  One step advances the wavefront by
// a block of four columns; a block of a boundary row is two words (H and F of
// two columns each).
struct StreamStripe {
    uint32_t cols;                 // blocks of database columns
    int4 * row;                    // the alignment's boundary row
    const uint32_t * above;        // progress of the stripe above, nullptr: the first stripe
    uint32_t * mine;               // this stripe's progress
    bool last;                     // no stripe below
    unsigned * error_flags;
};

// Sweeps one stripe, 16 steps (a chunk) at a time.  limit() reads the last block
// worth computing, which may shrink while the stripes run (lane 0's value
// counts).  refill( s0 ) runs before the steps s0 .. s0 + 15; the first
// stripe's leaves the alignment's top row in st.in.  block( s, edge, cols )
// computes wavefront step s: edge says that some lane may be on a block outside
// 0 .. cols - 1, or on the last one.  Lane 0 finds the row above block s in st.in
// (words 2 (s % 16) and the next), lane 31 leaves the row below block s - 31 in
// the same place of st.out.  Returns the blocks swept; the caller publishes the
// end with stream_end().
//
// The progress of the stripe above is read in the course of a chunk and counts
// from the chunk's end: the fence that publishes this stripe's row also orders
// that read before the loads of the row it covers.  An acquire of its own at
// every chunk is a round trip to L2 that nothing hides where a warp is alone
// on its sub-partition, and little where it is not.
template <class Limit, class Refill, class Block>
__device__ __forceinline__ uint32_t stream_columns( const StreamStripe & sp, StreamStage & st, int lane,
        const Limit & limit, Refill && refill, Block && block ) {
    constexpr uint32_t CHUNK = STREAM_CHUNK, POLL = STREAM_CHUNK - 5;
    uint32_t cols = sp.cols;
    uint32_t avail = 0;            // blocks of the row above known to be written
    bool have = false;             // pf holds the next chunk of it
    int4 pf = make_int4( 0, 0, 0, 0 );
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
                const uint32_t need = min( s0 + CHUNK, cols );
                if( avail < need ) {
                    const uint32_t v = stream_wait( sp.above, need, lane, sp.error_flags );
                    avail = v & ~STREAM_DONE;
                    if( avail < need )             // the stripe above has ended there
                        cols = min( cols, avail );
                }
                if( lane < (int) (2 * CHUNK) && s0 * 2 + (uint32_t) lane < cols * 2 )
                    pf = __ldcg( sp.row + (uint64_t) s0 * 2 + lane );
            }
            __syncwarp();
            if( lane < (int) (2 * CHUNK) )
                st.in[lane] = pf;
            // the next chunk now if it is there, so that its load is not on
            // the critical path; else after a wait at the next turn
            const uint32_t s2 = s0 + CHUNK;
            have = s2 < cols && avail >= min( s2 + CHUNK, cols );
            if( have && lane < (int) (2 * CHUNK) && s2 * 2 + (uint32_t) lane < cols * 2 )
                pf = __ldcg( sp.row + (uint64_t) s2 * 2 + lane );
        }
        const uint32_t steps = cols + 31u;
        if( cols == 0 || s0 >= steps )
            break;
        __syncwarp();
        refill( s0 );
        __syncwarp();
        const uint32_t s1 = min( s0 + CHUNK, steps );
        const bool poll = sp.above && avail < cols;
        uint32_t seen = 0;
        uint32_t s = s0;
        for( uint32_t stop = min( s0 + POLL, s1 );; stop = s1 ) {
            if( s0 >= 31u && s1 < cols ) {
                for( ; s < stop; s++ )
                    block( s, false, cols );
            }
            else {
                for( ; s < stop; s++ )
                    block( s, true, cols );
            }
            if( s >= s1 )
                break;
            if( poll && lane == 0 )
                seen = load_relaxed( sp.above );
        }
        __syncwarp();
        if( !sp.last ) {
            const int32_t c = (int32_t) s0 - 31 + lane / 2;
            if( lane < (int) (2 * CHUNK) && c >= 0 && c < (int32_t) s1 - 31 )
                __stcg( sp.row + (uint64_t) c * 2 + lane % 2, st.out[lane] );
            __syncwarp();
        }
        if( lane == 0 && (poll || !sp.last) ) {
            fence_acq_rel();
            if( !sp.last && s1 > 31u )
                store_relaxed( sp.mine, s1 - 31u );
        }
        if( poll )
            avail = max( avail, __shfl_sync( 0xffffffffu, seen, 0 ) & ~STREAM_DONE );
        __syncwarp();
        if( s1 == steps )
            break;
    }
    return cols;
}

// The stripe has ended after `cols` columns; whatever the warp wrote before is
// visible to a warp that sees this.
__device__ __forceinline__ void stream_end( const StreamStripe & sp, uint32_t cols, int lane ) {
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
