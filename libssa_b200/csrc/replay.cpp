// replay.cpp -- reproduces the order in which the CPU library inserts scores
// into its top-hit heap, and the heap itself.
//
// The GPU computes every (query, sequence) score at once, but the CPU
// library's result set depends on insertion order whenever scores tie at the
// heap boundary: its min-heap replaces the root only on a strictly greater
// score (reference: src/util/minheap.c:50-91), so which of several tied
// sequences survive depends on when each arrived.  The arrival order is fixed
// by the database chunks (ID ranges of chunk_size records, empty records
// skipped; src/db_adapter.c:212-239), by the SIMD channel scheduler inside
// each chunk (a sequence enters the lowest free lane at a block where some
// lane finished, and reports at the first block after its last one;
// src/algo/simd/search_simd_sw.c:338-428), and by the overflow cascade, which
// inserts a chunk's 8-bit reports first, then its 16-bit re-run reports in
// their own schedule, then the 64-bit re-runs in order
// (src/algo/8/search_8.c:94-124, src/algo/16/search_16.c:92-114,
// src/algo/64/search_64.c:44-56).  This file replays exactly that, from the
// per-sequence scores and the block counts the GPU passes return.
#include "ssa_internal.h"

#include <algorithm>
#include <cstring>

namespace ssa {

// When every sequence of a list scheduled on `lanes` channels reports, where
// sequence k occupies nb[k] blocks: the sequences report in ascending key
// order.  A sequence enters the channel that frees first, the lowest among
// equals; key = its last block, then its channel.  The channels are kept as a
// binary heap of (free block, channel), so a sequence costs log2(lanes) steps.
static void simulate_lanes( int lanes, const std::vector<int32_t> & nb, std::vector<int64_t> & key ) {
    const size_t n = nb.size();
    key.resize( n );
    int64_t heap[64];                              // free block << 6 | channel
    if( lanes > 64 )
        fatal( "Internal error: %d channels.", lanes );
    for( int c = 0; c < lanes; c++ )
        heap[c] = c;
    for( size_t k = 0; k < n; k++ ) {
        const int64_t v = heap[0] + ((int64_t) nb[k] << 6);
        key[k] = v;
        int at = 0;
        for( int c = 1; c < lanes; c = 2 * at + 1 ) {
            if( c + 1 < lanes && heap[c + 1] < heap[c] )
                c++;
            if( heap[c] >= v )
                break;
            heap[at] = heap[c];
            at = c;
        }
        heap[at] = v;
    }
}

// The indices of `pick` in report order: by key, then position in the list (a
// channel that takes a sequence of no blocks reports twice at the same block).
static void report_order( const std::vector<int64_t> & key, std::vector<uint32_t> & pick ) {
    std::sort( pick.begin(), pick.end(),
            [&]( uint32_t x, uint32_t y ) { return key[x] != key[y] ? key[x] < key[y] : x < y; } );
}

void schedule_ranks( const HostDb & db, size_t chunk_size, int lanes, std::vector<uint32_t> & rank ) {
    rank.assign( db.n_ids, 0 );
    std::vector<uint32_t> ids;
    std::vector<int32_t> nb;
    std::vector<int64_t> key;
    std::vector<uint32_t> order;
    const uint64_t cs = (uint64_t) chunk_size * db.upi;    // a chunk of records, in units
    for( uint64_t start = 0; start < db.n_ids; start += cs ) {
        const uint64_t end = std::min<uint64_t>( db.n_ids, start + cs );
        ids.clear();
        nb.clear();
        for( uint64_t id = start; id < end; id++ ) {
            if( db.len[id] == 0 )
                continue;
            ids.push_back( (uint32_t) id );
            nb.push_back( (int32_t) ((db.len[id] + 3) / 4) );
        }
        simulate_lanes( lanes, nb, key );
        order.resize( ids.size() );
        for( size_t k = 0; k < order.size(); k++ )
            order[k] = (uint32_t) k;
        report_order( key, order );
        for( size_t k = 0; k < order.size(); k++ )
            rank[ids[order[k]]] = (uint32_t) k;
    }
}

namespace {

// Bit-identical restatement of the reference's fixed-size min-heap
// (reference: src/util/minheap.c:50-91).
struct MinHeap {
    struct Elem {
        uint32_t id;       // database unit
        int64_t score;
        uint32_t q = 0;    // query strand or frame
    };
    size_t alloc;
    std::vector<Elem> a;

    explicit MinHeap( size_t k ) : alloc( k ) { a.reserve( k ); }

    // the score that an element has to exceed to enter (INT64_MIN: any enters);
    // it never falls, so an element at or below it can be left out from here on
    int64_t bar() const { return a.size() < alloc ? INT64_MIN : alloc ? a[0].score : INT64_MAX; }

    void add( uint32_t id, int64_t score, uint32_t q = 0 ) {
        if( alloc == 0 )
            return;
        Elem n{ id, score, q };
        if( a.size() < alloc ) {
            size_t i = a.size();
            a.push_back( n );
            while( i > 0 && n.score < a[(i - 1) / 2].score ) {
                a[i] = a[(i - 1) / 2];
                i = (i - 1) / 2;
            }
            a[i] = n;
        }
        else if( a[0].score < n.score ) {
            size_t p = 0, c = 1;
            const size_t count = a.size();
            while( c < count ) {
                if( c + 1 < count && a[c + 1].score < a[c].score )
                    c++;
                if( a[c].score < n.score )
                    a[p] = a[c];
                else
                    break;
                p = c;
                c = 2 * p + 1;
            }
            a[p] = n;
        }
    }
};

// (id, blocks) lists sorted by id, looked up per chunk.
struct BlockMap {
    const std::vector<std::pair<uint32_t, int32_t>> & v;
    size_t lower( uint32_t id ) const {
        return (size_t) (std::lower_bound( v.begin(), v.end(), std::make_pair( id, INT32_MIN ) ) - v.begin());
    }
    bool find( uint32_t id, int32_t & nb ) const {
        size_t k = lower( id );
        if( k < v.size() && v[k].first == id ) {
            nb = v[k].second;
            return true;
        }
        return false;
    }
};

}  // namespace

void replay_query( const HostDb & db, const SearchRequest & req, const ReplayQuery & rq, const uint32_t * rank_entry,
        std::vector<Hit> & hits, ReplayCounts & counts ) {
    MinHeap heap( req.hitcount );
    const size_t cs = (req.chunk_size ? req.chunk_size : 1000) * (size_t) db.upi;   // records -> units
    const int lanes_entry = req.bit_width == 8 ? req.lanes8 : req.lanes16;
    BlockMap ovfE{ rq.ovf_entry }, ovf16{ rq.ovf16 };

    std::vector<std::pair<uint32_t, uint32_t>> cand;   // (rank, id)
    std::vector<uint32_t> ids, reports, order16, next, list64;
    std::vector<int32_t> nb;
    std::vector<int64_t> key, key16;

    for( uint64_t start = 0; start < db.n_ids; start += cs ) {
        const uint64_t end = std::min<uint64_t>( db.n_ids, start + cs );
        // a chunk without non-empty records ends the search: the reference's
        // drivers loop while the chunk is non-empty (src/algo/8/search_8.c:652,
        // src/algo/16/search_16.c:785, src/algo/64/search_64.c:963)
        if( db.nonempty_before[end] == db.nonempty_before[start] )
            break;
        const int64_t bar = heap.bar();
        const size_t e0 = ovfE.lower( (uint32_t) start );
        const bool has_ovf = req.bit_width != 64 && e0 < rq.ovf_entry.size() && rq.ovf_entry[e0].first < end;
        if( !has_ovf ) {
            // every sequence of the chunk reported at the entry pass: the
            // order is the query-independent schedule
            cand.clear();
            // The score first, which leaves few: 400,000 sequences 0.33 ms of one core,
            // 0.55 with the length and the state of the heap before it.  (No score is
            // INT64_MIN: a Smith-Waterman score is not negative, and a global alignment
            // may be all gaps.)
            for( uint64_t id = start; id < end; id++ ) {
                if( rq.score_of( (uint32_t) id ) <= bar || db.len[id] == 0 )
                    continue;
                cand.emplace_back( req.bit_width == 64 ? (uint32_t) (id - start) : rank_entry[id], (uint32_t) id );
            }
            if( cand.empty() )
                continue;
            std::sort( cand.begin(), cand.end() );
            for( auto & c : cand )
                heap.add( c.second, rq.score_of( c.second ) );
            continue;
        }
        // the chunk has overflowing sequences: its counters follow from the
        // lists alone, its schedules are re-run only when one of its
        // sequences can enter the heap
        const size_t e1 = ovfE.lower( (uint32_t) end );
        const size_t s0 = ovf16.lower( (uint32_t) start ), s1 = ovf16.lower( (uint32_t) end );
        (req.bit_width == 8 ? counts.overflow8 : counts.overflow16) += e1 - e0;
        if( req.bit_width == 8 )
            counts.overflow16 += s1 - s0;
        bool reported = false, overflowed = false;     // a candidate that reports / overflows at the entry width
        {
            size_t at = e0;
            for( uint64_t id = start; id < end && !overflowed; id++ ) {
                const bool ovf = at < e1 && rq.ovf_entry[at].first == id;
                at += ovf;
                if( db.len[id] == 0 || (bar != INT64_MIN && rq.score_of( (uint32_t) id ) <= bar) )
                    continue;
                (ovf ? overflowed : reported) = true;
            }
        }
        if( !reported && !overflowed )
            continue;
        ids.clear();
        nb.clear();
        reports.clear();
        next.clear();
        {
            size_t at = e0;
            for( uint64_t id = start; id < end; id++ ) {
                const bool ovf = at < e1 && rq.ovf_entry[at].first == id;
                const int32_t b = ovf ? rq.ovf_entry[at].second : (int32_t) ((db.len[id] + 3) / 4);
                at += ovf;
                if( db.len[id] == 0 )
                    continue;
                if( ovf )
                    next.push_back( (uint32_t) ids.size() );
                else if( bar == INT64_MIN || rq.score_of( (uint32_t) id ) > bar )
                    reports.push_back( (uint32_t) ids.size() );
                ids.push_back( (uint32_t) id );
                nb.push_back( b );
            }
        }
        simulate_lanes( lanes_entry, nb, key );
        report_order( key, reports );
        for( uint32_t k : reports )
            heap.add( ids[k], rq.score_of( ids[k] ) );
        if( !overflowed )
            continue;
        report_order( key, next );
        for( uint32_t & k : next )
            k = ids[k];
        if( req.bit_width == 8 ) {
            nb.clear();
            order16.clear();
            list64.clear();
            for( uint32_t k = 0; k < (uint32_t) next.size(); k++ ) {
                int32_t b;
                const bool ovf = s1 > s0 && ovf16.find( next[k], b );
                (ovf ? list64 : order16).push_back( k );
                nb.push_back( ovf ? b : (int32_t) ((db.len[next[k]] + 3) / 4) );
            }
            simulate_lanes( req.lanes16, nb, key16 );
            report_order( key16, order16 );
            report_order( key16, list64 );
            for( uint32_t k : order16 )
                heap.add( next[k], rq.score_of( next[k] ) );
            for( uint32_t k : list64 )
                heap.add( next[k], rq.score_of( next[k] ) );
        }
        else {
            for( uint32_t id : next )
                heap.add( id, rq.score_of( id ) );
        }
    }

    // sort by score, then ID, both descending (reference: src/util/minheap.c:93-106)
    std::vector<MinHeap::Elem> e = heap.a;
    std::sort( e.begin(), e.end(), []( const MinHeap::Elem & x, const MinHeap::Elem & y ) {
        if( x.score != y.score )
            return x.score > y.score;
        return x.id > y.id;
    } );
    hits.clear();
    hits.resize( e.size() );
    for( size_t k = 0; k < e.size(); k++ ) {
        hits[k].score = e[k].score;
        hits[k].unit = e[k].id;
        hits[k].id = e[k].id / db.upi;
        hits[k].db_strand = (uint8_t) (e[k].id % db.upi);
    }
}

// A query searched as several sequences (strands, or translated frames): the
// reference runs every chunk once per query sequence into the same heap, then
// re-runs the chunk's overflow list, which holds the overflowing units of all
// query sequences in report order, at 16 bits for every query sequence, and its
// 16-bit overflow list at 64 bits for every query sequence
// (src/algo/8/search_8.c:94-124, src/algo/16/search_16.c:92-114,
// src/algo/64/search_64.c:44-56).  Every report carries the pair's exact
// score, which the GPU passes leave in the score rows.
void replay_frames( const HostDb & db, const SearchRequest & req, const ReplayQuery * rq, uint32_t F,
        std::vector<Hit> & hits, ReplayCounts & counts ) {
    MinHeap heap( req.hitcount );
    const size_t cs = (req.chunk_size ? req.chunk_size : 1000) * (size_t) db.upi;
    const int lanes_entry = req.bit_width == 8 ? req.lanes8 : req.lanes16;
    std::vector<BlockMap> ovfE, ovf16;
    for( uint32_t q = 0; q < F; q++ ) {
        ovfE.push_back( BlockMap{ rq[q].ovf_entry } );
        ovf16.push_back( BlockMap{ rq[q].ovf16 } );
    }
    auto blocks = [&]( uint32_t u ) { return (int32_t) ((db.len[u] + 3) / 4); };
    std::vector<uint32_t> units, order, ovf_chunk, list64;
    std::vector<int32_t> nb;
    std::vector<int64_t> key;
    for( uint64_t start = 0; start < db.n_ids; start += cs ) {
        const uint64_t end = std::min<uint64_t>( db.n_ids, start + cs );
        if( db.nonempty_before[end] == db.nonempty_before[start] )
            break;
        units.clear();
        for( uint64_t u = start; u < end; u++ )
            if( db.len[u] )
                units.push_back( (uint32_t) u );
        // a chunk none of whose pairs can enter the heap leaves it as it is
        const int64_t bar = heap.bar();
        bool any = bar == INT64_MIN;
        for( uint32_t q = 0; q < F && !any; q++ )
            for( size_t k = 0; k < units.size() && !any; k++ )
                any = rq[q].score_of( units[k] ) > bar;
        if( req.bit_width == 64 ) {
            for( uint32_t q = 0; q < F && any; q++ )
                for( uint32_t u : units )
                    heap.add( u, rq[q].score_of( u ), q );
            continue;
        }
        // the chunk's overflow list: the overflowing units of every query
        // sequence, in report order (in list order where only its counters count)
        ovf_chunk.clear();
        for( uint32_t q = 0; q < F; q++ ) {
            const size_t e0 = ovfE[q].lower( (uint32_t) start ), e1 = ovfE[q].lower( (uint32_t) end );
            if( !any ) {
                for( size_t e = e0; e < e1; e++ )
                    ovf_chunk.push_back( ovfE[q].v[e].first );
                continue;
            }
            nb.clear();
            order.clear();
            size_t at = e0;
            for( uint32_t k = 0; k < (uint32_t) units.size(); k++ ) {
                const bool ovf = at < e1 && ovfE[q].v[at].first == units[k];
                nb.push_back( ovf ? ovfE[q].v[at].second : blocks( units[k] ) );
                at += ovf;
                if( ovf || rq[q].score_of( units[k] ) > bar || bar == INT64_MIN )
                    order.push_back( k );
            }
            simulate_lanes( lanes_entry, nb, key );
            report_order( key, order );
            for( uint32_t k : order ) {
                const uint32_t u = units[k];
                int32_t b;
                if( ovfE[q].find( u, b ) )
                    ovf_chunk.push_back( u );
                else
                    heap.add( u, rq[q].score_of( u ), q );
            }
        }
        if( ovf_chunk.empty() )
            continue;
        if( req.bit_width == 8 ) {
            counts.overflow8 += ovf_chunk.size();
            list64.clear();
            for( uint32_t q = 0; q < F; q++ ) {
                // a pair that did not overflow at 8 bits reports at 16 bits too
                const size_t s0 = ovf16[q].lower( (uint32_t) start );
                const bool none64 = s0 == ovf16[q].v.size() || ovf16[q].v[s0].first >= end;
                if( !any && none64 )
                    continue;
                nb.clear();
                order.clear();
                for( uint32_t k = 0; k < (uint32_t) ovf_chunk.size(); k++ ) {
                    int32_t b8, b16;
                    const uint32_t u = ovf_chunk[k];
                    nb.push_back( (!none64 && ovfE[q].find( u, b8 ) && ovf16[q].find( u, b16 )) ? b16 : blocks( u ) );
                    order.push_back( k );
                }
                simulate_lanes( req.lanes16, nb, key );
                report_order( key, order );
                for( uint32_t k : order ) {
                    const uint32_t u = ovf_chunk[k];
                    int32_t b8, b16;
                    if( !none64 && ovfE[q].find( u, b8 ) && ovf16[q].find( u, b16 ) )
                        list64.push_back( u );
                    else
                        heap.add( u, rq[q].score_of( u ), q );
                }
            }
            counts.overflow16 += list64.size();
            for( uint32_t q = 0; q < F && any; q++ )
                for( uint32_t u : list64 )
                    heap.add( u, rq[q].score_of( u ), q );
        }
        else {
            counts.overflow16 += ovf_chunk.size();
            for( uint32_t q = 0; q < F && any; q++ )
                for( uint32_t u : ovf_chunk )
                    heap.add( u, rq[q].score_of( u ), q );
        }
    }
    // score, then database ID, both descending; entries equal in both keep
    // their heap order (the reference's qsort of the heap array is a stable
    // merge sort: src/util/minheap.c:93-106)
    std::vector<MinHeap::Elem> e = heap.a;
    std::stable_sort( e.begin(), e.end(), [&]( const MinHeap::Elem & x, const MinHeap::Elem & y ) {
        if( x.score != y.score )
            return x.score > y.score;
        return x.id / db.upi > y.id / db.upi;
    } );
    hits.clear();
    hits.resize( e.size() );
    for( size_t k = 0; k < e.size(); k++ ) {
        hits[k].score = e[k].score;
        hits[k].unit = e[k].id;
        hits[k].id = e[k].id / db.upi;
        hits[k].db_strand = (uint8_t) (e[k].id % db.upi);
        hits[k].q_index = e[k].q;
    }
}

}  // namespace ssa
