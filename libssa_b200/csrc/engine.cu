// engine.cu -- host orchestration of the GPU search.
//
// One search call (one query through sw_align/nw_align, or a batch through
// the batched extension) runs as:
//
//   1. the database, read once through the libssa_extern_db.h plugin and
//      mapped to residue codes, is resident in HBM (re-packed only after
//      init_db or a change of symbol type);
//   2. the queries of the batch are uploaded and their substitution profiles
//      built on the device, one 32 x rows table per query and pass width;
//   3. the entry pass scores every (query, non-empty sequence) pair; pairs the
//      entry width cannot report go to a device-side re-queue list with the
//      block count they used, and the next width runs on that list
//      (8 -> 16 -> 64, reference: src/algo/8/search_8.c:94-124,
//      src/algo/16/search_16.c:92-114);
//   4. the final score of every pair and the re-queue lists come back to the
//      host, which replays the CPU channel schedule and min-heap per query
//      (replay.cpp) to get the exact CPU hit list;
//   5. for COMPUTE_ALIGNMENT the hits go through the traceback kernels.
#include "device_common.cuh"
#include "stream_stripes.cuh"
#include "ssa_internal.h"
#include "libssa_extern_db.h"

#include <algorithm>
#include <atomic>
#include <chrono>
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <map>
#include <mutex>
#include <unordered_map>
#include <thread>
#include <tuple>

namespace ssa {

static_assert( REPLAY_SCORE_IN_WIDE == SCORE_IN_WIDE, "one marker for scores held in int64" );

#define CUDA_CHECK( expr ) \
    do { \
        cudaError_t e_ = (expr); \
        if( e_ != cudaSuccess ) \
            fatal( "CUDA error %s at %s:%d: %s", cudaGetErrorName( e_ ), __FILE__, __LINE__, cudaGetErrorString( e_ ) ); \
    } while( 0 )

// Grow-only device buffer.
struct DevBuf {
    void * p = nullptr;
    size_t bytes = 0;
    void * ensure( size_t n ) {
        if( n > bytes ) {
            if( p )
                CUDA_CHECK( cudaFree( p ) );
            p = nullptr;
            size_t want = std::max( n, (size_t) 256 );
            CUDA_CHECK( cudaMalloc( &p, want ) );
            bytes = want;
        }
        return p;
    }
    // with an eighth to spare, so that a call on slightly longer sequences does
    // not allocate again (10 ms for 4 GB); without where that does not fit
    void * ensure_spare( size_t n ) {
        if( n > bytes ) {
            release();
            if( cudaMalloc( &p, n + n / 8 ) == cudaSuccess ) {
                bytes = n + n / 8;
                return p;
            }
            (void) cudaGetLastError();
            p = nullptr;
        }
        return ensure( n );
    }
    void release() {
        if( p )
            cudaFree( p );
        p = nullptr;
        bytes = 0;
    }
    template <class T>
    T * as() const {
        return (T *) p;
    }
};

struct PinnedBuf {
    void * p = nullptr;
    size_t bytes = 0;
    void * ensure( size_t n ) {
        if( n > bytes ) {
            if( p )
                CUDA_CHECK( cudaFreeHost( p ) );
            p = nullptr;
            size_t want = std::max( n, (size_t) 256 );
            CUDA_CHECK( cudaMallocHost( &p, want ) );
            bytes = want;
        }
        return p;
    }
    void release() {
        if( p )
            cudaFreeHost( p );
        p = nullptr;
        bytes = 0;
    }
};

// A device array inside a buffer that something else owns.
struct DevView {
    void * p = nullptr;
    template <class T>
    T * as() const {
        return (T *) p;
    }
};

// Most pinned memory that one buffer keeps for later calls, where its size follows
// from a call's work and not from the database (SSA_B200_PINNED_KEPT: another bound,
// for tests).
static size_t pinned_kept() {
    const char * e = getenv( "SSA_B200_PINNED_KEPT" );
    return e ? strtoull( e, nullptr, 10 ) : (size_t) 64 << 20;
}

// The small arrays of one call on their way to the device: gathered in pinned
// memory and sent in one copy.  (A copy from pageable memory costs the host
// several microseconds, and a call has a dozen of them.)
class Stager {
public:
    // A new call: the device has finished the one before.
    void begin() {
        used_ = sent_ = 0;
        if( h_.bytes > pinned_kept() ) {         // a call with very many pairs
            h_.release();
            d_.release();
        }
        for( auto & o : old_ ) {
            o.first.release();
            o.second.release();
        }
        old_.clear();
    }
    // Copies n elements of data; returns where they will be on the device.
    template <class T>
    T * add( const T * data, size_t n, cudaStream_t st ) {
        const size_t bytes = (n * sizeof(T) + 15) & ~(size_t) 15;
        if( used_ + bytes > h_.bytes || !h_.p ) {
            // arrays added before stay where they are until the next call
            send( st );
            const size_t want = std::max<size_t>( { 2 * h_.bytes, 2 * bytes, (size_t) 1 << 16 } );
            if( h_.p )
                old_.emplace_back( h_, d_ );
            h_ = PinnedBuf();
            d_ = DevBuf();
            h_.ensure( want );
            d_.ensure( want );
            used_ = sent_ = 0;
        }
        const size_t at = used_;
        if( n )
            memcpy( (char *) h_.p + at, data, n * sizeof(T) );
        used_ += bytes;
        return (T *) ((char *) d_.p + at);
    }
    void send( cudaStream_t st ) {
        if( used_ > sent_ )
            CUDA_CHECK( cudaMemcpyAsync( (char *) d_.p + sent_, (char *) h_.p + sent_, used_ - sent_,
                    cudaMemcpyHostToDevice, st ) );
        sent_ = used_;
    }
    void release() {
        begin();
        h_.release();
        d_.release();
    }

private:
    PinnedBuf h_;
    DevBuf d_;
    size_t used_ = 0, sent_ = 0;
    std::vector<std::pair<PinnedBuf, DevBuf>> old_;
};

class Engine {
public:
    static Engine & get() {
        static Engine e;
        return e;
    }

    void init_device() {
        if( ready_ )
            return;
        int dev = 0;
        if( const char * s = getenv( "SSA_B200_DEVICE" ) )
            dev = atoi( s );
        int n = 0;
        CUDA_CHECK( cudaGetDeviceCount( &n ) );
        if( n <= 0 )
            fatal( "No CUDA device available: the B200 libssa build has no CPU path." );
        CUDA_CHECK( cudaSetDevice( dev ) );
        cudaDeviceProp prop;
        CUDA_CHECK( cudaGetDeviceProperties( &prop, dev ) );
        if( prop.major < 10 )
            fatal( "libssa B200 build needs an sm_100 device, found %s (sm_%d%d).", prop.name, prop.major,
                    prop.minor );
        sms_ = prop.multiProcessorCount;
        device_memory_ = prop.totalGlobalMem;
        CUDA_CHECK( cudaStreamCreateWithFlags( &stream_, cudaStreamNonBlocking ) );
        CUDA_CHECK( cudaEventCreate( &ev0_ ) );
        CUDA_CHECK( cudaEventCreate( &ev1_ ) );
        CUDA_CHECK( cudaEventCreateWithFlags( &ev_ready_, cudaEventDisableTiming ) );
        for( auto & e : ev_phase_ )
            CUDA_CHECK( cudaEventCreate( &e ) );
        for( auto & e : ev_seg_ )
            CUDA_CHECK( cudaEventCreate( &e ) );
        for( auto & e : ev_tb_ )
            CUDA_CHECK( cudaEventCreate( &e ) );
        for( int i = 0; i < 4; i++ ) {
            CUDA_CHECK( cudaStreamCreateWithFlags( &class_stream_[i], cudaStreamNonBlocking ) );
            CUDA_CHECK( cudaEventCreateWithFlags( &ev_class_[i], cudaEventDisableTiming ) );
            CUDA_CHECK( cudaEventCreate( &ev_cls_t_[2 * i] ) );
            CUDA_CHECK( cudaEventCreate( &ev_cls_t_[2 * i + 1] ) );
        }
        int least = 0, greatest = 0;
        CUDA_CHECK( cudaDeviceGetStreamPriorityRange( &least, &greatest ) );
        CUDA_CHECK( cudaStreamCreateWithPriority( &long_stream_, cudaStreamNonBlocking, greatest ) );
        CUDA_CHECK( cudaEventCreateWithFlags( &ev_long_, cudaEventDisableTiming ) );
        CUDA_CHECK( cudaEventCreateWithFlags( &ev_items_, cudaEventDisableTiming ) );
        device_ = dev;
        ready_ = true;
    }

    // ---- database ------------------------------------------------------------
    const HostDb & database() {
        const Config & cfg = config();
        if( db_.symtype != cfg.symtype || db_.upi != units_per_record( cfg.symtype, cfg.strands ) || db_stale_ )
            pack_database();
        return db_;
    }

    void invalidate() { db_stale_ = true; }

    void pack_database() {
        const Config & cfg = config();
        HostDb db;
        const size_t n_rec = ssa_db_get_sequence_count();
        const uint32_t upi = units_per_record( cfg.symtype, cfg.strands );
        if( (uint64_t) n_rec * upi > UINT32_MAX )
            fatal( "Database has %zu sequences; at most %u are supported.", n_rec, UINT32_MAX / upi );
        const size_t n = n_rec * upi;
        db.n_records = (uint32_t) n_rec;
        db.upi = upi;
        db.n_ids = (uint32_t) n;
        db.len.assign( n, 0 );
        db.off.assign( n, 0 );
        const bool nt = cfg.symtype == NUCLEOTIDE;
        if( cfg.symtype == TRANS_DB || cfg.symtype == TRANS_BOTH )
            fatal( "Searches of a translated database (symbol type %d) are not supported by the B200 build.",
                    cfg.symtype );
        std::vector<p_seqinfo> infos( n_rec );
        for( size_t id = 0; id < n_rec; id++ ) {
            p_seqinfo info = ssa_db_get_sequence( id );
            if( !info )
                fatal( "Could not get sequence from DB: %zu", id );
            infos[id] = info;
            if( info->seqlen > (size_t) INT32_MAX / 2 )
                fatal( "Database sequence %zu is too long (%zu residues).", id, info->seqlen );
            for( uint32_t k = 0; k < upi; k++ )
                db.len[id * upi + k] = (uint32_t) info->seqlen;
            db.max_len = std::max( db.max_len, (uint32_t) info->seqlen );
            db.residues += (uint64_t) info->seqlen * upi;
        }
        db.nonempty_before.assign( (size_t) n + 1, 0 );
        for( uint32_t id = 0; id < db.n_ids; id++ ) {
            db.nonempty_before[id + 1] = db.nonempty_before[id] + (db.len[id] ? 1 : 0);
            if( db.len[id] )
                db.order_desc.push_back( id );
        }
        std::stable_sort( db.order_desc.begin(), db.order_desc.end(),
                [&]( uint32_t a, uint32_t b ) { return db.len[a] > db.len[b]; } );
        auto padded = [&]( uint32_t id ) { return ((uint64_t) db.len[id] + 15) & ~(uint64_t) 15; };

        // Resident layout: every ID in ID order, plus the interleaved pairs of
        // the single-query pass.  Streaming layout (the resident one does not
        // fit the database memory): segments of consecutive IDs in length
        // order, each a contiguous block that is copied to the device when its
        // turn comes; the device offsets are relative to the block.
        init_device();
        uint64_t codes_bytes = 0;
        for( uint32_t id = 0; id < db.n_ids; id++ )
            codes_bytes += padded( id );
        const uint64_t resident_bytes = 2 * codes_bytes + (uint64_t) n * (8 + 4 + 4) + 64;
        const uint64_t budget = db_budget();
        streaming_ = resident_bytes > budget;
        seg_lo_.clear();
        seg_hi_.clear();
        seg_off_.clear();
        seg_bytes_.clear();
        std::vector<uint64_t> dev_off( n, 0 );
        uint64_t total = 0;
        if( !streaming_ ) {
            for( uint32_t id = 0; id < db.n_ids; id++ ) {
                db.off[id] = total;
                dev_off[id] = total;
                total += padded( id );
            }
        }
        else {
            const uint64_t seg_cap = std::max<uint64_t>( 1, budget / 2 );
            uint64_t in_seg = 0;
            for( uint32_t pos = 0; pos < (uint32_t) db.order_desc.size(); pos++ ) {
                const uint32_t id = db.order_desc[pos];
                if( seg_lo_.empty() || (in_seg > 0 && in_seg + padded( id ) > seg_cap) ) {
                    if( !seg_lo_.empty() ) {
                        seg_hi_.push_back( pos );
                        seg_bytes_.push_back( in_seg );
                    }
                    seg_lo_.push_back( pos );
                    seg_off_.push_back( total );
                    in_seg = 0;
                }
                db.off[id] = total;
                dev_off[id] = in_seg;
                total += padded( id );
                in_seg += padded( id );
            }
            if( !seg_lo_.empty() ) {
                seg_hi_.push_back( (uint32_t) db.order_desc.size() );
                seg_bytes_.push_back( in_seg );
            }
        }
        db.codes.assign( total + 16, 0 );
        uint64_t unknown = 0;
        for( size_t id = 0; id < n_rec; id++ ) {
            // unknown symbols become code 0 (reference: src/util/util_sequence.c:298-318)
            const char * s = infos[id]->seq;
            const size_t L = infos[id]->seqlen;
            if( L == 0 )
                continue;
            uint8_t * o = db.codes.data() + db.off[id * upi];
            for( size_t k = 0; k < L; k++ ) {
                int m = nt ? map_nt16( (unsigned char) s[k] ) : map_aa( (unsigned char) s[k] );
                if( m < 0 ) {
                    m = 0;
                    unknown++;
                }
                o[k] = (uint8_t) m;
            }
            if( upi == 2 ) {
                // the reverse complement unit (reference: src/util/util_sequence.c:420-437)
                uint8_t * rc = db.codes.data() + db.off[id * upi + 1];
                for( size_t k = 0; k < L; k++ )
                    rc[k] = nt_complement( o[L - 1 - k] );
            }
        }
        if( unknown )
            print_warning( "%llu unknown symbols found and set to zero", (unsigned long long) unknown );
        db.symtype = cfg.symtype;
        db.strands = cfg.strands;
        db.generation = ++generation_;
        db.mean_len = db.order_desc.empty() ? 0.0 : (double) db.residues / (double) db.order_desc.size();

        d_off_.ensure( sizeof(uint64_t) * std::max<size_t>( 1, n ) );
        d_len_.ensure( sizeof(uint32_t) * std::max<size_t>( 1, n ) );
        d_order_.ensure( sizeof(uint32_t) * std::max<size_t>( 1, db.order_desc.size() ) );
        if( n ) {
            CUDA_CHECK( cudaMemcpy( d_off_.p, dev_off.data(), sizeof(uint64_t) * n, cudaMemcpyHostToDevice ) );
            CUDA_CHECK( cudaMemcpy( d_len_.p, db.len.data(), sizeof(uint32_t) * n, cudaMemcpyHostToDevice ) );
        }
        if( !db.order_desc.empty() )
            CUDA_CHECK( cudaMemcpy( d_order_.p, db.order_desc.data(), sizeof(uint32_t) * db.order_desc.size(),
                    cudaMemcpyHostToDevice ) );
        resident_seg_ = -1;
        if( streaming_ ) {
            DevBuf * big[] = { &d_codes_, &d_pair_res_, &d_pair_off_, &d_pair_cols_, &d_pair_ids_ };
            for( DevBuf * b : big )
                b->release();
            uint64_t max_seg = 0;
            for( uint64_t b : seg_bytes_ )
                max_seg = std::max( max_seg, b );
            for( DevBuf & b : d_seg_ )
                b.ensure( max_seg + 64 );
            db_ = std::move( db );
            db_stale_ = false;
            ranks_.clear();
            return;
        }
        for( DevBuf & b : d_seg_ )
            b.release();

        // pairs of consecutive sequences in length order share the 16x2 lanes
        // of the fast Smith-Waterman pass; columns past a sequence's last
        // 4-column block hold the neutral pad code
        const size_t n_pairs = (db.order_desc.size() + 1) / 2;
        db.pair_cols.resize( n_pairs );
        db.pair_a.resize( n_pairs );
        db.pair_b.resize( n_pairs );
        db.pair_blocks.assign( n_pairs + 1, 0 );
        std::vector<uint64_t> pair_off( n_pairs + 1, 0 );
        for( size_t pi = 0; pi < n_pairs; pi++ ) {
            db.pair_a[pi] = db.order_desc[2 * pi];
            db.pair_b[pi] = (2 * pi + 1 < db.order_desc.size()) ? db.order_desc[2 * pi + 1] : 0xffffffffu;
            db.pair_cols[pi] = (db.len[db.pair_a[pi]] + 7u) & ~7u;
            db.pair_blocks[pi + 1] = db.pair_blocks[pi] + db.pair_cols[pi] / 4u;
            pair_off[pi + 1] = pair_off[pi] + 2ull * db.pair_cols[pi];
        }
        std::vector<uint8_t> pair_res( pair_off[n_pairs] + 16, (uint8_t) FAST_PAD_CODE );
        for( size_t pi = 0; pi < n_pairs; pi++ ) {
            uint8_t * out = pair_res.data() + pair_off[pi];
            for( int half = 0; half < 2; half++ ) {
                const uint32_t id = half ? db.pair_b[pi] : db.pair_a[pi];
                if( id == 0xffffffffu )
                    continue;
                const uint32_t L = db.len[id], Lb = (L + 3u) & ~3u;
                const uint8_t * src = db.codes.data() + db.off[id];
                for( uint32_t j = 0; j < L; j++ )
                    out[2 * j + half] = src[j];
                for( uint32_t j = L; j < Lb; j++ )
                    out[2 * j + half] = 0;   // the reference's pad inside the last block
            }
        }
        d_codes_.ensure( db.codes.size() );
        CUDA_CHECK( cudaMemcpy( d_codes_.p, db.codes.data(), db.codes.size(), cudaMemcpyHostToDevice ) );
        {
            std::vector<uint2> ids( std::max<size_t>( 1, n_pairs ) );
            for( size_t pi = 0; pi < n_pairs; pi++ )
                ids[pi] = make_uint2( db.pair_a[pi], db.pair_b[pi] );
            d_pair_res_.ensure( pair_res.size() );
            d_pair_off_.ensure( sizeof(uint64_t) * (n_pairs + 1) );
            d_pair_cols_.ensure( sizeof(uint32_t) * std::max<size_t>( 1, n_pairs ) );
            d_pair_ids_.ensure( sizeof(uint2) * ids.size() );
            CUDA_CHECK( cudaMemcpy( d_pair_res_.p, pair_res.data(), pair_res.size(), cudaMemcpyHostToDevice ) );
            CUDA_CHECK( cudaMemcpy( d_pair_off_.p, pair_off.data(), sizeof(uint64_t) * (n_pairs + 1),
                    cudaMemcpyHostToDevice ) );
            if( n_pairs )
                CUDA_CHECK( cudaMemcpy( d_pair_cols_.p, db.pair_cols.data(), sizeof(uint32_t) * n_pairs,
                        cudaMemcpyHostToDevice ) );
            CUDA_CHECK( cudaMemcpy( d_pair_ids_.p, ids.data(), sizeof(uint2) * ids.size(), cudaMemcpyHostToDevice ) );
        }
        db_ = std::move( db );
        db_stale_ = false;
        ranks_.clear();
    }

    DbView db_view() const {
        DbView v;
        v.codes = streaming_ ? d_seg_[resident_seg_ & 1].as<uint8_t>() : d_codes_.as<uint8_t>();
        v.offsets = d_off_.as<uint64_t>();
        v.lens = d_len_.as<uint32_t>();
        v.n_ids = db_.n_ids;
        return v;
    }

    const uint32_t * ranks( size_t chunk_size, int lanes ) {
        for( auto & c : ranks_ )
            if( c.chunk_size == chunk_size && c.lanes == lanes && c.generation == db_.generation )
                return c.rank.data();
        ScheduleCache c;
        c.chunk_size = chunk_size;
        c.lanes = lanes;
        c.generation = db_.generation;
        schedule_ranks( db_, chunk_size, lanes, c.rank );
        ranks_.push_back( std::move( c ) );
        return ranks_.back().rank.data();
    }

    // ---- search ----------------------------------------------------------------
    void search( const SearchRequest & req, const std::vector<QueryCodes> & queries,
            const std::vector<uint32_t> & groups, std::vector<std::vector<Hit>> & out, SearchStats & stats );
    // query i against database unit units[i] alone
    void align_pairs( const SearchRequest & req, const std::vector<QueryCodes> & queries,
            const std::vector<uint32_t> & units, std::vector<std::vector<Hit>> & out, SearchStats & stats );
    // database-sharded search: entry pass and cascade of every query against
    // the records [id_lo, id_hi) only; per (query, record) the final score and
    // the blocks the entry-width and 16-bit lanes spent when they overflowed
    void shard_scores( const SearchRequest & req, const std::vector<QueryCodes> & queries, uint32_t id_lo,
            uint32_t id_hi, int64_t * scores, int32_t * blocks_entry, int32_t * blocks_16, SearchStats & stats );
    // traceback of replayed hit lists (out[q] for query q)
    void align_hits( const SearchRequest & req, const std::vector<QueryCodes> & queries,
            std::vector<std::vector<Hit>> & out, SearchStats & stats );
    void set_traceback_budget( uint64_t bytes ) { tb_budget_ = bytes; }
    void set_db_budget( uint64_t bytes ) {
        db_budget_ = bytes;
        db_stale_ = true;
    }
    bool streaming() const { return streaming_; }

    // Device memory for the database: the setting of ssa_b200_set_db_memory,
    // else 40% of the device memory (scores, re-queue lists, profiles and
    // traceback matrices take the rest).
    uint64_t db_budget() {
        if( db_budget_ )
            return db_budget_;
        size_t free_b = 0, total_b = 0;
        CUDA_CHECK( cudaMemGetInfo( &free_b, &total_b ) );
        return (uint64_t) total_b / 5 * 2;
    }

    // Segment s of a streamed database on the device (the other buffer keeps
    // the previous one); a no-op when it is there already.
    void make_resident( uint32_t sg, SearchStats & stats ) {
        if( !streaming_ || resident_seg_ == (int) sg )
            return;
        const uint64_t bytes = seg_bytes_[sg];
        uint8_t * stage = (uint8_t *) h_stage_.ensure( std::max<uint64_t>( bytes, 16 ) );
        // the staging buffer is reused: the previous copy must have finished
        CUDA_CHECK( cudaStreamSynchronize( stream_ ) );
        memcpy( stage, db_.codes.data() + seg_off_[sg], bytes );
        CUDA_CHECK( cudaMemcpyAsync( d_seg_[sg & 1].p, stage, bytes, cudaMemcpyHostToDevice, stream_ ) );
        resident_seg_ = (int) sg;
        stats.h2d_bytes += bytes;
    }

    // A device view of the given database IDs alone (in that order, view ID k =
    // ids[k]), for passes over a few sequences of a streamed database.
    DbView gather_view( const std::vector<uint32_t> & ids, SearchStats & stats ) {
        std::vector<uint64_t> off( ids.size() + 1, 0 );
        std::vector<uint32_t> len( std::max<size_t>( 1, ids.size() ), 0 );
        for( size_t k = 0; k < ids.size(); k++ ) {
            len[k] = db_.len[ids[k]];
            off[k + 1] = off[k] + (((uint64_t) len[k] + 15) & ~(uint64_t) 15);
        }
        std::vector<uint8_t> codes( off[ids.size()] + 64, 0 );
        for( size_t k = 0; k < ids.size(); k++ )
            memcpy( codes.data() + off[k], db_.codes.data() + db_.off[ids[k]], len[k] );
        d_gather_codes_.ensure( codes.size() );
        d_gather_off_.ensure( off.size() * sizeof(uint64_t) );
        d_gather_len_.ensure( len.size() * sizeof(uint32_t) );
        CUDA_CHECK( cudaMemcpyAsync( d_gather_codes_.p, codes.data(), codes.size(), cudaMemcpyHostToDevice, stream_ ) );
        CUDA_CHECK( cudaMemcpyAsync( d_gather_off_.p, off.data(), off.size() * sizeof(uint64_t),
                cudaMemcpyHostToDevice, stream_ ) );
        CUDA_CHECK( cudaMemcpyAsync( d_gather_len_.p, len.data(), len.size() * sizeof(uint32_t),
                cudaMemcpyHostToDevice, stream_ ) );
        CUDA_CHECK( cudaStreamSynchronize( stream_ ) );   // the host vectors go out of scope
        stats.h2d_bytes += codes.size() + off.size() * sizeof(uint64_t) + len.size() * sizeof(uint32_t);
        DbView v;
        v.codes = d_gather_codes_.as<uint8_t>();
        v.offsets = d_gather_off_.as<uint64_t>();
        v.lens = d_gather_len_.as<uint32_t>();
        v.n_ids = (uint32_t) ids.size();
        return v;
    }

    void shutdown() {
        DevBuf * bufs[] = { &d_codes_, &d_off_, &d_len_, &d_order_, &d_pair_res_, &d_pair_off_, &d_pair_cols_,
            &d_pair_ids_, &d_prof8_,
            &d_scratch_fast_[0], &d_scratch_fast_[1], &d_scratch_fast_[2], &d_scratch_fast_[3], &d_scratch_fast_[4],
            &d_scratch_fast_[5], &d_scratch_fast_[6], &d_scratch_fast_[7], &d_serve_block_, &d_prof_, &d_score_, &d_list_a_, &d_list_b_, &d_counts_, &d_scratch_,
            &d_tb_io_, &d_tb_last_, &d_tb_dirs_, &d_tb_sync_, &d_tb_result_, &d_tb_bnd_, &d_qp_prof_,
            &d_serve_score_, &d_list_c_, &d_sw_sync_, &d_sw_bnd_,
            &d_seg_[0], &d_seg_[1], &d_gather_codes_, &d_gather_off_, &d_gather_len_, &d_prof64_, &d_score64_ };
        for( DevBuf * b : bufs )
            b->release();
        stage_.release();
        h_counts_.release();
        h_score_.release();
        h_score64_.release();
        h_tb_in_.release();
        h_tb_out_.release();
        h_stage_.release();
        resident_seg_ = -1;
        streaming_ = false;
        db_ = HostDb();
        db_stale_ = true;
        ranks_.clear();
        serve_layout_ = false;
        serve_slots_ = 0;
        serve_codes_.clear();
    }

    uint64_t launches() const { return launches_.load(); }

    // ---- serving: fixed query slots, waves over database segments ---------------
    std::vector<uint32_t> serve_open( const SearchRequest & req, uint32_t slots, uint32_t segments );
    void serve_restore( const SearchRequest & req );
    void serve_load( uint32_t slot, const uint8_t * codes, uint32_t len );
    void serve_wave( const SearchRequest & req, const std::vector<uint32_t> & active, uint32_t seq_lo,
            uint32_t seq_hi, std::vector<PairTask> & ovf_entry, std::vector<PairTask> & ovf16, SearchStats & stats );
    void serve_finish( const SearchRequest & req, const std::vector<uint32_t> & done,
            std::vector<ReplayQuery> & rq, std::vector<std::vector<Hit>> & out, SearchStats & stats );

private:
    Engine() = default;

    void run_pass( int algo, int width, const SearchRequest & req, uint32_t n_slots, const PairTask * tasks,
            uint64_t n_tasks, bool implicit, PairTask * next, unsigned * next_count, uint32_t next_cap,
            const uint32_t * slot_list = nullptr, uint32_t n_sub = 0, uint32_t order_lo = 0 );
    void run_fast_entry( const SearchRequest & req, uint32_t nq, PairTask * next, unsigned * next_count, uint32_t cap );
    // marked: the 16-bit pass of the cascade, only the pairs that the 8-bit entry re-queued (Needleman-Wunsch)
    void run_qpair_entry( const SearchRequest & req, uint32_t nq, PairTask * next, unsigned * next_count,
            uint32_t cap, PairTask * redo_list, const std::vector<uint32_t> * slots = nullptr, uint32_t seq_lo = 0,
            uint32_t seq_hi = UINT32_MAX, bool marked = false );
    void run_stream( const SearchRequest & req, std::vector<SwStreamItem> & items, const PassSink & lists,
            cudaStream_t st, bool marked = false );
    // The passes after the entry width: list A holds n_a pairs that it re-queued.
    // Leaves their scores, and the lists on the host (appended).
    void run_cascade( const SearchRequest & req, uint32_t nq, uint32_t n_a, uint32_t cap,
            std::vector<PairTask> & list_entry, std::vector<PairTask> & list_16, const std::vector<uint32_t> * slots,
            uint32_t lo, uint32_t hi );
    static constexpr size_t LIST_HEAD = 1024;
    const unsigned * read_counts( bool head, void * scores_to = nullptr, size_t score_bytes = 0 );
    const unsigned * run_redo( const SearchRequest & req, uint32_t nq, const unsigned * c, PairTask * next,
            unsigned * next_count, uint32_t cap, const PairTask * redo_list, uint32_t redo_cap );
    int32_t * score_sink() { return serving_ ? d_serve_score_.as<int32_t>() : d_score_.as<int32_t>(); }
    void build_profiles( int width, uint32_t n_slots );
    // scores_from_regions: the hits carry no score yet; take it from the
    // forward pass (SW, symmetric table) or the direction pass (NW);
    // scores_only: score the hits' pairs exactly, no alignment
    void traceback( const SearchRequest & req, std::vector<std::vector<Hit>> & out,
            const std::vector<std::pair<uint32_t, uint32_t>> & lists, SearchStats & stats,
            bool scores_from_regions = false, bool scores_only = false );
    uint64_t traceback_budget();
    void upload_queries( const SearchRequest & req, const QueryCodes * queries, uint32_t nq, bool profiles,
            SearchStats & stats );

    bool ready_ = false;
    int device_ = 0;
    int sms_ = 148;
    uint64_t device_memory_ = 0;
    // (query, sequence) pairs of one sub-batch: its int32 scores (4 B) and, at
    // most, two re-queue lists of 16 B per pair; 2^29 pairs (19 GB) on devices
    // of 64 GB and more (a 1,024-query batch against 500,000 sequences in one
    // pass), 2^28 otherwise; halved when the 64-bit pass keeps int64 scores
    uint64_t pair_budget() const {
        const int log2 = device_memory_ >= ((uint64_t) 64 << 30) ? 29 : 28;
        return (uint64_t) 1 << (wide_ ? log2 - 1 : log2);
    }
    cudaStream_t stream_ = nullptr;
    cudaEvent_t ev0_ = nullptr, ev1_ = nullptr;
    HostDb db_;
    bool db_stale_ = true;
    uint64_t generation_ = 0;
    std::vector<ScheduleCache> ranks_;
    std::atomic<uint64_t> launches_{ 0 };

    // device buffers
    DevBuf d_codes_, d_off_, d_len_, d_order_;
    DevBuf d_pair_res_, d_pair_off_, d_pair_cols_, d_pair_ids_;
    DevBuf d_prof8_;
    DevBuf d_scratch_fast_[8];      // per class of the single-query pass
    DevBuf d_qp_prof_;
    // serving: fixed query slots and their own score rows
    DevBuf d_serve_score_;
    bool serving_ = false;           // passes write d_serve_score_
    bool serve_layout_ = false;      // the query buffers hold the serving slots
    uint32_t serve_slots_ = 0;
    std::vector<std::vector<uint8_t>> serve_codes_;   // per slot, to restore the layout after a search
    std::vector<uint32_t> serve_new_;                 // slots whose query the device does not have yet
    cudaStream_t class_stream_[4] = { nullptr, nullptr, nullptr, nullptr };
    cudaEvent_t ev_class_[4] = { nullptr, nullptr, nullptr, nullptr };
    cudaEvent_t ev_cls_t_[8] = {};   // per class start / end, timed (SSA_B200_TIMING)
    cudaStream_t long_stream_ = nullptr;      // an entry pass's longest pairs
    cudaEvent_t ev_long_ = nullptr;
    cudaEvent_t ev_items_ = nullptr;     // the streamed pairs' inputs are there
    cudaEvent_t ev_ready_ = nullptr;
    cudaEvent_t ev_phase_[6] = {};
    cudaEvent_t ev_seg_[2] = {};     // around one segment's entry pass
    cudaEvent_t ev_tb_[5] = {};   // batch start, entry pass done, cascade done, copies done, traceback
    // the current queries and score table: in the stager, or the server's own block
    DevView d_qcodes_, d_qoff_, d_qlen_, d_qpad_, d_prof_off_, d_matrix_;
    DevBuf d_prof_, d_serve_block_;
    std::vector<uint64_t> blocks_before_;             // of an entry pass
    Stager stage_;
    PinnedBuf h_counts_;
    DevBuf d_score_, d_list_a_, d_list_b_, d_counts_, d_scratch_, d_list_c_, d_sw_sync_, d_sw_bnd_;
    DevBuf d_tb_io_, d_tb_last_, d_tb_dirs_, d_tb_sync_, d_tb_result_, d_tb_bnd_;
    PinnedBuf h_score_, h_tb_in_, h_tb_out_;
public:
    // entry-pass shapes of the last search call: kernel, (R, CTAs per SM) for
    // the query-pair kernel or (G, R) for the single-query one, queries or
    // query pairs, database bucket
    struct ShapeUse {
        const char * kernel;
        int a, b;
        uint32_t n;
        int bucket;
    };
    std::vector<ShapeUse> last_shapes_;
private:
    // the 64-bit pass in int64 arithmetic (wide_): exact profiles and scores
    DevBuf d_prof64_, d_score64_;
    PinnedBuf h_score64_;
    bool wide_ = false;
    int prof64_width_ = -1;
    uint64_t tb_budget_ = 0;         // traceback direction memory per wave (0 = automatic)
    // streaming: the database does not fit its device memory budget; segments
    // of consecutive positions of the length order take turns on the device
    uint64_t db_budget_ = 0;         // database device memory (0 = automatic)
    bool streaming_ = false;
    std::vector<uint32_t> seg_lo_, seg_hi_;     // per segment: positions in order_desc
    std::vector<uint64_t> seg_off_, seg_bytes_; // per segment: block in db_.codes
    DevBuf d_seg_[2];
    int resident_seg_ = -1;
    PinnedBuf h_stage_;
    DevBuf d_gather_codes_, d_gather_off_, d_gather_len_;

    // per-batch query layout
    std::vector<uint64_t> h_qoff_;
    std::vector<uint32_t> h_qlen_, h_qpad_;
    std::vector<uint64_t> h_prof_off_;
    int prof_width_ = -1;
    uint32_t prof_slots_ = 0;
    uint32_t max_qlen_ = 0;

    friend void engine_shutdown();
};

void Engine::build_profiles( int width, uint32_t n_slots ) {
    if( wide_ && width == 64 ) {
        // exact int64 table (same offsets as the int32 one, twice the bytes)
        if( prof_width_ == 64 && prof64_width_ == 64 && prof_slots_ == n_slots )
            return;
        uint64_t elems = 0;
        for( uint32_t s = 0; s < n_slots && s < h_prof_off_.size(); s++ )
            elems = std::max<uint64_t>( elems, h_prof_off_[s] + 32ull * h_qpad_[s] );
        d_prof64_.ensure( std::max<uint64_t>( elems, 1 ) * sizeof(int64_t) );
        CUDA_CHECK( launch_build_profile64( d_qcodes_.as<uint8_t>(), d_qoff_.as<uint64_t>(), d_qlen_.as<uint32_t>(),
                d_qpad_.as<uint32_t>(), d_prof_off_.as<uint64_t>(), d_matrix_.as<int64_t>(), d_prof64_.as<int64_t>(),
                n_slots, stream_ ) );
        launches_++;
        prof_width_ = 64;
        prof64_width_ = 64;
        prof_slots_ = n_slots;
        return;
    }
    if( prof_width_ == width && prof_slots_ == n_slots && prof64_width_ != 64 )
        return;
    launch_build_profile32( d_qcodes_.as<uint8_t>(), d_qoff_.as<uint64_t>(), d_qlen_.as<uint32_t>(),
            d_qpad_.as<uint32_t>(), d_prof_off_.as<uint64_t>(), d_matrix_.as<int64_t>(), width,
            d_prof_.as<int32_t>(), n_slots, stream_ );
    CUDA_CHECK( cudaGetLastError() );
    launches_++;
    prof_width_ = width;
    prof64_width_ = -1;
    prof_slots_ = n_slots;
}

void Engine::run_pass( int algo, int width, const SearchRequest & req, uint32_t n_slots, const PairTask * tasks,
        uint64_t n_tasks, bool implicit, PairTask * next, unsigned * next_count, uint32_t next_cap,
        const uint32_t * slot_list, uint32_t n_sub, uint32_t order_lo ) {
    if( n_tasks == 0 )
        return;
    stage_.send( stream_ );
    build_profiles( width, n_slots );
    EmulParams p;
    p.db = db_view();
    p.qv.prof32 = d_prof_.as<int32_t>();
    p.qv.prof32_off = d_prof_off_.as<uint64_t>();
    p.qv.qlen = d_qlen_.as<uint32_t>();
    p.qv.qpad = d_qpad_.as<uint32_t>();
    p.qv.n_slots = n_slots;
    p.tasks = implicit ? nullptr : tasks;
    p.order = d_order_.as<uint32_t>() + order_lo;
    p.slot_list = slot_list;
    p.n_sub = n_sub;
    p.n_tasks = n_tasks;
    unsigned long long * counter = d_counts_.as<unsigned long long>() + 4;
    CUDA_CHECK( cudaMemsetAsync( counter, 0, sizeof(unsigned long long), stream_ ) );
    p.counter = counter;
    p.gap_open = req.gap_open;
    p.gap_extend = req.gap_extend;
    p.sink.score = score_sink();
    p.sink.score_stride = db_.n_ids;
    p.sink.next = next;
    p.sink.next_count = next_count;
    p.sink.next_cap = next_cap;
    p.sink.error_flags = d_counts_.as<unsigned>() + 2;
    const bool wide = wide_ && width == 64;
    if( wide ) {
        if( serving_ )
            fatal( "Internal error: int64 scoring is not available to the server." );
        p.qv.prof64 = d_prof64_.as<int64_t>();
        p.sink.score64 = d_score64_.as<int64_t>();
    }
    const int grid = sms_ * 2;
    const uint32_t cols = ((db_.max_len + 3u) & ~3u) + 4;
    if( max_qlen_ > 256 ) {
        // a boundary column is 4 values: 16 bytes in int32, 32 in int64
        const size_t col_bytes = wide ? 2 * sizeof(int4) : sizeof(int4);
        p.scratch = (int4 *) d_scratch_.ensure( (size_t) grid * 8 * cols * col_bytes );
        p.scratch_cols = cols;
    }
    else {
        p.scratch = nullptr;
        p.scratch_cols = 0;
    }
    CUDA_CHECK( launch_emul( algo, width, p, grid, stream_, wide ) );
    launches_++;
}

// Whether the 64-bit pass needs int64 arithmetic: a DP value is bounded by the
// number of steps of a path (query rows + columns + a few boundary terms) times
// the largest magnitude of one step (a score-table entry, or gapO + gapE); at
// or below the int32 range (with a factor 2 of margin for the sums formed
// before each max) int32 is exact.
static bool needs_int64( const SearchRequest & req, uint32_t max_qlen, uint32_t max_dlen ) {
    int64_t m = std::llabs( (int64_t) req.gap_open ) + std::llabs( (int64_t) req.gap_extend );
    for( int k = 0; k < 1024; k++ )
        m = std::max<int64_t>( m, req.matrix[k] == INT64_MIN ? INT64_MAX / 4 : std::llabs( req.matrix[k] ) );
    const int64_t steps = (int64_t) max_qlen + max_dlen + 8;
    return m > (int64_t) INT32_MAX / 2 || steps * (m + 1) * 2 > (int64_t) INT32_MAX;
}

// Needleman-Wunsch at the 16-bit entry: the query-pair kernel scores exactly
// the sequences short enough that no value can come near the int16 limits
// (nw_qpair_kernel); it needs non-positive gap costs, and at 16 bits a cost for
// a gap of one: the lane's overflow line, -32768 - gapO - gapE - 1 in 16 bits,
// wraps to 32767 where that is 0, and every sequence then overflows in its first
// block.  The 64-bit entry takes the same kernel where the score table fits int16.
static bool nw_fast_eligible( const SearchRequest & req ) {
    if( req.algo != 1 || req.bit_width == 8 || getenv( "SSA_B200_NO_FAST" ) )
        return false;
    if( req.bit_width == 16 && req.gap_open + req.gap_extend == 0 )
        return false;
    for( int k = 0; k < 1024 && req.bit_width == 64; k++ )
        if( req.matrix[k] != (int16_t) req.matrix[k] )
            return false;
    return req.gap_open <= 0 && req.gap_extend <= 0;
}

// The running maximum at which the 16x2 Smith-Waterman kernels end a
// sequence, 0 where they do not apply.  They reproduce the 8-bit lanes exactly
// when the gap extension is not positive and the truncated 8-bit open+extend cost
// lies in [-128, gapE]; other parameters run the exact lane emulation.  8-bit entry: 255, the lane's own
// overflow.  At 16 and 64 bits the lane saturates far above (65535) or not at
// all, and the kernels are exact up to where a 16-bit half could leave its
// range: a cell below the limit plus one score-table entry stays below 0x7c00
// (the bound of the fp16 maximum, under the integer one of 32767 - bias); the
// few sequences that reach it are scored by the lane emulation.  Measured on a
// B200 against the lane emulation of every pair, which carries one cell per
// 32-bit lane and reads its profile through L1: 24 queries x 20,000 proteins at
// the 16-bit entry 98.9 -> 18.8 ms a call (entry pass 92 -> 12 ms), one query of
// 375 x 10,000 at 64 bits 1.51 -> 0.86 ms.
static int sw_fast_limit( const SearchRequest & req ) {
    if( req.algo != 0 || getenv( "SSA_B200_NO_FAST" ) )
        return 0;
    // the kernels also use gapO + gapE <= gapE (at the entry width) to let the
    // next row's F depend on Hdiag + V and E only
    const int goe = req.bit_width == 8 ? (int8_t) (req.gap_open + req.gap_extend) : req.gap_open + req.gap_extend;
    if( req.gap_extend > 0 || goe > 0 || goe > req.gap_extend )
        return 0;
    if( req.bit_width == 8 )
        return 255;
    int64_t most = 0;
    for( int k = 0; k < 1024; k++ ) {
        const int64_t v = (int16_t) req.matrix[k];
        if( req.bit_width == 64 && v != req.matrix[k] )
            return 0;
        most = std::max( most, v );
        // the kernels score a last block's pad columns (code 0), which the
        // 64-bit code does not have: they must not raise a score
        if( req.bit_width == 64 && k < 32 && v > 0 )
            return 0;
    }
    return most <= 8192 ? (int) (0x7c00 - 1024 - most) : 0;
}

static bool fast_eligible( const SearchRequest & req ) { return sw_fast_limit( req ) > 0; }

// The single-query kernels keep the profile in int8.
static bool fast_single_eligible( const SearchRequest & req ) {
    if( !fast_eligible( req ) )
        return false;
    for( int k = 0; k < 1024 && req.bit_width != 8; k++ )
        if( (req.bit_width == 16 ? (int16_t) req.matrix[k] : req.matrix[k]) != (int8_t) req.matrix[k] )
            return false;
    return true;
}

struct FastShape {
    int G, R, P;
    int C;      // columns per step: 1 (sw_fast_kernel) or 4 (sw_fast4_kernel)
};

constexpr uint32_t FAST_MAX_ROWS = 8192;    // longer queries run the lane emulation
constexpr uint32_t FAST_MAX_PASS_ROWS = 512; // G x R: 16 KiB profile slice per warp

// Threads per group G, rows per thread R, passes P and columns per step C for
// a query of Q rows: without a measured table, the one-column kernel with the
// smallest estimated issue cost per database column, counting the wavefront
// fill (G - 1 steps per pass) and a per-step overhead.  With a measured shape
// table for the database's bucket (tuning.cpp) the cost of a shape is
// passes x its measured cost per pass and column, over both kernels; on a
// small database that measurement includes the latency of the longest pairs,
// so it favours wide groups there.
static FastShape choose_shape( uint32_t Q, double mean_len, int bucket ) {
    FastShape best{ 0, 0, 0, 1 };
    double best_cost = 1e300;
    const int Gs[] = { 8, 16, 32 };
    const int G4s[] = { 4, 8, 16, 32 };
    const int Rs[] = { 8, 16, 24, 32 };
    const TuningTable & tt = tuning();
    bool measured = false, measured4 = false;
    for( int gi = 0; gi < 3 && tt.has_fast; gi++ )
        for( int ri = 0; ri < 4; ri++ )
            measured |= tt.fast[bucket][gi][ri] > 0;
    for( int gi = 0; gi < 4 && tt.has_fast4; gi++ )
        for( int ri = 0; ri < 4; ri++ )
            measured4 |= tt.fast4[bucket][gi][ri] > 0;
    auto fits = []( int G, int R, uint32_t Q, uint32_t * P ) {
        const uint32_t per = (uint32_t) (G * R);
        *P = (Q + per - 1) / per;
        return per <= FAST_MAX_PASS_ROWS && (uint64_t) *P * per <= FAST_MAX_ROWS;
    };
    // the model's cost units are not the table's: with only the 4-column
    // kernel measured, the one-column kernel is not a candidate
    if( measured || !measured4 ) {
        for( int gi = 0; gi < 3; gi++ ) {
            const int G = Gs[gi];
            for( int ri = 0; ri < 4; ri++ ) {
                const int R = Rs[ri];
                uint32_t P;
                if( !fits( G, R, Q, &P ) )
                    continue;
                if( measured && tt.fast[bucket][gi][ri] <= 0 )
                    continue;
                const double cost = measured ? (double) P * tt.fast[bucket][gi][ri]
                                             : (double) P * G * (mean_len + G - 1) * (8.0 * R + 24.0);
                if( cost < best_cost ) {
                    best_cost = cost;
                    best = FastShape{ G, R, (int) P, 1 };
                }
            }
        }
    }
    for( int gi = 0; gi < 4 && measured4; gi++ ) {
        const int G = G4s[gi];
        for( int ri = 0; ri < 3; ri++ ) {     // R = 8, 16, 24
            const int R = Rs[ri];
            uint32_t P;
            if( !fits( G, R, Q, &P ) || tt.fast4[bucket][gi][ri] <= 0 )
                continue;
            const double cost = (double) P * tt.fast4[bucket][gi][ri];
            if( cost < best_cost ) {
                best_cost = cost;
                best = FastShape{ G, R, (int) P, 4 };
            }
        }
    }
    return best;
}

// Which of an entry pass's pairs go to the streamed stripes (run_stream).  A group
// of threads of the entry kernel takes the passes x blocks steps of a pair one
// after the other; the whole pass takes `share` steps of every resident group,
// and a pair of more steps than that still runs when the rest is done.  On
// streamed stripes it ends sooner, but costs more instructions (stripes of 128
// rows and more, 31 steps to fill each) and host time per item.  So the pairs of
// more steps than the share, and than 64, are streamed where an estimate of the
// pass's time says that this pays; none where the longest has less than half as
// many again.  Needleman-Wunsch queries without a partner, for which the entry
// kernel computes an empty half, may go there whole.
// Calls on a B200, none streamed / always those above the share (lone
// Needleman-Wunsch queries whole) / chosen: Smith-Waterman, 30 x 20,000 nucleotide
// records of 100-1,500 0.56 / 0.83 / 0.56 ms, 300 x 1,500 proteins 0.60 / 0.35 /
// 0.36, 2 of 30 x 20,000 nucleotide records 0.91 / 1.36 / 0.92; Needleman-Wunsch,
// 30 x 100,000 reads of 80-150 0.74 / 1.85 / 0.76, 300 x 5,000 proteins 1.65 / 0.49 /
// 0.50, 32 of 30 x 1,000 nucleotide records 1.65 / 2.18 / 1.63.  Over 1,600 calls of 1 to
// 32 queries of 30-2,500 against 150-100,000 records, forced both ways, the choice
// loses 0.4% to the better of the two on average.
class StreamLine {
public:
    // Cycles of an SM sub-partition's ALU: `step` x (26 R + 20) for a warp's step of
    // R rows over a block of four columns, at least alone0 + alone1 R while it has
    // the sub-partition to itself; `stream` for a streamed step.  All fitted to the
    // calls above, each forced both ways, so that the choice between them is right.
    struct Costs {
        double step, alone0, alone1, stream;
    };
    static constexpr Costs SW_SINGLE{ 2.8, 1430, 30, 520 }, SW_PAIRS{ 2.4, 1500, 25, 225 }, NW_PAIRS{ 1.3, 700, 60, 130 };
    // A query, or pair of queries, of the entry kernel.
    struct Query {
        uint64_t passes;
        int R;                       // rows per thread
        bool one_column;             // a step is one column, not a block of four
        uint32_t rows[2];            // query lengths (0: none)
        uint32_t from;               // the units before this one are not streamed
    };
    // blocks[k]: blocks of four columns of the units (sequences, or pairs of them;
    // longest first) before unit k; a streamed item holds item_units of them.
    // lone_whole: queries without a partner may be streamed whole.
    StreamLine( const Costs & costs, bool lone_whole, int sms, int groups_per_warp, uint32_t item_units,
            const std::vector<uint64_t> & blocks, const std::vector<Query> & queries )
        : costs_( costs ), sms_( sms ), groups_( groups_per_warp ), item_units_( item_units ), blocks_( blocks ),
          queries_( queries ) {
        uint64_t steps = 0, longest = 0;
        for( const Query & q : queries_ ) {
            steps += q.passes * blocks_[units()];
            longest = std::max( longest, q.passes * unit( first( q ) ) );
        }
        const uint64_t share = std::max<uint64_t>( 64, steps / ((uint64_t) sms_ * 16 * (uint64_t) groups_) );
        // SSA_B200_STREAM_SHARE pins the line (tests)
        if( const char * pin = getenv( "SSA_B200_STREAM_SHARE" ) ) {
            line_ = strtoull( pin, nullptr, 10 );
            return;
        }
        double least = cycles( {} );
        auto consider = [&]( const Choice & c ) {
            const double t = cycles( c );
            if( t < least ) {
                least = t;
                line_ = c;
            }
        };
        const bool uneven = 2 * longest > 3 * share;
        if( uneven )
            consider( { share } );
        // (the estimate is not fitted to longer passes: 300 x 200,000 proteins, a share
        // of 2,800 steps, 9.3 ms and whole 14.2)
        if( lone_whole && share < 2048 )
            consider( { uneven ? share : UINT64_MAX, true } );
    }
    // the first unit that stays with the entry kernel
    uint32_t end( const Query & q ) const { return end( q, line_ ); }

private:
    struct Choice {
        uint64_t line = UINT64_MAX;      // pairs of more steps are streamed
        bool lone = false;               // queries without a partner whole
        Choice( uint64_t l = UINT64_MAX, bool w = false ) : line( l ), lone( w ) {}
    };
    uint32_t units() const { return (uint32_t) blocks_.size() - 1; }
    uint64_t unit( uint32_t k ) const { return k < units() ? blocks_[k + 1] - blocks_[k] : 0; }
    uint32_t first( const Query & q ) const { return std::min( q.from, units() ); }
    uint32_t end( const Query & q, const Choice & c ) const {
        const uint64_t line = c.lone && q.rows[1] == 0 ? 0 : c.line;
        uint32_t a = first( q ), b = units();
        while( a < b ) {
            const uint32_t mid = (a + b) / 2;
            if( q.passes * unit( mid ) <= line )
                b = mid;
            else
                a = mid + 1;
        }
        return a;
    }
    // The pass's time with the choice's pairs streamed: the work of a
    // sub-partition, four warps of the entry kernel side by side, and what is then
    // left of the longest kept pair; at least the longest streamed pair, or the
    // longest one beyond the kernels' range in the lane emulation.
    double cycles( const Choice & c ) const {
        double work = 0, items = 0, last = 0, tail = 0;
        auto step = [&]( const Query & q ) { return costs_.step * (26.0 * q.R + (q.one_column ? 80.0 : 20.0)); };
        for( const Query & q : queries_ ) {
            const uint32_t from = first( q ), to = end( q, c );
            const double n = to - from, cols = (double) (blocks_[to] - blocks_[from]);
            work += (double) q.passes * ((double) (blocks_[units()] - blocks_[from]) - cols) * step( q ) /
                    (groups_ * 4.0 * sms_);
            if( from )
                last = std::max( last, (q.rows[0] + 255u) / 256u * 4.0 * (double) unit( 0 ) * EMULATED_COLUMN );
            for( uint32_t rows : q.rows ) {
                if( rows == 0 || to == from )
                    continue;
                const double stripes = (rows + 127u) / 128u;
                work += stripes * (cols + 31.0 * n) / item_units_ * costs_.stream / (4.0 * sms_);
                items += n / item_units_;
                last = std::max( last, ((double) unit( from ) + STREAM_LAG * stripes) * STREAM_ALONE );
            }
        }
        for( const Query & q : queries_ ) {
            const double alone = costs_.alone0 + costs_.alone1 * q.R;
            const double left = (double) (q.passes * unit( end( q, c ) )) - work / std::max( alone, 4.0 * step( q ) );
            tail = std::max( tail, left * alone );
        }
        return ITEM * items + std::max( work + tail, last );
    }
    static constexpr double STREAM_ALONE = 200.0;     // a streamed step with the sub-partition to itself
    static constexpr double EMULATED_COLUMN = 800.0;  // a column of 256 rows in the lane emulation
    static constexpr double ITEM = 40.0;              // host time

    Costs costs_;
    int sms_, groups_;
    uint32_t item_units_;
    const std::vector<uint64_t> & blocks_;
    const std::vector<Query> & queries_;
    Choice line_;
};

void Engine::run_fast_entry( const SearchRequest & req, uint32_t nq, PairTask * next, unsigned * next_count,
        uint32_t cap ) {
    const uint32_t n_pairs = (uint32_t) db_.pair_cols.size();
    if( n_pairs == 0 )
        return;
    // shape per slot; queries too long for the shared-memory profile run the
    // exact lane emulation instead
    std::vector<FastShape> shape( nq );
    std::vector<uint32_t> rows_of( nq, 0 );
    std::vector<uint32_t> fallback;
    // classes: [columns per step 1 or 4][R = 8, 16, 24, 32]
    std::vector<std::vector<uint32_t>> by_r( 8 );
    // The table's costs of a small database include the latency of its longest
    // pairs, which are streamed here, so those of a large one choose better before
    // 50,000 sequences, as long as that shape's groups each have work: at least five
    // pairs and passes for four groups.  Where it has fewer, its more rows per thread
    // only make every pair slower (80 x 30,000 proteins: 18,944 groups of 4 threads
    // and 24 rows for 15,000 pairs, 0.68 ms; the small database's shape 0.60).
    // Mean lengths 250-500, queries of 30-2,000: calls on 30,000 / 38,000 / 49,999
    // sequences 1.22 / 1.28 / 1.33 times as fast, none slower than 0.98.  From 30,000
    // on, and for these mean lengths: at 20,000 a call gains 1.11 on average and the
    // slowest is 0.98; mean length 60 loses up to 0.54, 150 0.82, 800 0.90 and 1,500
    // 0.85 for one query or another, and keep the table's line.
    const size_t n_ne = db_.order_desc.size();
    const int bucket = db_bucket( db_.mean_len, n_ne );
    const bool middling = db_.mean_len >= 250.0 && db_.mean_len < 500.0 && n_ne >= 30000;
    const int crowded = middling ? db_bucket( db_.mean_len, std::max<size_t>( n_ne, 50000 ) ) : bucket;
    auto shape_of = [&]( uint32_t Q ) {
        const FastShape f = choose_shape( Q, db_.mean_len, crowded );
        if( crowded == bucket || !f.G ||
                4ull * n_pairs * (uint64_t) f.P >= 5ull * (uint64_t) sms_ * 16 * (uint64_t) (32 / f.G) )
            return f;
        return choose_shape( Q, db_.mean_len, bucket );
    };
    // SSA_B200_FAST_SHAPE=G,R[,C] pins the shape and the kernel (tuning, tests)
    int pin_g = 0, pin_r = 0, pin_c = 1;
    if( const char * pin = getenv( "SSA_B200_FAST_SHAPE" ) ) {
        const int n = sscanf( pin, "%d,%d,%d", &pin_g, &pin_r, &pin_c );
        const bool g_ok = pin_c == 4 ? (pin_g == 4 || pin_g == 8 || pin_g == 16 || pin_g == 32)
                                     : (pin_g == 8 || pin_g == 16 || pin_g == 32);
        const int r_max = pin_c == 4 ? 24 : 32;
        if( n < 2 || (n == 3 && pin_c != 1 && pin_c != 4) || !g_ok || pin_r < 8 || pin_r > r_max || pin_r % 8 )
            pin_g = pin_r = 0;
    }
    for( uint32_t s = 0; s < nq; s++ ) {
        shape[s] = shape_of( h_qlen_[s] );
        if( pin_g && shape[s].G ) {
            const uint32_t per = (uint32_t) (pin_g * pin_r);
            const uint32_t P = (h_qlen_[s] + per - 1) / per;
            if( per <= FAST_MAX_PASS_ROWS && (uint64_t) P * per <= FAST_MAX_ROWS )
                shape[s] = FastShape{ pin_g, pin_r, (int) P, pin_c };
        }
        if( shape[s].G == 0 ) {
            fallback.push_back( s );
            continue;
        }
        rows_of[s] = (uint32_t) (shape[s].G * shape[s].R * shape[s].P);
        by_r[(shape[s].C == 4 ? 4 : 0) + shape[s].R / 8 - 1].push_back( s );
    }
    // profiles: one 32 x rows int8 table per slot
    std::vector<uint64_t> prof_off( nq, 0 );
    uint64_t total = 0;
    std::vector<uint32_t> slots;
    for( auto & v : by_r )
        for( uint32_t s : v ) {
            prof_off[s] = total;
            total += 32ull * rows_of[s];
            slots.push_back( s );
        }
    const size_t n_shaped = slots.size();
    for( uint32_t s : fallback )
        slots.push_back( s );
    d_prof8_.ensure( total + 16 );
    const uint64_t * dev_prof_off = stage_.add( prof_off.data(), nq, stream_ );
    const uint32_t * dev_rows = stage_.add( rows_of.data(), nq, stream_ );
    const uint32_t * dev_slots = stage_.add( slots.data(), slots.size(), stream_ );
    // work units: ranges of length-sorted pairs holding about equal numbers
    // of columns, the longest first; every query of a class gets every range.
    // A warp takes one unit at a time and runs its pairs 32 / G at a time, so
    // a unit holds at least one such round for the smallest group of the call
    // (no idle groups) and, where the columns allow, no more: on a small
    // database the longest pairs then run side by side in separate warps
    // instead of one after another in the same warp.
    const uint64_t total_cols = 4 * db_.pair_blocks[n_pairs];
    int g_min = 32;
    for( uint32_t s = 0; s < nq; s++ )
        if( shape[s].G )
            g_min = std::min( g_min, shape[s].G );
    const uint32_t min_pairs = 32u / (uint32_t) g_min;
    const uint64_t want_units = (uint64_t) sms_ * 16 * 24;   // ~24 units per resident warp
    const uint64_t target = std::max<uint64_t>( 1, total_cols * std::max<size_t>( 1, n_shaped ) / want_units );
    std::vector<uint32_t> bounds{ 0 };
    {
        uint64_t acc = 0;
        uint32_t cnt = 0;
        for( uint32_t pi = 0; pi < n_pairs; pi++ ) {
            acc += db_.pair_cols[pi];
            cnt++;
            if( acc >= target && cnt >= min_pairs ) {
                bounds.push_back( pi + 1 );
                acc = 0;
                cnt = 0;
            }
        }
        if( bounds.back() != n_pairs )
            bounds.push_back( n_pairs );
    }
    const uint32_t n_chunks = (uint32_t) bounds.size() - 1;
    std::vector<uint16_t> group_of( nq, 32 );
    for( uint32_t s = 0; s < nq; s++ )
        if( shape[s].G )
            group_of[s] = (uint16_t) shape[s].G;
    const uint32_t * dev_bounds = stage_.add( bounds.data(), bounds.size(), stream_ );
    const uint16_t * dev_group = stage_.add( group_of.data(), nq, stream_ );
    stage_.send( stream_ );
    if( n_shaped ) {
        CUDA_CHECK( launch_build_profile8( d_qcodes_.as<uint8_t>(), d_qoff_.as<uint64_t>(), d_qlen_.as<uint32_t>(),
                dev_slots, (uint32_t) n_shaped, dev_rows, d_matrix_.as<int64_t>(),
                d_prof8_.as<int8_t>(), dev_prof_off, stream_ ) );
        launches_++;
    }
    const uint32_t cols_max = ((db_.max_len + 7u) & ~7u) + 8;
    unsigned * redo_count = d_counts_.as<unsigned>() + 5;
    if( req.bit_width != 8 )
        CUDA_CHECK( cudaMemsetAsync( redo_count, 0, sizeof(unsigned), stream_ ) );
    // the longest pairs on streamed stripes
    uint32_t pair_skip = 0;
    std::vector<SwStreamItem> items;
    if( nq == 1 && n_shaped == 1 && (!pin_g || getenv( "SSA_B200_STREAM_SHARE" )) ) {
        const FastShape & fs = shape[0];
        const std::vector<StreamLine::Query> queries{ { (uint64_t) fs.P, fs.R, fs.C != 4, { h_qlen_[0], 0 }, 0 } };
        pair_skip = StreamLine( StreamLine::SW_SINGLE, false, sms_, 32 / fs.G, 1, db_.pair_blocks, queries )
                .end( queries[0] );
        for( uint32_t k = 0; k < pair_skip; k++ )
            items.push_back( SwStreamItem{ 0, db_.pair_a[k], db_.pair_b[k], 0 } );
    }
    if( getenv( "SSA_B200_TIMING" ) )
        fprintf( stderr, "[ssa timing] entry pass: %zu items streamed\n", items.size() );
    CUDA_CHECK( cudaEventRecord( ev_ready_, stream_ ) );
    if( pair_skip ) {
        PassSink lists{};
        lists.next = next;
        lists.next_count = next_count;
        lists.next_cap = cap;
        if( req.bit_width != 8 ) {
            lists.redo = d_list_b_.as<PairTask>();
            lists.redo_count = redo_count;
            lists.redo_cap = cap;
        }
        CUDA_CHECK( cudaStreamWaitEvent( long_stream_, ev_ready_, 0 ) );
        run_stream( req, items, lists, long_stream_ );
        CUDA_CHECK( cudaEventRecord( ev_long_, long_stream_ ) );
        CUDA_CHECK( cudaStreamWaitEvent( stream_, ev_long_, 0 ) );
    }
    size_t class_first = 0;
    for( int ci = 0; ci < 8; ci++ ) {
        const std::vector<uint32_t> & cls = by_r[ci];
        if( cls.empty() )
            continue;
        const bool four = ci >= 4;
        const int ri = ci % 4;                 // classes of equal R share a stream
        const int R = 8 * (ri + 1);
        bool multi = false;
        uint32_t slice_rows = 0;
        for( uint32_t s : cls ) {
            multi |= shape[s].P > 1;
            slice_rows = std::max( slice_rows, (uint32_t) (shape[s].G * R) );
        }
        {
            std::map<int, uint32_t> by_g;
            for( uint32_t s : cls )
                by_g[shape[s].G]++;
            for( auto & kv : by_g )
                last_shapes_.push_back( { four ? "sw_fast4" : "sw_fast", kv.first, R, kv.second, bucket } );
        }
        auto launch = [&]( const FastParams & fp, int g, int * per ) {
            return four ? launch_sw_fast4( R, fp, g, class_stream_[ri], per )
                        : launch_sw_fast( R, fp, g, class_stream_[ri], per );
        };
        FastParams p{};
        p.slice_rows = slice_rows;
        int per_sm = 0;
        CUDA_CHECK( launch( p, 0, &per_sm ) );
        // SSA_B200_FAST_CTAS=n caps the resident CTAs per SM (tuning)
        if( const char * cap_env = getenv( "SSA_B200_FAST_CTAS" ) )
            per_sm = std::min( per_sm, std::max( 1, atoi( cap_env ) ) );
        const int grid = sms_ * std::max( 1, per_sm );
        // after the streamed pairs, which are the longest: a grid that fills the GPU
        // before they start would have them wait for its end
        CUDA_CHECK( cudaStreamWaitEvent( class_stream_[ri], pair_skip ? ev_items_ : ev_ready_, 0 ) );
        unsigned long long * unit_counter = d_counts_.as<unsigned long long>() + 8 + ri;   // bytes 64..95
        CUDA_CHECK( cudaMemsetAsync( unit_counter, 0, sizeof(unsigned long long), class_stream_[ri] ) );
        p.pair_res = d_pair_res_.as<uint8_t>();
        p.pair_off = d_pair_off_.as<uint64_t>();
        p.pair_cols = d_pair_cols_.as<uint32_t>();
        p.pair_ids = d_pair_ids_.as<uint2>();
        p.prof8 = d_prof8_.as<int8_t>();
        p.prof8_off = dev_prof_off;
        p.slot_group = dev_group;
        p.slot_rows = dev_rows;
        p.unit_slots = dev_slots + class_first;
        p.n_class = (uint32_t) cls.size();
        p.chunk_bounds = dev_bounds;
        p.n_units = (uint64_t) n_chunks * cls.size();
        p.unit_counter = unit_counter;
        p.gap_oe = req.bit_width == 8 ? (int8_t) (req.gap_open + req.gap_extend) : req.gap_open + req.gap_extend;
        p.gap_e = req.gap_extend;
        p.limit = sw_fast_limit( req );
        p.pair_skip = pair_skip;
        if( req.bit_width != 8 ) {
            p.sink.redo = d_list_b_.as<PairTask>();
            p.sink.redo_count = redo_count;
            p.sink.redo_cap = cap;
        }
        p.sink.score = score_sink();
        p.sink.score_stride = db_.n_ids;
        p.sink.next = next;
        p.sink.next_count = next_count;
        p.sink.next_cap = cap;
        p.sink.error_flags = d_counts_.as<unsigned>() + 2;
        if( multi ) {
            // a scratch row per group: 4 groups per warp (8 in the 4-column kernel)
            p.scratch = (int4 *) d_scratch_fast_[ci].ensure( (size_t) grid * (FAST_THREADS / 32) * (four ? 8 : 4) *
                    cols_max * sizeof(int4) );
            p.scratch_cols = cols_max;
        }
        CUDA_CHECK( launch( p, grid, nullptr ) );
        launches_++;
        CUDA_CHECK( cudaEventRecord( ev_class_[ri], class_stream_[ri] ) );
        CUDA_CHECK( cudaStreamWaitEvent( stream_, ev_class_[ri], 0 ) );
        class_first += cls.size();
    }
    if( !fallback.empty() ) {
        const uint64_t n_ne = db_.order_desc.size();
        run_pass( 0, req.bit_width, req, nq, nullptr, (uint64_t) fallback.size() * n_ne, true, next, next_count, cap,
                dev_slots + n_shaped, (uint32_t) fallback.size() );
    }
}

// Batches: queries sorted by length are paired, the two queries of a pair
// share the 16x2 lanes (sw_qpair_kernel.cu).  Rows per thread R for a pair of
// Q rows (the longer query): the smallest estimated time per column pair,
// passes x cost(R), with QP_G x R rows per pass.  cost(R) is the measured
// device time of one pass per column pair on a B200 (relative units; 64
// queries of 375 residues against 10,000 sequences, each R pinned): R = 16
// pays for 2-way shared-memory bank conflicts inside a group, R = 28 for a
// few spilled registers.
// The costs come from the measured shape table (tuning.cpp): per pass and
// database column of a query pair, for each rows-per-thread R and resident
// CTAs per SM (4 or 5); the smallest passes x cost wins.  pinned_r / pinned_mb
// (SSA_B200_QP_R, SSA_B200_QP_MB) force a shape, as the tuner does.
struct QpVariant {
    int mb;         // resident CTAs per SM
    int cols;       // columns per step
    bool hmax;      // running maximum in fp16x2 (4 columns, 4 CTAs per SM)
    bool g8;        // 8 threads of 12 rows per sequence (R = 24, 4 columns)
    double cost;    // measured cost, 0 = none
};

// The cheapest measured variant of the query-pair kernel for rows-per-thread
// R (pinned_mb / pinned_c / pinned_h / pinned_g8 force one; pinned_h and
// pinned_g8: 0 or 1, -1 = free).
static QpVariant qpair_variant( int bucket, int R, int pinned_mb, int pinned_c, int pinned_h, int pinned_g8 ) {
    QpVariant best{ 4, 2, false, false, 0 };
    for( int mi = 0; mi < 2; mi++ )
        for( int vi = 0; vi < 4; vi++ ) {
            const int mb = 4 + mi, cols = vi ? 4 : 2;
            const bool hm = vi == 2, g8 = vi == 3;
            if( (hm && mb != 4) || (g8 && R != 24) )
                continue;
            if( (pinned_mb == 4 || pinned_mb == 5) && mb != pinned_mb )
                continue;
            if( (pinned_c == 2 || pinned_c == 4) && cols != pinned_c )
                continue;
            if( pinned_h >= 0 && hm != (pinned_h == 1) )
                continue;
            if( pinned_g8 >= 0 && g8 != (pinned_g8 == 1) )
                continue;
            const double c = tuning().qpair[bucket][R / 4 - 4][mi][vi];
            if( c > 0 && (best.cost <= 0 || c < best.cost) )
                best = QpVariant{ mb, cols, hm, g8, c };
        }
    if( best.cost <= 0 ) {
        if( pinned_mb == 4 || pinned_mb == 5 )
            best.mb = pinned_mb;
        if( pinned_c == 2 || pinned_c == 4 )
            best.cols = pinned_c;
        if( pinned_h == 1 ) {
            best.cols = 4;
            best.mb = 4;
            best.hmax = true;
        }
        else if( pinned_g8 == 1 && R == 24 ) {
            best.cols = 4;
            best.g8 = true;
        }
    }
    return best;
}

static int choose_qpair_rows( uint32_t Q, uint32_t * passes, int pinned, int bucket, int pinned_mb, int pinned_c,
        int pinned_h, int pinned_g8 ) {
    static const int rs[4] = { 16, 20, 24, 28 };
    int best_r = 0;
    double best_cost = 1e300;
    for( int i = 0; i < 4; i++ ) {
        const int R = rs[i];
        if( pinned && R != pinned )
            continue;
        const uint32_t per = (uint32_t) (QP_G * R);
        const uint32_t P = std::max<uint32_t>( 1, (Q + per - 1) / per );
        if( (uint64_t) P * per > FAST_MAX_ROWS )
            continue;
        const double unit = qpair_variant( bucket, R, pinned_mb, pinned_c, pinned_h, pinned_g8 ).cost;
        if( unit <= 0 && !pinned )
            continue;                   // not measured
        const double c = (double) P * (unit > 0 ? unit : 1.0);
        if( c < best_cost ) {
            best_cost = c;
            best_r = R;
            *passes = P;
        }
    }
    if( best_r == 0 && pinned )         // the pinned R does not fit this query
        return choose_qpair_rows( Q, passes, 0, bucket, pinned_mb, pinned_c, pinned_h, pinned_g8 );
    if( best_r == 0 ) {                 // an empty table: 20 rows per thread
        best_r = 20;
        *passes = std::max<uint32_t>( 1, (Q + QP_G * 20 - 1) / (QP_G * 20) );
    }
    return best_r;
}

// The counters of a pass on the host: [0] re-queued pairs, [1] those of the
// 16-bit pass, [2] error flags, [5] pairs for the lane emulation.  head: also
// the first entries of list A, which are all of them in most calls, and
// (scores_to) that many bytes of scores.  One wait for all.
const unsigned * Engine::read_counts( bool head, void * scores_to, size_t score_bytes ) {
    unsigned * c = (unsigned *) h_counts_.ensure( 64 + LIST_HEAD * sizeof(PairTask) );
    CUDA_CHECK( cudaMemcpyAsync( c, d_counts_.p, 6 * sizeof(unsigned), cudaMemcpyDeviceToHost, stream_ ) );
    if( head )
        CUDA_CHECK( cudaMemcpyAsync( (char *) c + 64, d_list_a_.p,
                std::min<size_t>( d_list_a_.bytes, LIST_HEAD * sizeof(PairTask) ), cudaMemcpyDeviceToHost, stream_ ) );
    if( scores_to )
        CUDA_CHECK( cudaMemcpyAsync( scores_to, d_score_.p, score_bytes, cudaMemcpyDeviceToHost, stream_ ) );
    CUDA_CHECK( cudaStreamSynchronize( stream_ ) );
    return c;
}

// The pairs that the 16x2 kernels left out of their range (16- and 64-bit
// passes), by the lane emulation.  c: the pass's counters; returns them as they
// are afterwards.
const unsigned * Engine::run_redo( const SearchRequest & req, uint32_t nq, const unsigned * c, PairTask * next,
        unsigned * next_count, uint32_t cap, const PairTask * redo_list, uint32_t redo_cap ) {
    const uint32_t n_redo = std::min( c[5], redo_cap );
    if( req.bit_width == 8 || n_redo == 0 )
        return c;
    run_pass( req.algo, req.bit_width, req, nq, redo_list, n_redo, false, next, next_count, cap );
    return read_counts( true );
}

void Engine::run_qpair_entry( const SearchRequest & req, uint32_t nq, PairTask * next, unsigned * next_count,
        uint32_t cap, PairTask * redo_list, const std::vector<uint32_t> * slots, uint32_t seq_lo, uint32_t seq_hi,
        bool marked ) {
    // the sequences order_desc[seq_lo, seq_hi) (all by default)
    const uint32_t n_all = (uint32_t) db_.order_desc.size();
    const uint32_t lo = std::min( seq_lo, n_all ), hi = std::min( seq_hi, n_all );
    const uint32_t n_seq = hi - lo;
    if( n_seq == 0 )
        return;
    const bool nw = req.algo == 1;
    // pair the queries that fit, longest first; longer ones run the emulation
    std::vector<uint32_t> fit, fallback;
    if( slots ) {
        for( uint32_t s : *slots )
            (h_qlen_[s] <= FAST_MAX_ROWS ? fit : fallback).push_back( s );
    }
    else {
        for( uint32_t s = 0; s < nq; s++ )
            (h_qlen_[s] <= FAST_MAX_ROWS ? fit : fallback).push_back( s );
    }
    std::stable_sort( fit.begin(), fit.end(), [&]( uint32_t a, uint32_t b ) { return h_qlen_[a] > h_qlen_[b]; } );
    const uint32_t n_qp = (uint32_t) ((fit.size() + 1) / 2);
    // SSA_B200_QP_R=16|20|24|28 and SSA_B200_QP_MB=4|5 pin the shape (tuning)
    const char * pin = getenv( "SSA_B200_QP_R" );
    const int pinned_r = pin ? atoi( pin ) : 0;
    const char * pin_mb = getenv( "SSA_B200_QP_MB" );
    const int pinned_mb = pin_mb ? atoi( pin_mb ) : 0;
    const char * pin_c = getenv( "SSA_B200_QP_C" );      // 2|4 columns per step
    const int pinned_c = pin_c ? atoi( pin_c ) : 0;
    const char * pin_h = getenv( "SSA_B200_QP_HMAX" );   // 0|1 running maximum in fp16x2
    const int pinned_h = pin_h ? (atoi( pin_h ) ? 1 : 0) : -1;
    const char * pin_g8 = getenv( "SSA_B200_QP_G8" );    // 0|1 8 threads per sequence (R = 24)
    const int pinned_g8 = pin_g8 ? (atoi( pin_g8 ) ? 1 : 0) : -1;
    // the database bucket of the shape table: these sequences' mean length and count
    uint64_t seq_res = 0;
    for( uint32_t i = lo; i < hi; i++ )
        seq_res += db_.len[db_.order_desc[i]];
    const int bucket = db_bucket( (double) seq_res / std::max<uint32_t>( 1, n_seq ), n_seq );
    std::vector<uint32_t> qp_slots( 2 * std::max<uint32_t>( 1, n_qp ), 0xffffffffu );
    std::vector<uint32_t> qp_rows( std::max<uint32_t>( 1, n_qp ), 0 );
    std::vector<uint64_t> qp_off( std::max<uint32_t>( 1, n_qp ), 0 );
    std::vector<std::vector<uint32_t>> by_r( 4 );     // R = 16, 20, 24, 28
    uint64_t total = 0;
    for( uint32_t i = 0; i < n_qp; i++ ) {
        qp_slots[2 * i] = fit[2 * i];
        if( 2 * i + 1 < fit.size() )
            qp_slots[2 * i + 1] = fit[2 * i + 1];
        uint32_t P = 1;
        const int R = choose_qpair_rows( h_qlen_[fit[2 * i]], &P, pinned_r, bucket, pinned_mb, pinned_c, pinned_h,
                pinned_g8 );
        qp_rows[i] = P * (uint32_t) (QP_G * R);
        by_r[R / 4 - 4].push_back( i );
    }
    // NW: per pair, the longest sequence whose matrix (padded rows and the last
    // block's pad columns included) stays within +-30000: every step of a path
    // changes a value by at most m, and a path has at most rows + L + 4 steps
    // and two gap openings
    std::vector<uint32_t> qp_lmax( std::max<uint32_t>( 1, n_qp ), 0 );
    int64_t nw_step = std::max<int64_t>( 1, std::llabs( (int64_t) req.gap_extend ) );
    const int64_t nw_budget = 30000 - 2 * std::llabs( (int64_t) req.gap_open );
    bool nw_table8 = true;       // the scores at the pass width fit int8
    if( nw ) {
        for( int c = 0; c < 1024; c++ ) {
            const int64_t v = (int16_t) req.matrix[c];
            nw_step = std::max<int64_t>( nw_step, std::llabs( v ) );
            nw_table8 = nw_table8 && v == (int8_t) v;
        }
        for( uint32_t i = 0; i < n_qp; i++ ) {
            const int64_t l = nw_budget / nw_step - (int64_t) qp_rows[i] - 4;
            qp_lmax[i] = (uint32_t) std::max<int64_t>( 0, l );
        }
    }
    // Needleman-Wunsch: 4 columns per step unless SSA_B200_QP_C=2 pins the
    // 2-column kernel (4 resident CTAs per SM either way)
    QpVariant variant[4];
    for( int ri = 0; ri < 4; ri++ )
        variant[ri] = nw ? QpVariant{ 4, pinned_c == 2 ? 2 : 4, false, false, 0 }
                         : qpair_variant( bucket, 4 * (ri + 4), pinned_mb, pinned_c, pinned_h, pinned_g8 );
    // profiles (16-byte aligned: rows % 16 == 0): QP_CODES x rows words per
    // pair, twice that in the layout of the 4-column kernels with 4 threads
    std::vector<uint32_t> lane_rows( std::max<uint32_t>( 1, n_qp ), 0 );
    for( int ri = 0; ri < 4; ri++ )
        for( uint32_t i : by_r[ri] ) {
            qp_off[i] = total;
            lane_rows[i] = variant[ri].cols == 2 ? 0 : variant[ri].g8 ? 12 : 4 * (ri + 4);
            total += (uint64_t) QP_CODES * qp_rows[i] * (lane_rows[i] && !variant[ri].g8 ? 2 : 1);
        }
    std::vector<uint32_t> units;                  // pairs grouped by class, longest first
    for( auto & v : by_r ) {
        std::stable_sort( v.begin(), v.end(), [&]( uint32_t a, uint32_t b ) { return qp_rows[a] > qp_rows[b]; } );
        units.insert( units.end(), v.begin(), v.end() );
    }
    d_qp_prof_.ensure( std::max<uint64_t>( total, 4 ) * sizeof(uint32_t) );
    const uint64_t * dev_off = stage_.add( qp_off.data(), qp_off.size(), stream_ );
    const uint32_t * dev_rows = stage_.add( qp_rows.data(), qp_rows.size(), stream_ );
    const uint32_t * dev_lane_rows = stage_.add( lane_rows.data(), lane_rows.size(), stream_ );
    const uint32_t * dev_qslots = stage_.add( qp_slots.data(), qp_slots.size(), stream_ );
    const uint32_t * dev_units = stage_.add( units.data(), units.size(), stream_ );
    const uint32_t * dev_lmax = stage_.add( qp_lmax.data(), qp_lmax.size(), stream_ );
    // Pairs outside the kernels' range, for the lane emulation (the 8-bit entry has
    // none).  Needleman-Wunsch: the sequences longer than a pair of queries' limit,
    // which the emulation scores beside the entry pass (run_beyond); of a marked pass
    // only the device knows which of them it wants.
    const bool redo = nw ? marked : req.bit_width != 8;
    unsigned * redo_count = d_counts_.as<unsigned>() + 5;
    if( req.bit_width != 8 )
        CUDA_CHECK( cudaMemsetAsync( redo_count, 0, sizeof(unsigned), stream_ ) );
    // work units: ranges of length-sorted sequences (multiples of what a CTA
    // holds side by side) with about equal numbers of columns, the longest
    // first; every pair of a class gets every range.  A CTA takes one unit at a
    // time (a warp, in the 2-column kernels).
    std::vector<uint64_t> & blocks = blocks_before_;     // of four columns, of the sequences before each
    blocks.resize( n_seq + 1 );
    blocks[0] = 0;
    for( uint32_t k = 0; k < n_seq; k++ )
        blocks[k + 1] = blocks[k] + (db_.len[db_.order_desc[lo + k]] + 3u) / 4u;
    const uint64_t total_cols = 4 * blocks[n_seq];
    constexpr uint32_t CTA_SEQS = QP_THREADS_PER_CTA / QP_G;
    const uint64_t want_units = (uint64_t) sms_ * 16 * 24;
    const uint64_t target = std::max<uint64_t>( 1, total_cols * std::max<uint32_t>( 1, n_qp ) / want_units );
    std::vector<uint32_t> bounds{ 0 };
    {
        uint64_t acc = 0;
        for( uint32_t i = 0; i < n_seq; i++ ) {
            acc += 4 * (blocks[i + 1] - blocks[i]);
            if( acc >= target && (i + 1) % CTA_SEQS == 0 ) {
                bounds.push_back( i + 1 );
                acc = 0;
            }
        }
        if( bounds.back() != n_seq )
            bounds.push_back( n_seq );
    }
    const uint32_t n_chunks = (uint32_t) bounds.size() - 1;
    const uint32_t * dev_bounds = stage_.add( bounds.data(), bounds.size(), stream_ );
    stage_.send( stream_ );
    if( n_qp ) {
        CUDA_CHECK( launch_build_profile_qp( d_qcodes_.as<uint8_t>(), d_qoff_.as<uint64_t>(), d_qlen_.as<uint32_t>(),
                dev_qslots, n_qp, dev_rows, dev_lane_rows, d_matrix_.as<int64_t>(),
                d_qp_prof_.as<uint32_t>(), dev_off, req.bit_width == 8 ? 8 : 16, stream_ ) );
        launches_++;
    }
    CUDA_CHECK( cudaEventRecord( ev_ready_, stream_ ) );
    const uint32_t scratch_cols = (((db_.max_len + 3u) & ~3u) >> 1) + 2u;
    const bool timing = getenv( "SSA_B200_TIMING" ) != nullptr;
    // the longest sequences against the longest queries on streamed stripes
    const bool table8 = nw ? nw_table8 : fast_single_eligible( req );
    const bool pinned = pin || pin_mb || pin_c || pin_h || pin_g8;      // a pinned shape keeps the entry kernel
    std::vector<uint2> qp_skip( std::max<uint32_t>( 1, n_qp ), make_uint2( 0, 0 ) );
    std::vector<SwStreamItem> items;
    if( n_qp && table8 && (!pinned || getenv( "SSA_B200_STREAM_SHARE" )) ) {
        std::vector<StreamLine::Query> queries( n_qp );
        for( int ri = 0; ri < 4; ri++ )
            for( uint32_t i : by_r[ri] ) {
                StreamLine::Query & q = queries[i];
                q = StreamLine::Query{ qp_rows[i] / (uint64_t) (QP_G * 4 * (ri + 4)), 4 * (ri + 4), false, { 0, 0 }, 0 };
                for( int h = 0; h < 2; h++ )
                    if( qp_slots[2 * i + h] != 0xffffffffu )
                        q.rows[h] = h_qlen_[qp_slots[2 * i + h]];
                // Needleman-Wunsch: within the exact range for stripes of 128
                // rows (the entry kernel sends the longer ones to the redo list)
                const int64_t most = nw ? nw_budget / nw_step - (int64_t) ((q.rows[0] + 127u) & ~127u) - 4 : INT64_MAX;
                while( q.from < n_seq && (int64_t) db_.len[db_.order_desc[lo + q.from]] > most )
                    q.from++;
            }
        const StreamLine line( nw ? StreamLine::NW_PAIRS : StreamLine::SW_PAIRS, nw, sms_, QP_GPW, 2, blocks, queries );
        for( uint32_t i = 0; i < n_qp; i++ ) {
            const uint32_t from = queries[i].from;
            uint32_t to = line.end( queries[i] );
            if( to < n_seq && ((to - from) & 1u) )
                to++;
            qp_skip[i] = make_uint2( from, to );
            for( int h = 0; h < 2; h++ ) {
                const uint32_t slot = qp_slots[2 * i + h];
                for( uint32_t k = from; k < to && slot != 0xffffffffu; k += 2 )
                    items.push_back( SwStreamItem{ slot, db_.order_desc[lo + k],
                            k + 1 < to ? db_.order_desc[lo + k + 1] : 0xffffffffu, 0 } );
            }
        }
    }
    if( timing )
        fprintf( stderr, "[ssa timing] entry pass: %zu items streamed\n", items.size() );
    const uint2 * dev_skip = stage_.add( qp_skip.data(), qp_skip.size(), stream_ );
    stage_.send( stream_ );
    CUDA_CHECK( cudaEventRecord( ev_ready_, stream_ ) );
    // The pairs beyond the range, longest first.  A warp of the emulation takes all of
    // a pair's rows and columns one after the other, so a few long pairs run beside
    // the entry kernels; more than four per resident warp keep the GPU busy alone and
    // follow, because the entry kernels' shared memory leaves them little L1 cache.
    // After the pass / beside it, one query against proteins of mean length 350
    // (calls on a B200): 64-bit entry 1,300 x 1,000 6.4 / 4.0 ms, 2,000 x 10,000 12.2 /
    // 7.9; 16-bit entry 2,000 x 10,000 15.4 / 11.6; 15,289 pairs of 2,500 28.0 / 30.6.
    uint64_t n_beyond = 0;
    std::vector<uint32_t> beyond_end( n_qp, 0 );     // the first sequence within each pair's range
    for( uint32_t i = 0; i < n_qp && nw && !marked; i++ ) {
        beyond_end[i] = (uint32_t) (std::partition_point( db_.order_desc.begin() + lo, db_.order_desc.begin() + hi,
                [&]( uint32_t id ) { return db_.len[id] > qp_lmax[i]; } ) - (db_.order_desc.begin() + lo));
        n_beyond += (uint64_t) beyond_end[i] * (qp_slots[2 * i + 1] == 0xffffffffu ? 1 : 2);
    }
    const bool beside = n_beyond <= (uint64_t) sms_ * 64;
    // in lists of at most this many, so that a query longer than the range itself,
    // whose pairs are all beyond, takes no memory of the database's size
    const size_t beyond_cap = std::min<size_t>( cap, (size_t) 1 << 20 );
    auto run_beyond = [&]() {
        std::vector<PairTask> tasks;
        auto flush = [&]() {
            if( tasks.empty() )
                return;
            const PairTask * dev;
            if( beside ) {
                dev = stage_.add( tasks.data(), tasks.size(), stream_ );
            }
            else {
                dev = (const PairTask *) d_list_c_.ensure( beyond_cap * sizeof(PairTask) );
                CUDA_CHECK( cudaMemcpyAsync( d_list_c_.p, tasks.data(), tasks.size() * sizeof(PairTask),
                        cudaMemcpyHostToDevice, stream_ ) );
            }
            run_pass( 1, req.bit_width, req, nq, dev, tasks.size(), false, next, next_count, cap );
            tasks.clear();
        };
        const uint32_t last = n_qp ? *std::max_element( beyond_end.begin(), beyond_end.end() ) : 0;
        for( uint32_t k = 0; k < last; k++ )
            for( uint32_t i = 0; i < n_qp; i++ )
                for( int h = 0; h < 2 && k < beyond_end[i] && (k < qp_skip[i].x || k >= qp_skip[i].y); h++ ) {
                    if( qp_slots[2 * i + h] == 0xffffffffu )
                        continue;
                    tasks.push_back( PairTask{ qp_slots[2 * i + h], db_.order_desc[lo + k], 0, 0 } );
                    if( tasks.size() == beyond_cap )
                        flush();
                }
        flush();
    };
    if( beside )
        run_beyond();
    if( !items.empty() ) {
        PassSink lists{};
        lists.next = next;
        lists.next_count = next_count;
        lists.next_cap = cap;
        if( redo ) {
            lists.redo = redo_list;
            lists.redo_count = redo_count;
            lists.redo_cap = cap;
        }
        CUDA_CHECK( cudaStreamWaitEvent( long_stream_, ev_ready_, 0 ) );
        run_stream( req, items, lists, long_stream_, marked );
        CUDA_CHECK( cudaEventRecord( ev_long_, long_stream_ ) );
        CUDA_CHECK( cudaStreamWaitEvent( stream_, ev_long_, 0 ) );
    }
    // classes launched heaviest first (most rows per thread: the longest
    // queries), so that the last class to finish is the lightest
    bool launched[4] = { false, false, false, false };
    size_t class_start[4] = { 0, 0, 0, 0 };
    for( int ri = 1; ri < 4; ri++ )
        class_start[ri] = class_start[ri - 1] + by_r[ri - 1].size();
    for( int k = 0; k < 4; k++ ) {
        const int ri = 3 - k;
        const size_t class_first = class_start[ri];
        const std::vector<uint32_t> & cls = by_r[ri];
        bool work = false;       // sequences that the streamed stripes leave
        for( uint32_t i : cls )
            work = work || qp_skip[i].y - qp_skip[i].x < n_seq;
        if( !work )
            continue;
        launched[ri] = true;
        const int R = 4 * (ri + 4);
        const QpVariant var = variant[ri];
        const int mb = var.mb;
        auto launch = [&]( const QPairParams & pp, int grid, int * per ) {
            if( nw )
                return var.cols == 4 ? launch_nw_qpair4( R, pp, grid, class_stream_[ri], per )
                                     : launch_nw_qpair( R, pp, grid, class_stream_[ri], per );
            return var.cols == 4 ? launch_sw_qpair4( R, mb, var.hmax, var.g8, pp, grid, class_stream_[ri], per )
                                 : launch_sw_qpair( R, mb, pp, grid, class_stream_[ri], per );
        };
        bool multi = false;
        for( uint32_t i : cls )
            multi |= qp_rows[i] > (uint32_t) (QP_G * R);
        last_shapes_.push_back( { nw ? (var.cols == 4 ? "nw_qpair4" : "nw_qpair") : var.hmax ? "sw_qpair4h"
                : var.g8 ? "sw_qpair4g8"
                : var.cols == 4 ? "sw_qpair4" : "sw_qpair", R, mb,
                (uint32_t) cls.size(), bucket } );
        QPairParams p{};
        int per_sm = 0;
        CUDA_CHECK( launch( p, 0, &per_sm ) );
        const int grid = sms_ * std::max( 1, per_sm );
        // after the streamed pairs, which are the longest: a grid that fills the GPU
        // before they start would have them wait for its end
        CUDA_CHECK( cudaStreamWaitEvent( class_stream_[ri], !items.empty() ? ev_items_ : ev_ready_, 0 ) );
        unsigned long long * unit_counter = d_counts_.as<unsigned long long>() + 8 + ri;   // bytes 64..95
        CUDA_CHECK( cudaMemsetAsync( unit_counter, 0, sizeof(unsigned long long), class_stream_[ri] ) );
        p.db = db_view();
        p.order = d_order_.as<uint32_t>() + lo;
        p.prof = d_qp_prof_.as<uint32_t>();
        p.prof_off = dev_off;
        p.qp_slots = dev_qslots;
        p.qp_rows = dev_rows;
        p.unit_pairs = dev_units + class_first;
        p.n_class = (uint32_t) cls.size();
        p.n_chunks = n_chunks;
        p.chunk_bounds = dev_bounds;
        p.n_units = (uint64_t) n_chunks * cls.size();
        p.unit_counter = unit_counter;
        // the 8-bit Smith-Waterman lanes add the int8 truncation of gapO + gapE
        p.gap_oe = req.bit_width != 8 ? req.gap_open + req.gap_extend : (int8_t) (req.gap_open + req.gap_extend);
        p.gap_e = req.gap_extend;
        p.limit = nw ? 0 : sw_fast_limit( req );
        p.sink.score = score_sink();
        p.sink.score_stride = db_.n_ids;
        p.sink.next = next;
        p.sink.next_count = next_count;
        p.sink.next_cap = cap;
        p.sink.error_flags = d_counts_.as<unsigned>() + 2;
        if( multi ) {
            p.scratch = (int4 *) d_scratch_fast_[ri].ensure( (size_t) grid * (QP_THREADS_PER_CTA / 32) * QP_GPW *
                    scratch_cols * sizeof(int4) );
            p.scratch_cols = scratch_cols;
        }
        p.gap_open = req.gap_open;
        p.qlen = d_qlen_.as<uint32_t>();
        p.qp_lmax = dev_lmax;
        p.marked_only = marked;
        p.qp_skip = dev_skip;
        if( redo ) {
            p.sink.redo = redo_list;
            p.sink.redo_count = redo_count;
            p.sink.redo_cap = cap;
        }
        if( timing )
            CUDA_CHECK( cudaEventRecord( ev_cls_t_[2 * ri], class_stream_[ri] ) );
        CUDA_CHECK( launch( p, grid, nullptr ) );
        launches_++;
        if( timing )
            CUDA_CHECK( cudaEventRecord( ev_cls_t_[2 * ri + 1], class_stream_[ri] ) );
        CUDA_CHECK( cudaEventRecord( ev_class_[ri], class_stream_[ri] ) );
        CUDA_CHECK( cudaStreamWaitEvent( stream_, ev_class_[ri], 0 ) );
    }
    if( timing ) {
        for( int ri = 0; ri < 4; ri++ ) {
            if( !launched[ri] )
                continue;
            float ms = 0;
            CUDA_CHECK( cudaEventSynchronize( ev_cls_t_[2 * ri + 1] ) );
            CUDA_CHECK( cudaEventElapsedTime( &ms, ev_cls_t_[2 * ri], ev_cls_t_[2 * ri + 1] ) );
            double cells = 0, padded = 0;
            for( uint32_t i : by_r[ri] ) {
                const uint32_t a = qp_slots[2 * i], b = qp_slots[2 * i + 1];
                cells += (double) (h_qlen_[a] + (b == 0xffffffffu ? 0u : h_qlen_[b])) * (double) seq_res;
                padded += 2.0 * qp_rows[i] * (double) total_cols;
            }
            fprintf( stderr, "[ssa timing] qpair class R=%d: %zu pairs, %.3f ms, %.3e cells (%.1f%% of computed), "
                    "%.1f GCUPS\n", 4 * (ri + 4), by_r[ri].size(), ms, cells, 100.0 * cells / padded,
                    cells / (ms * 1e-3) / 1e9 );
        }
    }
    if( timing )
        fprintf( stderr, "[ssa timing] %llu pairs beyond the 16-bit range, %s the entry pass\n",
                (unsigned long long) n_beyond, beside ? "beside" : "after" );
    if( !beside )
        run_beyond();
    if( !fallback.empty() ) {
        const uint32_t * dev_slots = stage_.add( fallback.data(), fallback.size(), stream_ );
        run_pass( req.algo, req.bit_width, req, nq, nullptr, (uint64_t) fallback.size() * n_seq, true, next,
                next_count, cap, dev_slots, (uint32_t) fallback.size(), lo );
    }
}

// Scores of `items` at the request's width (two sequences of a
// query per register, sw_stream_kernel.cu) on stream st; lists: where the pairs
// that the kernel does not report go.
void Engine::run_stream( const SearchRequest & req, std::vector<SwStreamItem> & items, const PassSink & lists,
        cudaStream_t st, bool marked ) {
    const bool nw = req.algo == 1;
    // queries with the most rows first: their items have the most stripes
    auto longer = [&]( const SwStreamItem & x, const SwStreamItem & y ) { return h_qlen_[x.slot] > h_qlen_[y.slot]; };
    if( !std::is_sorted( items.begin(), items.end(), longer ) )
        std::stable_sort( items.begin(), items.end(), longer );
    // the items' lengths, and per run of items of one query their number, steps
    // of a stripe in all and the most of one
    struct Run {
        uint64_t qlen, items, columns, longest;
    };
    std::vector<Run> runs;
    std::vector<uint32_t> len( items.size() );
    for( size_t k = 0; k < items.size(); k++ ) {
        if( k == 0 || items[k].slot != items[k - 1].slot )
            runs.push_back( Run{ h_qlen_[items[k].slot], 0, 0, 0 } );
        Run & r = runs.back();
        len[k] = db_.len[items[k].id_a];              // A is the longer
        const uint64_t c = len[k] / 4 + 31;
        r.items++;
        r.columns += c;
        r.longest = std::max( r.longest, c );
    }
    // Rows per lane: 4 while every stripe of 128 rows can be resident (16 warps per
    // SM), else whichever of 4 .. 6 computes the items' stripes in the fewest
    // instructions (a step of R rows is 26 R + 20 of the ALU's).  964 items of 300
    // rows on 2 CTAs per SM: 5.47 ms with 4 (384 rows computed), 3.94 with 5 (320);
    // 7 and 8 were never the best on batches of 30-1,800 rows (7.3 with 5, 7.4 with
    // 6, 8.3 and 8.8 ms).  SSA_B200_STREAM_ROWS pins it.
    auto stripes = []( const Run & q, int r ) { return (q.qlen + 32u * (uint64_t) r - 1u) / (32u * (uint64_t) r); };
    uint64_t stripes128 = 0;
    for( const Run & q : runs )
        stripes128 += q.items * stripes( q, 4 );
    int R = 4;
    const char * pinned = getenv( "SSA_B200_STREAM_ROWS" );
    if( !nw && pinned && atoi( pinned ) >= 4 && atoi( pinned ) <= 6 )
        R = atoi( pinned );
    else if( !nw && stripes128 > (uint64_t) sms_ * 16 ) {
        uint64_t least = UINT64_MAX;
        for( int r = 4; r <= 6; r++ ) {
            uint64_t cost = 0;
            for( const Run & q : runs )
                cost += stripes( q, r ) * q.columns;
            cost *= 26u * (uint64_t) r + 20u;
            if( cost < least ) {
                least = cost;
                R = r;
            }
        }
    }
    // CTAs per SM: a step takes as long as the warps of the sub-partition (one of
    // each CTA) share its ALU, so the longest item ends in time where there are
    // no more of them than its steps go into the sub-partition's share of all
    // steps; at least 2, which keep the ALU busy, at most the 4 that fit.  On 2 / 3
    // / 4: 964 items of 300 x 8,000-35,000 (2.0 times) 3.9 / 4.8 / 5.7 ms, 1,031 of
    // 30-1,800 rows (3.6) 7.4 / 7.1 / 7.1 ms, Needleman-Wunsch of 10,000 (5.6) 1.11
    // / 1.01 / 0.99 ms; fewer items than warps the same on all.
    uint64_t steps = 0, longest = 1;
    for( const Run & q : runs ) {
        steps += stripes( q, R ) * q.columns;
        longest = std::max( longest, q.longest + STREAM_LAG * stripes( q, R ) );
    }
    const int ctas = (int) std::min<uint64_t>( 4, std::max<uint64_t>( 2, steps / ((uint64_t) sms_ * 4 * longest) ) );
    const uint32_t rows = 32u * (uint32_t) R;
    const uint32_t ni = (uint32_t) items.size();
    const bool blocks = req.bit_width == 8;       // Smith-Waterman 8-bit entry
    // Launches of as many items as 1 GB of boundary rows and ticket words holds
    // (SSA_B200_STREAM_MEMORY: another limit, for tests).  The buffers are those of the
    // largest: growing one would free it behind the launch before.
    uint64_t most = (uint64_t) 1 << 30;
    if( const char * m = getenv( "SSA_B200_STREAM_MEMORY" ) )
        most = strtoull( m, nullptr, 10 );
    std::vector<uint64_t> bnd( ni );             // per item, from the start of its launch's rows
    std::vector<uint32_t> part_end;
    uint64_t most_words = 0, most_sync = 0;
    {
        uint64_t words = 0, sync = 16;
        for( uint32_t i = 0; i < ni; i++ ) {
            const uint32_t q = h_qlen_[items[i].slot];
            const uint64_t w = q > rows ? 2ull * ((len[i] + 3u) / 4u) : 0;
            // progress and result of every stripe, and the first crossings
            const uint64_t t = (uint64_t) ((q + rows - 1u) / rows) * 2 * sizeof(uint32_t) + (blocks ? 2 * sizeof(int32_t) : 0);
            if( i > (part_end.empty() ? 0 : part_end.back()) && (words + w) * sizeof(int4) + sync + t > most ) {
                part_end.push_back( i );
                words = 0;
                sync = 16;
            }
            bnd[i] = words;
            words += w;
            sync += t;
            most_words = std::max( most_words, words );
            most_sync = std::max( most_sync, sync );
        }
        part_end.push_back( ni );
    }
    uint8_t * sy = (uint8_t *) d_sw_sync_.ensure( most_sync );
    int4 * boundary = (int4 *) d_sw_bnd_.ensure( most_words * sizeof(int4) + 16 );
    if( getenv( "SSA_B200_TIMING" ) )
        fprintf( stderr, "[ssa timing] %u items on streamed stripes in %zu launches\n", ni, part_end.size() );
    uint32_t i0 = 0;
    for( const uint32_t i1 : part_end ) {
        const uint32_t n = i1 - i0;
        std::vector<uint32_t> cum{ 0 };
        for( uint32_t left = n, i = 0;; i++ ) {
            while( left && (uint64_t) i * rows >= h_qlen_[items[i0 + left - 1].slot] )
                left--;
            if( left == 0 )
                break;
            cum.push_back( cum.back() + left );
        }
        const SwStreamItem * dev_items = stage_.add( items.data() + i0, n, st );
        const uint64_t * dev_bnd = stage_.add( bnd.data() + i0, n, st );
        const uint32_t * dev_cum = stage_.add( cum.data(), cum.size(), st );
        stage_.send( st );
        const uint32_t nt = cum.back();
        // ticket counter, progress, results, and per sequence its first crossing
        const size_t b_zero = 16 + (size_t) nt * sizeof(uint32_t), b_cross = blocks ? n * 2 * sizeof(int32_t) : 0;
        CUDA_CHECK( cudaMemsetAsync( sy, 0, b_zero, st ) );
        SwStreamParams p{};
        p.db = db_view();
        p.qcodes = d_qcodes_.as<uint8_t>();
        p.qoff = d_qoff_.as<uint64_t>();
        p.qlen = d_qlen_.as<uint32_t>();
        p.matrix = d_matrix_.as<int64_t>();
        p.gap_oe = blocks ? (int8_t) (req.gap_open + req.gap_extend) : req.gap_open + req.gap_extend;
        p.gap_e = req.gap_extend;
        p.limit = nw ? 0 : sw_fast_limit( req );
        p.gap_open = req.gap_open;
        p.marked_only = marked;
        p.items = dev_items;
        p.bnd_off = dev_bnd;
        p.cum = dev_cum;
        p.levels = (uint32_t) cum.size() - 1;
        p.n_tickets = nt;
        p.ctas_per_sm = ctas;
        p.counter = (unsigned long long *) sy;
        p.progress = (uint32_t *) (sy + 16);
        p.result = p.progress + nt;
        if( blocks ) {
            p.cross = (int32_t *) (p.result + nt);
            CUDA_CHECK( cudaMemsetAsync( p.cross, 0x7f, b_cross, st ) );
        }
        p.boundary = boundary;
        p.sink = lists;
        p.sink.score = score_sink();
        p.sink.score_stride = db_.n_ids;
        p.sink.error_flags = d_counts_.as<unsigned>() + 2;
        if( i0 == 0 )
            CUDA_CHECK( cudaEventRecord( ev_items_, st ) );
        CUDA_CHECK( nw ? launch_nw_stream( p, sms_, st ) : launch_sw_stream( R, p, sms_, st ) );
        launches_++;
        i0 = i1;
    }
}

void Engine::run_cascade( const SearchRequest & req, uint32_t nq, uint32_t n_a, uint32_t cap,
        std::vector<PairTask> & list_entry, std::vector<PairTask> & list_16, const std::vector<uint32_t> * slots,
        uint32_t lo, uint32_t hi ) {
    unsigned * cnt = d_counts_.as<unsigned>();
    PairTask * list_a = d_list_a_.as<PairTask>();
    PairTask * list_b = d_list_b_.as<PairTask>();
    const size_t first = list_entry.size();
    list_entry.resize( first + n_a );
    if( n_a <= LIST_HEAD )              // came with the counters
        memcpy( list_entry.data() + first, (const char *) h_counts_.p + 64, n_a * sizeof(PairTask) );
    else
        CUDA_CHECK( cudaMemcpyAsync( list_entry.data() + first, list_a, n_a * sizeof(PairTask), cudaMemcpyDeviceToHost,
                stream_ ) );
    if( req.bit_width != 8 ) {
        run_pass( req.algo, 64, req, nq, list_a, n_a, false, nullptr, cnt + 3, 0 );
        CUDA_CHECK( cudaStreamSynchronize( stream_ ) );     // the host list
        return;
    }
    // the 16-bit pass: the 16x2 kernels where they are exact, and the lane
    // emulation for the pairs that leave their range
    SearchRequest r16 = req;
    r16.bit_width = 16;
    const bool queries_fit = max_qlen_ <= FAST_MAX_ROWS;
    const uint64_t searched = (uint64_t) (slots ? slots->size() : nq) * (hi - lo);
    PairTask * redo = nullptr;
    if( fast_single_eligible( r16 ) ) {
        redo = (PairTask *) d_list_c_.ensure( (size_t) n_a * sizeof(PairTask) );
        CUDA_CHECK( cudaMemsetAsync( cnt + 5, 0, sizeof(unsigned), stream_ ) );
        if( n_a > LIST_HEAD )
            CUDA_CHECK( cudaStreamSynchronize( stream_ ) );
        // the re-queued sequences of a query, longest first, in pairs
        std::vector<PairTask> tasks( list_entry.begin() + first, list_entry.end() );
        std::sort( tasks.begin(), tasks.end(), [&]( const PairTask & a, const PairTask & b ) {
            if( a.qslot != b.qslot )
                return a.qslot < b.qslot;
            return db_.len[a.id] != db_.len[b.id] ? db_.len[a.id] > db_.len[b.id] : a.id < b.id;
        } );
        std::vector<SwStreamItem> items;
        for( size_t k = 0; k < tasks.size(); ) {
            const bool two = k + 1 < tasks.size() && tasks[k + 1].qslot == tasks[k].qslot;
            items.push_back( SwStreamItem{ tasks[k].qslot, tasks[k].id, two ? tasks[k + 1].id : 0xffffffffu, 0 } );
            k += two ? 2 : 1;
        }
        PassSink lists{};
        lists.redo = redo;
        lists.redo_count = cnt + 5;
        lists.redo_cap = n_a;
        run_stream( r16, items, lists, stream_ );
    }
    else if( nw_fast_eligible( r16 ) && queries_fit && n_a >= searched / 4 ) {
        // most pairs overflowed: the query-pair kernel over all of them, which
        // scores the marked ones.  It computes a pair an order of magnitude
        // faster than the emulation of the list, so it wins from a quarter on.
        redo = (PairTask *) d_list_c_.ensure( (size_t) n_a * sizeof(PairTask) );
        run_qpair_entry( r16, nq, list_b, cnt + 1, std::min( cap, n_a ), redo, slots, lo, hi, true );
    }
    else {
        run_pass( req.algo, 16, req, nq, list_a, n_a, false, list_b, cnt + 1, cap );
    }
    const unsigned * c = read_counts( false );
    if( redo )
        c = run_redo( r16, nq, c, list_b, cnt + 1, cap, redo, n_a );
    const uint32_t n_b = std::min( c[1], cap );
    if( n_b ) {
        const size_t at = list_16.size();
        list_16.resize( at + n_b );
        run_pass( req.algo, 64, req, nq, list_b, n_b, false, nullptr, cnt + 3, 0 );
        CUDA_CHECK( cudaMemcpyAsync( list_16.data() + at, list_b, n_b * sizeof(PairTask), cudaMemcpyDeviceToHost,
                stream_ ) );
        CUDA_CHECK( cudaStreamSynchronize( stream_ ) );
    }
}

void Engine::search( const SearchRequest & req, const std::vector<QueryCodes> & queries,
        const std::vector<uint32_t> & groups_in, std::vector<std::vector<Hit>> & out, SearchStats & stats ) {
    init_device();
    const HostDb & db = database();
    serving_ = false;
    serve_layout_ = false;      // the query buffers are reused for this batch
    // groups of query sequences (strands or frames of one query)
    std::vector<uint32_t> groups = groups_in;
    if( groups.empty() )
        groups.assign( queries.size(), 1u );
    std::vector<uint64_t> gstart( groups.size() + 1, 0 );
    for( size_t g = 0; g < groups.size(); g++ )
        gstart[g + 1] = gstart[g] + groups[g];
    if( gstart.back() != queries.size() )
        fatal( "Internal error: query groups do not cover the queries." );
    out.assign( groups.size(), {} );
    stats.query_overflow.assign( groups.size(), { 0, 0 } );
    last_shapes_.clear();
    if( queries.empty() )
        return;
    const uint64_t n_ne = db.order_desc.size();


    // the 64-bit pass in int64 arithmetic when the values can leave the int32 range
    {
        uint32_t qmax = 0;
        for( const QueryCodes & q : queries )
            qmax = std::max( qmax, q.len );
        wide_ = needs_int64( req, qmax, db.max_len );
    }
    // sub-batches bounded by the per-pair result memory (int32 scores, plus
    // int64 ones in the wide case)
    const uint64_t pair_budget = this->pair_budget();
    const uint64_t per_query = std::max<uint64_t>( 1, std::max<uint64_t>( n_ne, db.n_ids ) );
    const size_t batch = (size_t) std::max<uint64_t>(
            1, std::min<uint64_t>( std::min<uint64_t>( queries.size(), pair_budget / per_query ), 65535 ) );

    CUDA_CHECK( cudaEventRecord( ev0_, stream_ ) );
    for( size_t g0 = 0; g0 < groups.size(); ) {
        // whole groups, at most `batch` query sequences (at least one group)
        size_t g1 = g0 + 1;
        while( g1 < groups.size() && gstart[g1 + 1] - gstart[g0] <= batch )
            g1++;
        const size_t b0 = gstart[g0];
        const uint32_t nq = (uint32_t) (gstart[g1] - b0);
        // ---- upload queries
        stage_.begin();
        upload_queries( req, queries.data() + b0, nq, true, stats );
        for( uint32_t q = 0; q < nq; q++ )
            stats.cells += (uint64_t) h_qlen_[q] * db.residues;

        // ---- result and re-queue buffers
        const uint64_t n_pairs = (uint64_t) nq * n_ne;
        const size_t score_bytes = (size_t) nq * db.n_ids * sizeof(int32_t);
        d_score_.ensure( std::max<size_t>( score_bytes, 4 ) );
        if( wide_ )
            d_score64_.ensure( std::max<size_t>( 2 * score_bytes, 8 ) );
        // re-queue lists sized for the overflows a search expects (a few per
        // query): 1/32 of the pairs, at least 4M entries; an entry pass that
        // re-queues more runs again with lists of its count
        const uint64_t all_pairs = std::min<uint64_t>( std::max<uint64_t>( n_pairs, 1 ), 0xffffffffull );
        uint32_t cap = (uint32_t) std::min<uint64_t>( all_pairs, std::max<uint64_t>( (uint64_t) 1 << 22,
                all_pairs >> 5 ) );
        if( const char * c0 = getenv( "SSA_B200_REQUEUE_CAP" ) )   // a smaller first size (tests of the regrowth)
            cap = (uint32_t) std::max<uint64_t>( 1, std::min<uint64_t>( cap, strtoull( c0, nullptr, 10 ) ) );
        d_list_a_.ensure( (size_t) cap * sizeof(PairTask) );
        d_list_b_.ensure( (size_t) cap * sizeof(PairTask) );
        d_counts_.ensure( 32 * sizeof(unsigned long long) );
        CUDA_CHECK( cudaMemsetAsync( d_counts_.p, 0, 32 * sizeof(unsigned long long), stream_ ) );
        unsigned * cnt = d_counts_.as<unsigned>();   // [0] list a, [1] list b, [2] errors, [5] NW redo

        // ---- passes
        const bool timing = getenv( "SSA_B200_TIMING" ) != nullptr;
        CUDA_CHECK( cudaEventRecord( ev_phase_[0], stream_ ) );
        const int entry = req.bit_width;
        std::vector<PairTask> list_entry, list_16;   // host copies for the replay
        // few scores come back with the entry pass's counts: they are final when
        // nothing was re-queued, and the call then waits for the device once
        int32_t * hs = (int32_t *) h_score_.ensure( std::max<size_t>( score_bytes, 4 ) );
        const bool early = !streaming_ && !wide_ && score_bytes && score_bytes <= ((size_t) 1 << 20);
        bool redone = false;    // scores written after the entry pass's
        float entry_ms = 0;     // the entry passes of all segments
        // a resident database is one segment; a streamed one runs the entry pass
        // and the cascade of each segment while it is on the device
        const uint32_t n_seg = streaming_ ? (uint32_t) seg_lo_.size() : 1;
        for( uint32_t sg = 0; sg < n_seg; sg++ ) {
            const uint32_t lo = streaming_ ? seg_lo_[sg] : 0;
            const uint32_t hi = streaming_ ? seg_hi_[sg] : (uint32_t) n_ne;
            if( streaming_ ) {
                make_resident( sg, stats );
                CUDA_CHECK( cudaMemsetAsync( cnt, 0, 2 * sizeof(unsigned), stream_ ) );
            }
            const uint64_t seg_pairs = (uint64_t) nq * (hi - lo);
            CUDA_CHECK( cudaEventRecord( ev_seg_[0], stream_ ) );
            auto run_entry = [&]() {
                if( (fast_eligible( req ) && (nq >= 2 || streaming_ || !fast_single_eligible( req )) &&
                            !getenv( "SSA_B200_NO_QPAIR" )) ||
                        nw_fast_eligible( req ) )
                    run_qpair_entry( req, nq, d_list_a_.as<PairTask>(), cnt + 0, cap, d_list_b_.as<PairTask>(), nullptr,
                            lo, hi );
                else if( fast_single_eligible( req ) )
                    run_fast_entry( req, nq, d_list_a_.as<PairTask>(), cnt + 0, cap );
                else
                    run_pass( req.algo, entry, req, nq, nullptr, seg_pairs, true, d_list_a_.as<PairTask>(), cnt + 0,
                            cap, nullptr, 0, lo );
            };
            run_entry();
            uint32_t n_req = 0;     // pairs the entry pass re-queued
            for( ;; ) {
                // the counters of the entry list and the redo list count every
                // append, kept or not
                const unsigned * c = read_counts( true, early ? hs : nullptr, score_bytes );
                if( std::max( c[0], c[5] ) <= cap && !(c[2] & ERR_REQUEUE_OVERFLOW) && c[5] ) {
                    c = run_redo( req, nq, c, d_list_a_.as<PairTask>(), cnt + 0, cap, d_list_b_.as<PairTask>(), cap );
                    redone = true;
                }
                const uint64_t need = std::max<uint64_t>( c[0], c[5] );
                if( need <= cap && !(c[2] & ERR_REQUEUE_OVERFLOW) ) {
                    n_req = c[0];
                    break;
                }
                cap = (uint32_t) std::min<uint64_t>( all_pairs, std::max<uint64_t>( need, 2ull * cap ) );
                d_list_a_.ensure( (size_t) cap * sizeof(PairTask) );
                d_list_b_.ensure( (size_t) cap * sizeof(PairTask) );
                CUDA_CHECK( cudaMemsetAsync( cnt, 0, 6 * sizeof(unsigned), stream_ ) );
                run_entry();
            }
            CUDA_CHECK( cudaEventRecord( ev_seg_[1], stream_ ) );
            CUDA_CHECK( cudaEventSynchronize( ev_seg_[1] ) );
            float seg_ms = 0;
            CUDA_CHECK( cudaEventElapsedTime( &seg_ms, ev_seg_[0], ev_seg_[1] ) );
            entry_ms += seg_ms;
            if( entry == 64 || n_req == 0 )
                continue;
            run_cascade( req, nq, n_req, cap, list_entry, list_16, nullptr, lo, hi );
            if( streaming_ )
                CUDA_CHECK( cudaStreamSynchronize( stream_ ) );   // the lists are reused by the next segment
        }
        CUDA_CHECK( cudaEventRecord( ev_phase_[2], stream_ ) );
        const uint64_t n_a = list_entry.size(), n_b = list_16.size();
        stats.d2h_bytes += score_bytes + (n_a + n_b) * sizeof(PairTask);
        const bool have_scores = early && n_a == 0 && !redone;
        if( score_bytes && !have_scores )
            CUDA_CHECK( cudaMemcpyAsync( hs, d_score_.p, score_bytes, cudaMemcpyDeviceToHost, stream_ ) );
        int64_t * hs64 = nullptr;
        if( wide_ && score_bytes ) {
            hs64 = (int64_t *) h_score64_.ensure( 2 * score_bytes );
            CUDA_CHECK( cudaMemcpyAsync( hs64, d_score64_.p, 2 * score_bytes, cudaMemcpyDeviceToHost, stream_ ) );
            stats.d2h_bytes += 2 * score_bytes;
        }
        unsigned * err = (unsigned *) h_counts_.p + 2;
        if( !have_scores )
            CUDA_CHECK( cudaMemcpyAsync( err, cnt + 2, sizeof(unsigned), cudaMemcpyDeviceToHost, stream_ ) );
        CUDA_CHECK( cudaEventRecord( ev_phase_[3], stream_ ) );
        if( !have_scores )
            CUDA_CHECK( cudaStreamSynchronize( stream_ ) );
        if( *err )
            fatal( "Internal error in the GPU search (flags 0x%x).", *err );
        const auto t_replay0 = std::chrono::steady_clock::now();

        // ---- host replay, one query (group of query sequences) per worker
        std::vector<ReplayQuery> rq( nq );
        for( uint32_t s = 0; s < nq; s++ ) {
            rq[s].score = hs + (size_t) s * db.n_ids;
            if( hs64 )
                rq[s].score64 = hs64 + (size_t) s * db.n_ids;
        }
        for( const PairTask & t : list_entry )
            rq[t.qslot].ovf_entry.emplace_back( t.id, t.nb_prev );
        for( const PairTask & t : list_16 )
            rq[t.qslot].ovf16.emplace_back( t.id, t.nb_prev );
        for( auto & r : rq ) {
            std::sort( r.ovf_entry.begin(), r.ovf_entry.end() );
            std::sort( r.ovf16.begin(), r.ovf16.end() );
        }
        const uint32_t * rank_entry = (entry == 64) ? nullptr : ranks( req.chunk_size, entry == 8 ? req.lanes8 : req.lanes16 );
        {
            const uint32_t ng = (uint32_t) (g1 - g0);
            const unsigned hw = std::max( 1u, std::thread::hardware_concurrency() );
            const unsigned nthreads = std::min<unsigned>( hw, ng );
            std::atomic<uint32_t> next{ 0 };
            std::vector<ReplayCounts> counts( ng );
            auto work = [&]() {
                for( ;; ) {
                    const uint32_t i = next.fetch_add( 1 );
                    if( i >= ng )
                        break;
                    const size_t g = g0 + i;
                    const uint32_t s0 = (uint32_t) (gstart[g] - b0);
                    if( groups[g] == 1 && db.upi == 1 )
                        replay_query( db, req, rq[s0], rank_entry, out[g], counts[i] );
                    else
                        replay_frames( db, req, &rq[s0], groups[g], out[g], counts[i] );
                }
            };
            if( nthreads <= 1 ) {
                work();
            }
            else {
                std::vector<std::thread> th;
                for( unsigned k = 0; k < nthreads; k++ )
                    th.emplace_back( work );
                for( auto & t : th )
                    t.join();
            }
            for( uint32_t i = 0; i < ng; i++ ) {
                stats.overflow8 += counts[i].overflow8;
                stats.overflow16 += counts[i].overflow16;
                stats.query_overflow[g0 + i] = { counts[i].overflow8, counts[i].overflow16 };
            }
        }
        const auto t_replay1 = std::chrono::steady_clock::now();
        CUDA_CHECK( cudaEventRecord( ev_phase_[4], stream_ ) );
        if( req.align_type == COMPUTE_ALIGNMENT ) {
            std::vector<std::pair<uint32_t, uint32_t>> lists;   // (out index, slot of its first sequence)
            for( size_t g = g0; g < g1; g++ )
                lists.emplace_back( (uint32_t) g, (uint32_t) (gstart[g] - b0) );
            traceback( req, out, lists, stats );
        }
        CUDA_CHECK( cudaEventRecord( ev_phase_[5], stream_ ) );
        {
            CUDA_CHECK( cudaEventSynchronize( ev_phase_[5] ) );
            float ms[5];
            // [0] entry passes, [1] cascades (and segment copies), [2] result copies, [3] traceback
            float passes = 0;
            CUDA_CHECK( cudaEventElapsedTime( &passes, ev_phase_[0], ev_phase_[2] ) );
            ms[0] = entry_ms;
            ms[1] = std::max( 0.0f, passes - entry_ms );
            CUDA_CHECK( cudaEventElapsedTime( &ms[2], ev_phase_[2], ev_phase_[3] ) );
            CUDA_CHECK( cudaEventElapsedTime( &ms[3], ev_phase_[4], ev_phase_[5] ) );
            const double rep = std::chrono::duration<double, std::milli>( t_replay1 - t_replay0 ).count();
            stats.entry_seconds += ms[0] * 1e-3;
            stats.kernel_seconds += (ms[0] + ms[1] + ms[3]) * 1e-3;
            if( timing )
            fprintf( stderr,
                    "[ssa timing] queries %u pairs %llu: entry %.3f ms, cascade %.3f ms (%llu+%llu re-queued), "
                    "copies %.3f ms, replay %.3f ms, traceback %.3f ms\n",
                    nq, (unsigned long long) n_pairs, ms[0], ms[1], (unsigned long long) n_a,
                    (unsigned long long) n_b, ms[2], rep, ms[3] );
        }
        g0 = g1;
    }
    CUDA_CHECK( cudaEventRecord( ev1_, stream_ ) );
    CUDA_CHECK( cudaEventSynchronize( ev1_ ) );
    float ms = 0;
    CUDA_CHECK( cudaEventElapsedTime( &ms, ev0_, ev1_ ) );
    stats.seconds_gpu += ms * 1e-3;
    stats.kernel_launches = launches_.load();
}

// Query codes of one batch to the device (slot s = queries[s]); profiles: also
// size the int32 profile buffer of the lane emulation.
void Engine::upload_queries( const SearchRequest & req, const QueryCodes * queries, uint32_t nq, bool profiles,
        SearchStats & stats ) {
    h_qoff_.assign( nq, 0 );
    h_qlen_.assign( nq, 0 );
    h_qpad_.assign( nq, 0 );
    h_prof_off_.assign( nq, 0 );
    uint64_t qtotal = 0, ptotal = 0;
    max_qlen_ = 0;
    for( uint32_t s = 0; s < nq; s++ ) {
        const QueryCodes & q = queries[s];
        h_qoff_[s] = qtotal;
        h_qlen_[s] = q.len;
        h_qpad_[s] = std::max<uint32_t>( 256, (q.len + 255u) & ~255u );
        h_prof_off_[s] = ptotal;
        qtotal += (q.len + 15u) & ~15u;
        ptotal += 32ull * h_qpad_[s];
        max_qlen_ = std::max( max_qlen_, q.len );
    }
    std::vector<uint8_t> hq( qtotal + 16, 0 );
    for( uint32_t s = 0; s < nq; s++ )
        memcpy( hq.data() + h_qoff_[s], queries[s].codes, queries[s].len );
    if( profiles )
        d_prof_.ensure( ptotal * sizeof(int32_t) );
    stats.h2d_bytes += hq.size() + nq * (2 * sizeof(uint64_t) + 2 * sizeof(uint32_t));
    // sent with the arrays of the pass that reads them
    d_matrix_.p = stage_.add( req.matrix, 1024, stream_ );
    d_qcodes_.p = stage_.add( hq.data(), hq.size(), stream_ );
    d_qoff_.p = stage_.add( h_qoff_.data(), nq, stream_ );
    d_prof_off_.p = stage_.add( h_prof_off_.data(), nq, stream_ );
    d_qlen_.p = stage_.add( h_qlen_.data(), nq, stream_ );
    d_qpad_.p = stage_.add( h_qpad_.data(), nq, stream_ );
    prof_width_ = -1;
}

// Largest magnitude of one DP step: a score-table entry or a gap cost.
static int64_t max_abs_step( const SearchRequest & req ) {
    int64_t m = std::llabs( (int64_t) req.gap_open ) + std::llabs( (int64_t) req.gap_extend );
    for( int k = 0; k < 1024; k++ )
        m = std::max<int64_t>( m, std::llabs( req.matrix[k] ) );
    return m;
}

// Most direction memory that is kept for later calls.
constexpr uint64_t TB_KEPT = (uint64_t) 8 << 30;
// Least direction memory of one traceback wave (automatic budget).
constexpr uint64_t TB_MIN_BUDGET = (uint64_t) 256 << 20;

void Engine::traceback( const SearchRequest & req, std::vector<std::vector<Hit>> & out,
        const std::vector<std::pair<uint32_t, uint32_t>> & lists, SearchStats & stats, bool scores_from_regions,
        bool scores_only ) {
    std::vector<TbHit> hits;
    std::vector<std::pair<uint32_t, uint32_t>> where;   // (list index, hit index)
    for( const auto & l : lists ) {
        auto & hl = out[l.first];
        for( uint32_t k = 0; k < hl.size(); k++ ) {
            // the hit's query sequence; the database record's first unit (the
            // reference aligns a reverse-complement hit on the forward strand:
            // src/util/util_sequence.c:384-402)
            const uint32_t fwd_unit = hl[k].unit - hl[k].unit % db_.upi;
            hits.push_back( TbHit{ l.second + hl[k].q_index, fwd_unit, (int32_t) hl[k].score, req.algo } );
            where.emplace_back( l.first, k );
        }
    }
    const uint32_t nh = (uint32_t) hits.size();
    if( nh == 0 )
        return;
    // value range guard: every DP value is bounded by (q + d) * max |step|
    const int64_t mabs = max_abs_step( req );
    std::vector<TbRegion> regions( nh );
    std::vector<uint64_t> last_off( nh + 1, 0 );
    for( uint32_t h = 0; h < nh; h++ ) {
        const uint32_t A = h_qlen_[hits[h].qslot], B = db_.len[hits[h].id];
        if( (int64_t) (A + B + 4) * (mabs + 1) * 2 > INT32_MAX )
            fatal( "Alignment of %u x %u residues exceeds the supported score range.", A, B );
        TbRegion rg{};
        if( req.algo == 1 ) {
            rg.a_begin = 0;
            rg.a_end = (int32_t) A - 1;
            rg.b_begin = 0;
            rg.b_end = (int32_t) B - 1;
            rg.status = (A && B) ? 0 : 1;
        }
        regions[h] = rg;
        last_off[h + 1] = last_off[h] + A;
    }
    uint32_t stripe_rows = 0;                // of the waves: 32 x rows per lane
    bool p8 = true;
    for( int k = 0; k < 1024; k++ )
        p8 = p8 && req.matrix[k] == (int8_t) req.matrix[k];
    TbParams p{};
    // the hits as the device sees them: with a streamed database their
    // sequences are gathered into a view of their own and renumbered
    std::vector<TbHit> dev_hits = hits;
    if( streaming_ ) {
        std::vector<uint32_t> ids;
        std::unordered_map<uint32_t, uint32_t> index;
        for( TbHit & t : dev_hits ) {
            auto it = index.find( t.id );
            if( it == index.end() ) {
                it = index.emplace( t.id, (uint32_t) ids.size() ).first;
                ids.push_back( t.id );
            }
            t.id = it->second;
        }
        p.db = gather_view( ids, stats );
    }
    else {
        p.db = db_view();
    }
    p.qcodes = d_qcodes_.as<uint8_t>();
    p.qoff = d_qoff_.as<uint64_t>();
    p.qlen = d_qlen_.as<uint32_t>();
    p.matrix = d_matrix_.as<int64_t>();
    p.gap_open = req.gap_open;
    p.gap_extend = req.gap_extend;
    int32_t * last_all = (int32_t *) d_tb_last_.ensure( 2 * last_off[nh] * sizeof(int32_t) + 16 );
    p.last_h = last_all;
    p.last_e = last_all + last_off[nh];

    // Smith-Waterman with a symmetric score table: the forward region pass and
    // the direction pass run as one sweep per hit, then the reverse pass and
    // the walk.  It needs every hit's last database column past the initial E
    // terms: (B - 1) x gapE < gapO + gapE with B >= 2, and initial E and F
    // values that are not above zero (gapO <= 0).
    bool fused = req.algo == 0 && req.gap_extend < 0 && req.gap_open <= 0;
    for( int d = 0; d < 32 && fused; d++ )
        for( int q = 0; q < 32 && fused; q++ )
            fused = req.matrix[(d << 5) + q] == req.matrix[(q << 5) + d];
    for( uint32_t h = 0; h < nh && fused; h++ )
        fused = db_.len[hits[h].id] >= 2 &&
                ((int64_t) db_.len[hits[h].id] - 1) * req.gap_extend < (int64_t) req.gap_open + req.gap_extend;
    const bool timing = getenv( "SSA_B200_TIMING" ) != nullptr;
    float t_fwd = 0, t_rev = 0, t_dir = 0, t_walk = 0;
    uint64_t total_dir = 0;
    size_t n_waves = 0;

    // One wave: the hits of `wave`, most stripes first (rows[h] query rows and
    // cols[h] database columns each).  All its arrays travel in one copy each
    // way: hits, regions and offsets down; regions, move counts, error flags
    // and move strings up.
    struct Layout {
        size_t bytes = 0;
        size_t add( size_t n ) {
            const size_t at = bytes;
            bytes += (n + 15) & ~(size_t) 15;
            return at;
        }
    };
    enum Mode { REGIONS, PATHS, SCORES };
    auto run_wave = [&]( const std::vector<uint32_t> & wave, const std::vector<uint32_t> & rows,
            const std::vector<uint32_t> & cols, Mode mode ) {
        const uint32_t nw = (uint32_t) wave.size();
        const bool paths = mode == PATHS;
        const bool reverse = req.algo == 0 && (mode == REGIONS || (fused && paths));
        // tickets stripe by stripe: stripe i exists in the first n_i hits
        std::vector<uint32_t> cum{ 0 };
        for( uint32_t left = nw, i = 0;; i++ ) {
            while( left && (uint64_t) i * stripe_rows >= rows[wave[left - 1]] )
                left--;
            if( left == 0 )
                break;
            cum.push_back( cum.back() + left );
        }
        uint64_t dir_words = 0, bnd_words = 0, ops_bytes = 0;
        Layout in, res;
        const size_t o_hits = in.add( nw * sizeof(TbHit) ), o_last = in.add( nw * sizeof(uint64_t) ),
                o_dir = in.add( nw * sizeof(uint64_t) ), o_ops = in.add( (nw + 1) * sizeof(uint64_t) ),
                o_bnd = in.add( nw * sizeof(uint64_t) ), o_cum = in.add( cum.size() * sizeof(uint32_t) ),
                o_reg = in.add( nw * sizeof(TbRegion) ), o_err = in.add( sizeof(unsigned) );
        uint8_t * hin = (uint8_t *) h_tb_in_.ensure( in.bytes );
        memset( hin + o_err, 0, sizeof(unsigned) );
        for( uint32_t k = 0; k < nw; k++ ) {
            const uint32_t h = wave[k];
            const uint64_t stripes = (rows[h] + stripe_rows - 1) / stripe_rows;
            TbRegion rg = regions[h];
            rg.dir_steps = (int32_t) ((cols[h] + 3u) / 4u) + 31;
            ((TbHit *) (hin + o_hits))[k] = dev_hits[h];
            ((TbRegion *) (hin + o_reg))[k] = rg;
            ((uint64_t *) (hin + o_last))[k] = last_off[h];
            ((uint64_t *) (hin + o_dir))[k] = dir_words;
            ((uint64_t *) (hin + o_ops))[k] = ops_bytes;
            ((uint64_t *) (hin + o_bnd))[k] = bnd_words;
            if( paths ) {
                dir_words += stripes * (uint64_t) rg.dir_steps * 32;
                ops_bytes += (uint64_t) rows[h] + cols[h] + 1;
            }
            if( stripes > 1 )
                bnd_words += 2ull * ((cols[h] + 3u) / 4u);
        }
        ((uint64_t *) (hin + o_ops))[nw] = ops_bytes;
        memcpy( hin + o_cum, cum.data(), cum.size() * sizeof(uint32_t) );
        const uint32_t n_tickets = cum.back();
        // device side: inputs (regions and error flags last, updated in place),
        // then the passes' results in the order they are copied back
        const size_t r_reg = res.add( nw * sizeof(TbRegion) ), r_err = res.add( sizeof(unsigned) ),
                r_len = res.add( nw * sizeof(uint32_t) ), r_ops = res.add( paths ? ops_bytes : 0 );
        uint8_t * din = (uint8_t *) d_tb_io_.ensure( in.bytes + res.bytes );
        uint8_t * dout = din + o_reg;            // the regions and flags of the inputs are the first results
        // (the moves of a wave of chromosome-sized hits: pageable, and given back)
        std::vector<uint8_t> large( res.bytes > pinned_kept() ? res.bytes : 0 );
        uint8_t * hout = large.empty() ? (uint8_t *) h_tb_out_.ensure( res.bytes ) : large.data();
        p.error_flags = (unsigned *) (dout + r_err);
        // progress of both sweeps, ticket counters and column limits: cleared
        // by one memset (the limits to a large positive number)
        Layout sy;
        const size_t s_prog = sy.add( (size_t) n_tickets * 2 * sizeof(uint32_t) ),
                s_cnt = sy.add( 2 * sizeof(unsigned long long) );
        const size_t s_zero = sy.bytes;
        const size_t s_lim = sy.add( nw * sizeof(int32_t) );
        uint8_t * dsy = (uint8_t *) d_tb_sync_.ensure( sy.bytes );
        p.hits = (const TbHit *) (din + o_hits);
        p.n_hits = nw;
        p.last_off = (const uint64_t *) (din + o_last);
        p.dir_off = (const uint64_t *) (din + o_dir);
        p.ops_off = (const uint64_t *) (din + o_ops);
        p.bnd_off = (const uint64_t *) (din + o_bnd);
        p.cum = (const uint32_t *) (din + o_cum);
        p.regions = (TbRegion *) (dout + r_reg);
        p.ops_len = (uint32_t *) (dout + r_len);
        p.ops = (char *) (dout + r_ops);
        p.levels = (uint32_t) cum.size() - 1;
        p.n_tickets = n_tickets;
        p.result = (int4 *) d_tb_result_.ensure( std::max<size_t>( 16, (size_t) n_tickets * sizeof(int4) ) );
        p.boundary = (int4 *) d_tb_bnd_.ensure( bnd_words * sizeof(int4) + 16 );
        p.limit = (int32_t *) (dsy + s_lim);
        if( paths ) {
            const size_t n = dir_words * sizeof(uint32_t) + 16;
            p.dirs = (uint32_t *) (tb_budget_ || n + n / 8 > TB_KEPT ? d_tb_dirs_.ensure( n ) : d_tb_dirs_.ensure_spare( n ));
        }
        stage_.send( stream_ );
        CUDA_CHECK( cudaMemcpyAsync( din, hin, in.bytes, cudaMemcpyHostToDevice, stream_ ) );
        CUDA_CHECK( cudaMemsetAsync( dsy, 0, s_zero, stream_ ) );
        if( reverse )
            CUDA_CHECK( cudaMemsetAsync( dsy + s_lim, 0x7f, nw * sizeof(int32_t), stream_ ) );
        auto sweep = [&]( int k ) {
            p.progress = (uint32_t *) (dsy + s_prog) + (size_t) k * n_tickets;
            p.counter = (unsigned long long *) (dsy + s_cnt) + k;
            launches_++;
        };
        if( timing )
            CUDA_CHECK( cudaEventRecord( ev_tb_[0], stream_ ) );
        sweep( 0 );
        CUDA_CHECK( mode == SCORES ? launch_tb_scores( p, req.algo == 1, p8, sms_, stream_ )
                    : mode == REGIONS ? launch_tb_forward( p, p8, sms_, stream_ )
                    : fused ? launch_tb_fwddir( p, p8, sms_, stream_ )
                            : launch_tb_directions( p, req.algo == 1, p8, sms_, stream_ ) );
        if( timing )
            CUDA_CHECK( cudaEventRecord( ev_tb_[1], stream_ ) );
        if( reverse ) {
            sweep( 1 );
            CUDA_CHECK( launch_tb_reverse( p, p8, sms_, stream_ ) );
        }
        if( paths ) {
            launches_++;
            CUDA_CHECK( launch_tb_walk( p, stream_ ) );
        }
        if( timing )
            CUDA_CHECK( cudaEventRecord( ev_tb_[2], stream_ ) );
        CUDA_CHECK( cudaMemcpyAsync( hout, dout, res.bytes, cudaMemcpyDeviceToHost, stream_ ) );
        CUDA_CHECK( cudaStreamSynchronize( stream_ ) );
        unsigned err = 0;
        memcpy( &err, hout + r_err, sizeof err );
        if( err )
            fatal( "Internal error in the GPU traceback (flags 0x%x).", err );
        stats.h2d_bytes += in.bytes;
        stats.d2h_bytes += res.bytes;
        total_dir += dir_words * sizeof(uint32_t);
        n_waves++;
        if( timing ) {
            float x = 0, y = 0;
            CUDA_CHECK( cudaEventElapsedTime( &x, ev_tb_[0], ev_tb_[1] ) );
            CUDA_CHECK( cudaEventElapsedTime( &y, ev_tb_[1], ev_tb_[2] ) );
            (paths ? t_dir : t_fwd) += x;
            (paths ? t_walk : t_rev) += y;
        }
        for( uint32_t k = 0; k < nw; k++ ) {
            const uint32_t h = wave[k];
            const TbRegion & rg = regions[h] = ((const TbRegion *) (hout + r_reg))[k];
            if( rg.status == 2 )
                fatal( "Internal error in align function." );   // reference: src/algo/align.c:131
            if( mode == SCORES )
                out[where[h].first][where[h].second].score = rg.fwd_score;
            if( !paths )
                continue;
            Hit & hit = out[where[h].first][where[h].second];
            hit.has_cigar = true;
            if( scores_from_regions )
                hit.score = rg.fwd_score;
            if( rg.status != 0 ) {
                // no positive cell: the reference leaves the region undefined here
                hit.q_start = hit.q_end = hit.d_start = hit.d_end = 0;
                hit.cigar.clear();
                continue;
            }
            hit.q_start = (uint32_t) rg.a_begin;
            hit.q_end = (uint32_t) rg.a_end;
            hit.d_start = (uint32_t) rg.b_begin;
            hit.d_end = (uint32_t) rg.b_end;
            // run-length encode the moves in alignment order; counts of 1 are
            // omitted (reference: src/algo/cigar.c:221-263)
            const uint64_t * off = (const uint64_t *) (hin + o_ops);
            const char * mv = (const char *) (hout + r_ops) + off[k];
            uint32_t i = (uint32_t) std::min<uint64_t>( ((const uint32_t *) (hout + r_len))[k], off[k + 1] - off[k] );
            std::string cig;
            while( i > 0 ) {
                const char op = mv[i - 1];
                uint32_t run = 0;
                while( i > 0 && mv[i - 1] == op ) {
                    run++;
                    i--;
                }
                if( run > 1 )
                    cig += std::to_string( run );
                cig += op;
            }
            hit.cigar = std::move( cig );
        }
    };
    // Waves: runs of the hits in (most stripes first, most columns first) order
    // whose direction bytes and boundary rows fit the traceback memory.
    auto run_waves = [&]( const std::vector<uint32_t> & rows, const std::vector<uint32_t> & cols, Mode mode ) {
        std::vector<uint32_t> order( nh );
        for( uint32_t h = 0; h < nh; h++ )
            order[h] = h;
        auto stripes = [&]( uint32_t h ) { return (rows[h] + stripe_rows - 1) / stripe_rows; };
        auto need = [&]( uint32_t h ) {
            const uint64_t blocks = (cols[h] + 3u) / 4u;
            return (mode == PATHS ? (uint64_t) stripes( h ) * (blocks + 31) * 32 * sizeof(uint32_t) : 0) +
                    (stripes( h ) > 1 ? 2 * blocks * sizeof(int4) : 0);
        };
        // Rows per lane: 4, or 2 in the Smith-Waterman sweep of a few long hits.  A
        // warp alone on its sub-partition takes 352 ns for a step of 4 rows and 274
        // for one of 2 (Needleman-Wunsch: 270 for both), but 2 make twice the
        // stripes, each 48 steps behind the one above: it pays from hits five
        // times as long as high, while each stripe has a sub-partition and the
        // twice as many direction words are one wave.  10 hits of 300 x 33,000:
        // 3.8 ms with 4, 2.9 with 2; of 375 x 380 0.12 and 0.16.  SSA_B200_TB_ROWS
        // pins it.
        uint64_t total = 0, stripes64 = 0, columns = 0;
        stripe_rows = 64;
        for( uint32_t h = 0; h < nh; h++ ) {
            total += need( h );
            stripes64 += stripes( h );
            columns += cols[h];
        }
        const char * pinned = getenv( "SSA_B200_TB_ROWS" );
        if( !p8 || !fused || mode != PATHS || (pinned ? atoi( pinned ) != 2 : stripes64 > (uint64_t) sms_ * 4 ||
                columns < 5 * 64 * stripes64 || total > (tb_budget_ ? tb_budget_ : TB_MIN_BUDGET)) ) {
            stripe_rows = 128;
            total = 0;
            for( uint32_t h = 0; h < nh; h++ )
                total += need( h );
        }
        p.rows_per_lane = (int) stripe_rows / 32;
        std::stable_sort( order.begin(), order.end(), [&]( uint32_t x, uint32_t y ) {
            return stripes( x ) != stripes( y ) ? stripes( x ) > stripes( y ) : cols[x] > cols[y];
        } );
        // matrices within the smallest automatic budget make one wave whatever
        // the free memory is: asking the driver for it costs up to milliseconds
        const uint64_t budget = (!tb_budget_ && total <= TB_MIN_BUDGET) ? TB_MIN_BUDGET : traceback_budget();
        std::vector<uint32_t> wave;
        uint64_t load = 0;
        for( uint32_t h : order ) {
            if( !wave.empty() && load + need( h ) > budget ) {
                run_wave( wave, rows, cols, mode );
                wave.clear();
                load = 0;
            }
            wave.push_back( h );
            load += need( h );
        }
        run_wave( wave, rows, cols, mode );
    };
    std::vector<uint32_t> rows( nh ), cols( nh );
    for( uint32_t h = 0; h < nh; h++ ) {
        rows[h] = h_qlen_[hits[h].qslot];
        cols[h] = db_.len[hits[h].id];
    }
    if( req.algo == 0 && !fused && !scores_only ) {
        // the end and begin cell of every hit, then rows 0 .. a_end and columns
        // 0 .. b_end of the direction matrix
        run_waves( rows, cols, REGIONS );
        for( uint32_t h = 0; h < nh; h++ ) {
            rows[h] = regions[h].status == 0 ? (uint32_t) regions[h].a_end + 1 : 1;
            cols[h] = regions[h].status == 0 ? (uint32_t) regions[h].b_end + 1 : 1;
        }
    }
    run_waves( rows, cols, scores_only ? SCORES : PATHS );
    // a very large direction buffer (long pairs) is not kept for later calls,
    // whose scores, lists and database segments need the device memory
    if( d_tb_dirs_.bytes > TB_KEPT )
        d_tb_dirs_.release();
    if( d_tb_bnd_.bytes > ((uint64_t) 1 << 30) )
        d_tb_bnd_.release();
    if( timing ) {
        uint64_t max_cells = 0;
        uint32_t max_a = 0, max_b = 0;
        for( uint32_t h = 0; h < nh; h++ ) {
            const uint64_t A = h_qlen_[hits[h].qslot], B = db_.len[hits[h].id];
            if( A * B > max_cells ) {
                max_cells = A * B;
                max_a = (uint32_t) A;
                max_b = (uint32_t) B;
            }
        }
        if( fused )
            fprintf( stderr, "[ssa timing] traceback %u hits: forward with directions %.3f ms, reverse and walk "
                    "%.3f ms in %zu wave(s) (%.3f GB of directions); largest hit %u x %u\n", nh, t_dir, t_walk,
                    n_waves, total_dir * 1e-9, max_a, max_b );
        else
            fprintf( stderr, "[ssa timing] traceback %u hits: forward %.3f ms, reverse %.3f ms, directions %.3f ms, "
                    "walk %.3f ms in %zu wave(s) (%.3f GB of directions); largest hit %u x %u\n", nh, t_fwd, t_rev,
                    t_dir, t_walk, n_waves, total_dir * 1e-9, max_a, max_b );
    }
}

// Device memory for the direction words of one traceback wave: the setting of
// ssa_b200_set_traceback_memory, else the free device memory (plus what the
// direction buffer holds already) less a reserve.
uint64_t Engine::traceback_budget() {
    if( tb_budget_ )
        return tb_budget_;
    size_t free_b = 0, total_b = 0;
    CUDA_CHECK( cudaMemGetInfo( &free_b, &total_b ) );
    const uint64_t avail = (uint64_t) free_b + d_tb_dirs_.bytes;
    const uint64_t reserve = std::max<uint64_t>( (uint64_t) 4 << 30, (uint64_t) total_b / 16 );
    return avail > reserve + TB_MIN_BUDGET ? avail - reserve : TB_MIN_BUDGET;
}

// ---- long pairs -------------------------------------------------------------------
// Query i against database unit units[i] alone: what sw_align / nw_align return
// for the query against a database holding only that sequence (one hit, or
// none for an empty sequence).  The traceback's sweep scores each pair exactly;
// the hits then go through the traceback like a search's.
void Engine::align_pairs( const SearchRequest & req, const std::vector<QueryCodes> & queries,
        const std::vector<uint32_t> & units, std::vector<std::vector<Hit>> & out, SearchStats & stats ) {
    const HostDb & db = database();
    serving_ = false;
    serve_layout_ = false;      // the query buffers are reused for this batch
    const uint32_t n = (uint32_t) queries.size();
    out.assign( n, {} );
    if( n == 0 )
        return;
    if( units.size() != n )
        fatal( "Internal error: pairs without a database sequence." );
    const int64_t mabs = max_abs_step( req );
    bool any = false;               // pairs with a non-empty sequence
    for( uint32_t i = 0; i < n; i++ ) {
        if( units[i] >= db.n_ids )
            fatal( "Internal error: database unit %u out of range.", units[i] );
        const uint32_t A = queries[i].len, B = db.len[units[i]];
        if( (int64_t) (A + B + 4) * (mabs + 1) * 2 > INT32_MAX )
            fatal( "Alignment of %u x %u residues exceeds the supported score range.", A, B );
        stats.cells += (uint64_t) A * B;
        if( B == 0 )
            continue;       // the reference never searches an empty sequence
        any = true;
        Hit h;
        h.unit = units[i];
        h.id = units[i] / db.upi;
        out[i].push_back( h );
    }
    CUDA_CHECK( cudaEventRecord( ev0_, stream_ ) );
    stage_.begin();
    upload_queries( req, queries.data(), n, false, stats );
    stage_.send( stream_ );
    d_counts_.ensure( 32 * sizeof(unsigned long long) );
    CUDA_CHECK( cudaMemsetAsync( d_counts_.p, 0, 32 * sizeof(unsigned long long), stream_ ) );
    // With alignments the traceback passes compute the score themselves: the
    // direction pass ends on cell (A - 1, B - 1) of the same recurrence
    // (Needleman-Wunsch), the forward region pass finds the same maximum when
    // the score table is symmetric (Smith-Waterman; it scores [query][db])
    bool symmetric = true;
    for( int d = 0; d < 32; d++ )
        for( int q = 0; q < 32; q++ )
            symmetric = symmetric && req.matrix[(d << 5) + q] == req.matrix[(q << 5) + d];
    const bool scores_in_traceback = req.align_type == COMPUTE_ALIGNMENT && (req.algo == 1 || symmetric);
    if( any && !scores_in_traceback ) {
        std::vector<std::pair<uint32_t, uint32_t>> lists;
        for( uint32_t i = 0; i < n; i++ )
            if( !out[i].empty() )
                lists.emplace_back( i, i );
        const auto t0 = std::chrono::steady_clock::now();
        traceback( req, out, lists, stats, false, true );
        const double seconds = std::chrono::duration<double>( std::chrono::steady_clock::now() - t0 ).count();
        stats.entry_seconds += seconds;
        stats.kernel_seconds += seconds;
    }
    if( req.align_type == COMPUTE_ALIGNMENT && any ) {
        std::vector<std::pair<uint32_t, uint32_t>> lists;
        for( uint32_t i = 0; i < n; i++ )
            if( !out[i].empty() )
                lists.emplace_back( i, i );
        const auto t0 = std::chrono::steady_clock::now();
        traceback( req, out, lists, stats, scores_in_traceback );
        stats.kernel_seconds += std::chrono::duration<double>( std::chrono::steady_clock::now() - t0 ).count();
    }
    CUDA_CHECK( cudaEventRecord( ev1_, stream_ ) );
    CUDA_CHECK( cudaEventSynchronize( ev1_ ) );
    float ms = 0;
    CUDA_CHECK( cudaEventElapsedTime( &ms, ev0_, ev1_ ) );
    stats.seconds_gpu += ms * 1e-3;
    stats.kernel_launches = launches_.load();
}

// ---- serving -------------------------------------------------------------------
// A server keeps a fixed number of query slots resident: slot s owns the codes at
// s * SERVE_QSTRIDE, its int32 profile at s * 32 * SERVE_MAX_QUERY and the score
// row s of d_serve_score_.  Each wave runs the entry pass and the cascade of every
// occupied slot over one segment of the length-sorted database; a slot that has
// seen every segment is finished (score rows to the host, schedule replay, heap,
// traceback) and freed for the next request.
constexpr uint32_t SERVE_QSTRIDE = SERVE_MAX_QUERY + 16;

// ---- database-sharded searches (one process per GPU, contiguous record
// ranges; the per-record results are gathered to one replaying process) ----
void Engine::shard_scores( const SearchRequest & req, const std::vector<QueryCodes> & queries, uint32_t id_lo,
        uint32_t id_hi, int64_t * scores, int32_t * blocks_entry, int32_t * blocks_16, SearchStats & stats ) {
    init_device();
    const HostDb & db = database();
    if( db.upi != 1 )
        fatal( "Database-sharded searches support one database strand." );
    if( streaming_ )
        fatal( "Database-sharded searches need the database resident on the device." );
    serving_ = false;
    serve_layout_ = false;
    last_shapes_.clear();
    id_hi = std::min( id_hi, db.n_ids );
    id_lo = std::min( id_lo, id_hi );
    const uint64_t width = id_hi - id_lo;
    const uint32_t nq_all = (uint32_t) queries.size();
    for( uint64_t k = 0; k < (uint64_t) nq_all * width; k++ ) {
        scores[k] = 0;
        blocks_entry[k] = -1;
        blocks_16[k] = -1;
    }
    if( width == 0 || queries.empty() )
        return;
    // this shard's non-empty records, longest first: the entry passes see it as
    // their whole database
    std::vector<uint32_t> shard;
    for( uint32_t id : db.order_desc )
        if( id >= id_lo && id < id_hi )
            shard.push_back( id );
    const uint64_t n_sh = shard.size();
    {
        uint32_t qmax = 0;
        for( const QueryCodes & q : queries )
            qmax = std::max( qmax, q.len );
        wide_ = needs_int64( req, qmax, db.max_len );
    }
    std::vector<uint32_t> full_order;
    full_order.swap( db_.order_desc );
    db_.order_desc = shard;
    if( n_sh )
        CUDA_CHECK( cudaMemcpyAsync( d_order_.p, shard.data(), n_sh * sizeof(uint32_t), cudaMemcpyHostToDevice,
                stream_ ) );
    const uint64_t pair_budget = this->pair_budget();
    const uint32_t batch = (uint32_t) std::max<uint64_t>( 1, std::min<uint64_t>( nq_all,
            pair_budget / std::max<uint64_t>( 1, db.n_ids ) ) );
    for( uint32_t b0 = 0; b0 < nq_all && n_sh; b0 += batch ) {
        const uint32_t nq = std::min( batch, nq_all - b0 );
        stage_.begin();
        upload_queries( req, queries.data() + b0, nq, true, stats );
        for( uint32_t q = 0; q < nq; q++ ) {
            uint64_t res = 0;
            for( uint32_t id : shard )
                res += db.len[id];
            stats.cells += (uint64_t) h_qlen_[q] * res;
        }
        const size_t score_bytes = (size_t) nq * db.n_ids * sizeof(int32_t);
        d_score_.ensure( std::max<size_t>( score_bytes, 4 ) );
        if( wide_ )
            d_score64_.ensure( std::max<size_t>( 2 * score_bytes, 8 ) );
        const uint32_t cap = (uint32_t) std::min<uint64_t>( std::max<uint64_t>( (uint64_t) nq * n_sh, 1 ),
                0xffffffffull );
        d_list_a_.ensure( (size_t) cap * sizeof(PairTask) );
        d_list_b_.ensure( (size_t) cap * sizeof(PairTask) );
        d_counts_.ensure( 32 * sizeof(unsigned long long) );
        CUDA_CHECK( cudaMemsetAsync( d_counts_.p, 0, 32 * sizeof(unsigned long long), stream_ ) );
        unsigned * cnt = d_counts_.as<unsigned>();
        const int entry = req.bit_width;
        CUDA_CHECK( cudaEventRecord( ev_seg_[0], stream_ ) );
        if( fast_eligible( req ) || nw_fast_eligible( req ) )
            run_qpair_entry( req, nq, d_list_a_.as<PairTask>(), cnt + 0, cap, d_list_b_.as<PairTask>(), nullptr, 0,
                    (uint32_t) n_sh );
        else
            run_pass( req.algo, entry, req, nq, nullptr, (uint64_t) nq * n_sh, true, d_list_a_.as<PairTask>(),
                    cnt + 0, cap );
        CUDA_CHECK( cudaEventRecord( ev_seg_[1], stream_ ) );
        std::vector<PairTask> list_entry, list_16;
        const unsigned * c = read_counts( true );
        c = run_redo( req, nq, c, d_list_a_.as<PairTask>(), cnt + 0, cap, d_list_b_.as<PairTask>(), cap );
        if( entry != 64 && std::min( c[0], cap ) )
            run_cascade( req, nq, std::min( c[0], cap ), cap, list_entry, list_16, nullptr, 0, (uint32_t) n_sh );
        int32_t * hs = (int32_t *) h_score_.ensure( std::max<size_t>( score_bytes, 4 ) );
        CUDA_CHECK( cudaMemcpyAsync( hs, d_score_.p, score_bytes, cudaMemcpyDeviceToHost, stream_ ) );
        int64_t * hs64 = nullptr;
        if( wide_ ) {
            hs64 = (int64_t *) h_score64_.ensure( 2 * score_bytes );
            CUDA_CHECK( cudaMemcpyAsync( hs64, d_score64_.p, 2 * score_bytes, cudaMemcpyDeviceToHost, stream_ ) );
        }
        unsigned err = 0;
        CUDA_CHECK( cudaMemcpyAsync( &err, cnt + 2, sizeof(unsigned), cudaMemcpyDeviceToHost, stream_ ) );
        CUDA_CHECK( cudaStreamSynchronize( stream_ ) );
        if( err )
            fatal( "Internal error in the GPU search (flags 0x%x).", err );
        float ms = 0;
        CUDA_CHECK( cudaEventElapsedTime( &ms, ev_seg_[0], ev_seg_[1] ) );
        stats.entry_seconds += ms * 1e-3;
        stats.d2h_bytes += score_bytes + (list_entry.size() + list_16.size()) * sizeof(PairTask);
        for( uint32_t q = 0; q < nq; q++ ) {
            const uint64_t row = (uint64_t) (b0 + q) * width;
            ReplayQuery rq;
            rq.score = hs + (size_t) q * db.n_ids;
            rq.score64 = hs64 ? hs64 + (size_t) q * db.n_ids : nullptr;
            for( uint32_t id : shard )
                scores[row + (id - id_lo)] = rq.score_of( id );
        }
        for( const PairTask & t : list_entry )
            blocks_entry[(uint64_t) (b0 + t.qslot) * width + (t.id - id_lo)] = t.nb_prev;
        for( const PairTask & t : list_16 )
            blocks_16[(uint64_t) (b0 + t.qslot) * width + (t.id - id_lo)] = t.nb_prev;
    }
    db_.order_desc.swap( full_order );
    if( !db_.order_desc.empty() )
        CUDA_CHECK( cudaMemcpyAsync( d_order_.p, db_.order_desc.data(), db_.order_desc.size() * sizeof(uint32_t),
                cudaMemcpyHostToDevice, stream_ ) );
    CUDA_CHECK( cudaStreamSynchronize( stream_ ) );
    stats.kernel_launches = launches_.load();
}

void Engine::align_hits( const SearchRequest & req, const std::vector<QueryCodes> & queries,
        std::vector<std::vector<Hit>> & out, SearchStats & stats ) {
    init_device();
    database();
    serving_ = false;
    serve_layout_ = false;
    const uint32_t nq = (uint32_t) queries.size();
    const uint32_t batch = 65535;
    for( uint32_t b0 = 0; b0 < nq; b0 += batch ) {
        const uint32_t n = std::min( batch, nq - b0 );
        CUDA_CHECK( cudaStreamSynchronize( stream_ ) );
        stage_.begin();
        upload_queries( req, queries.data() + b0, n, false, stats );
        std::vector<std::pair<uint32_t, uint32_t>> lists;
        for( uint32_t q = 0; q < n; q++ )
            lists.emplace_back( b0 + q, q );
        traceback( req, out, lists, stats );
    }
    CUDA_CHECK( cudaStreamSynchronize( stream_ ) );
}

void Engine::serve_restore( const SearchRequest & req ) {
    const uint32_t S = serve_slots_;
    h_qoff_.assign( S, 0 );
    h_qlen_.assign( S, 0 );
    h_qpad_.assign( S, 256 );
    h_prof_off_.assign( S, 0 );
    for( uint32_t s = 0; s < S; s++ ) {
        const uint32_t len = (uint32_t) serve_codes_[s].size();
        h_qoff_[s] = (uint64_t) s * SERVE_QSTRIDE;
        h_qlen_[s] = len;
        h_qpad_[s] = std::max<uint32_t>( 256, (len + 255u) & ~255u );
        h_prof_off_[s] = (uint64_t) s * 32 * SERVE_MAX_QUERY;
    }
    // one block: score table, offsets, lengths, codes
    const size_t at_qoff = 1024 * sizeof(int64_t), at_poff = at_qoff + S * sizeof(uint64_t),
            at_len = at_poff + S * sizeof(uint64_t), at_pad = at_len + S * sizeof(uint32_t),
            at_codes = (at_pad + S * sizeof(uint32_t) + 15) & ~(size_t) 15;
    char * block = (char *) d_serve_block_.ensure( at_codes + (size_t) S * SERVE_QSTRIDE + 16 );
    d_matrix_.p = block;
    d_qoff_.p = block + at_qoff;
    d_prof_off_.p = block + at_poff;
    d_qlen_.p = block + at_len;
    d_qpad_.p = block + at_pad;
    d_qcodes_.p = block + at_codes;
    d_prof_.ensure( (size_t) S * 32 * SERVE_MAX_QUERY * sizeof(int32_t) );
    d_counts_.ensure( 32 * sizeof(unsigned long long) );
    std::vector<char> head( at_codes, 0 );
    memcpy( head.data(), req.matrix, 1024 * sizeof(int64_t) );
    memcpy( head.data() + at_qoff, h_qoff_.data(), S * sizeof(uint64_t) );
    memcpy( head.data() + at_poff, h_prof_off_.data(), S * sizeof(uint64_t) );
    memcpy( head.data() + at_len, h_qlen_.data(), S * sizeof(uint32_t) );
    memcpy( head.data() + at_pad, h_qpad_.data(), S * sizeof(uint32_t) );
    CUDA_CHECK( cudaMemcpyAsync( block, head.data(), head.size(), cudaMemcpyHostToDevice, stream_ ) );
    for( uint32_t s = 0; s < S; s++ )
        if( !serve_codes_[s].empty() )
            CUDA_CHECK( cudaMemcpyAsync( d_qcodes_.as<uint8_t>() + h_qoff_[s], serve_codes_[s].data(),
                    serve_codes_[s].size(), cudaMemcpyHostToDevice, stream_ ) );
    CUDA_CHECK( cudaStreamSynchronize( stream_ ) );
    prof_width_ = -1;
    serve_layout_ = true;
    serve_new_.clear();
}

std::vector<uint32_t> Engine::serve_open( const SearchRequest & req, uint32_t slots, uint32_t segments ) {
    init_device();
    const HostDb & db = database();
    if( needs_int64( req, SERVE_MAX_QUERY, db.max_len ) )
        fatal( "The server scores in int32: the score table and gap penalties can exceed that range on this "
               "database; use sw_align/nw_align." );
    wide_ = false;
    serve_slots_ = slots;
    serve_codes_.assign( slots, {} );
    d_serve_score_.ensure( std::max<size_t>( 4, (size_t) slots * db.n_ids * sizeof(int32_t) ) );
    serve_layout_ = false;
    serve_restore( req );
    // the query-independent lane schedule of the entry width, computed once here
    // rather than in the first request's latency
    if( req.bit_width != 64 )
        ranks( req.chunk_size, req.bit_width == 8 ? req.lanes8 : req.lanes16 );
    // segments of the length-sorted sequences holding about equal residues
    const uint32_t n = (uint32_t) db.order_desc.size();
    segments = std::max<uint32_t>( 1, std::min<uint32_t>( segments, std::max<uint32_t>( 1, n ) ) );
    std::vector<uint32_t> bounds{ 0 };
    uint64_t acc = 0;
    for( uint32_t i = 0; i < n && bounds.size() < segments; i++ ) {
        acc += db.len[db.order_desc[i]];
        if( acc * segments >= db.residues * (uint64_t) bounds.size() )
            bounds.push_back( i + 1 );
    }
    if( bounds.back() != n )
        bounds.push_back( n );
    return bounds;
}

void Engine::serve_load( uint32_t slot, const uint8_t * codes, uint32_t len ) {
    serve_codes_[slot].assign( codes, codes + len );
    if( !serve_layout_ )
        return;     // restored before the next wave
    h_qlen_[slot] = len;
    h_qpad_[slot] = std::max<uint32_t>( 256, (len + 255u) & ~255u );
    serve_new_.push_back( slot );       // sent with the next wave
    prof_width_ = -1;
}

void Engine::serve_wave( const SearchRequest & req, const std::vector<uint32_t> & active, uint32_t seq_lo,
        uint32_t seq_hi, std::vector<PairTask> & ovf_entry, std::vector<PairTask> & ovf16, SearchStats & stats ) {
    ovf_entry.clear();
    ovf16.clear();
    if( active.empty() || seq_hi <= seq_lo )
        return;
    if( !serve_layout_ )
        serve_restore( req );
    stage_.begin();
    // the queries admitted since the last wave
    if( !serve_new_.empty() ) {
        for( uint32_t slot : serve_new_ ) {
            const uint8_t * codes = stage_.add( serve_codes_[slot].data(), serve_codes_[slot].size(), stream_ );
            stage_.send( stream_ );
            CUDA_CHECK( cudaMemcpyAsync( d_qcodes_.as<uint8_t>() + h_qoff_[slot], codes, serve_codes_[slot].size(),
                    cudaMemcpyDeviceToDevice, stream_ ) );
        }
        const uint32_t * len = stage_.add( h_qlen_.data(), h_qlen_.size(), stream_ );
        const uint32_t * pad = stage_.add( h_qpad_.data(), h_qpad_.size(), stream_ );
        stage_.send( stream_ );
        CUDA_CHECK( cudaMemcpyAsync( d_qlen_.p, len, h_qlen_.size() * sizeof(uint32_t), cudaMemcpyDeviceToDevice,
                stream_ ) );
        CUDA_CHECK( cudaMemcpyAsync( d_qpad_.p, pad, h_qpad_.size() * sizeof(uint32_t), cudaMemcpyDeviceToDevice,
                stream_ ) );
        serve_new_.clear();
    }
    serving_ = true;
    wide_ = false;                 // the server's settings were checked at serve_open
    const uint32_t n_seg = seq_hi - seq_lo;
    max_qlen_ = 0;
    uint64_t seg_res = 0;
    for( uint32_t i = seq_lo; i < seq_hi; i++ )
        seg_res += db_.len[db_.order_desc[i]];
    for( uint32_t s : active ) {
        max_qlen_ = std::max( max_qlen_, h_qlen_[s] );
        stats.cells += (uint64_t) h_qlen_[s] * seg_res;
    }
    const uint64_t n_pairs = (uint64_t) active.size() * n_seg;
    const uint32_t cap = (uint32_t) std::min<uint64_t>( std::max<uint64_t>( n_pairs, 1 ), 0xffffffffull );
    d_list_a_.ensure( (size_t) cap * sizeof(PairTask) );
    d_list_b_.ensure( (size_t) cap * sizeof(PairTask) );
    CUDA_CHECK( cudaMemsetAsync( d_counts_.p, 0, 32 * sizeof(unsigned long long), stream_ ) );
    unsigned * cnt = d_counts_.as<unsigned>();
    const int entry = req.bit_width;
    CUDA_CHECK( cudaEventRecord( ev_phase_[0], stream_ ) );
    if( fast_eligible( req ) || nw_fast_eligible( req ) ) {
        run_qpair_entry( req, serve_slots_, d_list_a_.as<PairTask>(), cnt + 0, cap, d_list_b_.as<PairTask>(), &active,
                seq_lo, seq_hi );
    }
    else {
        const uint32_t * dev_slots = stage_.add( active.data(), active.size(), stream_ );
        run_pass( req.algo, entry, req, serve_slots_, nullptr, n_pairs, true, d_list_a_.as<PairTask>(), cnt + 0, cap,
                dev_slots, (uint32_t) active.size(), seq_lo );
    }
    CUDA_CHECK( cudaEventRecord( ev_phase_[1], stream_ ) );
    const unsigned * c = read_counts( true );
    c = run_redo( req, serve_slots_, c, d_list_a_.as<PairTask>(), cnt + 0, cap, d_list_b_.as<PairTask>(), cap );
    if( entry != 64 && std::min( c[0], cap ) )
        run_cascade( req, serve_slots_, std::min( c[0], cap ), cap, ovf_entry, ovf16, &active, seq_lo, seq_hi );
    CUDA_CHECK( cudaEventRecord( ev_phase_[2], stream_ ) );
    const unsigned err = read_counts( false )[2];
    serving_ = false;
    if( err )
        fatal( "Internal error in the GPU search (flags 0x%x).", err );
    float ms[2];
    CUDA_CHECK( cudaEventElapsedTime( &ms[0], ev_phase_[0], ev_phase_[1] ) );
    CUDA_CHECK( cudaEventElapsedTime( &ms[1], ev_phase_[1], ev_phase_[2] ) );
    stats.entry_seconds += ms[0] * 1e-3;
    stats.kernel_seconds += (ms[0] + ms[1]) * 1e-3;
    stats.overflow8 += ovf_entry.size();
    stats.overflow16 += ovf16.size();
}

void Engine::serve_finish( const SearchRequest & req, const std::vector<uint32_t> & done,
        std::vector<ReplayQuery> & rq, std::vector<std::vector<Hit>> & out, SearchStats & stats ) {
    out.assign( serve_slots_, {} );
    if( done.empty() )
        return;
    if( !serve_layout_ )
        serve_restore( req );
    const uint32_t nd = (uint32_t) done.size();
    const size_t row = (size_t) db_.n_ids;
    int32_t * hs = (int32_t *) h_score_.ensure( std::max<size_t>( 4, nd * row * sizeof(int32_t) ) );
    for( uint32_t i = 0; i < nd; i++ )
        CUDA_CHECK( cudaMemcpyAsync( hs + i * row, d_serve_score_.as<int32_t>() + (size_t) done[i] * row,
                row * sizeof(int32_t), cudaMemcpyDeviceToHost, stream_ ) );
    CUDA_CHECK( cudaStreamSynchronize( stream_ ) );
    stats.d2h_bytes += nd * row * sizeof(int32_t);
    const int entry = req.bit_width;
    const uint32_t * rank_entry =
            (entry == 64) ? nullptr : ranks( req.chunk_size, entry == 8 ? req.lanes8 : req.lanes16 );
    {
        std::atomic<uint32_t> next{ 0 };
        std::vector<ReplayCounts> counts( nd );
        auto work = [&]() {
            for( ;; ) {
                const uint32_t i = next.fetch_add( 1 );
                if( i >= nd )
                    break;
                rq[i].score = hs + i * row;
                std::sort( rq[i].ovf_entry.begin(), rq[i].ovf_entry.end() );
                std::sort( rq[i].ovf16.begin(), rq[i].ovf16.end() );
                replay_query( db_, req, rq[i], rank_entry, out[done[i]], counts[i] );
            }
        };
        const unsigned nthreads = std::min<unsigned>( std::max( 1u, std::thread::hardware_concurrency() ), nd );
        std::vector<std::thread> th;
        for( unsigned k = 1; k < nthreads; k++ )
            th.emplace_back( work );
        work();
        for( auto & t : th )
            t.join();
    }
    if( req.align_type == COMPUTE_ALIGNMENT ) {
        max_qlen_ = 0;
        for( uint32_t s : done )
            max_qlen_ = std::max( max_qlen_, h_qlen_[s] );
        std::vector<std::pair<uint32_t, uint32_t>> lists;
        for( uint32_t sl : done )
            lists.emplace_back( sl, sl );
        traceback( req, out, lists, stats );
    }
}

// ---- free functions ------------------------------------------------------------
// One engine per process; the search entry points and a server's waves take
// turns on it.
static std::mutex g_engine_mutex;

void engine_search( const SearchRequest & req, const std::vector<QueryCodes> & queries,
        const std::vector<uint32_t> & groups, std::vector<std::vector<Hit>> & out, SearchStats & stats ) {
    std::lock_guard<std::mutex> lock( g_engine_mutex );
    Engine::get().search( req, queries, groups, out, stats );
}

void engine_align_pairs( const SearchRequest & req, const std::vector<QueryCodes> & queries,
        const std::vector<uint32_t> & units, std::vector<std::vector<Hit>> & out, SearchStats & stats ) {
    std::lock_guard<std::mutex> lock( g_engine_mutex );
    Engine::get().align_pairs( req, queries, units, out, stats );
}

void engine_set_traceback_memory( uint64_t bytes ) {
    std::lock_guard<std::mutex> lock( g_engine_mutex );
    Engine::get().set_traceback_budget( bytes );
}

void engine_set_db_memory( uint64_t bytes ) {
    std::lock_guard<std::mutex> lock( g_engine_mutex );
    Engine::get().set_db_budget( bytes );
}

bool engine_streaming() {
    std::lock_guard<std::mutex> lock( g_engine_mutex );
    Engine & e = Engine::get();
    e.database();
    return e.streaming();
}

const HostDb & engine_database() {
    std::lock_guard<std::mutex> lock( g_engine_mutex );
    return Engine::get().database();
}

void engine_invalidate_database() {
    std::lock_guard<std::mutex> lock( g_engine_mutex );
    Engine::get().invalidate();
}

void engine_shutdown() {
    std::lock_guard<std::mutex> lock( g_engine_mutex );
    Engine::get().shutdown();
}

std::vector<uint32_t> engine_serve_open( const SearchRequest & req, uint32_t slots, uint32_t segments ) {
    std::lock_guard<std::mutex> lock( g_engine_mutex );
    return Engine::get().serve_open( req, slots, segments );
}

void engine_serve_load( uint32_t slot, const uint8_t * codes, uint32_t len ) {
    std::lock_guard<std::mutex> lock( g_engine_mutex );
    Engine::get().serve_load( slot, codes, len );
}

void engine_serve_wave( const SearchRequest & req, const std::vector<uint32_t> & active, uint32_t seq_lo,
        uint32_t seq_hi, std::vector<ServeOverflow> & ovf_entry, std::vector<ServeOverflow> & ovf16,
        SearchStats & stats ) {
    std::vector<PairTask> a, b;
    {
        std::lock_guard<std::mutex> lock( g_engine_mutex );
        Engine::get().serve_wave( req, active, seq_lo, seq_hi, a, b, stats );
    }
    ovf_entry.clear();
    ovf16.clear();
    for( const PairTask & t : a )
        ovf_entry.push_back( ServeOverflow{ t.qslot, t.id, t.nb_prev } );
    for( const PairTask & t : b )
        ovf16.push_back( ServeOverflow{ t.qslot, t.id, t.nb_prev } );
}

void engine_serve_finish( const SearchRequest & req, const std::vector<uint32_t> & done,
        std::vector<ReplayQuery> & rq, std::vector<std::vector<Hit>> & out, SearchStats & stats ) {
    std::lock_guard<std::mutex> lock( g_engine_mutex );
    Engine::get().serve_finish( req, done, rq, out, stats );
}

void engine_shard_scores( const SearchRequest & req, const std::vector<QueryCodes> & queries, uint32_t id_lo,
        uint32_t id_hi, int64_t * scores, int32_t * blocks_entry, int32_t * blocks_16, SearchStats & stats ) {
    std::lock_guard<std::mutex> lock( g_engine_mutex );
    Engine::get().shard_scores( req, queries, id_lo, id_hi, scores, blocks_entry, blocks_16, stats );
}

void engine_align_hits( const SearchRequest & req, const std::vector<QueryCodes> & queries,
        std::vector<std::vector<Hit>> & out, SearchStats & stats ) {
    std::lock_guard<std::mutex> lock( g_engine_mutex );
    Engine::get().align_hits( req, queries, out, stats );
}

// Host-only: the database's record lengths through the plugin (no device),
// as the schedule replay needs them.
void lengths_db( HostDb & db ) {
    db = HostDb();
    const size_t n = ssa_db_get_sequence_count();
    if( n > UINT32_MAX )
        fatal( "Database has %zu sequences; at most %u are supported.", n, UINT32_MAX );
    db.n_ids = db.n_records = (uint32_t) n;
    db.upi = 1;
    db.len.assign( n, 0 );
    for( size_t id = 0; id < n; id++ ) {
        p_seqinfo info = ssa_db_get_sequence( id );
        if( !info )
            fatal( "Could not get sequence from DB: %zu", id );
        db.len[id] = (uint32_t) info->seqlen;
        db.max_len = std::max( db.max_len, db.len[id] );
        db.residues += info->seqlen;
    }
    db.nonempty_before.assign( n + 1, 0 );
    for( uint32_t id = 0; id < db.n_ids; id++ ) {
        db.nonempty_before[id + 1] = db.nonempty_before[id] + (db.len[id] ? 1 : 0);
        if( db.len[id] )
            db.order_desc.push_back( id );
    }
    std::stable_sort( db.order_desc.begin(), db.order_desc.end(),
            [&]( uint32_t a, uint32_t b ) { return db.len[a] > db.len[b]; } );
    db.mean_len = db.order_desc.empty() ? 0.0 : (double) db.residues / (double) db.order_desc.size();
}

std::string tuning_report() {
    const TuningTable & t = tuning();
    std::string out = "{\"source\": \"";
    for( char c : t.source )
        if( c != '"' && c != '\\' )
            out += c;
    out += "\", \"version\": " + std::to_string( t.version ) + ", \"device\": \"";
    for( char c : t.device )
        if( c != '"' && c != '\\' )
            out += c;
    out += "\", \"last_call\": [";
    std::lock_guard<std::mutex> lock( g_engine_mutex );
    bool first = true;
    for( const auto & u : Engine::get().last_shapes_ ) {
        char buf[160];
        const bool qp = strncmp( u.kernel, "sw_fast", 7 ) != 0;
        snprintf( buf, sizeof buf, "%s{\"kernel\": \"%s\", \"%s\": %d, \"%s\": %d, \"%s\": %u, \"bucket\": %d}",
                first ? "" : ", ", u.kernel, qp ? "R" : "G", u.a, qp ? "ctas_per_sm" : "R", u.b,
                qp ? "query_pairs" : "queries", u.n, u.bucket );
        out += buf;
        first = false;
    }
    out += "]}";
    return out;
}

uint64_t engine_kernel_launches() {
    return Engine::get().launches();
}

}  // namespace ssa
