// readback.cu -- device-to-host copies of diagnostics.
//
// A driver copy into pageable memory goes through one staging thread: 16 GB/s
// into pages that the process has just used, 2 to 8 into pages that it has to
// fault in, of the link's 55.  So a copy goes through two pinned chunks here, and
// a large one is cut into LANES parts, each with its own stream, chunks and host
// thread, so that the copies over the link, the page faults of the destination
// and the host-side copies overlap: 35.8 MB (one field of 2048x1024 cells) into
// fresh memory takes 2.5 ms instead of 7.9, 1.1 MB 0.43 instead of 0.55.
#include <cuda_runtime.h>
#include <sys/mman.h>

#include <algorithm>
#include <cstdint>
#include <cstring>
#include <map>
#include <memory>
#include <mutex>
#include <thread>
#include <vector>

namespace zb {

namespace {

constexpr int LANES = 4;
constexpr size_t CHUNK = 512 * 1024;          // pinned bytes per slot (two slots per lane)
constexpr size_t CHUNK_FIRST = 160 * 1024;    // those of the further lanes until they have copied PAYS bytes
constexpr size_t PAYS = 256 << 20;
constexpr size_t SMALL = 64 * 1024;           // the driver's own path is as good below
// All lanes into fresh pages, and into pages that are there, from this many bytes
// on, one below.  Waking a thread costs up to 0.25 ms.  With one lane, four lanes
// and by the driver: 4.4 MB of fresh pages 1.3, 0.9 and 1.7 ms; an array in memory
// just given back 0.49, 0.70 to 0.88 and 0.71, 13.4 MB there 1.5, 1.7 and 1.9;
// one buffer again and again 2.1 MB 0.15, 0.40 and 0.15, 4.4 MB 0.30, 0.25 to
// 0.94 and 0.28; 2.1 MB of fresh pages 0.82, 0.58 and 1.0.
constexpr size_t WIDE_FRESH = 2 << 20, WIDE = 12 << 20;

struct Lane {
    cudaStream_t st = nullptr;                // none for the first lane: it copies on the caller's stream
    cudaEvent_t done[2] = { nullptr, nullptr };
    char * buf = nullptr;                     // two chunks
    size_t chunk = 0;
};

// The lanes of one device, made when they are first used and given back when the
// device's last simulation is destroyed.  The first read-out of a simulation
// pays for them, so they are made to cost little: the first lane needs no stream,
// and the driver cuts pinned buffers from blocks of 2 MB, 1.3 ms each, of which
// every simulation holds one for its scratch: the lanes' 1.94 MB fit the rest of
// it (4 MB of buffers and four streams made at once took 2.1 to 5 ms, and 0.9 ms
// when they were given back; now 0.01 ms, and 0.2 for the three streams of a wide
// copy).  Small chunks cost a wide copy a tenth, so that after PAYS bytes, 25 ms of
// copying, the further lanes get large ones as well.
struct Pool {
    std::mutex busy;
    Lane lane[LANES];
    cudaEvent_t ready = nullptr;
    int made = 0;
    size_t wide_bytes = 0;
    int users = 0;

    // lanes [0, n) are there, or as many as could be made
    void make( int n ) {
        cudaError_t e = cudaSuccess;
        if ( !ready && n > 1 ) e = cudaEventCreateWithFlags( &ready, cudaEventDisableTiming );
        for ( int k = 0; k < n && e == cudaSuccess; k++ ) {
            Lane & l = lane[k];
            const size_t chunk = k == 0 || wide_bytes >= PAYS ? CHUNK : CHUNK_FIRST;
            if ( l.chunk == chunk ) continue;
            if ( l.buf ) { cudaFreeHost( l.buf ); l.buf = nullptr; }        // (larger chunks)
            if ( k > 0 && !l.st ) e = cudaStreamCreateWithFlags( &l.st, cudaStreamNonBlocking );
            for ( int i = 0; i < 2; i++ )
                if ( e == cudaSuccess && !l.done[i] ) e = cudaEventCreateWithFlags( &l.done[i], cudaEventDisableTiming );
            if ( e == cudaSuccess ) e = cudaHostAlloc( (void **) &l.buf, 2 * chunk, cudaHostAllocPortable );
            if ( e == cudaSuccess ) { l.chunk = chunk; made = std::max( made, k + 1 ); }
            else { free_lane( l ); made = std::min( made, k ); }
        }
        if ( e != cudaSuccess ) cudaGetLastError();
    }
    void free_lane( Lane & l ) {
        if ( l.st ) { cudaStreamSynchronize( l.st ); cudaStreamDestroy( l.st ); }
        for ( int k = 0; k < 2; k++ ) if ( l.done[k] ) cudaEventDestroy( l.done[k] );
        if ( l.buf ) cudaFreeHost( l.buf );
        l = Lane{};
    }
    void drop() {
        for ( auto & l : lane ) free_lane( l );
        if ( ready ) cudaEventDestroy( ready );
        ready = nullptr;
        made = 0;
        wide_bytes = 0;
    }
};

std::mutex g_pools_mutex;
std::map<int, std::unique_ptr<Pool>> g_pools;

// One lane's part: chunk k comes over the link while chunk k - 1 is copied out.
cudaError_t run_lane( int device, Lane & l, cudaStream_t st, char * dst, const char * src, size_t bytes ) {
    cudaError_t e = cudaSetDevice( device );
    if ( e != cudaSuccess ) return e;
    const size_t n = ( bytes + l.chunk - 1 ) / l.chunk;
    for ( size_t k = 0; k <= n; k++ ) {
        const int b = (int) ( k & 1 );
        if ( k < n ) {
            const size_t at = k * l.chunk, len = std::min( l.chunk, bytes - at );
            e = cudaMemcpyAsync( l.buf + b * l.chunk, src + at, len, cudaMemcpyDeviceToHost, st );
            if ( e == cudaSuccess ) e = cudaEventRecord( l.done[b], st );
            if ( e != cudaSuccess ) break;
        }
        if ( k > 0 ) {
            const size_t at = ( k - 1 ) * l.chunk, len = std::min( l.chunk, bytes - at );
            e = cudaEventSynchronize( l.done[1 - b] );
            if ( e != cudaSuccess ) break;
            std::memcpy( dst + at, l.buf + ( 1 - b ) * l.chunk, len );
        }
    }
    if ( e != cudaSuccess ) cudaStreamSynchronize( st );       // nothing of this copy is left in flight
    return e;
}

cudaError_t copy_plain( cudaStream_t st, void * dst, const void * src, size_t bytes ) {
    const cudaError_t e = cudaMemcpyAsync( dst, src, bytes, cudaMemcpyDeviceToHost, st );
    return e != cudaSuccess ? e : cudaStreamSynchronize( st );
}

// Whether the destination's pages have still to be faulted in (by a few of them).
bool fresh_pages( const void * dst, size_t bytes ) {
    constexpr uintptr_t PAGE = 4096, SAMPLES = 8;
    for ( uintptr_t k = 0; k < SAMPLES; k++ ) {
        const uintptr_t at = ( reinterpret_cast<uintptr_t>( dst ) + ( 2 * k + 1 ) * ( bytes / ( 2 * SAMPLES ) ) ) & ~( PAGE - 1 );
        unsigned char there = 0;
        if ( mincore( reinterpret_cast<void *>( at ), PAGE, &there ) == 0 && ( there & 1 ) ) return false;
    }
    return true;
}

}  // namespace

// Called for every simulation made on and destroyed from a device.
void readback_retain( int device ) {
    std::lock_guard<std::mutex> g( g_pools_mutex );
    auto & p = g_pools[ device ];
    if ( !p ) p = std::make_unique<Pool>();
    p->users++;
}
void readback_release( int device ) {
    std::lock_guard<std::mutex> g( g_pools_mutex );
    auto it = g_pools.find( device );
    if ( it == g_pools.end() || --it->second->users > 0 ) return;
    std::lock_guard<std::mutex> b( it->second->busy );
    it->second->drop();
}

// bytes of device memory to host memory in the order of stream st; returns
// when they have arrived.  Pinned destinations, small copies and copies that
// find the lanes in use by another thread go to the driver directly.
cudaError_t copy_to_host( int device, cudaStream_t st, void * dst, const void * src, size_t bytes ) {
    if ( bytes == 0 ) return cudaStreamSynchronize( st );
    if ( bytes <= SMALL ) return copy_plain( st, dst, src, bytes );
    cudaPointerAttributes a{};
    if ( cudaPointerGetAttributes( &a, dst ) != cudaSuccess ) cudaGetLastError();
    else if ( a.type != cudaMemoryTypeUnregistered ) return copy_plain( st, dst, src, bytes );
    Pool * pool = nullptr;
    {
        std::lock_guard<std::mutex> g( g_pools_mutex );
        auto it = g_pools.find( device );
        if ( it != g_pools.end() ) pool = it->second.get();
    }
    if ( !pool ) return copy_plain( st, dst, src, bytes );
    std::unique_lock<std::mutex> own( pool->busy, std::try_to_lock );
    if ( !own.owns_lock() ) return copy_plain( st, dst, src, bytes );
    const bool wide = ( bytes >= WIDE || ( bytes >= WIDE_FRESH && fresh_pages( dst, bytes ) ) ) &&
                      std::thread::hardware_concurrency() >= LANES;
    if ( wide && pool->wide_bytes < PAYS ) pool->wide_bytes += bytes;
    pool->make( wide ? LANES : 1 );
    if ( pool->made == 0 ) return copy_plain( st, dst, src, bytes );
    const int lanes = wide ? pool->made : 1;
    cudaError_t e = cudaSuccess;
    if ( lanes > 1 ) e = cudaEventRecord( pool->ready, st );
    for ( int k = 1; k < lanes && e == cudaSuccess; k++ ) e = cudaStreamWaitEvent( pool->lane[k].st, pool->ready, 0 );
    if ( e != cudaSuccess ) return e;
    const size_t part = ( ( bytes + lanes - 1 ) / lanes + 4095 ) & ~(size_t) 4095;
    cudaError_t err[LANES];
    auto work = [&]( int k ) {
        const size_t at = std::min( bytes, k * part ), len = std::min( part, bytes - at );
        err[k] = len ? run_lane( device, pool->lane[k], k ? pool->lane[k].st : st, (char *) dst + at, (const char *) src + at, len ) : cudaSuccess;
    };
    std::thread th[LANES];
    int started = 1;
    try {
        for ( ; started < lanes; started++ ) th[started] = std::thread( work, started );
    } catch ( ... ) {
        // no more threads to be had: this one does the remaining parts
    }
    work( 0 );
    for ( int k = started; k < lanes; k++ ) work( k );
    for ( int k = 1; k < started; k++ ) th[k].join();
    for ( int k = 0; k < lanes; k++ ) if ( e == cudaSuccess ) e = err[k];
    return e;
}

}  // namespace zb
