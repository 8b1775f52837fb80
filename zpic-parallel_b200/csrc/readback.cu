// readback.cu -- device-to-host copies of diagnostics.
//
// A driver copy into pageable memory goes through one staging thread: 8 GB/s
// into fresh memory, of the link's 55.  Here a copy is cut into up to LANES
// parts, each with its own stream, two pinned chunks and host thread, so
// that the copies over the link, the page faults of the destination and the
// host-side copies overlap: 35.8 MB (one field of 2048x1024 cells) into fresh
// memory takes 2.5 ms instead of 7.9.
#include <cuda_runtime.h>

#include <algorithm>
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
constexpr size_t SMALL = 64 * 1024;           // the driver's own path is as good below
constexpr size_t PER_LANE = 1024 * 1024;      // a further lane (host thread) pays from this many bytes on

struct Lane {
    cudaStream_t st = nullptr;
    cudaEvent_t done[2] = { nullptr, nullptr };
    char * buf = nullptr;                     // two chunks
};

// The lanes of one device: 4 MB of pinned memory, made at the first copy that
// uses them and given back when the device's last simulation is destroyed.
struct Pool {
    std::mutex busy;
    Lane lane[LANES];
    cudaEvent_t ready = nullptr;
    bool made = false;
    int users = 0;

    cudaError_t make() {
        if ( made ) return cudaSuccess;
        cudaError_t e = cudaEventCreateWithFlags( &ready, cudaEventDisableTiming );
        for ( auto & l : lane ) {
            if ( e == cudaSuccess ) e = cudaStreamCreateWithFlags( &l.st, cudaStreamNonBlocking );
            for ( int k = 0; k < 2; k++ )
                if ( e == cudaSuccess ) e = cudaEventCreateWithFlags( &l.done[k], cudaEventDisableTiming );
            if ( e == cudaSuccess ) e = cudaHostAlloc( (void **) &l.buf, 2 * CHUNK, cudaHostAllocPortable );
        }
        made = true;
        if ( e != cudaSuccess ) drop();
        return e;
    }
    void drop() {
        if ( !made ) return;
        for ( auto & l : lane ) {
            if ( l.st ) { cudaStreamSynchronize( l.st ); cudaStreamDestroy( l.st ); }
            for ( int k = 0; k < 2; k++ ) if ( l.done[k] ) cudaEventDestroy( l.done[k] );
            if ( l.buf ) cudaFreeHost( l.buf );
            l = Lane{};
        }
        if ( ready ) cudaEventDestroy( ready );
        ready = nullptr;
        made = false;
    }
};

std::mutex g_pools_mutex;
std::map<int, std::unique_ptr<Pool>> g_pools;

// One lane's part: chunk k comes over the link while chunk k - 1 is copied out.
cudaError_t run_lane( int device, Lane & l, char * dst, const char * src, size_t bytes ) {
    cudaError_t e = cudaSetDevice( device );
    if ( e != cudaSuccess ) return e;
    const size_t n = ( bytes + CHUNK - 1 ) / CHUNK;
    for ( size_t k = 0; k <= n; k++ ) {
        const int b = (int) ( k & 1 );
        if ( k < n ) {
            const size_t at = k * CHUNK, len = std::min( CHUNK, bytes - at );
            e = cudaMemcpyAsync( l.buf + b * CHUNK, src + at, len, cudaMemcpyDeviceToHost, l.st );
            if ( e == cudaSuccess ) e = cudaEventRecord( l.done[b], l.st );
            if ( e != cudaSuccess ) break;
        }
        if ( k > 0 ) {
            const size_t at = ( k - 1 ) * CHUNK, len = std::min( CHUNK, bytes - at );
            e = cudaEventSynchronize( l.done[1 - b] );
            if ( e != cudaSuccess ) break;
            std::memcpy( dst + at, l.buf + ( 1 - b ) * CHUNK, len );
        }
    }
    if ( e != cudaSuccess ) cudaStreamSynchronize( l.st );     // nothing of this copy is left in flight
    return e;
}

cudaError_t copy_plain( cudaStream_t st, void * dst, const void * src, size_t bytes ) {
    const cudaError_t e = cudaMemcpyAsync( dst, src, bytes, cudaMemcpyDeviceToHost, st );
    return e != cudaSuccess ? e : cudaStreamSynchronize( st );
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
    if ( !own.owns_lock() || pool->make() != cudaSuccess ) { cudaGetLastError(); return copy_plain( st, dst, src, bytes ); }
    const unsigned cores = std::thread::hardware_concurrency();
    const int lanes = (int) std::max<size_t>( 1, std::min<size_t>( { (size_t) LANES, bytes / PER_LANE, (size_t) std::max( 1u, cores ) } ) );
    cudaError_t e = cudaEventRecord( pool->ready, st );
    for ( int k = 0; k < lanes && e == cudaSuccess; k++ ) e = cudaStreamWaitEvent( pool->lane[k].st, pool->ready, 0 );
    if ( e != cudaSuccess ) return e;
    const size_t part = ( ( bytes + lanes - 1 ) / lanes + 4095 ) & ~(size_t) 4095;
    cudaError_t err[LANES];
    auto work = [&]( int k ) {
        const size_t at = std::min( bytes, k * part ), len = std::min( part, bytes - at );
        err[k] = len ? run_lane( device, pool->lane[k], (char *) dst + at, (const char *) src + at, len ) : cudaSuccess;
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
