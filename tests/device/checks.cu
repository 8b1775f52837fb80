// Device functions of the library under test on their own: the pair arithmetic against the GPU's IEEE operations,
// the bounded wait on a phase that completes and on one that never does.  Built beside the library.
#include <cuda_runtime.h>

#include <cstdint>

#include "zpic_dev.cuh"
#include "pair_math.cuh"

using namespace zb;

namespace {

constexpr int THREADS = 256, BLOCKS = 148 * 16;

__device__ void halves( F2 x, float & a, float & b ) { unpack2( x, a, b ); }
__device__ bool differ( float a, float b ) { return __float_as_uint( a ) != __float_as_uint( b ); }
__device__ uint32_t mix( uint64_t x ) {              // splitmix64
    x += 0x9E3779B97F4A7C15ull;
    x = ( x ^ ( x >> 30 ) ) * 0xBF58476D1CE4E5B9ull;
    x = ( x ^ ( x >> 27 ) ) * 0x94D049BB133111EBull;
    return (uint32_t) ( ( x ^ ( x >> 31 ) ) >> 16 );
}

// bad[0]: roots, bad[1]: reciprocals of the floats with bits [first, last) that differ; the other half of each pair
// holds another float of the range
__global__ void k_roots( uint32_t first, uint32_t last, unsigned long long * bad ) {
    unsigned long long r = 0, q = 0;
    for ( uint64_t i = (uint64_t) first + blockIdx.x * THREADS + threadIdx.x; i < last; i += (uint64_t) gridDim.x * THREADS ) {
        const float x = __uint_as_float( (uint32_t) i ), y = __uint_as_float( last - 1 - (uint32_t) ( i - first ) );
        float a, b;
        halves( sqrt2( pack2( x, y ) ), a, b );
        r += differ( a, __fsqrt_rn( x ) ) + differ( b, __fsqrt_rn( y ) );
        halves( recip2( pack2( x, y ) ), a, b );
        q += differ( a, __frcp_rn( x ) ) + differ( b, __frcp_rn( y ) );
    }
    if ( r ) atomicAdd( bad, r );
    if ( q ) atomicAdd( bad + 1, q );
}

// utsq / ( sqrt( 1 + utsq ) + 1 ), the energy term, for the floats with bits [first, last)
__global__ void k_energy_terms( uint32_t first, uint32_t last, unsigned long long * bad ) {
    unsigned long long r = 0;
    for ( uint64_t i = (uint64_t) first + blockIdx.x * THREADS + threadIdx.x; i < last; i += (uint64_t) gridDim.x * THREADS ) {
        const float x = __uint_as_float( (uint32_t) i ), y = __uint_as_float( last - 1 - (uint32_t) ( i - first ) );
        const F2 t = pack2( x, y ), one = both( 1.0f );
        const F2 g1 = sqrt2( one + t ) + one;
        float a, b;
        halves( quot2( t, g1, recip2( g1 ) ), a, b );
        r += differ( a, __fdiv_rn( x, __fsqrt_rn( 1.0f + x ) + 1.0f ) ) + differ( b, __fdiv_rn( y, __fsqrt_rn( 1.0f + y ) + 1.0f ) );
    }
    if ( r ) atomicAdd( bad, r );
}

// alpha / gamma: every significand of gamma with exponents of [0, 48), n numerators each with any significand and
// magnitudes of (1e-18, 1e18)
__global__ void k_quotients( int n, unsigned long long * bad ) {
    unsigned long long r = 0;
    for ( uint32_t m = blockIdx.x * THREADS + threadIdx.x; m < 1u << 23; m += gridDim.x * THREADS )
        for ( int k = 0; k < n; k++ ) {
            const uint32_t h = mix( (uint64_t) m * n + k ), g = mix( ~( (uint64_t) m * n + k ) );
            const float d = __uint_as_float( ( 127u + h % 48u ) << 23 | m );
            const float e = __uint_as_float( ( 127u + g % 48u ) << 23 | ( ~m & 0x7fffffu ) );
            // 2^-59 > 1e-18, 2^59 < 1e18
            const float x = __uint_as_float( ( 127u - 59u + ( h >> 8 ) % 118u ) << 23 | ( g >> 9 ) );
            const float y = -__uint_as_float( ( 127u - 59u + ( g >> 8 ) % 118u ) << 23 | ( h >> 9 ) );
            const F2 p = pack2( d, e );
            float a, b;
            halves( quot2( pack2( x, y ), p, recip2( p ) ), a, b );
            r += differ( a, __fdiv_rn( x, d ) ) + differ( b, __fdiv_rn( y, e ) );
        }
    if ( r ) atomicAdd( bad, r );
}

// out[0]: the wait's answer, out[1]: nanoseconds it took, out[2]: the status word.  The phase completes before the
// wait (arrive != 0), or nothing ever completes it; no copy is in flight in either case.
__global__ void k_wait( int arrive, int limit, int * out ) {
    __shared__ uint64_t bar;
    if ( threadIdx.x == 0 ) {
        mbar_init( &bar, 1 );
        fence_mbar_init();
        if ( arrive ) mbar_arrive_expect_tx( &bar, 0 );
    }
    __syncthreads();
    unsigned long long t0, t1;
    asm volatile( "mov.u64 %0, %globaltimer;" : "=l"( t0 ) );
    const bool ok = mbar_wait_bounded( &bar, 0, out + 2, limit );
    asm volatile( "mov.u64 %0, %globaltimer;" : "=l"( t1 ) );
    if ( threadIdx.x == 0 ) { out[0] = ok; out[1] = (int) ( t1 - t0 ); }
}

template < class T, class F > int run( T * host, int n, F launch ) {
    T * d = nullptr;
    cudaError_t e = cudaMalloc( &d, n * sizeof( T ) );
    if ( e == cudaSuccess ) e = cudaMemset( d, 0, n * sizeof( T ) );
    if ( e == cudaSuccess ) { launch( d ); e = cudaGetLastError(); }
    if ( e == cudaSuccess ) e = cudaMemcpy( host, d, n * sizeof( T ), cudaMemcpyDeviceToHost );
    cudaFree( d );
    return (int) e;
}

}  // namespace

extern "C" int check_roots( uint32_t first, uint32_t last, unsigned long long bad[2] ) {
    return run( bad, 2, [&]( unsigned long long * d ) { k_roots<<< BLOCKS, THREADS >>>( first, last, d ); } );
}
extern "C" int check_energy_terms( uint32_t first, uint32_t last, unsigned long long bad[1] ) {
    return run( bad, 1, [&]( unsigned long long * d ) { k_energy_terms<<< BLOCKS, THREADS >>>( first, last, d ); } );
}
extern "C" int check_quotients( int n, unsigned long long bad[1] ) {
    return run( bad, 1, [&]( unsigned long long * d ) { k_quotients<<< BLOCKS, THREADS >>>( n, d ); } );
}
extern "C" int check_wait( int arrive, int limit, int out[3] ) {
    return run( out, 3, [&]( int * d ) { k_wait<<< 1, 64 >>>( arrive, limit, d ); } );
}
