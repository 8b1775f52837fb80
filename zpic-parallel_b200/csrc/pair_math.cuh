// pair_math.cuh -- FP32 arithmetic on two particles at a time, for sm_100a.
#pragma once

namespace zb {

// ---------------------------------------------------------------------------
// Two particles at a time
//
// A thread pushes, moves and deposits its two particles together, their FP32
// values in the two halves of 64-bit registers, with sm_100's packed
// instructions (add, mul and fma .f32x2): one instruction slot for two
// particles, each half rounded as the scalar instruction rounds it.  The
// particle kernel is bound by instruction issue.
// ---------------------------------------------------------------------------
struct F2 { unsigned long long v; };
__device__ __forceinline__ F2 pack2( float a, float b ) { F2 r; asm( "mov.b64 %0, {%1, %2};" : "=l"( r.v ) : "f"( a ), "f"( b ) ); return r; }
__device__ __forceinline__ F2 both( float a ) { return pack2( a, a ); }
__device__ __forceinline__ void unpack2( F2 x, float & a, float & b ) { asm( "mov.b64 {%0, %1}, %2;" : "=f"( a ), "=f"( b ) : "l"( x.v ) ); }
__device__ __forceinline__ F2 operator+( F2 a, F2 b ) { F2 r; asm( "add.rn.f32x2 %0, %1, %2;" : "=l"( r.v ) : "l"( a.v ), "l"( b.v ) ); return r; }
__device__ __forceinline__ F2 operator-( F2 a, F2 b ) { F2 r; asm( "sub.rn.f32x2 %0, %1, %2;" : "=l"( r.v ) : "l"( a.v ), "l"( b.v ) ); return r; }
__device__ __forceinline__ F2 operator*( F2 a, F2 b ) { F2 r; asm( "mul.rn.f32x2 %0, %1, %2;" : "=l"( r.v ) : "l"( a.v ), "l"( b.v ) ); return r; }
__device__ __forceinline__ F2 fma2( F2 a, F2 b, F2 c ) { F2 r; asm( "fma.rn.f32x2 %0, %1, %2, %3;" : "=l"( r.v ) : "l"( a.v ), "l"( b.v ), "l"( c.v ) ); return r; }
// The product that a sum takes up.  The assembler contracts a packed product and
// the sum that uses it into one fused operation, whatever it is told about
// contraction, and the reference rounds in between: nz is {-0, -0} from memory,
// so that it cannot know that adding it changes nothing.
__device__ __forceinline__ F2 mul2( F2 a, F2 b, F2 nz ) { return fma2( a, b, nz ); }
// (folded into the consuming instruction's operand)
__device__ __forceinline__ F2 neg2( F2 a ) { float x, y; unpack2( a, x, y ); return pack2( -x, -y ); }

// Correctly rounded square root, reciprocal and quotient for arguments in
// [1, QLIM): an approximation by the special-function unit, then one Newton
// step on the exact remainder that fma gives (P. Markstein, "Computation of
// elementary functions on the IBM RISC System/6000 processor", IBM J. Res.
// Dev. 34, 1990).  The same floats as the IEEE operations, without their tests
// of the argument's range at each call: tests/test_device_functions_gpu.py
// compares every float of [1, 2^96) for the root and the reciprocal, and for the
// quotient every significand of the divisor with 64 numerators each.  The
// theorem behind the last step asks for a quotient and a remainder that are
// normal numbers.  The kernel's two quotients are alpha / gamma, with |alpha| in
// (1e-18, 1e18), and the energy term utsq / (gamma + 1): where utsq is too small
// for that, gamma is 1 and the divisor exactly 2, and the same test compares that
// term for every float utsq of [0, 2^96).
constexpr float QLIM = 7.9e28f;             // about 2^96
__device__ __forceinline__ F2 sqrt2( F2 x ) {
    float a, b, ra, rb;
    unpack2( x, a, b );
    asm( "rsqrt.approx.ftz.f32 %0, %1;" : "=f"( ra ) : "f"( a ) );
    asm( "rsqrt.approx.ftz.f32 %0, %1;" : "=f"( rb ) : "f"( b ) );
    const F2 r = pack2( ra, rb );
    const F2 g = x * r;
    return fma2( fma2( g, neg2( g ), x ), r * both( 0.5f ), g );
}
__device__ __forceinline__ F2 recip2( F2 d ) {
    float a, b, ra, rb;
    unpack2( d, a, b );
    asm( "rcp.approx.ftz.f32 %0, %1;" : "=f"( ra ) : "f"( a ) );
    asm( "rcp.approx.ftz.f32 %0, %1;" : "=f"( rb ) : "f"( b ) );
    const F2 r = pack2( ra, rb );
    return fma2( r, fma2( d, neg2( r ), both( 1.0f ) ), r );
}
// a / d, with y = recip2( d )
__device__ __forceinline__ F2 quot2( F2 a, F2 d, F2 y ) {
    const F2 q = a * y;
    return fma2( fma2( d, neg2( q ), a ), y, q );
}

}  // namespace zb
