// One warp's device code on the host: its 32 lanes are contexts of one thread, each run to its next warp-wide operation
// before the next lane, so a lane reads there what the others brought -- enough for code whose lanes meet at every such
// operation (the full mask) and share memory only across them.
#pragma once
#include <algorithm>
#include <cmath>
#include <cstdlib>
#include <cstring>
#include <cuda_runtime.h>
#include <functional>
#include <ucontext.h>
#include <vector>

namespace warp_on_host {
inline int lane = 0, parity[ 32 ];
inline unsigned long long brought[ 2 ][ 32 ];        // two sets: a fast lane may bring to the next operation
inline ucontext_t here[ 32 ], caller;
inline std::function<void( int )> body;

inline void next_lane() {
    const int me = lane;
    lane = ( me + 1 ) % 32;
    swapcontext( &here[ me ], &here[ lane ] );
}
template<class X> const unsigned long long *meet( X v ) {
    static_assert( sizeof( X ) <= 8, "a register pair at most" );
    unsigned long long *set = brought[ parity[ lane ] ];
    parity[ lane ] ^= 1;
    set[ lane ] = 0;
    std::memcpy( &set[ lane ], &v, sizeof( X ) );
    next_lane();
    return set;
}
template<class X> X from( X v, int src ) {
    const unsigned long long *set = meet( v );
    X r;
    std::memcpy( &r, &set[ src & 31 ], sizeof( X ) );
    return r;
}
inline void entry() {
    body( lane );
    if ( lane == 31 ) setcontext( &caller );          // (the lanes leave in order, the last one back to run())
    ++lane;
    setcontext( &here[ lane ] );
}
// f( lane ) on the 32 lanes
inline void run( std::function<void( int )> f ) {
    static std::vector<char> stack( 32 << 16 );
    body = f;
    for ( int l = 0; l < 32; ++l ) {
        getcontext( &here[ l ] );
        here[ l ].uc_stack.ss_sp = stack.data() + ( size_t( l ) << 16 );
        here[ l ].uc_stack.ss_size = 1 << 16;
        makecontext( &here[ l ], entry, 0 );
        parity[ l ] = 0;
    }
    lane = 0;
    swapcontext( &caller, &here[ 0 ] );
    if ( lane != 31 ) std::abort();                   // the lanes did not meet the same operations
}
struct Index { struct { operator unsigned() const { return unsigned( lane ); } } x; };
} // namespace warp_on_host

static warp_on_host::Index threadIdx;
static const dim3 blockIdx( 0 ), blockDim( 32 );

template<class X> X __shfl_sync( unsigned, X v, int src ) { return warp_on_host::from( v, src ); }
template<class X> X __shfl_xor_sync( unsigned, X v, int o ) { return warp_on_host::from( v, warp_on_host::lane ^ o ); }
template<class X> X __shfl_up_sync( unsigned, X v, int o ) { const int l = warp_on_host::lane; return warp_on_host::from( v, l < o ? l : l - o ); }
template<class X> X __shfl_down_sync( unsigned, X v, int o ) { const int l = warp_on_host::lane; return warp_on_host::from( v, l + o > 31 ? l : l + o ); }
inline unsigned __ballot_sync( unsigned, bool b ) {
    const unsigned long long *set = warp_on_host::meet( b );
    unsigned r = 0;
    for ( int l = 0; l < 32; ++l ) r |= unsigned( set[ l ] ) << l;
    return r;
}
inline int __any_sync( unsigned m, bool b ) { return __ballot_sync( m, b ) != 0; }
inline int __all_sync( unsigned m, bool b ) { return __ballot_sync( m, b ) == m; }
inline int __reduce_min_sync( unsigned, int v ) {
    const unsigned long long *set = warp_on_host::meet( v );
    int r = v;
    for ( int l = 0; l < 32; ++l ) r = std::min( r, int( unsigned( set[ l ] ) ) );
    return r;
}
inline void __syncwarp() { warp_on_host::meet( 0 ); }
inline void __syncthreads() { warp_on_host::meet( 0 ); }          // (a block of one warp)
inline void __threadfence() {}
inline int __popc( unsigned x ) { return __builtin_popcount( x ); }
inline int __ffs( unsigned x ) { return __builtin_ffs( int( x ) ); }
template<class To, class From> To bits_as( From v ) { To r; std::memcpy( &r, &v, sizeof( To ) ); return r; }
inline int __float_as_int( float x ) { return bits_as<int>( x ); }
inline long long __double_as_longlong( double x ) { return bits_as<long long>( x ); }
inline double __longlong_as_double( long long x ) { return bits_as<double>( x ); }
inline float rsqrtf( float x ) { return 1 / std::sqrt( x ); }
template<class X> X atomicAdd( X *p, X v ) { const X o = *p; *p += v; return o; }
using std::max;
using std::min;
// (last: the standard headers spell the attribute so, too; include them before this one)
#define __noinline__ __attribute__( ( noinline ) )
