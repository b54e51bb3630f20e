// How the launches number a block's sites and faces: quotients by fixed extents
// and the tiles built on them.  Compiles for the host alone too.
#pragma once

#include <algorithm>
#include <cstdint>

#ifdef __CUDACC__
#define KR_HD __host__ __device__ __forceinline__
#else
#define KR_HD inline
#endif

namespace kr
{
// Quotient of n < 2^31 by a fixed d >= 2 with one multiply-high and a shift
// (Granlund and Montgomery, "Division by invariant integers using
// multiplication", PLDI 1994): with 2^s < d <= 2^(s+1) and m = ceil( 2^(32+s) / d ),
// m fits 32 bits and m d exceeds 2^(32+s) by less than d <=
// 2^(s+1), which times n stays under 2^(32+s): exact for every such n.
// A block has fewer sites than 2^31 (each takes 100 bytes and more).
struct udiv_t { unsigned d, m, s; };
static inline udiv_t make_udiv( unsigned d )
{
    unsigned s = 0;
    while( ( 2ull << s ) < d )
        ++ s;
    return { d, unsigned( ( ( 1ull << ( 32 + s ) ) + d - 1 ) / d ), s };
}
KR_HD unsigned udiv_q( unsigned n, const udiv_t & v )
{
#ifdef __CUDA_ARCH__
    return __umulhi( n, v.m ) >> v.s;
#else
    return unsigned( uint64_t( n ) * v.m >> 32 ) >> v.s;
#endif
}

KR_HD unsigned udiv_q1( unsigned n, const udiv_t & v )   // d >= 1
{
    return v.d == 1 ? n : udiv_q( n, v );
}

// The sites of a block (e0 x e1 x e2, x fastest) as one index over CTAs of 256
// threads, so small planes share CTAs (the 17 x 17 edge sites of a 16^3 block's
// plane filled 56% of two CTAs, its 17 planes fill 96% of 20).
struct tile_t
{
    int e0, e1, e2;
    udiv_t d0, d01;
};
static inline tile_t make_tile( int e0, int e1, int e2 )
{
    return { e0, e1, e2, make_udiv( unsigned( e0 ) ), make_udiv( unsigned( e0 ) * unsigned( e1 ) ) };
}
static inline unsigned tile_ctas( const tile_t & t )
{
    return unsigned( ( ( long long ) t.e0 * t.e1 * t.e2 + 255 ) / 256 );
}

// Site s; false past the block's last site.
KR_HD bool tile_site( const tile_t & t, unsigned s, int * i )
{
    const unsigned p = udiv_q( s, t.d01 ), r = s - p * t.d01.d;
    const unsigned q = udiv_q( r, t.d0 );
    i[ 0 ] = int( r - q * t.d0.d );
    i[ 1 ] = int( q );
    i[ 2 ] = int( p );
    return i[ 2 ] < t.e2;
}
}   // namespace kr
