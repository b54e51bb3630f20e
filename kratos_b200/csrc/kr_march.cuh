// MHD flux sweeps along y and z that march: a thread walks a run of faces of one
// column and keeps the primitives around them in its own ring in shared memory,
// filled by 16-byte asynchronous copies one cell ahead of the arithmetic.
//
// The per-face kernel k_flux fetches every cell of a y or z stencil four times
// from the L2 (the four cells lie in four rows or planes; 10% to 36% L1 hits) and
// waits for it at the start of every face; here a cell is fetched once per sweep
// while the face before it is solved, and its limited slope is formed once for
// both of its faces.  Along x the four cells share cache lines and k_flux stays.
// Sweeps z / y of the 256^3 mesh (64 blocks of 64^3), us per step, k_flux -> march:
// FP32 717 / 726 -> 597 / 643, FP64 1276 / 1226 -> 1096 / 1085.  Hydro sweeps (5
// words) gained nothing in FP64 (632 us per step of 128^3 against 626) and lost on
// small meshes, so they stay face by face.
// Included by kr_core.cu; the same arithmetic per face as k_flux.

// Resident CTAs of 128 threads per SM (ring: 24 KB per CTA in FP32, 44 KB in
// FP64).  FP32: 80 registers, nothing spilled; at 7 CTAs (72) the 256^3 sweeps
// took 631 / 667 us, at 8 (64, 16 to 28 bytes spilled) 651 / 937.
template< class R > __host__ __device__ constexpr int march_ctas(  ) { return sizeof( R ) == 4 ? 6 : 4; }

__device__ __forceinline__ void cp_async16( void * s, const void * g )
{
    asm volatile( "cp.async.cg.shared.global [%0], [%1], 16;" :: "r"( unsigned( __cvta_generic_to_shared( s ) ) ), "l"( g ) : "memory" );
}
__device__ __forceinline__ void cp_async8( void * s, const void * g )
{
    asm volatile( "cp.async.ca.shared.global [%0], [%1], 8;" :: "r"( unsigned( __cvta_generic_to_shared( s ) ) ), "l"( g ) : "memory" );
}

// Lower (q - s) and upper (q + s) states of a cell's 8 words from it and its two
// neighbours (rings of 16-byte groups, strided by 128); the normal field's word
// is left out in FP64.  plm_face_fast's and plm_face_fast2's operations; without a
// slope the cell's own value is selected, so a neighbour that is no number (or a
// donor's, the VL2 predictor) leaves it alone.
template< int AXIS > __device__ __forceinline__
void plm_cell( const float4 * qm, const float4 * q, const float4 * qp, bool donor, float * lo, float * hi )
{
    const float2 m1 = make_float2( -1.f, -1.f );
#pragma unroll
    for( int k = 0; k < 2; ++ k )
    {
        const float4 a = qm[ 128 * k ], c = q[ 128 * k ], d = qp[ 128 * k ];
#pragma unroll
        for( int h = 0; h < 2; ++ h )
        {
            const float2 x = h ? make_float2( a.z, a.w ) : make_float2( a.x, a.y );
            const float2 y = h ? make_float2( c.z, c.w ) : make_float2( c.x, c.y );
            const float2 z = h ? make_float2( d.z, d.w ) : make_float2( d.x, d.y );
            const float2 dl = __ffma2_rn( x, m1, y ), dr = __ffma2_rn( y, m1, z );
            const float2 p = __fmul2_rn( dl, dr ), s = __fadd2_rn( dl, dr );
            const float2 t = __fmul2_rn( dr, make_float2( rcp( s.x ), rcp( s.y ) ) );
            const float2 u = __ffma2_rn( dl, t, y ), l = __ffma2_rn( dl, __fmul2_rn( t, m1 ), y );
            const bool px = p.x > 0.f && ! donor, py = p.y > 0.f && ! donor;
            const int w = 4 * k + 2 * h;
            lo[ w ] = px ? l.x : y.x; lo[ w + 1 ] = py ? l.y : y.y;
            hi[ w ] = px ? u.x : y.x; hi[ w + 1 ] = py ? u.y : y.y;
        }
    }
}
template< int AXIS > __device__ __forceinline__
void plm_cell( const double2 * qm, const double2 * q, const double2 * qp, bool donor, double * lo, double * hi )
{
#pragma unroll
    for( int k = 0; k < 4; ++ k )
    {
        const double2 a = qm[ 128 * k ], c = q[ 128 * k ], d = qp[ 128 * k ];
        if( 2 * k != BCC + AXIS )
        {
            const double s = donor ? 0.0 : plm_slope( a.x, c.x, d.x );
            lo[ 2 * k ] = c.x - s;
            hi[ 2 * k ] = c.x + s;
        }
        if( 2 * k + 1 != BCC + AXIS )
        {
            const double s = donor ? 0.0 : plm_slope( a.y, c.y, d.y );
            lo[ 2 * k + 1 ] = c.y - s;
            hi[ 2 * k + 1 ] = c.y + s;
        }
    }
}

// Faces [f0, f1) of the column at transverse position t (x fastest, then the
// other transverse axis O).  ring: four cells per thread, three in use and one in
// flight, and a slot for the first cell, which only the start reads; a slot is
// refilled after the face that last read it has been stored, so a thread waits
// only for its own copies and nothing is synchronised.
template< class R, int MODE, bool XL, int AXIS > __device__ __forceinline__
void march_column( const args_t< R > & a, int step, udiv_t dv, int b, unsigned t, int f0, int f1,
                   typename w_vec< R >::type ( * ring )[ 8 / w_group< R >(  ) ][ 128 ], double ( * ringb )[ 128 ] )
{
    constexpr int G = w_group< R >(  ), NQ = 8 / G, O = 3 - AXIS;
    typedef typename w_vec< R >::type V;
    const int nn[ 3 ] = { a.n0, a.n1, a.n2 };
    const int e0 = a.n0 + 2, eo = nn[ O ] + 2;
    const unsigned q = udiv_q( t, dv );
    int ii[ 3 ];
    ii[ 0 ] = int( t - q * unsigned( e0 ) ) - 1;
    ii[ O ] = int( q ) - 1;
    const bool ox = ii[ 0 ] < 0 || ii[ 0 ] >= a.n0, oo = ii[ O ] < 0 || ii[ O ] >= nn[ O ];
    if( t >= unsigned( e0 * eo ) || ( ox && oo ) )
        return;                        // past the plane, or an edge line that nothing reads
    const int th = threadIdx.x;
    const int sw = AXIS == 1 ? a.sw1 : a.sw2, sb = AXIS == 1 ? a.sb1 : a.sb2, sf = AXIS == 1 ? a.sf1 : a.sf2;
    ii[ AXIS ] = f0;
    const int pos = w_pos( a, ii[ 0 ], ii[ 1 ], ii[ 2 ] ) - 2 * sw;        // cell f0 - 2
    const V * wp = reinterpret_cast< const V * >( a.w + ( size_t ) b * 11 * a.ngw ) + pos;
    const double * bp = a.bf[ step ] + ibf( a, b, AXIS, ii[ 0 ], ii[ 1 ], ii[ 2 ] );
    R * F = a.f[ AXIS ] + ifx( a, b, 0, 7, ii[ 0 ], ii[ 1 ], ii[ 2 ] );
    const int nfb = int( a.nfb );
    bool cross = false;
    if constexpr( XL )
    {   // next to a side whose neighbours are on another level (normal_b)
        const int x = a.geo[ b ].xlev;
        cross = ( ox && ( x >> ( ii[ 0 ] < 0 ? 0 : 1 ) & 1 ) )
             || ( oo && ( x >> ( 2 * O + ( ii[ O ] < 0 ? 0 : 1 ) ) & 1 ) );
    }
    const unsigned dstep = ( ( unsigned( e0 * eo ) + 127u ) >> 7 ) * 4u;   // choices per face of the march
    const unsigned * dec = nullptr;
    if constexpr( MODE == FLUX_APPLY )
        dec = a.sel_dec + ( ( size_t ) AXIS * a.nblk + b ) * a.sel_wcap + ( size_t ) f0 * dstep + ( t >> 5 );
    const bool donor = a.vl2 && step == 0;      // VL2 predictor: piecewise-constant states
    const eos_c< R > e = { R( a.gamma ), R( a.gm1 ), R( a.cv ) };
    const int nf = f1 - f0;
    auto load = [ & ]( int j )                  // cell f0 - 2 + j and, from j = 3, the normal B of face f0 + j - 3
    {
        if( j < nf + 3 )
        {
            const int s = j ? j & 3 : 4;
#pragma unroll
            for( int k = 0; k < NQ; ++ k )
                cp_async16( & ring[ s ][ k ][ th ], wp + ( long long ) k * a.ngw + j * sw );
            if( j >= 3 )
                cp_async8( & ringb[ j & 3 ][ th ], bp + ( j - 3 ) * sb );
        }
        asm volatile( "cp.async.commit_group;" ::: "memory" );
    };
    auto wait = [  ] { asm volatile( "cp.async.wait_group 1;" ::: "memory" ); };
#pragma unroll
    for( int j = 0; j < 4; ++ j )
        load( j );
    wait(  );
    R hi[ 8 ];
    {
        R drop[ 8 ];
        plm_cell< AXIS >( & ring[ 4 ][ 0 ][ th ], & ring[ 1 ][ 0 ][ th ], & ring[ 2 ][ 0 ][ th ], donor, drop, hi );
    }
#pragma unroll 1
    for( int i = 0; i < nf; ++ i )
    {
        load( i + 4 );
        wait(  );
        bool cheap = false;
        if constexpr( MODE == FLUX_APPLY )
            cheap = ( dec[ ( size_t ) i * dstep ] >> ( t & 31u ) ) & 1u;
        R l[ 8 ], r[ 8 ], flx[ 8 ];
#pragma unroll
        for( int k = 0; k < 8; ++ k )
            l[ k ] = hi[ k ];
        plm_cell< AXIS >( & ring[ ( i + 1 ) & 3 ][ 0 ][ th ], & ring[ ( i + 2 ) & 3 ][ 0 ][ th ],
                          & ring[ ( i + 3 ) & 3 ][ 0 ][ th ], donor, r, hi );
        R bn = R( ringb[ ( i + 3 ) & 3 ][ th ] );
        if( XL && cross )
            bn = reinterpret_cast< const R * >( & ring[ ( i + 2 ) & 3 ][ ( BCC + AXIS ) / G ][ th ] )[ ( BCC + AXIS ) % G ];
        l[ BCC + AXIS ] = r[ BCC + AXIS ] = bn;
        idx_swap( l + MOM, AXIS ); idx_swap( r + MOM, AXIS );
        idx_swap( l + BCC, AXIS ); idx_swap( r + BCC, AXIS );
        if constexpr( MODE == KR_RIEMANN_HLLE ) hlle_fast< R >( flx, l, r, e );
        else if constexpr( MODE == FLUX_APPLY ) hll_pick_fast< R >( flx, l, r, e, cheap );
        else                                    hlld_fast< R >( flx, l, r, e );
        idx_swap( flx + MOM, 3 - AXIS );
#pragma unroll
        for( int k = 0; k < 5; ++ k )
            F[ k * nfb ] = flx[ k ];
        F[ 5 * nfb ] =  flx[ BCC + 2 ];
        F[ 6 * nfb ] = -flx[ BCC + 1 ];
        F += sf;
    }
}

// One CTA's share: its warps number the (segment, 32 transverse positions) pairs
// of block b; a segment is `seg` faces of the columns.
template< class R, int MODE, bool XL, int AXIS > __device__ __forceinline__
void march_tile( const args_t< R > & a, int step, udiv_t dv, unsigned warps, int seg, int b, unsigned tile )
{
    __shared__ typename w_vec< R >::type ring[ 5 ][ 8 / w_group< R >(  ) ][ 128 ];
    __shared__ double ringb[ 4 ][ 128 ];
    const unsigned w = tile * 4u + ( threadIdx.x >> 5 ), s = w / warps;
    const int f0 = int( s ) * seg, f1 = min( f0 + seg, ( AXIS == 1 ? a.n1 : a.n2 ) + 1 );
    if( f0 < f1 )
        march_column< R, MODE, XL, AXIS >( a, step, dv, b, ( w - s * warps ) * 32u + ( threadIdx.x & 31u ), f0, f1, ring, ringb );
}

template< class R, int MODE, bool XL, int AXIS >
__global__ void __launch_bounds__( 128, ( march_ctas< R >(  ) ) )
k_march( const args_t< R > a, int step, udiv_t dv, unsigned warps, int seg )
{
    if constexpr( MODE == FLUX_APPLY )
        if( step == 0 && sel_eval_step( a.s, a.sel_period ) )
            return;                    // the network's sweep (k_flux_eval) solves this one
    march_tile< R, MODE, XL, AXIS >( a, step, dv, warps, seg, blockIdx.z, blockIdx.x );
}

// The march on one block: the row length and the warps of its transverse plane,
// the faces per segment and the CTAs per block.  The segment trades the march's
// start (three cells to wait for and a slope more, about two faces' time) against
// the last wave: the length with the least (waves + 1) (length + 2).  FP64 256^3:
// 22 faces 2.4% faster per step than whole columns of 65.
struct march_t { unsigned row, warps; int seg; unsigned tiles; };

static inline march_t march_shape( const int * n, int axis, long long nblk, int resident )
{
    march_t s;
    s.row = unsigned( n[ 0 ] + 2 );
    s.warps = ( s.row * unsigned( n[ 3 - axis ] + 2 ) + 31u ) / 32u;
    const int faces = n[ axis ] + 1;
    double best = 0;
    for( int k = 1; k <= faces; ++ k )
    {
        const int len = ( faces + k - 1 ) / k;
        const double ctas = double( s.warps ) * ( ( faces + len - 1 ) / len ) / 4 * nblk;
        const double cost = ( ctas / resident + 1 ) * ( len + 2 );
        if( k == 1 || cost < best )
        {
            best = cost;
            s.seg = len;
        }
    }
    s.tiles = ( s.warps * unsigned( ( faces + s.seg - 1 ) / s.seg ) + 3u ) / 4u;
    return s;
}

// Whether blocks n march along y and z: at least 32 warps per SM with eight faces
// each (24 are resident in FP32, 16 in FP64); smaller meshes need k_flux's one
// thread per face to fill the chip.  The mesh's own block count, not a rank's, so that every rank of a
// sharded mesh and an unsharded one run the same kernels.  Measured per step, load
// over the line, k_flux -> march: 1.87 (8 blocks of 64^3) FP32 659 -> 639 us, FP64
// 987 -> 969; 1.80 (one block of 128^3) FP32 620 -> 598, FP64 934 -> 905.  With the
// scalar-load march of an earlier form, FP64: 0.25 (8 blocks of 32^3) 186 -> 189,
// 0.23 (one of 64^3) 168 -> 174, 0.29 (64 of 16^3) 237 -> 240, 2.0 (64 of 32^3)
// 1205 -> 1127.
static inline double march_load( const int * n, int axis, long long nblk )
{
    return double( ( n[ 0 ] + 2 ) * ( long long )( n[ 3 - axis ] + 2 ) ) / 32 * ( n[ axis ] + 1 ) / 8 * double( nblk );
}
static inline bool march_pays( double load, int n_sm ) { return load >= 32.0 * n_sm; }
