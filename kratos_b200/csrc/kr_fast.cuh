// Face arithmetic of the step, arranged for the FP64 / FP32 pipes of sm_100a.
//
// Same mathematics as kr_math.cuh (which restates the reference expression by
// expression), with every division by a shared denominator replaced by one
// reciprocal: 1 / rho per state, 1 / (gamma - 1) and gamma - 1 from the host,
// rsqrt for the star-state densities, one reciprocal per HLLD star denominator,
// and the van Leer PLM slope (dl dc / (dl + dc), algebraically the reference's
// dl dc (dl + dc) / (dl^2 + dc^2 + 2 dl dc)).
// Results differ from the reference by rounding only; the GPU parity tests state
// the bound.  FP64 divides are long dependent DFMA sequences, so this is what
// moves the FP64 flux kernel off its latency floor.
#pragma once

#include "kr_math.cuh"

namespace kr
{
template< class R > struct eos_c
{
    R gamma, gm1, cv;        // gamma, gamma - 1, 1 / (gamma - 1)
};

// Reciprocals and roots without the library functions' branches for zero,
// subnormal, infinite and NaN arguments, so that a face's independent ones overlap.
//
// FP32: the hardware approximations, one instruction each (rcp 1 ulp, rsqrt 2^-22.9
// relative by the PTX ISA), in their .ftz forms: the others carry a compare and two
// scalings for subnormal inputs.  Arguments: densities, pressures and differences of
// wave speeds between 2^-126 and 2^126; a square below FLT_MIN counts as zero (a
// speed below 1.1e-19 in code units, and in the fast speed's root, which takes
// fourth powers, one below 3e-10).
//
// FP64: Newton-Raphson from the hardware approximations (about 20 bits).
//  - reciprocal, from f( y ) = 1 / y - x: y += y ( 1 - x y ), twice: 2^-40, 2^-80;
//    what is left is the last rounding, 2^-53.
//  - reciprocal root: with e = 1 - x y^2, x^-1/2 = y ( 1 - e )^-1/2 = y ( 1 + e / 2 +
//    3 e^2 / 8 + ... ) (the binomial series), first to e^2 (5 / 16 e^3 is left, 2^-58),
//    then to e: the last rounding and half of x y's, 1.5 x 2^-53.
//  - root: g = x y, then Newton-Raphson on g^2 = x, g += ( x - g^2 ) / ( 2 g ) with
//    1 / g = y: the last rounding, 2^-53.
// Arguments: 2^-1021 to 2^1021 in size (positive for the roots); a square below
// 1e-290 counts as zero; NaN stays NaN; zero and infinity give NaN, and callers
// select such results away.
__device__ __forceinline__ float rcp( float x )
{
    float y;
    asm( "rcp.approx.ftz.f32 %0, %1;" : "=f"( y ) : "f"( x ) );
    return y;
}
__device__ __forceinline__ float rsq( float x )
{
    float y;
    asm( "rsqrt.approx.ftz.f32 %0, %1;" : "=f"( y ) : "f"( x ) );
    return y;
}
__device__ __forceinline__ float fsqrt( float x ) { return x >= FLT_MIN ? x * rsq( x ) : 0.f; }
__device__ __forceinline__ double rcp( double x )
{
    double y;
    asm( "rcp.approx.ftz.f64 %0, %1;" : "=d"( y ) : "d"( x ) );
    y = fma( y, fma( -x, y, 1.0 ), y );
    return fma( y, fma( -x, y, 1.0 ), y );
}
__device__ __forceinline__ double rsq3( double x )
{
    double y;
    asm( "rsqrt.approx.ftz.f64 %0, %1;" : "=d"( y ) : "d"( x ) );
    const double e = fma( -x * y, y, 1.0 );
    return fma( y * e, fma( 0.375, e, 0.5 ), y );
}
__device__ __forceinline__ double rsq( double x )
{
    const double y = rsq3( x );
    return fma( 0.5 * y, fma( -x * y, y, 1.0 ), y );
}
__device__ __forceinline__ double fsqrt( double x )
{
    const double y = rsq3( x ), g = x * y;
    return x < 1e-290 ? 0.0 : fma( 0.5 * y, fma( -g, g, x ), g );
}

// Limited slope of a cell (half its van Leer difference, plm.h:116-153
// mathematics), FP64: q + s is its state at the upper face, q - s at the lower.
__device__ __forceinline__ double plm_slope( double qm, double q, double qp )
{
    const double dl = q - qm, dr = qp - q, p = dl * dr;
    const bool pos = p > 0;
    const double s = p * rcp( pos ? dl + dr : 1.0 );
    return pos ? s : 0.0;
}

// PLM on one face from the four cells around it (plm.h:116-153 mathematics).
template< class R > __device__ __forceinline__
void plm_face_fast( R q_ll, R q_l, R q_r, R q_rr, R & ql, R & qr )
{
    R dql = q_l - q_ll, dqc = q_r - q_l, dqr = q_rr - q_r;
    if constexpr( sizeof( R ) == 4 )
    {   // Scale-free form of the same limiter: dl dr / ( dl + dr ) =
        // dl * ( dr / ( dl + dr ) ), whose quotient lies in ( 0, 1 ) when dl
        // and dr share a sign, so the slope never forms the product of two
        // differences -- no FP32 overflow for huge differences (the
        // reference's FP32 path rescales by max |d| for the same purpose).
        // Same sign is a positive product of the two differences (the limited
        // slope itself is formed scale-free below).  A positive product needs
        // one difference of normal size, so the sum is normal and its SFU
        // reciprocal finite (a subnormal sum would give 1 / 0 = inf); two
        // differences whose product underflows (both below ~1e-23) give no
        // slope.  plm_face_fast2 makes the same test on pairs.
        const bool lpos = dql * dqc > R( 0 );
        const bool rpos = dqr * dqc > R( 0 );
        ql = lpos ? q_l + dql * ( dqc * rcp( dql + dqc ) ) : q_l;
        qr = rpos ? q_r - dqc * ( dqr * rcp( dqc + dqr ) ) : q_r;
        return;
    }
    ql = q_l + plm_slope( q_ll, q_l, q_r );
    qr = q_r - plm_slope( q_l, q_r, q_rr );
}

// The FP32 limiter of plm_face_fast on two variables at once (.x, .y): the
// differences, sums and products as paired FP32 instructions (sm_100's
// FADD2 / FMUL2 / FFMA2), the sign tests and reciprocals per element.  Same
// operations per element as the scalar form.
__device__ __forceinline__
void plm_face_fast2( float2 q_ll, float2 q_l, float2 q_r, float2 q_rr, float2 & ql, float2 & qr )
{
    const float2 m1 = make_float2( -1.f, -1.f );
    const float2 dql = __ffma2_rn( q_ll, m1, q_l );      // q_l - q_ll, exact
    const float2 dqc = __ffma2_rn( q_l, m1, q_r );
    const float2 dqr = __ffma2_rn( q_r, m1, q_rr );
    // same sign: a positive product (paired multiply, one compare each).  A
    // positive product needs one difference of normal size, so the sum below
    // is normal and its SFU reciprocal finite; differences whose product
    // underflows (both below ~1e-23) give no slope
    const float2 pl = __fmul2_rn( dql, dqc ), pr = __fmul2_rn( dqr, dqc );
    const bool lx = pl.x > 0.f, ly = pl.y > 0.f, rx = pr.x > 0.f, ry = pr.y > 0.f;
    const float2 sl = __fadd2_rn( dql, dqc ), sr = __fadd2_rn( dqc, dqr );
    const float2 il = make_float2( rcp( sl.x ), rcp( sl.y ) ), ir = make_float2( rcp( sr.x ), rcp( sr.y ) );
    const float2 tl = __fmul2_rn( dqc, il );
    const float2 tr = __fmul2_rn( __fmul2_rn( dqr, ir ), m1 );
    // a cell's slope is its lower difference times the upper one's share of their
    // sum, at both of its faces (as the march forms it, once for both)
    const float2 cl = __ffma2_rn( dql, tl, q_l );        // q_l + dql ( dqc / ( dql + dqc ) )
    const float2 cr = __ffma2_rn( dqc, tr, q_r );        // q_r - dqc ( dqr / ( dqc + dqr ) )
    ql = make_float2( lx ? cl.x : q_l.x, ly ? cl.y : q_l.y );
    qr = make_float2( rx ? cr.x : q_r.x, ry ? cr.y : q_r.y );
}

////////////////////////////////////////////////////////////
// HLLC on rotated primitive states (hllc.h:262-379 mathematics).

template< class R > __device__ __forceinline__
void hllc_fast( R * flx, const R * wl, const R * wr, const eos_c< R > & e )
{
    const R irl = rcp( wl[ RHO ] ), irr = rcp( wr[ RHO ] );
    R v2l = wl[ MOM ] * wl[ MOM ] + wl[ MOM + 1 ] * wl[ MOM + 1 ] + wl[ MOM + 2 ] * wl[ MOM + 2 ];
    R v2r = wr[ MOM ] * wr[ MOM ] + wr[ MOM + 1 ] * wr[ MOM + 1 ] + wr[ MOM + 2 ] * wr[ MOM + 2 ];
    const R el = wl[ ENE ] * e.cv + wl[ RHO ] * v2l * R( 0.5f );
    const R er = wr[ ENE ] * e.cv + wr[ RHO ] * v2r * R( 0.5f );
    const R cl = fsqrt( e.gamma * rmax( wl[ ENE ] * irl, R( 0 ) ) );
    const R cr = fsqrt( e.gamma * rmax( wr[ ENE ] * irr, R( 0 ) ) );
    const R rsl = rsq( wl[ RHO ] ), rsr = rsq( wr[ RHO ] );
    const R sqrtdl = wl[ RHO ] * rsl, sqrtdr = wr[ RHO ] * rsr;
    const R isdlpdr = rcp( sqrtdl + sqrtdr );
    R wroe[ 5 ];
    for( int n = MOM; n < MOM + 3; ++ n )
        wroe[ n ] = ( sqrtdl * wl[ n ] + sqrtdr * wr[ n ] ) * isdlpdr;
    const R hroe = isdlpdr * ( ( el + wl[ ENE ] ) * rsl + ( er + wr[ ENE ] ) * rsr );
    const R gam1_roe = e.gm1;            // constant gamma: the Roe average is gamma - 1
    const R v2roe = wroe[ MOM ] * wroe[ MOM ] + wroe[ MOM + 1 ] * wroe[ MOM + 1 ]
                  + wroe[ MOM + 2 ] * wroe[ MOM + 2 ];
    const R q = hroe - R( 0.5f ) * v2roe;
    const R a = ( q <= 0 ) ? R( 0 ) : fsqrt( gam1_roe * q );
    const R al = rmin( wroe[ MOM ] - a, wl[ MOM ] - cl );
    const R ar = rmax( wroe[ MOM ] + a, wr[ MOM ] + cr );
    const R bp = ar > 0 ? ar : R( 0 );
    const R bm = al < 0 ? al : R( 0 );
    const R vxl = wl[ MOM ] - al, vxr = wr[ MOM ] - ar;
    const R tl  = wl[ ENE ] + vxl * wl[ RHO ] * wl[ MOM ];
    const R tr  = wr[ ENE ] + vxr * wr[ RHO ] * wr[ MOM ];
    const R ml  =  wl[ RHO ] * vxl;
    const R mr  = -wr[ RHO ] * vxr;
    R cp, am;
    const R f_max = R( FLT_MAX / 1e1f ), f_min = R( FLT_MIN * 1e1f );
    if( uabs( ml + mr ) < f_min )
        cp = am = 0;
    else if( ( tr != 0 && uabs( ml ) > f_max / uabs( tr ) ) ||
             ( tl != 0 && uabs( mr ) > f_max / uabs( tl ) ) )
    {
        const R mli = R( sgn( ml ) ) / rmax( uabs( ml ), f_min );
        const R mri = R( sgn( mr ) ) / rmax( uabs( mr ), f_min );
        am = ( tl - tr ) / ( ml + mr );
        cp = rmax( ( mri * tr + mli * tl ) / ( mli + mri ), R( 0 ) );
    }
    else
    {
        const R im = rcp( ml + mr );
        am = ( tl - tr ) * im;
        cp = rmax( ( ml * tr + mr * tl ) * im, R( 0 ) );
    }
    const R d_am_bm = rmax( uabs( am - bm ), f_min ) * R( am > bm ? 1 : -1 );
    const R d_am_bp = rmax( uabs( am - bp ), f_min ) * R( am > bp ? 1 : -1 );
    const R i_bm = rcp( d_am_bm ), i_bp = rcp( d_am_bp );
    const R sl = am >= 0 ? am * i_bm : R( 0 );
    const R sr = am <  0 ? am * i_bp : R( 0 );
    const R sm = am >  0 ? -bm * i_bm : -bp * i_bp;
    R fl[ 5 ], fr[ 5 ];
    f_lr_hyd( fl, wl, wl[ MOM ] - bm, el );
    f_lr_hyd( fr, wr, wr[ MOM ] - bp, er );
    for( int n = RHO; n < MOM + 3; ++ n )
        flx[ n ] = sl * fl[ n ] + sr * fr[ n ];
    flx[ MOM ] += sm * cp;
    flx[ ENE ] += sm * cp * am;
}

////////////////////////////////////////////////////////////
// HLLD and HLLE on rotated primitive states (hlld.h:31-298 mathematics).
//
// The left and right states go through the same arithmetic up to the contact
// speed and the star states, so they are kept as pairs (.x left, .y right) and
// FP32 uses sm_100's paired instructions: one issue slot for both sides (the
// sweep is bound by instruction issue in FP32, by latency in FP64).  The HLLD
// flux of a star region is the physical flux of its state -- the star states
// satisfy the jump conditions across the outer and the Alfven waves -- so
// instead of F + S (U* - U) + ... over eight conserved words of both sides, one
// side's region state is selected and put through one flux; energies are formed
// for that side only, and no branch on the contact's side is left.  Where a star
// state is degenerate (f_tiny below) the reference keeps the outer transverse
// field, whose jump the contact speed does not satisfy: the field flux then takes
// the difference B_t (v_n - S_M).
// FP32 forms the star states as the outer state plus a difference that is itself
// made of the states' differences: S_M - v_n = ( m' dv_n - dp_T ) / dm (m' the other
// side's rho ( S - v_n )), rho* - rho, E* - E, B_t* - B_t and v_t** - v_t* all carry
// it as a factor.  Formed directly, S_M and the star states each bring the rounding
// of large sums into a flux whose outer wave may be nearly at rest: one step of
// Mach 5 turbulence at beta 0.1 (96^3) moved the face fields 2.5e-8 to 2.9e-8 (L1)
// from FP64, the outer flux plus jumps of directly formed states 1.3e-8 to 1.4e-8,
// this 1.0e-8 to 1.3e-8.  Over turbulence, vortices, boxes and VL2, 5 to 12 steps,
// every field's 2-norm error is 0.3 to 0.95 of that two-sided form's.
// Flux sweeps z / y / x of the 256^3 mesh in 64 blocks of 64^3, ms per launch, one
// thread per face, two-sided -> one-sided with the reciprocals above: FP64 1.62 /
// 1.50 / 1.41 -> 0.67 / 0.65 / 0.58, FP32 0.48 / 0.45 / 0.37 -> 0.35 / 0.33 / 0.31
// (direct and difference forms, us per step with the march: 598 / 643 / 701 and
// 598 / 643 / 714).

template< class R > struct lr_t;
template<> struct lr_t< float >  { typedef float2 type; };
template<> struct lr_t< double > { typedef double2 type; };
template< class R > using lr = typename lr_t< R >::type;

__device__ __forceinline__ float2  mk2( float a, float b )   { return make_float2( a, b ); }
__device__ __forceinline__ double2 mk2( double a, double b ) { return make_double2( a, b ); }
__device__ __forceinline__ float2 add2( float2 a, float2 b ) { return __fadd2_rn( a, b ); }
__device__ __forceinline__ float2 mul2( float2 a, float2 b ) { return __fmul2_rn( a, b ); }
__device__ __forceinline__ float2 mad2( float2 a, float2 b, float2 c ) { return __ffma2_rn( a, b, c ); }
__device__ __forceinline__ float2 sub2( float2 a, float2 b ) { return __ffma2_rn( b, make_float2( -1.f, -1.f ), a ); }
__device__ __forceinline__ double2 add2( double2 a, double2 b ) { return make_double2( a.x + b.x, a.y + b.y ); }
__device__ __forceinline__ double2 mul2( double2 a, double2 b ) { return make_double2( a.x * b.x, a.y * b.y ); }
__device__ __forceinline__ double2 mad2( double2 a, double2 b, double2 c ) { return make_double2( a.x * b.x + c.x, a.y * b.y + c.y ); }
__device__ __forceinline__ double2 sub2( double2 a, double2 b ) { return make_double2( a.x - b.x, a.y - b.y ); }
template< class P > __device__ __forceinline__ P rcp2( P a ) { return mk2( rcp( a.x ), rcp( a.y ) ); }
template< class P > __device__ __forceinline__ P rsq2( P a ) { return mk2( rsq( a.x ), rsq( a.y ) ); }
// Square roots of positive pairs
__device__ __forceinline__ float2 root2( float2 a ) { return mul2( a, rsq2( a ) ); }
__device__ __forceinline__ double2 root2( double2 a ) { return make_double2( fsqrt( a.x ), fsqrt( a.y ) ); }

// What both solvers start from: the states, total pressures and outer speeds.
template< class R > struct hll_prefix
{
    lr< R > rho, pre, vn, vt1, vt2, bt1, bt2, pm;
    R b_x, bx_2, spd_m2, spd_p2;
};

template< class R > __device__ __forceinline__
void hll_prefix_fast( hll_prefix< R > & h, const R * wl, const R * wr, const eos_c< R > & e )
{
    typedef lr< R > P;
    const P half = mk2( R( 0.5f ), R( 0.5f ) );
    h.rho = mk2( wl[ RHO ], wr[ RHO ] );
    h.pre = mk2( wl[ ENE ], wr[ ENE ] );
    h.vn  = mk2( wl[ MOM ], wr[ MOM ] );
    h.vt1 = mk2( wl[ MOM + 1 ], wr[ MOM + 1 ] );
    h.vt2 = mk2( wl[ MOM + 2 ], wr[ MOM + 2 ] );
    h.bt1 = mk2( wl[ BCC + 1 ], wr[ BCC + 1 ] );
    h.bt2 = mk2( wl[ BCC + 2 ], wr[ BCC + 2 ] );
    h.b_x = wl[ BCC ];
    h.bx_2 = h.b_x * h.b_x;
    const P b2 = mk2( h.bx_2, h.bx_2 );
    const P bt = mad2( h.bt1, h.bt1, mul2( h.bt2, h.bt2 ) );
    h.pm = mul2( half, add2( b2, bt ) );
    // fast magnetosonic speeds (mhd/eos/adiabatic.h:84-98)
    const P ir = rcp2( h.rho );
    const P cs = mul2( mul2( mk2( e.gamma, e.gamma ), h.pre ), ir );
    const P vt = mul2( bt, ir ), va = mul2( b2, ir );
    const P s = add2( va, vt ), q = add2( s, cs ), r = sub2( s, cs );
    P rad = mad2( r, r, mul2( mul2( mk2( R( 4 ), R( 4 ) ), cs ), vt ) );
    const R tiny = sizeof( R ) == 4 ? R( FLT_MIN ) : R( 1e-290 );
    rad = mk2( rmax( rad.x, tiny ), rmax( rad.y, tiny ) );       // its root: finite at zero
    const P cf = root2( mul2( half, mad2( rad, rsq2( rad ), q ) ) );
    const P sm = sub2( h.vn, cf ), sp = add2( h.vn, cf );
    h.spd_m2 = rmin( sm.x, sm.y );
    h.spd_p2 = rmax( sp.x, sp.y );
}

template< class R > __device__ __forceinline__
void hlld_tail( R * flx, const hll_prefix< R > & h, const eos_c< R > & e )
{
    typedef lr< R > P;
    const R b_x = h.b_x, bx_2 = h.bx_2;
    const R f_tiny = R( 1.00e-4f );
    constexpr bool F32 = sizeof( R ) == 4;
    const P nb2 = mk2( -bx_2, -bx_2 ), nbx = mk2( -b_x, -b_x );
    const P pt = add2( h.pre, h.pm );
    const P s2 = mk2( h.spd_m2, h.spd_p2 );
    const P sd = sub2( s2, h.vn );
    const P m = mul2( h.rho, sd );                              // rho ( S - v_n )
    const P u_m = mul2( h.rho, h.vn );
    P s0, w, sdm, ism;                                          // S_M, S_M - v_n, S - S_M
    if constexpr( F32 )
    {   // from the states' differences (above)
        const R dv = h.vn.y - h.vn.x, dp = pt.y - pt.x, i = rcp( m.y - m.x );
        w = mk2( ( m.y * dv - dp ) * i, ( m.x * dv - dp ) * i );
        s0 = add2( h.vn, w );
        sdm = sub2( sd, w );
        ism = rcp2( sdm );
    }
    else
    {
        const R sc = ( sd.y * u_m.y - pt.y - sd.x * u_m.x + pt.x ) * rcp( m.y - m.x );
        s0 = mk2( sc, sc );
        w = sub2( s0, h.vn );
        sdm = sub2( s2, s0 );
        const R i = rcp( sdm.x * sdm.y );                       // one reciprocal for both sides
        ism = mk2( sdm.y * i, sdm.x * i );
    }
    const R ptot_s = pt.x + m.x * w.x;
    const P rhos = mul2( m, ism );
    const P rs = rsq2( rhos );                                  // 1 / sqrt( rho* )
    const P sq = mul2( rhos, rs );
    const P denom = mad2( m, sdm, nb2 );
    const P id = rcp2( denom );
    P tv = mul2( mul2( nbx, w ), id );                          // v_t* = v_t + B_t tv
    P tb;                                                       // B_t* = B_t tb (FP32: B_t + B_t tb)
    if constexpr( F32 ) tb = mul2( mul2( m, w ), id );
    else                tb = mul2( mad2( m, sd, nb2 ), id );
    const R flat = f_tiny * ptot_s, keep = R( F32 ? 0 : 1 );
    const bool flat_l = uabs( denom.x ) < flat, flat_r = uabs( denom.y ) < flat;
    tv = mk2( flat_l ? R( 0 ) : tv.x, flat_r ? R( 0 ) : tv.y );
    tb = mk2( flat_l ? keep : tb.x, flat_r ? keep : tb.y );
    const P vs1 = mad2( h.bt1, tv, h.vt1 ), vs2 = mad2( h.bt2, tv, h.vt2 );
    P bs1, bs2;
    if constexpr( F32 ) { bs1 = mad2( h.bt1, tb, h.bt1 ); bs2 = mad2( h.bt2, tb, h.bt2 ); }
    else                { bs1 = mul2( h.bt1, tb ); bs2 = mul2( h.bt2, tb ); }
    const R spd_m1 = s0.x - uabs( b_x ) * rs.x, spd_p1 = s0.y + uabs( b_x ) * rs.y;
    // the side the face lies on, and whether outside its fan, in its star or
    // in its double-star region
    const bool out_l = h.spd_m2 >= 0, out_r = h.spd_p2 <= 0, outer = out_l || out_r;
    const bool left = out_l || ( ! out_r && s0.x >= 0 );
    const bool inner = ! outer && ( left ? spd_m1 < 0 : spd_p1 > 0 ) && bx_2 > flat;
    const R rho = left ? h.rho.x : h.rho.y;
    R vn = left ? h.vn.x : h.vn.y, p = left ? pt.x : pt.y;
    R v1 = left ? h.vt1.x : h.vt1.y, v2 = left ? h.vt2.x : h.vt2.y;
    R b1 = left ? h.bt1.x : h.bt1.y, bb2 = left ? h.bt2.x : h.bt2.y;
    const R pre = left ? h.pre.x : h.pre.y;
    const R vv = vn * vn + v1 * v1 + v2 * v2;
    R en;
    if constexpr( F32 ) en = ( p + pre * ( e.cv - 1 ) ) + rho * R( 0.5f ) * vv;   // (the magnetic pressure in p)
    else                en = pre * e.cv + rho * vv * R( 0.5f ) + ( left ? h.pm.x : h.pm.y );
    R vb = vn * b_x + v1 * b1 + v2 * bb2;
    R x1 = 0, x2 = 0, mass = left ? u_m.x : u_m.y, mn = mass;
    if( ! outer )
    {
        const R il = left ? ism.x : ism.y, ws = left ? w.x : w.y, ms = left ? m.x : m.y;
        const R so = left ? h.spd_m2 : h.spd_p2, sc = left ? s0.x : s0.y;
        const bool flt = left ? flat_l : flat_r;
        x1 = flt ? - b1 * ws : R( 0 );
        x2 = flt ? - bb2 * ws : R( 0 );
        v1 = left ? vs1.x : vs1.y; v2 = left ? vs2.x : vs2.y;
        b1 = left ? bs1.x : bs1.y; bb2 = left ? bs2.x : bs2.y;
        const R vbs = sc * b_x + v1 * b1 + v2 * bb2;
        if constexpr( F32 )
        {   // rho* - rho = rho ( S_M - v_n ) / ( S - S_M ), E* - E and p* - p alike
            mass += so * ( rho * ws * il );
            mn = mass;
            en += ( b_x * ( vb - vbs ) + ws * ( en + p + ms * sc ) ) * il;
            p += ms * ws;
        }
        else
        {   // FP64: the mass flux as the sum of its jumps.  Against a wall it is
            // rounding residue, whose sign the edge EMF's upwind switch reads:
            // the region's rho S_M is exactly zero there, which the reference's
            // sum is not
            const R si = left ? spd_m1 : spd_p1, rho_s = left ? rhos.x : rhos.y;
            mass += ( left ? si < 0 : si > 0 ) ? - so * rho - ( si - so ) * rho_s + si * rho_s
                                               : so * ( rho_s - rho );
            mn = rho_s * sc;
            en = ( b_x * ( vb - vbs ) - p * vn + ( left ? sd.x : sd.y ) * en + ptot_s * sc ) * il;
            p = ptot_s;
        }
        vb = vbs;
        vn = sc;
        if( inner )
        {
            const R sg = b_x > 0 ? R( 1 ) : R( -1 );
            const R rni = rcp( sq.x + sq.y ), ss = sg * sq.x * sq.y;
            const R dv1 = vs1.y - vs1.x, dv2 = vs2.y - vs2.x, db1 = bs1.y - bs1.x, db2 = bs2.y - bs2.x;
            if constexpr( F32 )
            {   // this side's star state plus the differences' share
                const R cv = left ? sq.y : - sq.x, cb = left ? sq.x : - sq.y;
                v1 += rni * ( cv * dv1 + sg * db1 );
                v2 += rni * ( cv * dv2 + sg * db2 );
                b1 += rni * ( cb * db1 + ss * dv1 );
                bb2 += rni * ( cb * db2 + ss * dv2 );
            }
            else
            {
                v1 = rni * ( sq.x * vs1.x + sq.y * vs1.y + sg * db1 );
                v2 = rni * ( sq.x * vs2.x + sq.y * vs2.y + sg * db2 );
                b1 = rni * ( sq.x * bs1.y + sq.y * bs1.x + ss * dv1 );
                bb2 = rni * ( sq.x * bs2.y + sq.y * bs2.x + ss * dv2 );
            }
            const R vbd = sc * b_x + v1 * b1 + v2 * bb2;
            en += ( left ? -sq.x : sq.y ) * sg * ( vb - vbd );
            vb = vbd;
        }
    }
    flx[ RHO ] = mass;
    flx[ ENE ] = ( en + p ) * vn - b_x * vb;
    flx[ MOM ] = mn * vn + p - bx_2;
    flx[ MOM + 1 ] = mn * v1 - b_x * b1;
    flx[ MOM + 2 ] = mn * v2 - b_x * bb2;
    flx[ BCC ] = 0;
    flx[ BCC + 1 ] = b1 * vn - b_x * v1 + x1;
    flx[ BCC + 2 ] = bb2 * vn - b_x * v2 + x2;
}

// HLLE with the HLLD outer speeds, from the prefix.
template< class R > __device__ __forceinline__
void hlle_tail( R * flx, const hll_prefix< R > & h, const eos_c< R > & e )
{
    typedef lr< R > P;
    const R s_l = rmin( h.spd_m2, R( 0 ) );
    const R s_r = rmax( h.spd_p2, R( 0 ) );
    const R inv = rcp( s_r - s_l ), slr = s_r * s_l;
    const P nbx = mk2( -h.b_x, -h.b_x ), half = mk2( R( 0.5f ), R( 0.5f ) );
    const P mn = mul2( h.rho, h.vn );
    const P v2 = mad2( h.vn, h.vn, mad2( h.vt1, h.vt1, mul2( h.vt2, h.vt2 ) ) );
    const P en = mad2( h.pre, mk2( e.cv, e.cv ), mad2( mul2( half, h.rho ), v2, h.pm ) );
    const P pt = sub2( add2( h.pre, h.pm ), mk2( h.bx_2, h.bx_2 ) );
    const P vb = mad2( h.vt1, h.bt1, mul2( h.vt2, h.bt2 ) );
    auto join = [ & ]( P f, P u ) { return ( s_r * f.x - s_l * f.y + slr * ( u.y - u.x ) ) * inv; };
    flx[ RHO ] = join( mn, h.rho );
    flx[ ENE ] = join( mad2( nbx, vb, mul2( h.vn, add2( pt, en ) ) ), en );
    flx[ MOM ] = join( mad2( mn, h.vn, pt ), mn );
    flx[ MOM + 1 ] = join( mad2( nbx, h.bt1, mul2( mn, h.vt1 ) ), mul2( h.rho, h.vt1 ) );
    flx[ MOM + 2 ] = join( mad2( nbx, h.bt2, mul2( mn, h.vt2 ) ), mul2( h.rho, h.vt2 ) );
    flx[ BCC ] = 0;
    flx[ BCC + 1 ] = join( mad2( nbx, h.vt1, mul2( h.bt1, h.vn ) ), h.bt1 );
    flx[ BCC + 2 ] = join( mad2( nbx, h.vt2, mul2( h.bt2, h.vn ) ), h.bt2 );
}

template< class R > __device__ __forceinline__
void hlld_fast( R * flx, const R * wl, const R * wr, const eos_c< R > & e )
{
    hll_prefix< R > h;
    hll_prefix_fast( h, wl, wr, e );
    hlld_tail( flx, h, e );
}

// HLLE with the HLLD outer speeds (cheap flux of the learned selector).
template< class R > __device__ __forceinline__
void hlle_fast( R * flx, const R * wl, const R * wr, const eos_c< R > & e )
{
    hll_prefix< R > h;
    hll_prefix_fast( h, wl, wr, e );
    hlle_tail( flx, h, e );
}

// The learned mode's solver of one face, HLLE where `cheap`, else HLLD, from
// one shared prefix (one copy of it in the kernel).
template< class R > __device__ __forceinline__
void hll_pick_fast( R * flx, const R * wl, const R * wr, const eos_c< R > & e, bool cheap )
{
    hll_prefix< R > h;
    hll_prefix_fast( h, wl, wr, e );
    if( cheap ) hlle_tail( flx, h, e );
    else        hlld_tail( flx, h, e );
}

}   // namespace kr
