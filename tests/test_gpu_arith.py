"""The rounding of the face arithmetic (kr_fast.cuh): its reciprocals and roots by
themselves, the mixed step's distance from the FP64 step where the star states
cancel, and every axis treated alike."""
import os
import shutil
import subprocess

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

GAMMA = 5 / 3


@pytest.mark.parametrize("seed", [4, 5])
def test_mixed_field_error_in_turbulence(seed):
    """One mixed step of Mach 5 turbulence at beta 0.1: the face fields' L1 distance
    from the FP64 step.  The primitives and face fluxes are stored with relative
    rounding 3e-8 on average (2^-25), the edge EMF averages eight of them and a step
    carries about a third (the CFL number) of one into the field: 1e-8 is what the
    storage alone costs.  Twice that is allowed; star states formed without the
    states' differences gave 2.5e-8 and more."""
    from kratos_b200 import Dynamics
    nb, n = (1, 1, 1), (96, 96, 96)
    out = []
    for precision in (2, 1):
        d = Dynamics(True, nb, n, gamma=GAMMA, precision=precision)
        d.init_problem("turb", seed)
        d.step(1)
        _, b = d.get_state()
        assert d.status() == 0
        out.append(b[:, 2:-3, 2:-3, 2:-3].copy())
        d.close()
    err = np.abs(out[1] - out[0]).sum() / np.abs(out[0]).sum()
    print("face field error %.2e" % err)
    assert err <= 2e-8


def test_mixed_hydro_treats_axes_alike():
    """A mixed hydro step of a state whose axes are turned (x, y, z) -> (y, z, x) is
    the turned step: every word goes through the same operations along every axis,
    and only the FP64 sums over axes round differently (1e-16 per term, 1e-13
    allowed; one word limited in another order moved it by FP32's 1e-8)."""
    from kratos_b200 import Dynamics
    rng = np.random.default_rng(3)
    n, gamma = 12, 1.4
    rho, p = np.exp(0.3 * rng.normal(size=(2, n, n, n)))
    v = 0.5 * rng.normal(size=(3, n, n, n))
    u0 = np.stack([rho, p / (gamma - 1) + 0.5 * rho * (v ** 2).sum(0)] + [rho * q for q in v], axis=-1)[None]

    def turn(u):
        return np.ascontiguousarray(u.transpose(0, 3, 1, 2, 4)[..., [0, 1, 3, 4, 2]])
    out = []
    for u in (u0, turn(u0)):
        d = Dynamics(False, (1, 1, 1), (n, n, n), gamma=gamma, precision=1)
        d.set_state(u)
        d.step(1)
        out.append(d.get_state()[0].copy())
        d.close()
    assert np.abs(turn(out[0]) - out[1]).max() <= 1e-13 * np.abs(out[0]).max()


# Largest relative errors, in units of 2^-53 (FP64) or 2^-24 (FP32): by the exact
# residual (a fused multiply-add of the result), and against CUDA's own functions.
ARITH = r"""
#include <cstdio>
#include <cmath>
#include "kr_fast.cuh"
using namespace kr;
__device__ unsigned long long worst[ 16 ];
__device__ void note( int k, double e )
{
    if( ! ( e <= 1e300 ) ) e = 1e300;                      // NaN, too
    atomicMax( & worst[ k ], (unsigned long long) __double_as_longlong( e ) );
}
__global__ void k64( unsigned long long seed )
{
    unsigned long long h = ( blockIdx.x * 256ull + threadIdx.x + seed ) * 0x9E3779B97F4A7C15ull;
    for( int k = 0; k < 64; ++ k )
    {
        h = ( h ^ ( h >> 30 ) ) * 0xBF58476D1CE4E5B9ull + 0x94D049BB133111EBull;
        h ^= h >> 27;
        // exponents -1021..1021, mantissas random, or at the ends of a binade
        const int ex = int( ( h >> 52 ) % 2043 ) - 1021;
        unsigned long long m = h & 0xfffffffffffffull;
        if( k % 16 == 0 ) m &= 7;
        if( k % 16 == 1 ) m |= 0xffffffffffff8ull;
        if( ex == 1021 ) m = 0;
        const double x = __longlong_as_double( ( (unsigned long long)( ex + 1023 ) << 52 ) | m );
        const double u = 9007199254740992.0;               // 2^53
        const double y = rcp( x ), yn = rcp( -x );
        note( 0, fabs( fma( -x, y, 1.0 ) ) * u );
        note( 1, fabs( y / __drcp_rn( x ) - 1 ) * u );
        note( 1, yn == -y ? 0.0 : 1e9 );
        const double r = rsq( x ), p = x * r;
        note( 2, fabs( fma( -p, r, 1.0 ) - fma( x, r, -p ) * r ) / 2 * u );
        note( 3, fabs( r / rsqrt( x ) - 1 ) * u );
        const double g = kr::fsqrt( x );
        if( x >= 1e-290 )
        {
            note( 4, fabs( fma( -g, g, x ) / x ) / 2 * u );
            note( 5, fabs( g / __dsqrt_rn( x ) - 1 ) * u );
        }
        else
            note( 6, g );
    }
}
__global__ void k32(  )
{   // every normal float whose reciprocal is one
    for( unsigned i = 0x00800000u + blockIdx.x * 256u + threadIdx.x; i < 0x7e800000u; i += gridDim.x * 256u )
    {
        const float x = __uint_as_float( i );
        const double u = 16777216.0;                       // 2^24
        note( 8, fabs( double( rcp( x ) ) * x - 1 ) * u );
        const double r = rsq( x );
        note( 9, fabs( r * sqrt( double( x ) ) - 1 ) * u );
        note( 10, fabs( kr::fsqrt( x ) / sqrt( double( x ) ) - 1 ) * u );
    }
}
__global__ void edges( double * o )
{
    const double z = o[ 0 ];
    o[ 1 ] = kr::fsqrt( z ); o[ 2 ] = kr::fsqrt( z + 1e-300 ); o[ 3 ] = kr::fsqrt( z - 1 ); o[ 4 ] = kr::fsqrt( z + 1e-290 );
    o[ 5 ] = kr::fsqrt( float( z ) ); o[ 6 ] = kr::fsqrt( float( z ) + 1e-40f ); o[ 7 ] = kr::fsqrt( float( z ) - 1 );
    o[ 8 ] = isnan( kr::fsqrt( o[ 9 ] ) );
}
int main(  )
{
    for( int k = 0; k < 8; ++ k ) k64<<< 2048, 256 >>>( k * 1000003ull );
    k32<<< 4096, 256 >>>(  );
    double * o, h[ 10 ] = { 0 }, e[ 16 ];
    h[ 9 ] = NAN;
    cudaMalloc( & o, sizeof( h ) );
    cudaMemcpy( o, h, sizeof( h ), cudaMemcpyHostToDevice );
    edges<<< 1, 1 >>>( o );
    if( cudaMemcpy( h, o, sizeof( h ), cudaMemcpyDeviceToHost ) != cudaSuccess ) return 1;
    cudaMemcpyFromSymbol( e, worst, sizeof( e ) );
    for( int k = 0; k < 11; ++ k ) std::printf( "%.4f ", e[ k ] );
    for( int k = 1; k < 9; ++ k ) std::printf( "%.17g ", h[ k ] );
    return 0;
}
"""


def test_reciprocals_and_roots(tmp_path):
    """FP64, 2^28 arguments over all exponents: the last rounding alone (1 unit of
    2^-53; the reciprocal root also half of a product's, 1.5), and so within one ulp
    (2 units) of CUDA's correctly rounded reciprocal and root and within 1.5 + 2 of
    its rsqrt (1 ulp by its documentation).  FP32, every normal float: 1 ulp (2 units
    of 2^-24) for the reciprocal and 2^-22.9 (2.15) for the reciprocal root, by the PTX
    ISA, and a rounding more (3.15) for the root."""
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    root = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
    src, exe = tmp_path / "arith.cu", tmp_path / "arith"
    src.write_text(ARITH)
    subprocess.check_call([nvcc, "-gencode", "arch=compute_100a,code=sm_100a", "-O3", "-std=c++17",
                           "-I", os.path.join(root, "kratos_b200", "csrc"), "-o", str(exe), str(src)])
    out = [float(x) for x in subprocess.run([str(exe)], capture_output=True, text=True, check=True).stdout.split()]
    print(out)
    worst, edge = out[:11], out[11:]
    for k, bound in ((0, 1.01), (1, 2.01), (2, 1.51), (3, 3.52), (4, 1.01), (5, 2.01), (6, 0.0),
                     (8, 2.0), (9, 2.15), (10, 3.15)):
        assert worst[k] <= bound, (k, worst[k])
    assert edge[:3] == [0, 0, 0] and abs(edge[3] / 1e-145 - 1) < 1e-15 and edge[4:7] == [0, 0, 0] and edge[7] == 1
