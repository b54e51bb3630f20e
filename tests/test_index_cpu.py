"""The numbering of a block's faces and sites, every one of them, on the host:
quotients by the row length of the planes that the sweeps number (x, y) or
(x, z), and the tiles of the cell and lattice launches, on shapes whose planes
go up to the largest that a block on one card has."""
import os
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

MAIN = r"""
#include <cstdio>
#include <cstdlib>
#include "kr_index.h"
using namespace kr;
// every divisor's quotients at, just below and just above multiples of it, up to 2^31
static long long quotients(  )
{
    long long bad = 0;
    for( unsigned k = 1; k < 40000; ++ k )
    {
        const unsigned d = k < 20000 ? k : unsigned( 1 + k * 53681ull % 2147483000ull );
        const udiv_t v = make_udiv( d );
        const unsigned top = 0x7fffffffu / d;
        for( unsigned j = 0; j < 400; ++ j )
        {
            const unsigned q = j < 200 ? std::min( j, top ) : top - std::min( j - 200, top );
            for( long long n = ( long long ) q * d - 1; n <= ( long long ) q * d + 1; ++ n )
                if( n >= 0 && n < ( 1LL << 31 ) )
                    bad += udiv_q1( unsigned( n ), v ) != unsigned( n ) / d;
        }
    }
    return bad;
}
int main( int argc, char ** argv )
{
    if( argc == 1 )
        return std::printf( "%lld\n", quotients(  ) ) < 0;
    const int n[ 3 ] = { atoi( argv[ 1 ] ), atoi( argv[ 2 ] ), atoi( argv[ 3 ] ) };
    long long rows = 0, sites = 0;
    const udiv_t dv = make_udiv( unsigned( n[ 0 ] + 2 ) );
    const long long face = ( long long )( n[ 0 ] + 2 ) * ( std::max( n[ 1 ], n[ 2 ] ) + 2 );
    for( unsigned t = 0; t < face + 128; ++ t )
        rows += udiv_q( t, dv ) != t / unsigned( n[ 0 ] + 2 );
    const tile_t tl = make_tile( n[ 0 ] + 1, n[ 1 ] + 1, n[ 2 ] + 1 );
    long long next = 0;
    for( unsigned s = 0; s < tile_ctas( tl ) * 256u; ++ s )
    {
        int i[ 3 ];
        if( tile_site( tl, s, i ) )
            sites += i[ 0 ] + ( long long ) tl.e0 * ( i[ 1 ] + ( long long ) tl.e1 * i[ 2 ] ) != next ++;
    }
    sites += next != ( long long ) tl.e0 * tl.e1 * tl.e2;
    std::printf( "%lld %lld\n", rows, sites );
}
"""


@pytest.fixture(scope="module")
def exe(tmp_path_factory):
    d = tmp_path_factory.mktemp("index")
    src, out = d / "index.cpp", d / "index"
    src.write_text(MAIN)
    subprocess.check_call(["g++", "-std=c++17", "-O2", "-I", os.path.join(ROOT, "kratos_b200", "csrc"),
                           str(src), "-o", str(out)])
    return str(out)


@pytest.mark.parametrize("n", [(4, 4, 4), (16, 16, 16), (33, 5, 19), (260, 252, 4), (30, 30, 2000), (4096, 8, 512),
                               (2000, 4, 2000), (2000, 2000, 4), (4000, 4, 400), (1920, 4, 1920), (9000, 4, 1800),
                               (4, 4, 400000), (4, 300000, 6), (5000000, 4, 4), (1025, 1023, 17)])
def test_every_site_and_row(exe, n):
    out = subprocess.run([exe] + [str(k) for k in n], capture_output=True, text=True, check=True).stdout.split()
    assert out == ["0", "0"], "wrong rows of the faces' planes, wrong sites of the tiles: %s" % out


def test_quotients_below_2_to_31(exe):
    out = subprocess.run([exe], capture_output=True, text=True, check=True).stdout.split()
    assert out == ["0"], "wrong quotients: %s" % out
