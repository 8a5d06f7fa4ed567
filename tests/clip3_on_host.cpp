// The 3D clip of the library (cells3d.cu up to its pyramid walk, in "clip3.inc") run on the host: a line per query.
//   links TRIALS       seeds at the limits of rounding: cuts made, cuts after which some link is not to a vertex of the cell that
//                      holds the reversed edge and links back across it, cells that end with a missing link
#include <array>
#include <cstdio>
#include <random>
#include "warp_on_host.h"
#include "internal.h"
namespace sdot {
#include "clip3.inc"
}
using namespace sdot;
using Cell = Cell3;
typedef std::vector<std::array<double, 3>> Seeds;        // the cell's own first

static const double lo[ 3 ] = { 0, 0, 0 }, hi[ 3 ] = { 1, 1, 1 };
static std::mt19937_64 gen;
static double uniform() { return std::uniform_real_distribution<double>( -1, 1 )( gen ); }

static bool links_hold( const Cell &C, bool &missing ) {
    missing = false;
    for ( int k = 0; k < C.nv; ++k ) {
        const int v[ 3 ] = { C.va[ k ], C.vb[ k ], C.vc[ k ] };
        for ( int q = 0; q < 3; ++q ) {
            const int t = C.ad[ q ][ k ];
            if ( t == Cell::NONE ) { missing = true; continue; }
            if ( t >= C.nv ) return false;
            const int u[ 3 ] = { C.va[ t ], C.vb[ t ], C.vc[ t ] };
            bool back = false;
            for ( int p = 0; p < 3; ++p ) back = back || ( u[ p ] == v[ ( q + 1 ) % 3 ] && u[ ( p + 1 ) % 3 ] == v[ q ] && C.ad[ p ][ t ] == k );
            if ( ! back ) return false;
        }
    }
    return true;
}

// a lattice (0: cubic, 1: face-centred) or rings about an axis through the seed (their bisectors meet on it), jittered at the
// rounding of the coordinates
static Seeds tied_seeds( int kind ) {
    const double h = 0.01 * std::pow( 10.0, 0.5 * ( 1 + uniform() ) ), jitter = 1e-15 * std::pow( 10.0, 0.6 * ( 1 + uniform() ) );
    double c[ 3 ];
    for ( double &x : c ) x = 0.5 + 0.3 * uniform();
    Seeds s;
    auto add = [&]( double x, double y, double z ) { s.push_back( { c[ 0 ] + x + jitter * uniform(), c[ 1 ] + y + jitter * uniform(), c[ 2 ] + z + jitter * uniform() } ); };
    add( 0, 0, 0 );
    if ( kind < 2 ) {
        for ( int i = -2; i <= 2; ++i ) for ( int j = -2; j <= 2; ++j ) for ( int k = -2; k <= 2; ++k )
            if ( ( i || j || k ) && ( kind == 0 || ( i + j + k ) % 2 == 0 ) ) add( h * i, h * j, h * k );
    } else {
        const int rings = 1 + int( gen() % 3 );
        for ( int r = 0; r < rings; ++r ) {
            const int m = 5 + int( gen() % 12 );
            const double turn = uniform();
            for ( int k = 0; k < m; ++k ) {
                const double t = turn + 2 * M_PI * k / m;
                add( h * std::cos( t ), h * std::sin( t ), h * ( 0.6 + 0.5 * r ) * ( r & 1 ? -1 : 1 ) );
            }
        }
    }
    std::shuffle( s.begin() + 1, s.end(), gen );
    return s;
}

static void links( int trials ) {
    static Cell C;
    long cuts = 0, wrong = 0, open = 0;
    for ( int t = 0; t < trials; ++t ) {
        const Seeds s = tied_seeds( t % 8 < 2 ? t % 8 : 2 );
        std::memset( ( void * ) &C, 0x5a, sizeof( C ) );
        const double *p = s[ 0 ].data();
        warp_on_host::run( [&]( int lane ) { init_box3( C, lane, lo, hi, p[ 0 ], p[ 1 ], p[ 2 ] ); } );
        bool missing = false;
        for ( size_t j = 1; j < s.size() && C.nv > 0; ++j ) {
            const double x = s[ j ][ 0 ] - p[ 0 ], y = s[ j ][ 1 ] - p[ 1 ], z = s[ j ][ 2 ] - p[ 2 ], off = 0.5 * ( x * x + y * y + z * z );
            bool ok = true;
            warp_on_host::run( [&]( int lane ) { ok = wclip3( C, lane, x, y, z, off, tie_tol3( x, y, z, off, C.L ), int( j ), int( j ) ); } );
            if ( ! ok ) break;
            ++cuts;
            wrong += ! links_hold( C, missing );
        }
        open += missing;
    }
    std::printf( "%ld %ld %ld\n", cuts, wrong, open );
}

int main( int argc, char **argv ) {
    gen.seed( 12345 );
    if ( argc == 3 && ! std::strcmp( argv[ 1 ], "links" ) ) links( std::atoi( argv[ 2 ] ) );
    else return 2;
}
