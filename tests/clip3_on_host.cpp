// The 3D clip of the library (cells3d.cu up to its pyramid walk, in "clip3.inc") run on the host: a line per query.
//   links TRIALS       seeds at the limits of rounding: cuts made, cuts after which some link is not to a vertex of the cell that
//                      holds the reversed edge and links back across it, cells that end with a missing link
//   volume H TRIALS    a seed in a cluster of extent H in the unit box: the largest relative error of its cell's volume
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
    auto add = [&]( double x, double y, double z ) {
        const double jx = jitter * uniform(), jy = jitter * uniform(), jz = jitter * uniform();
        s.push_back( { c[ 0 ] + x + jx, c[ 1 ] + y + jy, c[ 2 ] + z + jz } );
    };
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

// the cell's volume from its vertices, as the integration sums it
static double volume( const Cell &C ) {
    double v6 = 0;
    for ( int k = 0; k < C.nv; ++k ) {
        const int v[ 3 ] = { C.va[ k ], C.vb[ k ], C.vc[ k ] };
        for ( int q = 0; q < 3; ++q ) {
            const int f = v[ q ], t = C.ad[ q ][ k ];
            if ( t == Cell::NONE ) return NAN;
            const double n2 = C.nx[ f ] * C.nx[ f ] + C.ny[ f ] * C.ny[ f ] + C.nz[ f ] * C.nz[ f ], u = C.no[ f ] / n2;
            v6 -= u * ( C.nx[ f ] * ( C.vy[ k ] * C.vz[ t ] - C.vz[ k ] * C.vy[ t ] ) + C.ny[ f ] * ( C.vz[ k ] * C.vx[ t ] - C.vx[ k ] * C.vz[ t ] ) +
                        C.nz[ f ] * ( C.vx[ k ] * C.vy[ t ] - C.vy[ k ] * C.vx[ t ] ) );
        }
    }
    return v6 / 6;
}
// and face by face in 80 bits: a square of half side R in the face's plane, cut by every other half space
typedef long double Wide;
static Wide volume_of_faces( const Seeds &s, Wide R ) {
    struct Plane { Wide n[ 3 ], o; };
    std::vector<Plane> planes;
    for ( size_t j = 1; j < s.size(); ++j ) {
        Plane p;
        Wide l = 0;
        for ( int a = 0; a < 3; ++a ) { p.n[ a ] = Wide( s[ j ][ a ] ) - s[ 0 ][ a ]; l += p.n[ a ] * p.n[ a ]; }
        l = sqrtl( l );
        for ( Wide &x : p.n ) x /= l;
        p.o = l / 2;
        planes.push_back( p );
    }
    std::sort( planes.begin(), planes.end(), []( const Plane &a, const Plane &b ) { return a.o < b.o; } );
    Wide vol = 0;
    for ( size_t f = 0; f < planes.size(); ++f ) {
        const Wide *n = planes[ f ].n;
        Wide u[ 3 ] = { 0, n[ 2 ], -n[ 1 ] }, w[ 3 ];
        if ( fabsl( n[ 0 ] ) > 0.6L ) { u[ 0 ] = -n[ 2 ]; u[ 1 ] = 0; u[ 2 ] = n[ 0 ]; }
        const Wide l = sqrtl( u[ 0 ] * u[ 0 ] + u[ 1 ] * u[ 1 ] + u[ 2 ] * u[ 2 ] );
        for ( Wide &x : u ) x /= l;
        for ( int a = 0; a < 3; ++a ) w[ a ] = n[ ( a + 1 ) % 3 ] * u[ ( a + 2 ) % 3 ] - n[ ( a + 2 ) % 3 ] * u[ ( a + 1 ) % 3 ];
        std::vector<std::array<Wide, 2>> poly = { { -R, -R }, { R, -R }, { R, R }, { -R, R } }, cut;
        for ( size_t g = 0; g < planes.size() && ! poly.empty(); ++g ) {
            if ( g == f ) continue;
            const Plane &G = planes[ g ];
            Wide a = 0, b = 0, d = 0;
            for ( int q = 0; q < 3; ++q ) { a += G.n[ q ] * u[ q ]; b += G.n[ q ] * w[ q ]; d += G.n[ q ] * n[ q ]; }
            const Wide o = G.o - d * planes[ f ].o;
            cut.clear();
            for ( size_t i = 0; i < poly.size(); ++i ) {
                const auto A = poly[ i ], B = poly[ ( i + 1 ) % poly.size() ];
                const Wide sa = a * A[ 0 ] + b * A[ 1 ] - o, sb = a * B[ 0 ] + b * B[ 1 ] - o;
                if ( sa <= 0 ) cut.push_back( A );
                const Wide t = sa / ( sa - sb );
                if ( ( sa < 0 && sb > 0 ) || ( sa > 0 && sb < 0 ) ) cut.push_back( { A[ 0 ] + t * ( B[ 0 ] - A[ 0 ] ), A[ 1 ] + t * ( B[ 1 ] - A[ 1 ] ) } );
            }
            poly = cut;
        }
        Wide area = 0;
        for ( size_t i = 0; i < poly.size(); ++i ) {
            const auto A = poly[ i ], B = poly[ ( i + 1 ) % poly.size() ];
            area += ( A[ 0 ] * B[ 1 ] - A[ 1 ] * B[ 0 ] ) / 2;
        }
        vol += fabsl( area ) * planes[ f ].o / 3;
    }
    return vol;
}

static void volumes( double h, int trials ) {
    static Cell C;
    double worst = 0;
    for ( int t = 0; t < trials; ++t ) {
        Seeds s( 1 );
        for ( double &x : s[ 0 ] ) x = 0.5 + 0.4 * uniform();
        if ( t % 2 ) for ( int k = 0; k < 64; ++k ) s.push_back( { 0.5 + 0.5 * uniform(), 0.5 + 0.5 * uniform(), 0.5 + 0.5 * uniform() } );
        for ( int k = 0; k < 40; ++k ) s.push_back( { s[ 0 ][ 0 ] + h * uniform(), s[ 0 ][ 1 ] + h * uniform(), s[ 0 ][ 2 ] + h * uniform() } );
        ProbDev P = {};
        P.pos = s[ 0 ].data();
        std::memset( ( void * ) &C, 0x5a, sizeof( C ) );
        bool over = false;
        warp_on_host::run( [&]( int lane ) {
            const double *p = P.pos;
            int met = 0;
            bool overflow = false;
            init_box3( C, lane, lo, hi, p[ 0 ], p[ 1 ], p[ 2 ] );
            cut_by_ranges3<false>( C, P, lane, 0, p[ 0 ], p[ 1 ], p[ 2 ], 0.0, 0, lane == 0 ? int( s.size() ) : 0, met, overflow );
            resolve3( C, lane );
            if ( lane == 0 ) over = overflow;
        } );
        const Wide ref = volume_of_faces( s, 16 * Wide( h ) );
        const double err = over ? 1.0 : double( fabsl( volume( C ) - ref ) / ref );
        worst = err <= worst ? worst : err;
    }
    std::printf( "%.3e\n", worst );
}

int main( int argc, char **argv ) {
    gen.seed( 12345 );
    if ( argc == 3 && ! std::strcmp( argv[ 1 ], "links" ) ) links( std::atoi( argv[ 2 ] ) );
    else if ( argc == 4 && ! std::strcmp( argv[ 1 ], "volume" ) ) volumes( std::atof( argv[ 2 ] ), std::atoi( argv[ 3 ] ) );
    else return 2;
}
