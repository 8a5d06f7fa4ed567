// The preconditioned CG of a batch of systems in ONE launch: a TEAM of blocks per problem runs many iterations, its blocks
// meeting at barriers -- the hardware's cluster barrier for a team of up to 16 blocks, else a counter in memory (a
// cooperative launch, so that the blocks run together; the wait is bounded).
//
// What bounds it: latency.  An iteration of 2e4 rows moves 3 MB, half a microsecond of HBM, but as a launch per vector
// operation and per multigrid level it is 13 dependent launches of about 4 us (56 us an iteration at 20,011 rows; 27 us, 7
// launches, at 1,000).  Here the same steps are separated by barriers, and there are fewer of them:
//   1  p = z + beta p and q = A p together (a neighbour's p is made from its pair {z, p}: one 16-byte gather), p . q
//   2  x += alpha p, r -= alpha q, |r|^2, and the first half of the V-cycle's level 0 (pre-smoothing, residual,
//      restriction; a neighbour's r from its pair {r, q})
//   3  the V-cycle below level 0: the larger levels by the whole team, the others by its first block
//   4  the second half of level 0: z, the pairs {z, p}, r . z
// The convergence test runs on the device, so a launch ends with the iteration that converges.  A block's share is kept
// near PCG_SHARE rows where the GPU has the blocks: the gathers of a row cost its SM's L1 about four cycles an entry, so
// that 1,250 rows on one SM take 4 us a step and 128 half a microsecond.  A barrier empties the L1, and a step then waits for
// one L2 access after the other (row bounds, entries, vector); so each block holds its rows of the matrix and of the levels
// in shared memory, and the first block the vectors of its levels, too: one L2 access a step is left.
// Measured, us an iteration with the multigrid, before (launches in a graph) and now: 1,000 2D rows 27 -> 16, 10,000 53 -> 30,
// 20,011 60 -> 38, 100,003 78 -> 57, 1e6 307 -> 300; 3D 3,001 rows 62 -> 28, 20,000 107 -> 36.  What is left is the barriers
// (2 us each for a grid's team, most of it the writes becoming visible) and the first block's levels.  Tried and slower past
// 5,000 rows: the vectors spread over a cluster's shared memories, whose network takes one address every two cycles.
//
// Sums: the rows are cut in SHARES by the row count alone, each summed by one block in a fixed tree, and every block folds
// the shares' sums in another; a block that plays several shares sums each in the same tree (the trees of eight together, so
// that it does not wait at the end of each: 148 systems of 20,011 rows, a block each, 576 -> 469 ms of CG).  A solve is
// therefore bitwise the same whatever its team's size -- which follows the batch's load -- and whatever else shares the launch.
#include "internal.h"
#include <algorithm>

namespace sdot {

constexpr int PCG_T = 768;                   // threads a block
constexpr int PCG_W = PCG_T / 32;
constexpr int PCG_SG = 8;                    // shares whose sums a block folds together
constexpr int PCG_SMEM = 220 * 1024;         // dynamic shared memory of a block
// the levels of at most this many rows are the first block's: a barrier and the steps' latency cost the team more than a
// few rounds of the block's warps (1,251 rows: 6,000 cycles by one block, 8,000 with the team's two barriers)
constexpr int PCG_CHAIN_GRID = 1600, PCG_CHAIN_CLUSTER = 512;
constexpr float PCG_OMEGA = 0.8f, PCG_ALPHA = 1.5f;      // (the smoother's and the correction's factors of mg.cu)

// rows of a share: a function of the row count alone, at most 148 shares
__host__ __device__ inline int pcg_share_rows( int n ) {
    const int k = ( ( n + 147 ) / 148 + 31 ) / 32 * 32;
    return k < PCG_SHARE ? PCG_SHARE : k;
}

struct Team {
    int rank, size;                          // this block in its team
    unsigned *bar;                           // the team's counter; NULL: the team is a cluster
    int *dead;                               // (shared) set when a wait ran out, after `polls` of them
    unsigned polls;
    unsigned goal;                           // the arrivals that the next barrier waits for
    SDOT_DEV void sync() {
        if ( size == 1 ) { __syncthreads(); return; }
        if ( ! bar ) {
            asm volatile( "barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory" );
            return;
        }
        __syncthreads();
        goal += size;
        if ( threadIdx.x == 0 && ! *dead ) {
            asm volatile( "red.release.gpu.global.add.u32 [%0], 1;" ::"l"( bar ) : "memory" );
            unsigned now = 0, k = 0;
            for ( ; k < polls; ++k ) {
                asm volatile( "ld.acquire.gpu.global.u32 %0, [%1];" : "=r"( now ) : "l"( bar ) : "memory" );
                if ( int( now - goal ) >= 0 ) break;
            }
            if ( k == polls ) *dead = 1;
        }
        __syncthreads();
    }
};

// the shares' sums (at most 148) folded: every warp by itself, the same sums in every lane
SDOT_DEV double2 pcg_fold( const double2 *part, int ns ) {
    double2 v[ ( PCG_MAX_BLOCKS + 31 ) / 32 ];
    double a = 0, b = 0;
#pragma unroll
    for ( int q = 0; q < ( PCG_MAX_BLOCKS + 31 ) / 32; ++q ) {
        const int u = int( threadIdx.x & 31 ) + 32 * q;
        v[ q ] = u < ns ? part[ u ] : make_double2( 0, 0 );
    }
#pragma unroll
    for ( int q = 0; q < ( PCG_MAX_BLOCKS + 31 ) / 32; ++q ) { a += v[ q ].x; b += v[ q ].y; }
    return make_double2( warp_sum( a ), warp_sum( b ) );
}
// the sums of the block's shares: a warp's part of each goes to `sh`, and after PCG_SG of them (or the last) the block folds
// them together, a warp a share, and writes them to out[ share ] (a barrier of the team follows before they are read): a block
// of many shares does not wait at the end of each
SDOT_DEV void pcg_share( double a, double b, bool two, int s, int s0, int s1, double2 *out, double2 *sh ) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, at = ( s - s0 ) % PCG_SG;
    a = warp_sum( a );
    if ( two ) b = warp_sum( b );
    if ( lane == 0 ) sh[ at * PCG_W + warp ] = make_double2( a, b );
    if ( at + 1 < PCG_SG && s + 1 < s1 ) return;
    __syncthreads();
    if ( warp <= at ) {
        const double2 v = lane < PCG_W ? sh[ warp * PCG_W + lane ] : make_double2( 0, 0 );
        a = warp_sum( v.x );
        if ( two ) b = warp_sum( v.y );
        if ( lane == 0 ) out[ s - at + warp ] = make_double2( a, b );
    }
    __syncthreads();
}

// A level as a block sees it: the arrays of its rows in shared memory where they fit (offset so that they take the level's
// own row and entry numbers), else the level's own
struct SLev {
    int n, nn;
    const int *rp, *col;
    const float *val, *vd, *dia, *dinv;      // vd: val times the smoother's factor at the column (NULL: from dinv0)
    const float *dinv0;                      // the level's own, every row
    float *b, *x, *y, *bn;
    const float *xn, *inv;
    float *b0, *y0;                          // the first block's first level: the level's own rhs and solution, b and y their copies
};

struct Smem {
    char *at, *end;
    // `count` elements, NULL if they do not fit (the same answer in every thread)
    template<class X> SDOT_DEV X *take( long count ) {
        const long bytes = ( count * long( sizeof( X ) ) + 15 ) & ~15l;
        if ( bytes > end - at ) return nullptr;
        X *p = reinterpret_cast<X *>( at );
        at += bytes;
        return p;
    }
};

template<class X> SDOT_DEV const X *pcg_copy( Smem &S, const X *src, long a, long b ) {
    X *d = S.take<X>( b - a );
    if ( ! d ) return src;
    for ( long k = a + threadIdx.x; k < b; k += PCG_T ) d[ k - a ] = src[ k ];
    return d - a;
}
// the rows [ r0, r1 ) of level M
SDOT_DEV void pcg_stage( Smem &S, SLev &Z, const MgLevel &M, int r0, int r1 ) {
    if ( r1 <= r0 ) return;
    const int e0 = M.rp[ r0 ], e1 = M.rp[ r1 ];
    Z.rp = pcg_copy( S, M.rp, r0, long( r1 ) + 1 );
    Z.dia = pcg_copy( S, M.dia, r0, r1 );
    Z.dinv = pcg_copy( S, M.dinv, r0, r1 );
    Z.col = pcg_copy( S, M.col, e0, e1 );
    Z.val = pcg_copy( S, const_cast<const float *>( M.val ), e0, e1 );
    float *vd = S.take<float>( e1 - e0 );
    if ( vd ) {
        for ( int k = e0 + threadIdx.x; k < e1; k += PCG_T ) vd[ k - e0 ] = M.val[ k ] * ( PCG_OMEGA * M.dinv[ M.col[ k ] ] );
        Z.vd = vd - e0;
    }
}

// sum over the entries of row i that fall to lane `sub` of its LN lanes, f( entry, col ); the first NCH rounds are
// loaded together (a 2D row has 6 entries, a 3D row 16), the rest of a longer row one by one
template<int LN, int NCH, class S, class F>
SDOT_DEV S row_part( const int *rp, const int *col, int i, bool in, int sub, F f ) {
    int b = 0, e = 0;
    if ( in ) { b = rp[ i ]; e = rp[ i + 1 ]; }
    S t[ NCH ];
#pragma unroll
    for ( int q = 0; q < NCH; ++q ) {
        const int k = b + sub + q * LN;
        t[ q ] = k < e ? f( k, col[ k ] ) : S( 0 );
    }
    S s = t[ 0 ];
#pragma unroll
    for ( int q = 1; q < NCH; ++q ) s += t[ q ];
    for ( int k = b + sub + NCH * LN; k < e; k += LN ) s += f( k, col[ k ] );
    return s;
}

// LN lanes a row, PK rows an aggregate (2D: 4 and 4, 3D: 8 and 8).  An ITEM is what a warp does at a time: a whole number
// of aggregates, IR rows (8) in GP passes
template<int LN, int PK>
struct Pcg {
    static constexpr int NCH = LN == 8 ? 3 : 2;
    static constexpr int RPW = 32 / LN;                  // rows a warp holds at a time
    static constexpr int GL = LN * PK < 32 ? LN * PK : 32;      // lanes of one aggregate in a pass
    static constexpr int GP = LN * PK / GL;              // passes of one aggregate
    static constexpr int IR = RPW * GP;

    // level l's pre-smoothing from zero, residual and restriction for the fine rows of one item; bv( j ): the level's rhs at
    // row j (made from {r, q} at level 0); `own( i, b )` is called once a row by its first lane
    template<class B, class Own>
    SDOT_DEV static void down_item( const SLev &M, int item, int lane, B bv, Own own ) {
        const int sub = lane % LN;
        float acc = 0;
#pragma unroll
        for ( int h = 0; h < GP; ++h ) {
            const int i = IR * item + h * RPW + lane / LN;
            const bool in = i < M.n;
            const float *vd = M.vd, *val = M.val, *dinv0 = M.dinv0;
            acc += row_part<LN, 3, float>( M.rp, M.col, i, in, sub, [&]( int k, int j ) {
                return ( vd ? vd[ k ] : val[ k ] * ( PCG_OMEGA * dinv0[ j ] ) ) * bv( j );
            } );
            if ( in && sub == 0 ) {
                const float bi = bv( i ), xi = PCG_OMEGA * M.dinv[ i ] * bi, di = M.dia[ i ];
                own( i, bi );
                M.x[ i ] = xi;
                acc += bi - di * xi;
            }
        }
#pragma unroll
        for ( int o = 1; o < GL; o <<= 1 ) acc += __shfl_xor_sync( 0xffffffffu, acc, o );
        const int I = ( IR * item + lane / LN ) / PK;
        if ( lane % GL == 0 && I < M.nn ) M.bn[ I ] = acc;
    }

    // the correction of level l + 1 prolonged and post-smoothed on the rows of one item; `put( i, y )` once a row
    template<class Put>
    SDOT_DEV static void up_item( const SLev &M, int item, int lane, Put put ) {
        const int sub = lane % LN;
        const float *x = M.x, *xn = M.xn, *val = M.val;
#pragma unroll
        for ( int h = 0; h < GP; ++h ) {
            const int i = IR * item + h * RPW + lane / LN;
            const bool in = i < M.n;
            float s = row_part<LN, 3, float>( M.rp, M.col, i, in, sub,
                                                [&]( int k, int j ) { return val[ k ] * ( x[ j ] + PCG_ALPHA * xn[ j / PK ] ); } );
#pragma unroll
            for ( int o = 1; o < LN; o <<= 1 ) s += __shfl_xor_sync( 0xffffffffu, s, o );
            if ( in && sub == 0 ) {
                const float xi = x[ i ] + PCG_ALPHA * xn[ i / PK ];
                put( i, xi + PCG_OMEGA * M.dinv[ i ] * ( M.b[ i ] - ( M.dia[ i ] * xi - s ) ) );
            }
        }
    }

    // the items of a level that this block does: an equal run of them
    SDOT_DEV static int item0( int n, Team &T, int rank ) { return int( long( ( n + IR - 1 ) / IR ) * rank / T.size ); }

    // z = M^-1 r below level 0: b of level 1 in, y of level 1 out; the levels f and up by the first block
    static __device__ __noinline__ void coarse( const SLev *lv, int L, int f, Team &T ) {
        const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
        for ( int l = 1; l < f; ++l ) {
            const SLev &M = lv[ l ];
            const float *b = M.b;
            for ( int u = item0( M.n, T, T.rank ) + warp; u < item0( M.n, T, T.rank + 1 ); u += PCG_W )
                down_item( M, u, lane, [&]( int j ) { return b[ j ]; }, []( int, float ) {} );
            T.sync();
        }
        if ( T.rank == 0 ) {
            const SLev &F = lv[ f ];
            if ( F.b0 ) {
                for ( int i = threadIdx.x; i < F.n; i += PCG_T ) F.b[ i ] = F.b0[ i ];
                __syncthreads();
            }
            for ( int l = f; l + 1 < L; ++l ) {
                const SLev &M = lv[ l ];
                const float *b = M.b;
                for ( int u = warp; IR * u < M.n; u += PCG_W ) down_item( M, u, lane, [&]( int j ) { return b[ j ]; }, []( int, float ) {} );
                __syncthreads();
            }
            const SLev &M = lv[ L - 1 ];                          // the coarsest: its dense inverse, a warp a row
            for ( int i = warp; i < M.n; i += PCG_W ) {
                float s = lane < M.n ? M.inv[ i * M.n + lane ] * M.b[ lane ] : 0.0f;
#pragma unroll
                for ( int o = 16; o > 0; o >>= 1 ) s += __shfl_xor_sync( 0xffffffffu, s, o );
                if ( lane == 0 ) M.y[ i ] = s;
            }
            for ( int l = L - 2; l >= f; --l ) {
                __syncthreads();
                const SLev &N = lv[ l ];
                for ( int u = warp; IR * u < N.n; u += PCG_W ) up_item( N, u, lane, [&]( int i, float y ) { N.y[ i ] = y; } );
            }
            if ( F.y0 ) {
                __syncthreads();
                for ( int i = threadIdx.x; i < F.n; i += PCG_T ) F.y0[ i ] = F.y[ i ];
            }
        }
        T.sync();
        for ( int l = f - 1; l >= 1; --l ) {
            const SLev &M = lv[ l ];
            for ( int u = item0( M.n, T, T.rank ) + warp; u < item0( M.n, T, T.rank + 1 ); u += PCG_W )
                up_item( M, u, lane, [&]( int i, float y ) { M.y[ i ] = y; } );
            T.sync();
        }
    }

    static __device__ __forceinline__ void run( const VecDev &V, const MgLevel *glv, int L, int burst, int chain, Team &T, double2 *sh,
                                                SLev *lv, Smem S ) {
        const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, sub = lane % LN;
        const int n = V.n, rows = pcg_share_rows( n ), ns = ( n + rows - 1 ) / rows;
        // this block's shares
        const int s0 = int( ( long ) ns * T.rank / T.size ), s1 = int( ( long ) ns * ( T.rank + 1 ) / T.size );
        const int r0 = s0 * rows, r1 = min( n, s1 * rows );
        // the levels of at most `chain` rows (the coarsest always) are the first block's: their matrices and vectors first
        int f = 1;
        while ( f + 1 < L && T.size > 1 && glv[ f ].n > chain ) ++f;
        for ( int l = L - 1; l >= 0; --l ) {
            const MgLevel &M = glv[ l ];
            SLev Z;
            Z.n = M.n; Z.nn = M.nn; Z.rp = M.rp; Z.col = M.col; Z.val = M.val; Z.vd = nullptr; Z.dia = M.dia; Z.dinv = M.dinv; Z.dinv0 = M.dinv;
            Z.b = M.b; Z.x = M.x; Z.y = M.y; Z.bn = M.bn; Z.xn = M.xn; Z.inv = M.inv; Z.b0 = Z.y0 = nullptr;
            if ( l >= f && T.rank == 0 ) {
                if ( l == L - 1 ) Z.inv = pcg_copy( S, const_cast<const float *>( M.inv ), 0, long( M.n ) * M.n );
                else pcg_stage( S, Z, M, 0, M.n );
                if ( float *p = S.take<float>( M.n ) ) Z.x = p;
                const bool meets = l == f && T.size > 1;              // (level f's rhs and solution meet the other blocks)
                if ( float *p = S.take<float>( M.n ) ) { if ( meets ) Z.b0 = Z.b; Z.b = p; }
                if ( float *p = S.take<float>( M.n ) ) { if ( meets ) Z.y0 = Z.y; Z.y = p; }
            } else if ( l > 0 && l < f )
                pcg_stage( S, Z, M, IR * item0( M.n, T, T.rank ), min( M.n, IR * item0( M.n, T, T.rank + 1 ) ) );
            else if ( l == 0 )
                pcg_stage( S, Z, M, r0, r1 );
            __syncthreads();
            if ( threadIdx.x == 0 ) {
                if ( l + 1 < L ) {
                    const SLev &N = lv[ l + 1 ];
                    Z.bn = l >= f || ! N.b0 ? N.b : N.b0;
                    Z.xn = l >= f || ! N.y0 ? N.y : N.y0;
                }
                lv[ l ] = Z;
            }
            __syncthreads();
        }
        double2 *pz = V.pz, *rq = V.rq, *part2 = V.part2;
        double *x = V.x, *r = V.r, *p2 = V.p2, *sc = V.sc;
        const int *rp = V.row_ptr, *col = V.col;
        const double *val = V.val, *dia = V.dia;
        if ( r1 > r0 ) {
            const int e0 = rp[ r0 ], e1 = rp[ r1 ];
            val = pcg_copy( S, val, e0, e1 );
            dia = pcg_copy( S, dia, r0, r1 );
            if ( L > 0 ) { rp = lv[ 0 ].rp; col = lv[ 0 ].col; }
            else { rp = pcg_copy( S, rp, r0, long( r1 ) + 1 ); col = pcg_copy( S, col, e0, e1 ); }
        }
        __syncthreads();
        const double tol = V.tol, maxit = V.maxit;
        int par = 0;
        double rz = sc[ SC_RZ ], beta = sc[ SC_BETA ], bnorm = sc[ SC_BNORM ], it = sc[ SC_ITER ], rnorm = sc[ SC_RNORM ];
        double conv = 0, fail = 0;
        const bool start = it < 0;
        if ( start ) {
            const double mean = sc[ SC_MEAN ];
            for ( int i = r0 + threadIdx.x; i < r1; i += PCG_T ) {
                const double b = V.b[ i ] - mean;
                V.b[ i ] = b;
                x[ i ] = 0;
                rq[ i ] = make_double2( b, 0.0 );
                pz[ i ] = make_double2( 0.0, 0.0 );
            }
            T.sync();                        // (every block has read the scalars, too)
        }
        for ( int k = 0; k < burst || ( start && k == burst ); ++k ) {
            const bool first = start && k == 0;
            double alpha = 0;
            if ( ! first ) {
                // 1: p = z + beta p, q = A p
                for ( int s = s0; s < s1; ++s ) {
                    double pq = 0;
                    for ( int i0 = s * rows + warp * RPW; i0 < min( n, ( s + 1 ) * rows ); i0 += PCG_W * RPW ) {
                        const int i = i0 + lane / LN;
                        const bool in = i < n;
                        double t = row_part<LN, NCH, double>( rp, col, i, in, sub, [&]( int k, int j ) {
                            const double2 zp = pz[ j ];
                            return val[ k ] * ( zp.x + beta * zp.y );
                        } );
#pragma unroll
                        for ( int o = 1; o < LN; o <<= 1 ) t += __shfl_xor_sync( 0xffffffffu, t, o );
                        if ( in && sub == 0 ) {
                            const double2 zp = pz[ i ];
                            const double p = zp.x + beta * zp.y, q = dia[ i ] * p - t;
                            p2[ i ] = p;
                            rq[ i ] = make_double2( r[ i ], q );
                            pq += p * q;
                        }
                    }
                    pcg_share( pq, 0.0, false, s, s0, s1, part2 + par * ns, sh );
                }
                T.sync();
                const double pq = pcg_fold( part2 + par * ns, ns ).x;
                par ^= 1;
                if ( ! ( pq > 0 ) ) { conv = 2; fail = 1; break; }
                alpha = rz / pq;
            }
            // 2: x, r, |r|^2; with the multigrid its level 0 on the way down, else z = r / dia and r . z
            for ( int s = s0; s < s1; ++s ) {
                double rr = 0, zz = 0;
                if ( L > 0 ) {
                    const SLev &M = lv[ 0 ];
                    for ( int u = s * rows / IR + warp; IR * u < min( n, ( s + 1 ) * rows ); u += PCG_W )
                        down_item( M, u, lane, [&]( int j ) { const double2 v = rq[ j ]; return float( v.x - alpha * v.y ); },
                                   [&]( int i, float b ) {
                                       const double2 v = rq[ i ];
                                       const double ri = v.x - alpha * v.y;
                                       M.b[ i ] = b;
                                       r[ i ] = ri;
                                       if ( ! first ) x[ i ] += alpha * p2[ i ];
                                       rr += ri * ri;
                                   } );
                } else {
                    for ( int i = s * rows + threadIdx.x; i < min( n, ( s + 1 ) * rows ); i += PCG_T ) {
                        const double2 v = rq[ i ];
                        const double ri = v.x - alpha * v.y, z = ri / dia[ i ], p = first ? 0.0 : p2[ i ];
                        r[ i ] = ri;
                        if ( ! first ) x[ i ] += alpha * p;
                        pz[ i ] = make_double2( z, p );
                        rr += ri * ri;
                        zz += ri * z;
                    }
                }
                pcg_share( rr, zz, L == 0, s, s0, s1, part2 + par * ns, sh );
            }
            T.sync();
            const double2 s = pcg_fold( part2 + par * ns, ns );
            par ^= 1;
            rnorm = sqrt( s.x );
            if ( first ) {
                bnorm = rnorm;
                it = 0;
                if ( s.x == 0 ) conv = 1;
                if ( V.cap > 0 && sc[ SC_NNZ ] > double( n ) * V.cap ) { conv = 2; fail = 1; }     // (past the CSR's capacity)
            } else {
                it += 1;
                if ( rnorm <= tol * bnorm ) conv = 1;
                else if ( it >= maxit ) { conv = 2; fail = 1; }
            }
            if ( *T.dead ) { conv = 2; fail = 1; }      // (a barrier gave up: every block leaves, and the launch is an error)
            if ( conv != 0 ) break;
            double rz1 = s.y;
            if ( L > 0 ) {
                // 3, 4: the V-cycle's coarse levels, then level 0 on the way up
                coarse( lv, L, f, T );
                for ( int s = s0; s < s1; ++s ) {
                    double zz = 0;
                    const SLev &M = lv[ 0 ];
                    for ( int u = s * rows / IR + warp; IR * u < min( n, ( s + 1 ) * rows ); u += PCG_W )
                        up_item( M, u, lane, [&]( int i, float y ) {
                            const double z = double( y );
                            zz += r[ i ] * z;
                            pz[ i ] = make_double2( z, first ? 0.0 : p2[ i ] );
                        } );
                    pcg_share( zz, 0.0, false, s, s0, s1, part2 + par * ns, sh );
                }
                T.sync();
                rz1 = pcg_fold( part2 + par * ns, ns ).x;
                par ^= 1;
            }
            beta = first ? 0.0 : rz1 / rz;
            rz = rz1;
        }
        if ( T.rank == 0 && threadIdx.x == 0 ) {
            sc[ SC_RZ ] = rz; sc[ SC_BETA ] = beta; sc[ SC_BNORM ] = bnorm; sc[ SC_ITER ] = it; sc[ SC_RNORM ] = rnorm;
            sc[ SC_FAIL ] = fail; sc[ SC_CONV ] = conv;
        }
    }
};

// teams: each block's { problem, rank, team size, team }; bars: a counter per team, zeroed (NULL: the teams are clusters)
__global__ void __launch_bounds__( PCG_T, 1 ) k_pcg( const PcgProb *__restrict__ probs, const int4 *__restrict__ teams,
                                                 const MgLevel *__restrict__ chain, const VecDev *__restrict__ vs, int burst, unsigned *bars,
                                                 unsigned polls, ErrRec *err ) {
    extern __shared__ __align__( 16 ) char pcg_smem[];
    __shared__ double2 sh[ PCG_SG * PCG_W ];
    __shared__ SLev lv[ MG_MAX_LEVELS ];
    __shared__ int dead;
    const int4 t = teams[ blockIdx.x ];
    const PcgProb P = probs[ t.x ];
    const VecDev &V = vs[ P.vec ];
    if ( threadIdx.x == 0 ) dead = 0;
    Team T{ t.y, t.z, bars ? bars + t.w : nullptr, &dead, polls, 0u };
    const double done = V.sc[ SC_CONV ];
    __syncthreads();
    T.sync();                                // (read by every block before the first one's last write)
    if ( done != 0 ) return;                 // (the whole team)
    const int small = bars ? PCG_CHAIN_GRID : PCG_CHAIN_CLUSTER;
    const Smem S{ pcg_smem, pcg_smem + PCG_SMEM };
    if ( P.count > 0 && chain[ P.first ].pack == 8 ) Pcg<8, 8>::run( V, chain + P.first, P.count, burst, small, T, sh, lv, S );
    else Pcg<4, 4>::run( V, chain + P.first, P.count, burst, small, T, sh, lv, S );
    // a wait that ran out: the device did not run the team's blocks together -- not a failure of the system
    if ( threadIdx.x == 0 && dead && atomicCAS( &err->code, 0, 2 ) == 0 ) { err->kind = 0; err->prob = t.x; err->seed = -1; err->needed = 0; }
}

// the launch of `blocks` blocks, in clusters of `cluster` (0: cooperative)
static void pcg_config( cudaLaunchConfig_t &cfg, cudaLaunchAttribute &at, int blocks, int cluster ) {
    cfg = {};
    cfg.gridDim = dim3( blocks );
    cfg.blockDim = dim3( PCG_T );
    cfg.dynamicSmemBytes = PCG_SMEM;
    cudaFuncSetAttribute( k_pcg, cudaFuncAttributeMaxDynamicSharedMemorySize, PCG_SMEM );      // (per device: set for every launch)
    if ( cluster ) {
        if ( cluster > 8 ) cudaFuncSetAttribute( k_pcg, cudaFuncAttributeNonPortableClusterSizeAllowed, 1 );
        at.id = cudaLaunchAttributeClusterDimension;
        at.val.clusterDim.x = cluster; at.val.clusterDim.y = 1; at.val.clusterDim.z = 1;
    } else {
        at.id = cudaLaunchAttributeCooperative;
        at.val.cooperative = 1;
    }
    cfg.attrs = &at;
    cfg.numAttrs = 1;
}

PcgDevice pcg_device() {
    PcgDevice D{ 1, {} };
    int dev = 0, n = 0;
    if ( cudaGetDevice( &dev ) == cudaSuccess && cudaDeviceGetAttribute( &n, cudaDevAttrMultiProcessorCount, dev ) == cudaSuccess && n > 1 )
        D.blocks = std::min( n, PCG_MAX_BLOCKS );
    for ( int c = 0; c < 5; ++c ) {
        cudaLaunchConfig_t cfg;
        cudaLaunchAttribute at;
        pcg_config( cfg, at, 1 << c, 1 << c );
        if ( cudaOccupancyMaxActiveClusters( &D.clusters[ c ], k_pcg, &cfg ) != cudaSuccess ) { D.clusters[ c ] = 0; cudaGetLastError(); }
    }
    return D;
}

// the blocks of each of `np` problems of a launch of at most `D.blocks`: one, the others in proportion to its rows, none more than
// it has shares.  When no team passes 16 blocks, every team is a cluster instead if they all run at once (of 148 SMs 15
// clusters of 8 and 7 of 16) and a block's rows stay within PCG_CLUSTER_ROWS of that: a cluster's barriers are some 6 us an
// iteration cheaper, a row more on a block costs 0.02 to 0.04.  Returns the cluster's size, 0 for none, and the ROUNDS of the
// fullest block: a warp's turns over its shares
constexpr int PCG_CLUSTER_ROWS = 200, PCG_ROUND = 8 * PCG_W;
static int pcg_teams( const int *rows, int np, const PcgDevice &D, std::vector<int> &size, int &rounds ) {
    size.assign( np, 1 );
    long sum = 0;
    int big = 0, load = 0, widest = 0;
    for ( int k = 0; k < np; ++k ) { sum += rows[ k ]; widest = std::max( widest, rows[ k ] ); }
    auto per = []( int a, int b ) { return ( a + b - 1 ) / b; };
    auto shares = [&]( int k ) { return per( rows[ k ], pcg_share_rows( rows[ k ] ) ); };
    for ( int k = 0; k < np; ++k ) {
        size[ k ] = std::min( shares( k ), 1 + int( double( D.blocks - np ) * rows[ k ] / double( sum ) ) );
        big = std::max( big, size[ k ] );
        load = std::max( load, per( rows[ k ], size[ k ] ) );
    }
    int cluster = 0;
    if ( big <= 16 && D.clusters[ 0 ] >= np ) {
        int c = 0;
        while ( ( 1 << c ) < big && D.clusters[ c + 1 ] >= np ) ++c;
        if ( per( widest, 1 << c ) <= load + PCG_CLUSTER_ROWS ) { cluster = 1 << c; size.assign( np, cluster ); }
    }
    rounds = 0;
    for ( int k = 0; k < np; ++k ) rounds = std::max( rounds, per( shares( k ), size[ k ] ) * per( pcg_share_rows( rows[ k ] ), PCG_ROUND ) );
    return cluster;
}

// The launches of a batch.  A problem has a block at least, so with fewer problems a launch the SMs are shared out finer, but the
// launches run one after the other.  Taken: the cut whose iteration takes least, a launch of R rounds taking 36 + 3.5 R + 0.1 R^2
// us (its barriers and coarse levels; a round's latency; what no longer fits in shared memory).  Measured, ms of CG with so many
// systems a launch: 65 of 20,011 rows, all 259, 33 199, 16 182, 8 219, 4 320; 17 of 100,003, all 279, 9 255, 4 212, 2 280, 1 435;
// 33 of 50,003, all 264, 17 237, 8 183, 4 238
double pcg_plan( const std::vector<int> &rows, const PcgDevice &D, std::vector<PcgLaunch> &launches, std::vector<int4> &teams ) {
    const int np = int( rows.size() );
    launches.clear();
    teams.clear();
    std::vector<int> size;
    long least = -1;
    for ( int each = std::min( np, D.blocks ); each >= 1; each /= 2 ) {
        std::vector<PcgLaunch> plan;
        std::vector<int4> blocks;
        long time = 0;
        for ( int b = 0; b < np; b += each ) {
            PcgLaunch l{ b, std::min( np, b + each ) - b, int( blocks.size() ), 0, 0 };
            int R;
            l.cluster = pcg_teams( rows.data() + b, l.nprob, D, size, R );
            time += 360 + 35l * R + long( R ) * R;
            for ( int k = 0; k < l.nprob; ++k )
                for ( int q = 0; q < size[ k ]; ++q ) blocks.push_back( make_int4( k, q, size[ k ], k ) );
            l.nblock = int( blocks.size() ) - l.block;
            plan.push_back( l );
        }
        if ( least < 0 || time < least ) { least = time; launches = plan; teams = blocks; }
    }
    return 0.1 * double( least );
}

// the launches hold the stream until their slowest system has had its burst: 10 ms at most where the solve is alone and a request
// may come (256 iterations of up to 100,000 rows; 34 of 1e6), 4 ms where other solves wait, and half as many iterations
// where their diagrams do; not under 8, which a tick's copies and decisions (0.2 ms) cost a tenth of at most
int pcg_burst( double us, bool alone, bool diagrams ) {
    const int most = alone ? 256 : ( diagrams ? 32 : 64 );
    return std::max( 8, std::min( most, int( ( alone ? 10000 : 4000 ) / us ) ) );
}

cudaError_t launch_pcg( const Launch &L, const PcgProb *probs, const int4 *teams, int nblocks, int cluster, int nteams, const MgLevel *chain,
                        const VecDev *vs, int burst, unsigned *bars, unsigned polls, ErrRec *err ) {
    if ( nblocks <= 0 ) return cudaSuccess;
    cudaLaunchConfig_t cfg;
    cudaLaunchAttribute at;
    pcg_config( cfg, at, nblocks, cluster );
    cfg.stream = L.stream;
    if ( cluster ) bars = nullptr;
    else {
        const cudaError_t e = cudaMemsetAsync( bars, 0, size_t( nteams ) * sizeof( unsigned ), L.stream );
        if ( e != cudaSuccess ) return e;
    }
    const cudaError_t e = cudaLaunchKernelEx( &cfg, k_pcg, probs, teams, chain, vs, burst, bars, polls, err );
    ++*L.launches;
    return e;
}

} // namespace sdot
