// Fused MLS setup, FP64 form, with the reference's Jacobi on the integer
// pipes (sm_103a): the stages of dtk_setup_fp64.cu.
//
// What bounds it: GB300 issues one FP64 warp instruction per 64 cycles per SM
// sub-partition, and the FP64 Jacobi spends about 150 of them on each of about
// 113 rotations a target (FP64 pipe 79% busy).  Here the rotations run in
// 89-bit fixed point on the IMAD and ALU pipes (dtk_fixed.cuh), which leaves
// the gather passes to the FP64 pipe, and these are cut down too: the moments
// are the 35 distinct sums of monomials up to degree 4 (not 55 products), the
// weight's quotient takes 3 operations, and the second pass reads the weights
// the first one left in the coefficient array.  What is left is issue and
// latency: about 2.4k warp instructions a rotation at 53% of the issue slots
// with 10 warps an SM (shared memory), FP64 pipe 27%, ALU 37%.  The loop's code
// is kept small: with its two halves unrolled the 2M setup takes 44 ms in place
// of 37.6 (instruction fetch).  2M quadratic targets, k = 32: 84 -> 37.6 ms; 10k,
// k = 20: 1.20 -> 0.60 ms; 200k rows of 120 within a radius: 18.6 -> 8.9 ms; the
// batched setup of 1.5M targets 26 -> 15.
//
// Targets the fixed-point form hands back (near-singular moments, scales out
// of range, eigenvalues at the truncation threshold) are listed, and the FP64
// kernel runs them afterwards.
#include "dtk_common.cuh"
#include "dtk_fixed.cuh"
#include "dtk_moments.cuh"

#include <algorithm>

namespace dtk
{
namespace
{

constexpr unsigned FULL = 0xffffffffu;

// The support radius of a target, 1.1 * max(10 eps, max |x|) (computeRadius),
// and its reciprocal.
struct Support
{
    double radius, inv;
};
__device__ __forceinline__ Support support_of( double d2max )
{
    double distance = 10. * DBL_EPSILON;
    double const dmax = __dsqrt_rn( d2max );
    if ( dmax > distance )
        distance = dmax;
    double const radius = 1.1 * distance;
    return Support{radius, 1.0 / radius};
}

// A diagonal moment, and with it the smallest eigenvalue, is certainly below the
// truncation threshold: the least over the axes of the sum of phi x^2 (M = 4;
// phi x^2 y^2, M = 10) is at most 1/3 (1/9) of that of phi rho^2 (rho^4), and
// phi(q) q^2 1.1^2 / 3 < 0.125, phi(q) q^4 1.1^4 / 9 < 0.0125 for every positive
// phi.  Such a row is the FP64 kernel's, before its moments are summed.
template <int M>
__device__ __forceinline__ bool truncates_by_size( double d2max, int len )
{
    double const most = M == 10 ? 0.0125 * ( d2max * d2max ) : 0.125 * d2max;
    return M > 1 && len * most < 4.440892098500626e-16; // 2^FX_TRUNCATE
}

// phi of a neighbour, rounded as the reference rounds it: ill-conditioned rows
// carry an ulp of a weight into the twelfth digit of their coefficients.  The
// quotient |x| / radius comes from the reciprocal and one residual (3 FP64
// operations in place of 9).  The multiply-adds are spelled out, so that every
// kernel rounds alike.
__device__ __forceinline__ double weight_of( int rbf, double xx, double yy, double zz, Support const &s )
{
    double const dist = __dsqrt_rn( __dadd_rn( __dadd_rn( xx, yy ), zz ) );
    double const q = __dmul_rn( dist, s.inv );
    return rbf_eval<double>( rbf, fma( fma( -q, s.radius, dist ), s.inv, q ) );
}

// row0 . P
template <int M>
__device__ __forceinline__ double dot_basis( double const *row0, double x, double y, double z )
{
    double acc = row0[0];
    if constexpr ( M >= 4 )
    {
        acc = fma( row0[1], x, acc );
        acc = fma( row0[2], y, acc );
        acc = fma( row0[3], z, acc );
    }
    if constexpr ( M == 10 )
    {
        // x (r4 x + r5 y + r6 z) + y (r7 y + r8 z) + r9 z z
        acc = fma( x, fma( row0[4], x, fma( row0[5], y, row0[6] * z ) ), acc );
        acc = fma( y, fma( row0[7], y, row0[8] * z ), acc );
        acc = fma( row0[9] * z, z, acc );
    }
    return acc;
}

// The state of a warp's matrices in shared memory, interleaved by matrix: the
// two leading digits of a number as one 64-bit word, the third digits in a
// plane of their own, the exponents as bytes (712 B a matrix at M = 10).  With
// COLS = 32 every lane has a matrix (the fewest instructions: 10 warps an SM).
// With COLS = 16 lanes c and c + 16 share matrix c, each scanning half of the
// entries and rotating half of the columns, both computing the angle: 1.4
// times the instructions, but a shorter chain, for launches that do not fill
// the GPU.  Both give the same bits.  The rotation log lies in the global work
// area, interleaved by resident matrix.
template <int M>
struct FixedLayout
{
    static constexpr int OFF = M * ( M - 1 ) / 2;
    // a block's table of FxLayout::column: (up, uq) of pair u and index t as two
    // bytes at u * PITCH + t (the odd pitch spreads the lanes' rows over the
    // banks)
    static constexpr int PITCH = M > 2 ? ( M - 2 ) | 1 : 1;
    static constexpr size_t TABLE = ( OFF * PITCH * sizeof( uint16_t ) + 15 ) / 16 * 16;
    // bytes a matrix
    static constexpr size_t BYTES =
        ( OFF + 2 * M ) * sizeof( int2 ) + OFF * sizeof( int32_t ) + ( M + 3 ) / 4 * 4;
};

template <int M, int COLS_>
struct FixedState
{
    static constexpr int COLS = COLS_, PARTS = 32 / COLS, OFF = FixedLayout<M>::OFF;
    int2 *N;    // leading digits of F, its diagonal, V
    int32_t *L; // last digits of F
    int8_t *E;
    uint16_t const *T;
    double *W;
    int64_t ut, us;
    int part;
    __device__ FixedState( void *warp_smem, uint16_t const *table, int lane, double *work, int64_t warp,
                           int64_t warps )
        : N( (int2 *)warp_smem + lane % COLS )
        , L( (int32_t *)( (int2 *)warp_smem + ( OFF + 2 * M ) * COLS ) + lane % COLS )
        , E( (int8_t *)( (int32_t *)( (int2 *)warp_smem + ( OFF + 2 * M ) * COLS ) + OFF * COLS ) + lane % COLS )
        , T( table )
        , W( work )
        , ut( warp * COLS + lane % COLS )
        , us( warps * COLS )
        , part( lane / COLS )
    {
    }
    __device__ __forceinline__ double &a( int u ) const { return reinterpret_cast<double *>( N )[u * COLS]; }
    __device__ __forceinline__ FxNum<3> f( int u ) const
    {
        int2 const n = N[u * COLS];
        return FxNum<3>{{n.x, n.y, L[u * COLS]}};
    }
    __device__ __forceinline__ void set_f( int u, FxNum<3> const &x ) const
    {
        N[u * COLS] = make_int2( x.d[0], x.d[1] );
        L[u * COLS] = x.d[2];
    }
    __device__ __forceinline__ int64_t diag( int k ) const
    {
        return reinterpret_cast<int64_t *>( N )[( OFF + k ) * COLS];
    }
    __device__ __forceinline__ void set_diag( int k, int64_t x ) const
    {
        reinterpret_cast<int64_t *>( N )[( OFF + k ) * COLS] = x;
    }
    __device__ __forceinline__ FxNum<2> v( int k ) const
    {
        int2 const n = N[( OFF + M + k ) * COLS];
        return FxNum<2>{{n.x, n.y}};
    }
    __device__ __forceinline__ void set_v( int k, FxNum<2> const &x ) const
    {
        N[( OFF + M + k ) * COLS] = make_int2( x.d[0], x.d[1] );
    }
    __device__ __forceinline__ double &w( int k ) const { return a( OFF + M + k ); }
    __device__ __forceinline__ void column( int u, int, int, int t, int &up, int &uq ) const
    {
        int const x = T[u * FixedLayout<M>::PITCH + t];
        up = x & 255;
        uq = x >> 8;
    }
    __device__ __forceinline__ int exp( int k ) const { return E[k * COLS]; }
    __device__ __forceinline__ void set_exp( int k, int d ) const { E[k * COLS] = (int8_t)d; }
    __device__ __forceinline__ double2 &rot( int r ) const { return reinterpret_cast<double2 *>( W )[r * us + ut]; }
    __device__ __forceinline__ uint8_t &pivot( int r ) const
    {
        return reinterpret_cast<uint8_t *>( W + 2 * FX_LOG * us )[r * us + ut];
    }
    __device__ __forceinline__ void log( int r, double c, double s, int ls ) const
    {
        rot( r ) = make_double2( c, s );
        pivot( r ) = (uint8_t)ls;
    }
    template <class Fn>
    __device__ __forceinline__ void for_parts( Fn const &fn ) const
    {
        if constexpr ( PARTS == 2 )
            fn( part );
        else
        {
            // (rolled: the loop bodies compete for the instruction cache)
#pragma unroll 1
            for ( int h = 0; h < 2; ++h )
                fn( h );
        }
    }
    __device__ __forceinline__ void merge( int &k1, int &k2, float &sum ) const
    {
        if constexpr ( PARTS == 1 )
            return;
        int const o1 = __shfl_xor_sync( FULL, k1, COLS ), o2 = __shfl_xor_sync( FULL, k2, COLS );
        sum += __shfl_xor_sync( FULL, sum, COLS );
        k2 = max( min( k1, o1 ), max( k2, o2 ) );
        k1 = max( k1, o1 );
    }
    __device__ __forceinline__ void sync() const
    {
        if constexpr ( PARTS == 2 )
            __syncwarp();
    }
    __device__ __forceinline__ bool any( bool x ) const { return __any_sync( FULL, x ); }
    __device__ __forceinline__ bool both( bool x ) const
    {
        if constexpr ( PARTS == 1 )
            return x;
        unsigned const m = __ballot_sync( FULL, x );
        return ( m & ( m >> 16 | m << 16 ) ) >> ( threadIdx.x & 31 ) & 1u;
    }
};

// Fills a block's table (all its threads; a barrier follows).
template <int M>
__device__ __forceinline__ void fill_columns( uint16_t *table )
{
    if constexpr ( M > 2 )
    {
        using Lay = FxLayout<M>;
        for ( int x = threadIdx.x; x < Lay::OFF * ( M - 2 ); x += blockDim.x )
        {
            int p, q, up, uq;
            Lay::of_slot( x / ( M - 2 ), p, q );
            Lay::column( p, q, x % ( M - 2 ), up, uq );
            table[x / ( M - 2 ) * FixedLayout<M>::PITCH + x % ( M - 2 )] = (uint16_t)( up | uq << 8 );
        }
    }
}

constexpr int FX_WORK = 2 * FX_LOG + FX_LOG / 8; // doubles of the log a matrix

// Row 0 of the pseudo-inverse from the moments in the state's entries (as
// doubles), left in w, for the matrices that take part (live); false when the
// FP64 kernel has to take the target.  All lanes of a warp together.
template <int M, int COLS>
__device__ __forceinline__ bool fixed_row0( FixedState<M, COLS> const &st, int cap, int log_cap, bool live,
                                            unsigned &iters )
{
    if constexpr ( M == 1 )
    {
        double const e = live ? st.a( 0 ) : 1.0;
        __syncwarp();
        st.w( 0 ) = 1.0 / e; // (both lanes write the same)
        __syncwarp();
        return live && e > 1e-13; // well above the truncation threshold
    }
    else
    {
        live = fx_load<M>( st, live );
        __syncwarp();
        int const rotations = fx_jacobi<M>( st, cap, live );
        __syncwarp();
        if ( rotations > 0 && st.part == 0 )
            iters += rotations;
        bool const form = log_cap < JACOBI_LOG && rotations > log_cap;
        if ( __any_sync( FULL, form ) )
        {
            // (a lowered log, for tests: U formed in the reference's order for
            // the matrices that outrun it, row by row in the places of F)
            if ( form && st.part == 0 )
            {
                for ( int j = 0; j < M; ++j )
                {
                    for ( int k = 0; k < M; ++k )
                        st.a( k ) = j == k ? 1.0 : 0.0;
                    for ( int n = 0; n < rotations; ++n )
                    {
                        double2 const cs = st.rot( n );
                        int const l = st.pivot( n ) >> 4, s = st.pivot( n ) & 15;
                        double const zl = st.a( l ), zs = st.a( s );
                        st.a( min( l, s ) ) = fma( cs.x, zl, cs.y * zs );
                        st.a( max( l, s ) ) = fma( cs.x, zs, -( cs.y * zl ) );
                    }
                    double v = 0.0;
                    for ( int k = 0; k < M; ++k )
                        v = fma( st.a( k ), st.w( k ), v );
                    st.a( M + j ) = v;
                }
                for ( int j = 0; j < M; ++j )
                    st.w( j ) = st.a( M + j );
            }
            __syncwarp();
        }
        // U w = the logged rotations applied in reverse: X = c z_L + s z_S went
        // to row min(L, S), Y = c z_S - s z_L to the other (two lanes a matrix:
        // one of the two results a lane)
        int n = form ? 0 : rotations;
        while ( __any_sync( FULL, n > 0 ) )
        {
            double2 cs[4];
            int ls[4];
#pragma unroll
            for ( int u = 0; u < 4; ++u )
                if ( n - 1 - u >= 0 )
                {
                    cs[u] = st.rot( n - 1 - u );
                    ls[u] = st.pivot( n - 1 - u );
                }
#pragma unroll
            for ( int u = 0; u < 4; ++u )
            {
                bool const on = n - 1 - u >= 0;
                int const l = ls[u] >> 4, s = ls[u] & 15;
                double X = 0.0, Y = 0.0;
                if ( on )
                {
                    X = st.w( min( l, s ) );
                    Y = st.w( max( l, s ) );
                }
                st.sync();
                // L: c X - s Y, S: s X + c Y
                if ( on && ( st.PARTS == 1 || st.part == 0 ) )
                    st.w( l ) = fma( cs[u].x, X, -( cs[u].y * Y ) );
                if ( on && ( st.PARTS == 1 || st.part == 1 ) )
                    st.w( s ) = fma( cs[u].y, X, cs[u].x * Y );
                st.sync();
            }
            n -= 4;
        }
        return rotations >= 0;
    }
}

// Warps a block: one block of 10 an SM with 32 matrices a warp (shared memory
// allows 227 KB), or single warps, up to 16 an SM, with 16.
template <int COLS>
constexpr int FIXED_WARPS = COLS == 32 ? 10 : 1;
template <int COLS>
constexpr int FIXED_BLOCKS_PER_SM = COLS == 32 ? 1 : 16;

// Sums of A over the lanes that differ in the bits of `mask` (a power of two
// and all below it), scattered: at each step a lane keeps one half of its
// sums and sends the other, so 35 sums over 32 lanes take 37 adds in place of
// 175.  On return the lane holds sums base .. base + count - 1 in A[0 ..].
template <int N>
__device__ __forceinline__ void scatter_sums( double *A, int mask, int lane, int &base, int &count )
{
    if ( mask == 0 )
        return; // uniform
    if constexpr ( N > 1 )
    {
        constexpr int H = ( N + 1 ) / 2;
        bool const upper = lane & mask;
#pragma unroll
        for ( int k = 0; k < H; ++k )
        {
            double const low = A[k], high = k + H < N ? A[k + H] : 0.0;
            double const other = __shfl_xor_sync( FULL, upper ? low : high, mask );
            A[k] = ( upper ? high : low ) + other;
        }
        base += upper ? H : 0;
        count = upper ? max( 0, count - H ) : min( count, H );
        scatter_sums<H>( A, mask >> 1, lane, base, count );
    }
    else
    {
        // one sum left: the lanes of the remaining bits share it
        for ( ; mask; mask >>= 1 )
        {
            A[0] += __shfl_xor_sync( FULL, A[0], mask );
            count = lane & mask ? 0 : count;
        }
    }
}

// The targets of one warp: up to COLS, list[first ..] (null: the targets first
// ..), with G lanes a target in the gather phases (1 to 32; with G = 1 a lane
// sums its target's row alone, in entry order, as the reference does: the two
// lanes of a shared matrix both).  The targets handed back come as a mask.
// With the same G every kernel runs the same arithmetic, bit for bit.
template <int M, int COLS>
__device__ __forceinline__ unsigned fixed_targets( Neighbours const &nb, PointsView const &tgt, int32_t const *offset,
                                                   uint32_t const *list, int64_t first, int cnt, int rbf, int G,
                                                   bool rows_sorted, double *coeff64, float *coeff32,
                                                   unsigned *status, FixedState<M, COLS> const &st, void *wsm, int cap,
                                                   int log_cap, unsigned &iters, int lane )
{
    double *const cols = (double *)wsm; // entry u of matrix c: cols[u * COLS + c]
    int const per = min( 32 / G, COLS ), sub = lane & ( G - 1 );
    Support mine_s{1.0, 1.0};
    for ( int r = 0; r * per < cnt; ++r ) // warp-uniform
    {
        int const ti = r * per + lane / G % per;
        bool const active = ti < cnt;
        int64_t const i = active ? ( list ? (int64_t)list[first + ti] : first + ti ) : 0;
        int64_t const b = active ? offset[i] : 0;
        int len = active ? offset[i + 1] - (int)b : 0;
        double const tx = active ? tgt( i, 0 ) : 0.0, ty = active ? tgt( i, 1 ) : 0.0, tz = active ? tgt( i, 2 ) : 0.0;
        bool bad = false;
        for ( int j = sub; j < len; j += G )
            bad |= (uint32_t)nb.ref( b + j ) >= (uint64_t)nb.src.n;
        for ( int o = G >> 1; o; o >>= 1 )
            bad |= __shfl_xor_sync( FULL, (int)bad, o ) != 0;
        if ( bad )
        {
            if ( sub == 0 )
                atomicOr( status, DEV_BAD_INDEX );
            len = 0;
        }
        // the farthest neighbour (the last of a row sorted by distance)
        double d2max = 0.0;
        for ( int j = rows_sorted ? max( 0, len - 1 ) : sub; j < len; j += G )
        {
            double sx, sy, sz;
            nb.xyz( b + j, sx, sy, sz );
            d2max = fmax( d2max, dist2_rn( sx, sy, sz, tx, ty, tz ) );
        }
        for ( int o = rows_sorted ? 0 : G >> 1; o; o >>= 1 )
            d2max = fmax( d2max, __shfl_xor_sync( FULL, d2max, o ) );
        Support const sup = support_of( d2max );
        if ( truncates_by_size<M>( d2max, len ) )
            len = 0; // (no moments: handed back)
        double A[N_MOMENTS<M>];
#pragma unroll
        for ( int u = 0; u < N_MOMENTS<M>; ++u )
            A[u] = 0.0;
        for ( int j = sub; j < len; j += G )
        {
            double sx, sy, sz;
            nb.xyz( b + j, sx, sy, sz );
            double const x = sx - tx, y = sy - ty, z = sz - tz;
            double const xx = __dmul_rn( x, x ), yy = __dmul_rn( y, y ), zz = __dmul_rn( z, z );
            double const w = weight_of( rbf, xx, yy, zz, sup );
            if ( coeff64 )
                coeff64[b + j] = w; // (the lanes of a shared matrix: the same value)
            add_moments<M>( x, y, z, xx, yy, zz, w, A );
        }
        int base = 0, count = N_MOMENTS<M>;
        scatter_sums<N_MOMENTS<M>>( A, G >> 1, lane, base, count );
        if ( active )
#pragma unroll
            for ( int k = 0; k < N_MOMENTS<M>; ++k )
                if ( k < count )
                    cols[( base + k ) * COLS + ti] = A[k];
        // the radius to the matrix's own lanes
        Support const from{__shfl_sync( FULL, sup.radius, ( lane % COLS % per ) * G ),
                           __shfl_sync( FULL, sup.inv, ( lane % COLS % per ) * G )};
        if ( lane % COLS / per == r )
            mine_s = from;
    }
    __syncwarp();
    bool const mine = lane % COLS < cnt;
    {
        // the distinct sums to the moment matrix, in place (two lanes a
        // matrix: each reads all of them and writes half of the entries)
        double A[N_MOMENTS<M>];
#pragma unroll
        for ( int u = 0; u < N_MOMENTS<M>; ++u )
            A[u] = st.a( u );
        __syncwarp();
        if constexpr ( M == 1 )
            st.a( 0 ) = A[0];
        else
        {
            using Lay = FxLayout<M>;
#pragma unroll
            for ( int p = 0; p < M; ++p )
#pragma unroll
                for ( int q = p; q < M; ++q )
                    if ( st.PARTS == 1 || ( ( p + q ) & 1 ) == st.part )
                        st.a( p == q ? Lay::diag( p ) : Lay::pair( p, q ) ) = A[moment_index( p, q )];
        }
    }
    __syncwarp();
    bool const ok = fixed_row0<M, COLS>( st, cap, log_cap, mine, iters );
    unsigned const rest = __ballot_sync( FULL, mine && !ok ) & ( FULL >> ( 32 - COLS ) );
    // computePolynomialCoefficients, G lanes a target (all the lanes of a
    // shared matrix)
    int const gc = max( G, 32 / COLS ), per_c = 32 / gc, sub_c = lane & ( gc - 1 );
    for ( int r = 0; r * per_c < cnt; ++r )
    {
        int const ti = r * per_c + lane / gc;
        Support const sup{__shfl_sync( FULL, mine_s.radius, ti & ( COLS - 1 ) ),
                          __shfl_sync( FULL, mine_s.inv, ti & ( COLS - 1 ) )};
        if ( ti >= cnt || ( ( rest >> ti ) & 1u ) )
            continue;
        int64_t const i = list ? (int64_t)list[first + ti] : first + ti;
        int64_t const b = offset[i];
        int const len = offset[i + 1] - (int)b;
        double const tx = tgt( i, 0 ), ty = tgt( i, 1 ), tz = tgt( i, 2 );
        double row0[M];
#pragma unroll
        for ( int p = 0; p < M; ++p )
            row0[p] = cols[( st.OFF + M + p ) * COLS + ti];
        for ( int j = sub_c; j < len; j += gc )
        {
            if ( (uint32_t)nb.ref( b + j ) >= (uint64_t)nb.src.n )
                continue; // reported above
            double sx, sy, sz;
            nb.xyz( b + j, sx, sy, sz );
            double const x = sx - tx, y = sy - ty, z = sz - tz;
            double const d = dot_basis<M>( row0, x, y, z );
            if ( coeff64 )
                coeff64[b + j] *= d;
            else
                coeff32[b + j] =
                    (float)( weight_of( rbf, __dmul_rn( x, x ), __dmul_rn( y, y ), __dmul_rn( z, z ), sup ) * d );
        }
    }
    __syncwarp();
    return rest;
}

__device__ __forceinline__ void add_rotations( unsigned iters, unsigned long long *count )
{
    unsigned long long it64 = iters;
    for ( int o = 16; o; o >>= 1 )
        it64 += __shfl_xor_sync( FULL, it64, o );
    if ( ( threadIdx.x & 31 ) == 0 && it64 )
        atomicAdd( count, it64 );
}

// The single operator's kernel: a warp takes COLS targets at a time, in the
// given order.
template <int M, int COLS>
__global__ void __launch_bounds__( 32 * FIXED_WARPS<COLS>, FIXED_BLOCKS_PER_SM<COLS> )
    k_setup_fixed( Neighbours nb, PointsView tgt, int32_t const *offset, uint32_t const *order, int64_t n_tgt,
                   int rbf, bool rows_sorted, double *coeff, unsigned long long *rot_count, unsigned *status,
                   int cap, int log_cap, double *work, uint32_t *list, unsigned *count )
{
    extern __shared__ double smem[];
    int const lane = threadIdx.x & 31, wib = threadIdx.x >> 5;
    int64_t const warp = blockIdx.x * (int64_t)FIXED_WARPS<COLS> + wib,
                  warps = gridDim.x * (int64_t)FIXED_WARPS<COLS>;
    uint16_t *const table = (uint16_t *)smem;
    fill_columns<M>( table );
    __syncthreads();
    void *const wsm = (char *)smem + FixedLayout<M>::TABLE + wib * FixedLayout<M>::BYTES * COLS;
    FixedState<M, COLS> const st( wsm, table, lane, work, warp, warps );
    unsigned iters = 0;
    for ( int64_t g = warp * COLS; g < n_tgt; g += warps * COLS )
    {
        int const cnt = (int)min( (int64_t)COLS, n_tgt - g );
        unsigned const rest = fixed_targets<M, COLS>( nb, tgt, offset, order, g, cnt, rbf, 1, rows_sorted, coeff,
                                                      nullptr, status, st, wsm, cap, log_cap, iters, lane );
        if ( ( rest >> lane ) & 1u )
            list[atomicAdd( count, 1u )] = order ? order[g + lane] : (uint32_t)( g + lane );
    }
    add_rotations( iters, rot_count );
}

// One task of a batch: up to 32 targets of one bucket.
template <int M>
__device__ void fixed_task( BatchSetupArgs const &a, SetupTask const &t, int rbf, int G, void *wsm,
                            uint16_t const *table, int64_t warp, int64_t warps, int cap, unsigned &iters, int lane )
{
    FixedState<M, 32> const st( wsm, table, lane, a.u_work, warp, warps );
    unsigned rest = FULL >> ( 32 - t.count );
    if ( fixed_supported( rbf ) )
        rest = fixed_targets<M, 32>( a.nb, a.tgt, a.offset, a.list, t.first, t.count, rbf, G, a.rows_sorted,
                                     a.coeff64, a.coeff32, a.status, st, wsm, cap, a.jlog, iters, lane );
    // the targets handed back, as a task of their own with the same lanes
    if ( rest )
    {
        unsigned at = 0;
        if ( lane == 0 )
        {
            at = atomicAdd( &a.counters->rest, (unsigned)__popc( rest ) );
            int64_t const ta = (int64_t)atomicAdd( (unsigned long long *)&a.counters->rest_tasks, 1ull );
            SetupTask x = t;
            x.first = (int32_t)at;
            x.count = (uint8_t)__popc( rest );
            x.lanes = (uint8_t)G;
            a.rest_task[ta] = x;
        }
        at = __shfl_sync( FULL, at, 0 );
        if ( ( rest >> lane ) & 1u )
            a.rest_list[at + __popc( rest & ( ( 1u << lane ) - 1u ) )] = a.list[t.first + lane];
    }
}

// Persistent over the tasks (the warps take theirs from one counter).
__global__ void __launch_bounds__( 32 * FIXED_WARPS<32>, FIXED_BLOCKS_PER_SM<32> ) k_batch_fixed( BatchSetupArgs a )
{
    extern __shared__ double smem[];
    int const lane = threadIdx.x & 31, wib = threadIdx.x >> 5;
    int64_t const warp = blockIdx.x * (int64_t)FIXED_WARPS<32> + wib, warps = gridDim.x * (int64_t)FIXED_WARPS<32>;
    uint16_t *const table10 = (uint16_t *)smem, *const table4 = table10 + FixedLayout<10>::TABLE / sizeof( uint16_t );
    fill_columns<10>( table10 );
    fill_columns<4>( table4 );
    __syncthreads();
    void *const wsm =
        (char *)smem + FixedLayout<10>::TABLE + FixedLayout<4>::TABLE + wib * FixedLayout<10>::BYTES * 32;
    int64_t const t_end = a.t_end >= 0 ? a.t_end : *a.n_tasks;
    unsigned iters = 0;
    for ( ;; )
    {
        unsigned c = 0;
        if ( lane == 0 )
            c = atomicAdd( &a.counters->task[0], 1u );
        int64_t const ti = a.t_begin + __shfl_sync( FULL, c, 0 );
        if ( ti >= t_end )
            break;
        SetupTask const t = a.tasks[ti];
        int const key = t.key;
        int const basis = key / SETUP_PATHS / SETUP_RBFS, rbf = key / SETUP_PATHS % SETUP_RBFS;
        int const G = a.force_lanes ? a.force_lanes : t.lanes;
        // a task out of range is reported and skipped, never followed
        if ( key >= SETUP_KEYS || t.count < 1 || t.count > 32 || G < 1 || G > 32 || ( G & ( G - 1 ) ) ||
             t.first < 0 || (int64_t)t.first + t.count > a.n_list )
        {
            if ( lane == 0 )
                atomicOr( a.status, DEV_BAD_TASK );
            continue;
        }
        int const cap = (int)min( a.jcap[basis], (unsigned)FX_LOG );
        if ( basis == DTK_CONSTANT3 )
            fixed_task<1>( a, t, rbf, G, wsm, nullptr, warp, warps, cap, iters, lane );
        else if ( basis == DTK_LINEAR3 )
            fixed_task<4>( a, t, rbf, G, wsm, table4, warp, warps, cap, iters, lane );
        else
            fixed_task<10>( a, t, rbf, G, wsm, table10, warp, warps, cap, iters, lane );
    }
    add_rotations( iters, a.rotations );
}

// Two lanes a matrix while that runs all of them at once (a chain of about 150
// rotations: 0.59 ms against 0.78 for 10k quadratic targets), one beyond.
bool shared_matrices( int64_t n )
{
    return n <= 16 * FIXED_BLOCKS_PER_SM<16> * (int64_t)num_sms();
}

template <int COLS>
unsigned fixed_blocks( int64_t n )
{
    int64_t const per = COLS * FIXED_WARPS<COLS>;
    return (unsigned)std::max<int64_t>(
        1, std::min<int64_t>( ( n + per - 1 ) / per, FIXED_BLOCKS_PER_SM<COLS> * (int64_t)num_sms() ) );
}

template <int M, int COLS>
void launch_fixed( SetupArgs const &a, double *work, uint32_t *list, unsigned *count, cudaStream_t s )
{
    size_t const smem = FixedLayout<M>::TABLE + FixedLayout<M>::BYTES * COLS * FIXED_WARPS<COLS>;
    ensure_dynamic_smem( k_setup_fixed<M, COLS>, smem );
    Neighbours const nb{a.src, a.idx, a.pos, a.s2};
    int const cap = (int)std::min<unsigned long long>( jacobi_cap( M ), FX_LOG );
    k_setup_fixed<M, COLS><<<fixed_blocks<COLS>( a.n_tgt ), 32 * FIXED_WARPS<COLS>, smem, s>>>(
        nb, a.tgt, a.offset, a.order, a.n_tgt, a.rbf, a.rows_sorted, a.coeff64, a.rotations, a.status, cap,
        jacobi_log_cap(), work, list, count );
    check_launch( "k_setup_fixed" );
}

template <int M>
void launch_fixed( SetupArgs const &a, double *work, uint32_t *list, unsigned *count, cudaStream_t s )
{
    if ( shared_matrices( a.n_tgt ) )
        launch_fixed<M, 16>( a, work, list, count, s );
    else
        launch_fixed<M, 32>( a, work, list, count, s );
}

} // namespace

size_t fixed_work_doubles( int64_t n_tgt )
{
    return FX_WORK * ( shared_matrices( n_tgt ) ? 16 * (size_t)fixed_blocks<16>( n_tgt )
                                                : 32 * FIXED_WARPS<32> * (size_t)fixed_blocks<32>( n_tgt ) );
}

size_t batch_fixed_warps()
{
    return FIXED_WARPS<32> * FIXED_BLOCKS_PER_SM<32> * (size_t)num_sms();
}

size_t batch_fixed_work_doubles()
{
    return FX_WORK * 32 * batch_fixed_warps();
}

void setup_fixed( SetupArgs const &a, double *work, uint32_t *list, unsigned *count, cudaStream_t s )
{
    switch ( a.basis )
    {
    case DTK_CONSTANT3:
        launch_fixed<1>( a, work, list, count, s );
        break;
    case DTK_LINEAR3:
        launch_fixed<4>( a, work, list, count, s );
        break;
    default:
        launch_fixed<10>( a, work, list, count, s );
        break;
    }
}

void batch_fixed( BatchSetupArgs const &a, cudaStream_t s )
{
    size_t const smem =
        FixedLayout<10>::TABLE + FixedLayout<4>::TABLE + FixedLayout<10>::BYTES * 32 * FIXED_WARPS<32>;
    ensure_dynamic_smem( k_batch_fixed, smem );
    k_batch_fixed<<<(unsigned)( FIXED_BLOCKS_PER_SM<32> * num_sms() ), 32 * FIXED_WARPS<32>, smem, s>>>( a );
    check_launch( "k_batch_fixed" );
}

} // namespace dtk
