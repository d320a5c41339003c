// MLS apply: CSR gather-SpMV (sm_103a).
//
// Replaces MovingLeastSquaresOperator::apply
// (packages/Meshfree/src/DTK_MovingLeastSquaresOperator_def.hpp:121-141):
// the single-rank fetch (a gather of source values into per-neighbour
// order, DTK_DetailsNearestNeighborOperatorImpl.hpp:152-192), computeTargetValues
// (DTK_DetailsMovingLeastSquaresOperatorImpl.hpp:49-70) and the deep_copy fuse
// into one kernel that reads idx/coeff once and writes each target once.
//
// Rows of equal length R with R % 4 == 0 and R/4 a power of two (kNN rows,
// e.g. R = 32) use R/8 lanes per row (8 entries each) with 128-bit loads:
// int4 of indices and two double2 (FP64 form) or one float4 (mixed form) of
// coefficients per 4 entries, then a shuffle reduction; a group of lanes may
// take several rows.  Other rows use S lanes per row (S a power of two chosen
// from the mean row length) with coalesced scalar loads.  Source values are
// gathered through the read-only path; at 8M sources they are 64 MB and stay
// resident in the 129 MB L2 while the CSR streams from HBM.
#include "dtk_common.cuh"

#include <algorithm>
#include <type_traits>

namespace dtk
{
namespace
{

constexpr unsigned FULL = 0xffffffffu;

template <int L>
__device__ __forceinline__ double group_sum( double v )
{
#pragma unroll
    for ( int o = L / 2; o > 0; o >>= 1 )
        v += __shfl_xor_sync( FULL, v, o );
    return v;
}

// S lanes per row, strided scalar loads.
template <int S, bool F32>
__global__ void __launch_bounds__( 256 )
    k_apply_csr( int64_t n_tgt, int32_t const *__restrict__ offset,
                 int32_t const *__restrict__ idx, void const *__restrict__ coeff,
                 double const *__restrict__ values, double *__restrict__ target )
{
    int64_t const gt = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    int64_t const row = gt / S;
    int const sub = (int)( gt % S );
    double acc = 0.0;
    if ( row < n_tgt )
    {
        int const b = offset[row], e = offset[row + 1];
        for ( int j = b + sub; j < e; j += S )
        {
            double const c = F32 ? (double)static_cast<float const *>( coeff )[j]
                                 : static_cast<double const *>( coeff )[j];
            acc += c * __ldg( values + idx[j] );
        }
    }
    acc = group_sum<S>( acc );
    if ( row < n_tgt && sub == 0 )
        target[row] = acc;
}

template <bool F32>
void launch_csr( int S, int64_t n_tgt, int32_t const *offset, int32_t const *idx,
                 void const *coeff, double const *values, double *target, cudaStream_t s )
{
    int64_t const threads = n_tgt * S;
    unsigned const blocks = (unsigned)( ( threads + 255 ) / 256 );
    switch ( S )
    {
    case 1: k_apply_csr<1, F32><<<blocks, 256, 0, s>>>( n_tgt, offset, idx, coeff, values, target ); break;
    case 2: k_apply_csr<2, F32><<<blocks, 256, 0, s>>>( n_tgt, offset, idx, coeff, values, target ); break;
    case 4: k_apply_csr<4, F32><<<blocks, 256, 0, s>>>( n_tgt, offset, idx, coeff, values, target ); break;
    case 8: k_apply_csr<8, F32><<<blocks, 256, 0, s>>>( n_tgt, offset, idx, coeff, values, target ); break;
    case 16: k_apply_csr<16, F32><<<blocks, 256, 0, s>>>( n_tgt, offset, idx, coeff, values, target ); break;
    default: k_apply_csr<32, F32><<<blocks, 256, 0, s>>>( n_tgt, offset, idx, coeff, values, target ); break;
    }
    check_launch( "k_apply_csr" );
}

bool is_pow2( int v ) { return v > 0 && ( v & ( v - 1 ) ) == 0; }

} // namespace

// ---------------------------------------------------------------------------
// Apply over uniform rows.
//
// Mixed form, one component: the source values are first permuted into the
// tree's Morton order (one pass over the sources) as double-floats (hi =
// fl32(v), lo = fl32(v - hi)), and the rows gather them by sorted position, so a
// row's neighbours sit in a few sectors of an L2-resident array instead of 32
// scattered ones; c_j (hi_j + lo_j) is summed in double-float arithmetic on the
// FP32 pipe (TwoProd / TwoSum, the compensated scheme of the mixed setup): the
// FP32 coefficients are the only rounding left, as with an FP64 sum.  A row whose
// sum says that FP32's range was not enough (not finite, or below 2^-60, where a
// term's low part nears the subnormals) is summed again in FP64 from the field.
//
// FP64 sums, for the FP64 form and for fields of several components in both (a
// double-float has FP32's range and 48 bits): FP64 FMAs, whose pipe bounds them
// with the bytes (64 cycles an instruction a warp), by index from the field as
// it is, up to four components a thread, so that indices and coefficients are
// read once; FP32 coefficients are widened on the integer pipe.  Large fields of
// several components go through a sorted copy, a point's components side by
// side.  FP64 form, 2M rows of 32: 257 us by sorted position with a reduction
// a row of 4 entries a lane, 169 us so (118 us are the bytes); three components
// of 1M rows, mixed: 480 us with 8 lanes a row and scalar loads, 187 us so (269
// with the conversions on the FP64 pipe).
//
// Rows go in the targets' Morton order when the operator has it, so that
// consecutive rows share most of their neighbours' values in L1 (0.70 -> 0.59 ms
// for 8M rows of 32; 16 entries a lane instead of 8 was 1.26 ms, 4 no different).
// ---------------------------------------------------------------------------
namespace
{

// the biased exponent (integer pipe)
__device__ __forceinline__ int exponent_of( double v )
{
    return ( __double2hiint( v ) >> 20 ) & 0x7ff;
}

__device__ __forceinline__ void two_sum( float a, float b, float &s, float &e )
{
    s = __fadd_rn( a, b );
    float const bb = __fsub_rn( s, a );
    e = __fadd_rn( __fsub_rn( a, __fsub_rn( s, bb ) ), __fsub_rn( b, bb ) );
}

__device__ __forceinline__ void two_prod( float a, float b, float &p, float &e )
{
    p = __fmul_rn( a, b );
    e = __fmaf_rn( a, b, -p );
}

// sorted[p] = values[perm[p]] (perm null: the identity) as a double (FP64
// form) or a double-float; NaN for a value that FP32 products could lose (its
// rows are summed in FP64)
__global__ void k_permute_values( int64_t n, uint32_t const *__restrict__ perm, double const *__restrict__ values,
                                  double *__restrict__ sorted64, float2 *__restrict__ sorted32 )
{
    int64_t const p = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if ( p >= n )
        return;
    double const v = __ldg( values + ( perm ? (int64_t)__ldg( perm + p ) : p ) );
    if ( sorted32 )
    {
        float hi = __double2float_rn( v );
        float const lo = __double2float_rn( v - (double)hi );
        // 0 < |v| < 2^-100
        if ( exponent_of( v ) < 1023 - 100 && ( __double_as_longlong( v ) << 1 ) != 0 )
            hi = __int_as_float( 0x7fffffff );
        sorted32[p] = make_float2( hi, lo );
    }
    else
        sorted64[p] = v;
}

// c * (v.x + v.y) added to the double-float (s, c_acc)
__device__ __forceinline__ void df_axpy( float c, float2 v, float &s, float &cs )
{
    float p, e, t, f;
    two_prod( c, v.x, p, e );
    e = __fmaf_rn( c, v.y, e );
    two_sum( s, p, t, f );
    s = t;
    cs = __fadd_rn( cs, __fadd_rn( f, e ) );
}

// The double-floats (s, cs) of a group of L lanes added up, in every lane.
template <int L>
__device__ __forceinline__ void df_group_sum( float &s, float &cs )
{
#pragma unroll
    for ( int o = L / 2; o > 0; o >>= 1 )
    {
        float const os = __shfl_xor_sync( FULL, s, o ), oc = __shfl_xor_sync( FULL, cs, o );
        float t, f;
        two_sum( s, os, t, f );
        s = t;
        cs = __fadd_rn( cs, __fadd_rn( oc, f ) );
    }
}

// Exactly (double)c on the integer pipe: a conversion takes the FP64 pipe 64
// cycles a warp, as an FMA does, and where a condition turns it off as well.
__device__ __forceinline__ double widen( float c )
{
    unsigned const e = __float_as_uint( c ) & 0x7f800000u;
    // the exponent's bias 127 -> 1023; a subnormal is made normal first, 2^24
    // times as large, and an infinity or NaN goes to the largest exponent
    unsigned bias = 896u << 20;
    if ( e == 0u || e == 0x7f800000u )
    {
        bias = c == 0.f ? 0u : e ? 1792u << 20 : 872u << 20;
        c = e ? c : __fmul_rn( c, 16777216.f );
    }
    unsigned const b = __float_as_uint( c );
    return __hiloint2double( (int)( ( b & 0x80000000u ) | ( ( ( b & 0x7fffffffu ) >> 3 ) + bias ) ), (int)( b << 29 ) );
}

// Four consecutive coefficients as doubles.
__device__ __forceinline__ void load_coeff4( double const *p, double *c )
{
    double2 const c0 = __ldcs( reinterpret_cast<double2 const *>( p ) );
    double2 const c1 = __ldcs( reinterpret_cast<double2 const *>( p + 2 ) );
    c[0] = c0.x;
    c[1] = c0.y;
    c[2] = c1.x;
    c[3] = c1.y;
}
__device__ __forceinline__ void load_coeff4( float const *p, double *c )
{
    float4 const v = __ldcs( reinterpret_cast<float4 const *>( p ) );
    c[0] = widen( v.x );
    c[1] = widen( v.y );
    c[2] = widen( v.z );
    c[3] = widen( v.w );
}

// A row's sum in FP64 from the field (apart, so that the callers' loads stay
// together).
__device__ __noinline__ double row_sum64( int n, int32_t const *pos, float const *coeff, double const *values,
                                          uint32_t const *perm )
{
    double sum = 0.0;
    for ( int j = 0; j < n; ++j )
        sum = fma( (double)coeff[j], values[perm ? (int64_t)perm[pos[j]] : pos[j]], sum );
    return sum;
}

// Mixed form, one component: L lanes per row, each lane EPL consecutive entries
// (EPL a multiple of 4).  values, perm: the field and its order, for the rows
// that FP32's range does not hold.
template <int L, int EPL>
__global__ void __launch_bounds__( 256 )
    k_apply_pos( int64_t n_tgt, int32_t const *__restrict__ pos, float const *__restrict__ coeff,
                 float2 const *__restrict__ sorted, double const *__restrict__ values,
                 uint32_t const *__restrict__ perm, double *__restrict__ target, uint32_t const *__restrict__ order )
{
    constexpr int R = EPL * L;
    int64_t const gt = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    int64_t const row0 = gt / L;
    int64_t const row = ( order && row0 < n_tgt ) ? (int64_t)__ldg( order + row0 ) : row0;
    int const sub = (int)( gt % L );
    float s = 0.f, cs = 0.f;
    if ( row < n_tgt )
    {
#pragma unroll
        for ( int q = 0; q < EPL; q += 4 )
        {
            int64_t const e = row * R + EPL * sub + q;
            int4 const ix = __ldcs( reinterpret_cast<int4 const *>( pos + e ) );
            float4 const c = __ldcs( reinterpret_cast<float4 const *>( coeff + e ) );
            df_axpy( c.x, __ldg( sorted + ix.x ), s, cs );
            df_axpy( c.y, __ldg( sorted + ix.y ), s, cs );
            df_axpy( c.z, __ldg( sorted + ix.z ), s, cs );
            df_axpy( c.w, __ldg( sorted + ix.w ), s, cs );
        }
    }
    df_group_sum<L>( s, cs );
    if ( row < n_tgt && sub == 0 )
    {
        float const size = fabsf( s );
        bool const held = ( size >= 8.6736174e-19f && size <= 3.4028235e38f ) || ( s == 0.f && cs == 0.f ); // 2^-60
        target[row] = held ? (double)s + (double)cs : row_sum64( R, pos + row * R, coeff + row * R, values, perm );
    }
}

// FP64 sums of CB components from c0 on: L lanes take ROWS rows, each lane EPL
// consecutive entries of every row (EPL a multiple of 4).  mine: the row that
// this lane ends with, -1 for none.  PACKED: the field has CB components side by
// side.
template <int L, int EPL, int ROWS, int CB, bool PACKED, class Coeff>
__device__ __forceinline__ void rows64( int32_t const *__restrict__ at, Coeff const *__restrict__ coeff,
                                        FieldView const &in, FieldView const &out, int64_t c0, int64_t mine )
{
    constexpr int R = EPL * L, SHARE = L / ROWS; // lanes that end with the same row
    int const sub = threadIdx.x % L;
    double a[ROWS][CB];
#pragma unroll
    for ( int r = 0; r < ROWS; ++r )
    {
#pragma unroll
        for ( int k = 0; k < CB; ++k )
            a[r][k] = 0.0;
        int64_t const row = L > 1 ? __shfl_sync( FULL, mine, r * SHARE, L ) : mine;
        if ( row < 0 )
            continue;
#pragma unroll
        for ( int q = 0; q < EPL; q += 4 )
        {
            int64_t const e = row * R + EPL * sub + q;
            int4 const ix = __ldcs( reinterpret_cast<int4 const *>( at + e ) );
            int const p[4] = {ix.x, ix.y, ix.z, ix.w};
            double cj[4];
            load_coeff4( coeff + e, cj );
#pragma unroll
            for ( int j = 0; j < 4; ++j )
            {
                double const *v = PACKED ? in.base + (int64_t)CB * p[j] : in.base + p[j] * in.ps + c0 * in.cs;
#pragma unroll
                for ( int k = 0; k < CB; ++k )
                    a[r][k] = fma( cj[j], __ldg( v + ( PACKED ? k : k * in.cs ) ), a[r][k] );
            }
        }
    }
    // halve the rows a lane holds until one is left, then add up its lanes
#pragma unroll
    for ( int n = ROWS / 2, o = L / 2; n > 0; n >>= 1, o >>= 1 )
    {
        bool const upper = ( sub & o ) != 0;
#pragma unroll
        for ( int r = 0; r < n; ++r )
#pragma unroll
            for ( int k = 0; k < CB; ++k )
            {
                double const give = upper ? a[r][k] : a[r + n][k];
                double const keep = upper ? a[r + n][k] : a[r][k];
                a[r][k] = keep + __shfl_xor_sync( FULL, give, o );
            }
    }
#pragma unroll
    for ( int o = SHARE / 2; o > 0; o >>= 1 )
#pragma unroll
        for ( int k = 0; k < CB; ++k )
            a[0][k] += __shfl_xor_sync( FULL, a[0][k], o );
    if ( mine >= 0 && sub % SHARE == 0 )
#pragma unroll
        for ( int k = 0; k < CB; ++k )
            out.wbase[mine * out.ps + ( c0 + k ) * out.cs] = a[0][k];
}

// FP64 sums (the FP64 form, and every field of several components: a mixed
// operator's coefficients are widened, exactly) of n_full groups of CB
// components and others of CB - 1 behind them, in one launch (a component that
// is only masked out takes the FP64 pipe as long as a real one).  `at` indexes
// the values: a sorted copy of the field or the field itself.  A row's partial
// sums meet in the same order whatever ROWS is and wherever the values lie, so
// every path gives the same bits.
template <int L, int EPL, int ROWS, int CB, bool PACKED, class Coeff>
__global__ void __launch_bounds__( 256 )
    k_apply_rows64( int64_t n_rows, int32_t const *__restrict__ at, Coeff const *__restrict__ coeff, FieldView in,
                    FieldView out, int64_t n_full, uint32_t const *__restrict__ order )
{
    static_assert( ROWS <= L && L % ROWS == 0, "a lane ends with one row at most" );
    int64_t const gt = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    int64_t const first = gt / L * ROWS + threadIdx.x % L / ( L / ROWS ); // this lane's row in order
    int64_t const mine = first < n_rows ? ( order ? (int64_t)__ldg( order + first ) : first ) : -1;
    if constexpr ( PACKED )
    {
        rows64<L, EPL, ROWS, CB, true>( at, coeff, in, out, 0, mine );
        return;
    }
    for ( int64_t g = blockIdx.y;; g += gridDim.y )
    {
        int64_t const c0 = g < n_full ? g * CB : g * CB - ( g - n_full );
        if ( c0 >= in.n_comp )
            break;
        if ( g < n_full )
            rows64<L, EPL, ROWS, CB, false>( at, coeff, in, out, c0, mine );
        else if constexpr ( CB > 1 )
            rows64<L, EPL, ROWS, CB - 1, false>( at, coeff, in, out, c0, mine );
    }
}

// sorted[nc p + k] = component c0 + k < c0 + nc of source perm[p]
__global__ void k_permute_fields( FieldView in, int64_t c0, int nc, uint32_t const *__restrict__ perm,
                                  double *__restrict__ sorted )
{
    int64_t const p = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if ( p >= in.n )
        return;
    double const *v = in.base + (int64_t)__ldg( perm + p ) * in.ps + c0 * in.cs;
#pragma unroll
    for ( int k = 0; k < 4; ++k )
        if ( k < nc )
            sorted[nc * p + k] = __ldg( v + k * in.cs );
}

// fn( lanes a row, entries a lane ) of row length R (a lane of 8 entries reads a
// sector in two loads, which has to stay in L1 between them: rows of 8 by two
// lanes)
template <class Fn>
void for_row_shape( int R, Fn const &fn )
{
    std::integral_constant<int, 8> const eight;
    switch ( R )
    {
    case 4: fn( std::integral_constant<int, 1>{}, std::integral_constant<int, 4>{} ); break;
    case 8: fn( std::integral_constant<int, 2>{}, std::integral_constant<int, 4>{} ); break;
    case 16: fn( std::integral_constant<int, 2>{}, eight ); break;
    case 32: fn( std::integral_constant<int, 4>{}, eight ); break;
    case 64: fn( std::integral_constant<int, 8>{}, eight ); break;
    default: fn( std::integral_constant<int, 16>{}, eight ); break;
    }
}

// FP64 sums of every component in one launch, up to four components a thread.
// A group of lanes takes one row where the adds over its lanes are cheap beside
// the latency (up to two components, or few rows), otherwise up to four rows
// (us, one row / four: 2M rows of 32, FP64 form, 1 component 169 / 239, 2
// components 301 / 325, on a sorted copy 314 / 281; 3 components 423 / 406, mixed
// 421 / 368; 10k rows, 3 components 10.9 / 12.4).
template <int CB, class Coeff>
void launch_rows64( int64_t n_rows, int R, int32_t const *at, Coeff const *coeff, FieldView const &in,
                    FieldView const &out, int64_t groups, bool sorted, cudaStream_t s, uint32_t const *order )
{
    int64_t const n_full = in.n_comp - groups * ( CB - 1 );
    bool const packed = in.n_comp == CB && in.ps == CB && ( CB == 1 || in.cs == 1 );
    bool const several = n_rows >= 100000 && ( CB >= 3 || ( CB == 2 && sorted ) );
    for_row_shape( R, [&]( auto l, auto epl ) {
        constexpr int L = decltype( l )::value, EPL = decltype( epl )::value;
        constexpr int MOST = CB == 1 || L == 1 ? 1 : L < 4 ? L : 4;
        auto const run = [&]( auto rows, auto is_packed ) {
            constexpr int ROWS = decltype( rows )::value;
            dim3 const grid( (unsigned)( ( ( n_rows + ROWS - 1 ) / ROWS * L + 255 ) / 256 ),
                             (unsigned)std::min<int64_t>( groups, 65535 ) );
            k_apply_rows64<L, EPL, ROWS, CB, decltype( is_packed )::value>
                <<<grid, 256, 0, s>>>( n_rows, at, coeff, in, out, n_full, order );
            check_launch( "k_apply_rows64" );
        };
        auto const run_rows = [&]( auto rows ) {
            if ( packed )
                run( rows, std::true_type{} );
            else
                run( rows, std::false_type{} );
        };
        if ( several )
            run_rows( std::integral_constant<int, MOST>{} );
        else
            run_rows( std::integral_constant<int, 1>{} );
    } );
}

void apply_rows64( int64_t n_rows, int R, int32_t const *at, double const *coeff64, float const *coeff32,
                   FieldView const &in, FieldView const &out, bool sorted, cudaStream_t s, uint32_t const *order )
{
    int64_t const groups = ( in.n_comp + 3 ) / 4, cb = ( in.n_comp + groups - 1 ) / groups;
    auto const run = [&]( auto c ) {
        constexpr int CB = decltype( c )::value;
        if ( coeff32 )
            launch_rows64<CB>( n_rows, R, at, coeff32, in, out, groups, sorted, s, order );
        else
            launch_rows64<CB>( n_rows, R, at, coeff64, in, out, groups, sorted, s, order );
    };
    switch ( cb )
    {
    case 1: run( std::integral_constant<int, 1>{} ); break;
    case 2: run( std::integral_constant<int, 2>{} ); break;
    case 3: run( std::integral_constant<int, 3>{} ); break;
    default: run( std::integral_constant<int, 4>{} ); break;
    }
}

FieldView rank1( double const *values, double *target, int64_t n )
{
    return FieldView{values, target, n, 1, 1, 0};
}

} // namespace

bool apply_sorted_supported( int uniform_row )
{
    return uniform_row > 0 && uniform_row % 4 == 0 && is_pow2( uniform_row / 4 ) && uniform_row / 4 <= 32;
}

SortedValues permute_values( int64_t n_src, uint32_t const *perm, double const *values, bool f32,
                             cudaStream_t s )
{
    SortedValues v;
    if ( f32 )
        v.v32.allocate( std::max<int64_t>( 1, n_src ), s );
    else
        v.v64.allocate( std::max<int64_t>( 1, n_src ), s );
    if ( n_src > 0 )
    {
        k_permute_values<<<(unsigned)( ( n_src + 255 ) / 256 ), 256, 0, s>>>( n_src, perm, values, v.v64.get(),
                                                                            v.v32.get() );
        check_launch( "k_permute_values" );
    }
    return v;
}

void apply_pos( int64_t n_rows, int uniform_row, int32_t const *pos, double const *coeff64, float const *coeff32,
                SortedValues const &v, double const *values, uint32_t const *perm, double *target, cudaStream_t s, uint32_t const *order )
{
    if ( n_rows == 0 )
        return;
    if ( !coeff32 )
    {
        apply_rows64( n_rows, uniform_row, pos, coeff64, nullptr, rank1( v.v64.get(), nullptr, 0 ),
                      rank1( nullptr, target, n_rows ), true, s, order );
        return;
    }
    for_row_shape( uniform_row, [&]( auto l, auto epl ) {
        constexpr int L = decltype( l )::value, EPL = decltype( epl )::value;
        k_apply_pos<L, EPL><<<(unsigned)( ( n_rows * L + 255 ) / 256 ), 256, 0, s>>>( n_rows, pos, coeff32,
                                                                                      v.v32.get(), values, perm,
                                                                                      target, order );
        check_launch( "k_apply_pos" );
    } );
}

void apply_sorted( int64_t n_tgt, int uniform_row, int32_t const *idx, int32_t const *pos, double const *coeff64,
                   float const *coeff32, int64_t n_src, uint32_t const *perm, double const *values,
                   double *target, cudaStream_t s, uint32_t const *order )
{
    if ( n_tgt == 0 )
        return;
    if ( coeff64 )
    {
        apply_rows64( n_tgt, uniform_row, idx, coeff64, nullptr, rank1( values, nullptr, n_src ),
                      rank1( nullptr, target, n_tgt ), false, s, order );
        return;
    }
    uint32_t const *const by = pos ? perm : nullptr;
    SortedValues const v = permute_values( n_src, by, values, true, s );
    apply_pos( n_tgt, uniform_row, pos ? pos : idx, nullptr, coeff32, v, values, by, target, s, order );
}

void apply_sorted_multi( int64_t n_tgt, int uniform_row, int32_t const *idx, int32_t const *pos,
                         double const *coeff64, float const *coeff32, uint32_t const *perm, FieldView in,
                         FieldView out, cudaStream_t s, uint32_t const *order )
{
    if ( n_tgt == 0 )
        return;
    // A sorted copy pays from about 2M sources on, when the fields outgrow the
    // caches of L2's nearer half, with at least 16 entries a source (us, by
    // index / on a copy, as many targets: 2M, rows of 16, 3 components 274 / 261;
    // 4M, rows of 16, 2 components 539 / 466, 3 components 734 / 580, rows of 32
    // 882 / 789; but 1M, rows of 32, 3 components 202 / 206; 4M to 1M, rows of 32
    // 261 / 273; 4M to 30k 15 / 81)
    if ( !( pos && in.n_comp > 1 && in.n >= 2000000 && n_tgt * uniform_row >= 16 * in.n ) )
    {
        apply_rows64( n_tgt, uniform_row, idx, coeff64, coeff32, in, out, false, s, order );
        return;
    }
    int64_t const groups = ( in.n_comp + 3 ) / 4, cb = ( in.n_comp + groups - 1 ) / groups;
    DeviceBuffer<double> v( cb * in.n, s );
    for ( int64_t c0 = 0; c0 < in.n_comp; c0 += cb )
    {
        int64_t const nc = std::min( cb, in.n_comp - c0 );
        k_permute_fields<<<(unsigned)( ( in.n + 255 ) / 256 ), 256, 0, s>>>( in, c0, (int)nc, perm, v.get() );
        check_launch( "k_permute_fields" );
        apply_rows64( n_tgt, uniform_row, pos, coeff64, coeff32, FieldView{v.get(), nullptr, in.n, nc, nc, 1},
                      FieldView{nullptr, out.wbase + c0 * out.cs, n_tgt, nc, out.ps, out.cs}, true, s, order );
    }
}

// uniform_row > 0: every row has that length (offset[i] = i * uniform_row);
// otherwise mean_row picks the lanes per row.
namespace
{

// Rank-2 fields: 8 lanes per row, 4 components per pass; the row's indices
// and coefficients are read once per pass for 4 components.
template <bool F32>
__global__ void __launch_bounds__( 256 )
    k_apply_multi( int64_t n_tgt, int32_t const *__restrict__ offset, int32_t const *__restrict__ idx,
                   void const *__restrict__ coeff, FieldView in, FieldView out )
{
    constexpr int S = 8, CB = 4;
    int64_t const gt = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    int64_t const row = gt / S;
    int const sub = (int)( gt % S );
    bool const live = row < n_tgt;
    int const b = live ? offset[row] : 0, e = live ? offset[row + 1] : 0;
    for ( int c0 = 0; c0 < in.n_comp; c0 += CB ) // uniform across the warp
    {
        double acc[CB] = {0.0, 0.0, 0.0, 0.0};
        for ( int j = b + sub; j < e; j += S )
        {
            double const cj = F32 ? (double)__ldg( static_cast<float const *>( coeff ) + j )
                                  : __ldg( static_cast<double const *>( coeff ) + j );
            int64_t const sj = __ldg( idx + j );
#pragma unroll
            for ( int q = 0; q < CB; ++q )
                if ( c0 + q < in.n_comp )
                    acc[q] = fma( cj, __ldg( in.base + sj * in.ps + ( c0 + q ) * in.cs ), acc[q] );
        }
#pragma unroll
        for ( int q = 0; q < CB; ++q )
            acc[q] = group_sum<S>( acc[q] );
        if ( live && sub == 0 )
#pragma unroll
            for ( int q = 0; q < CB; ++q )
                if ( c0 + q < in.n_comp )
                    out.wbase[row * out.ps + ( c0 + q ) * out.cs] = acc[q];
    }
}

} // namespace

void apply_csr_multi( int64_t n_tgt, int32_t const *offset, int32_t const *idx, double const *coeff64,
                      float const *coeff32, FieldView in, FieldView out, cudaStream_t s )
{
    if ( n_tgt == 0 )
        return;
    unsigned const blocks = (unsigned)( ( n_tgt * 8 + 255 ) / 256 );
    if ( coeff32 )
        k_apply_multi<true><<<blocks, 256, 0, s>>>( n_tgt, offset, idx, coeff32, in, out );
    else
        k_apply_multi<false><<<blocks, 256, 0, s>>>( n_tgt, offset, idx, coeff64, in, out );
    check_launch( "k_apply_multi" );
}

void apply_csr( int64_t n_tgt, int32_t const *offset, int32_t const *idx, double const *coeff64,
                float const *coeff32, int uniform_row, int mean_row, double const *values,
                double *target, cudaStream_t s )
{
    if ( n_tgt == 0 )
        return;
    bool const f32 = coeff32 != nullptr;
    void const *coeff = f32 ? (void const *)coeff32 : (void const *)coeff64;
    if ( !f32 && apply_sorted_supported( uniform_row ) )
    {
        // (a saved operator has no positions: the same sums by index)
        apply_rows64( n_tgt, uniform_row, idx, coeff64, nullptr, rank1( values, nullptr, 0 ),
                      rank1( nullptr, target, n_tgt ), false, s, nullptr );
        return;
    }
    int const len = uniform_row > 0 ? uniform_row : mean_row;
    int S = 1;
    while ( S < 32 && S * 2 <= len )
        S *= 2;
    if ( f32 )
        launch_csr<true>( S, n_tgt, offset, idx, coeff, values, target, s );
    else
        launch_csr<false>( S, n_tgt, offset, idx, coeff, values, target, s );
}

} // namespace dtk
