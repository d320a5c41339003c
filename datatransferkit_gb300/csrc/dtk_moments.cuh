// The moment sums of the polynomial bases, shared by the FP64 setup and the
// adjoint.
#pragma once

#include "dtk_common.cuh"

namespace dtk
{

// Distinct moments sum phi x^a y^b z^c of the basis products, a + b + c <= 2
// deg: 1, 10 or 35.  moment_index( i, j ) is the sum that holds entry (i, j)
// of the moment matrix.
template <int M>
constexpr int N_MOMENTS = M == 10 ? 35 : M == 4 ? 10 : 1;

__host__ __device__ constexpr int mono_index( int a, int b, int c )
{
    // degree by degree; within a degree by descending power of x, then of y
    int const n = a + b + c, m = n - a;
    return n * ( n + 1 ) * ( n + 2 ) / 6 + m * ( m + 1 ) / 2 + c;
}
// powers of x, y and z in basis function i: 1 x y z xx xy xz yy yz zz
__host__ __device__ constexpr int pow_x( int i ) { return ( i == 1 ) + 2 * ( i == 4 ) + ( i == 5 ) + ( i == 6 ); }
__host__ __device__ constexpr int pow_y( int i ) { return ( i == 2 ) + ( i == 5 ) + 2 * ( i == 7 ) + ( i == 8 ); }
__host__ __device__ constexpr int pow_z( int i ) { return ( i == 3 ) + ( i == 6 ) + ( i == 8 ) + 2 * ( i == 9 ); }
__host__ __device__ constexpr int moment_index( int i, int j )
{
    return mono_index( pow_x( i ) + pow_x( j ), pow_y( i ) + pow_y( j ), pow_z( i ) + pow_z( j ) );
}
static_assert( moment_index( 9, 9 ) == 34 && moment_index( 0, 9 ) == 9 && moment_index( 3, 3 ) == 9 && moment_index( 1, 4 ) == 10 &&
                   moment_index( 5, 8 ) == 27 && moment_index( 6, 9 ) == 29 && moment_index( 2, 6 ) == 14,
               "moment order" );

// Adds one neighbour's phi x^a y^b z^c (x, y, z relative to the target).
template <int M>
__device__ __forceinline__ void add_moments( double x, double y, double z, double xx, double yy, double zz,
                                             double w, double *A )
{
    A[0] += w;
    if constexpr ( M >= 4 )
    {
        double const wx = w * x, wy = w * y, wz = w * z;
        A[1] = fma( w, x, A[1] );
        A[2] = fma( w, y, A[2] );
        A[3] = fma( w, z, A[3] );
        A[4] = fma( wx, x, A[4] );
        A[5] = fma( wx, y, A[5] );
        A[6] = fma( wx, z, A[6] );
        A[7] = fma( wy, y, A[7] );
        A[8] = fma( wy, z, A[8] );
        A[9] = fma( wz, z, A[9] );
    }
    if constexpr ( M == 10 )
    {
        double const xy = x * y, xz = x * z, yz = y * z;
        double const wxx = w * xx, wxy = w * xy, wyy = w * yy, wzz = w * zz;
        // degree 3: xxx xxy xxz xyy xyz xzz yyy yyz yzz zzz
        A[10] = fma( wxx, x, A[10] );
        A[11] = fma( wxx, y, A[11] );
        A[12] = fma( wxx, z, A[12] );
        A[13] = fma( wyy, x, A[13] );
        A[14] = fma( wxy, z, A[14] );
        A[15] = fma( wzz, x, A[15] );
        A[16] = fma( wyy, y, A[16] );
        A[17] = fma( wyy, z, A[17] );
        A[18] = fma( wzz, y, A[18] );
        A[19] = fma( wzz, z, A[19] );
        // degree 4: xxxx xxxy xxxz xxyy xxyz xxzz xyyy xyyz xyzz xzzz yyyy yyyz yyzz yzzz zzzz
        A[20] = fma( wxx, xx, A[20] );
        A[21] = fma( wxx, xy, A[21] );
        A[22] = fma( wxx, xz, A[22] );
        A[23] = fma( wxx, yy, A[23] );
        A[24] = fma( wxx, yz, A[24] );
        A[25] = fma( wxx, zz, A[25] );
        A[26] = fma( wyy, xy, A[26] );
        A[27] = fma( wyy, xz, A[27] );
        A[28] = fma( wzz, xy, A[28] );
        A[29] = fma( wzz, xz, A[29] );
        A[30] = fma( wyy, yy, A[30] );
        A[31] = fma( wyy, yz, A[31] );
        A[32] = fma( wyy, zz, A[32] );
        A[33] = fma( wzz, yz, A[33] );
        A[34] = fma( wzz, zz, A[34] );
    }
}

} // namespace dtk
