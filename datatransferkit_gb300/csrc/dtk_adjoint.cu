// Adjoint of the MLS transfer (extension; the reference has none).
//
// For L with dL/d(target values) = cot:
//   dL/d(source values) = C^T cot, C the operator's CSR coefficients.  The
//     transpose (source -> its entries) is built once per handle by a stable
//     radix sort of (source index, entry), so each source sums its entries
//     in ascending entry order: deterministic, no atomics.
//   dL/d(source coordinates): per target, with x_j = s_j - t, rho_j = |x_j|,
//     R = 1.1 max(10 eps, max rho), phi_j = rbf(rho_j / R),
//     A = sum phi P P^T, a = A^+ e0, z = A^+ b, b = sum phi_j v_j P_j, y = a.b,
//     and in the radius-scaled frame (x^ = x / R, P^ = P(x^), J^ = dP^/dx^):
//       dy/dx_j = (phi_j / R) J^_j^T (e_j a^ - alpha_j z^) + (g_j / R) u_j
//                 - [j farthest] 1.1 (sum_l g_l rho^_l) / R u_j
//     with alpha_j = a^.P^_j, e_j = v_j - P^_j.z^, g_j = alpha_j e_j rbf'(rho^_j),
//     u_j = x_j / rho_j; the radius max sends its gradient to the farthest
//     neighbour (the last of largest rho in row order): the only term that
//     needs the sum over the row, so one pass writes every entry's contribution
//     and the farthest one is corrected after it.  The contributions cot_i
//     dy/dx_j, with c_j beside them, are written at the entry's place in the
//     transpose (one 32-byte sector each), so each source sums a run of
//     consecutive sectors.  The pseudo-inverse is recomputed per target (never
//     stored) from FP64 scaled moments.  Well-conditioned targets take an
//     FP64 Cholesky (A^+ = A^-1 there); the rest take an FP32 round-robin
//     Jacobi, one FP64 sweep on B = V32^T A V32 and truncation at 2^-40 of
//     the largest eigenvalue.  Both end with one FP64 refinement step for a^
//     and z^ each.
#include "dtk_common.cuh"
#include "dtk_handle.cuh"
#include "dtk_jacobi.cuh"
#include "dtk_moments.cuh"

#include <algorithm>
#include <new>
#include <utility>

namespace dtk
{
namespace
{

constexpr int AB = 32; // threads per block of the coordinate kernel

__global__ void k_entry_pairs( int32_t const *idx, int64_t nnz, uint32_t *keys, uint32_t *vals )
{
    int64_t const e = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if ( e < nnz )
    {
        keys[e] = (uint32_t)idx[e];
        vals[e] = (uint32_t)e;
    }
}

__global__ void k_source_counts( uint32_t const *sorted_keys, int64_t nnz, int64_t *counts )
{
    int64_t const e = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if ( e < nnz )
        atomicAdd( reinterpret_cast<unsigned long long *>( counts + sorted_keys[e] ), 1ull );
}

__global__ void k_narrow( int64_t const *in, int32_t *out, int64_t n )
{
    int64_t const i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if ( i <= n )
        out[i] = (int32_t)in[i];
}

__global__ void k_entry_rows( int32_t const *offset, int64_t n_tgt, int32_t *row_of )
{
    int64_t const i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if ( i < n_tgt )
        for ( int e = offset[i]; e < offset[i + 1]; ++e )
            row_of[e] = (int32_t)i;
}

// t_place[e] = the place of entry e in the transpose
__global__ void k_entry_places( int32_t const *t_entry, int64_t nnz, int32_t *t_place )
{
    int64_t const q = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if ( q < nnz )
        t_place[t_entry[q]] = (int32_t)q;
}

// One thread per source: grad_values[s] = sum_e coeff[e] cot[row(e)] over the
// source's entries, ascending.  Bound by the coefficients' sectors in L1 (a
// source's entries lie in as many rows, and neighbouring sources use the same
// rows): two blocks of 704 threads an SM, where that fills the GPU, keep more of
// them there than 2048 threads do (1M sources of 32 entries 0.61 -> 0.52 ms, 3M
// of 24 1.78 -> 1.68; 1M of 8 0.103 -> 0.108, of 16 0.225 -> 0.207).
constexpr int GATHER_THREADS = 704;

template <bool F32>
__global__ void __launch_bounds__( GATHER_THREADS )
    k_transpose_gather( int64_t n_src, int32_t const *t_offset, int32_t const *t_entry, int uniform_row,
                        int32_t const *row_of, void const *coeff, double const *cot, double *grad_values )
{
    int64_t const s = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if ( s >= n_src )
        return;
    double gv = 0.0;
#pragma unroll 4
    for ( int q = t_offset[s]; q < t_offset[s + 1]; ++q )
    {
        unsigned const e = (unsigned)t_entry[q];
        int const row = uniform_row > 0 ? (int)( e / (unsigned)uniform_row ) : row_of[e];
        double const c = F32 ? (double)static_cast<float const *>( coeff )[e]
                             : static_cast<double const *>( coeff )[e];
        gv = fma( c, cot[row], gv );
    }
    grad_values[s] = gv;
}

// The same sums, bit for bit, and those of the coordinates from the entries'
// contributions, which lie in the transpose's order (x, y, z and the
// coefficient: 32 bytes an entry): four lanes a source, one a component, so that
// a warp reads whole lines; the lane of the values looks its entries' rows up.
// 1M x 1M, k = 32: 1.47 ms as gathers through the entries' indices (three cache
// lines an entry).
__global__ void k_transpose_sum( int64_t n_src, int32_t const *t_offset, int32_t const *t_entry, int uniform_row,
                                 int32_t const *row_of, double const *cot, double const *contrib, double *grad_values,
                                 double *grad_coords )
{
    int64_t const t = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    int64_t const s = t >> 2;
    int const c = (int)( t & 3 );
    if ( s >= n_src )
        return;
    int64_t const b = t_offset[s], e = t_offset[s + 1];
    double sum = 0.0;
#pragma unroll 4
    for ( int64_t q = b; q < e; ++q )
    {
        double by = 1.0;
        if ( c == 3 )
        {
            unsigned const at = (unsigned)__ldcs( t_entry + q );
            by = __ldg( cot + ( uniform_row > 0 ? (int)( at / (unsigned)uniform_row ) : row_of[at] ) );
        }
        sum = fma( __ldcs( contrib + 4 * q + c ), by, sum );
    }
    if ( c == 3 )
        grad_values[s] = sum;
    else
        grad_coords[3 * s + c] = sum;
}

// What the coordinate-adjoint kernels read and write.
struct AdjointView
{
    double const *src, *tgt;
    int32_t const *offset, *idx, *place; // place: of each entry in the transpose
    int64_t n_src;
    int rbf;
    double const *values, *cot;
    double const *coeff64;
    float const *coeff32;
    double *contrib; // 4 doubles an entry, in the transpose's order
    unsigned *status;
    __device__ __forceinline__ void put( int64_t e, double x, double y, double z ) const
    {
        double2 *const p = reinterpret_cast<double2 *>( contrib + 4 * (int64_t)place[e] );
        p[0] = make_double2( x, y );
        p[1] = make_double2( z, coeff32 ? (double)coeff32[e] : coeff64[e] );
    }
};

// Per-target pieces shared by the two coordinate-adjoint kernels.
struct AdjTarget
{
    int64_t i, b0;
    int len, far;
    bool radius_live;
    double tx, ty, tz, ci, inv_r;
};

// Returns false when the target needs no more work (no entries, a zero
// cotangent: its contributions are zero, or a bad index: reported).
__device__ __forceinline__ bool adjoint_prologue( int64_t i, AdjointView const &v, AdjTarget &T )
{
    T.i = i;
    T.b0 = v.offset[i];
    T.len = v.offset[i + 1] - (int)T.b0;
    T.ci = v.cot[i];
    if ( T.len == 0 )
        return false;
    for ( int j = 0; j < T.len; ++j )
        if ( (uint32_t)v.idx[T.b0 + j] >= (uint64_t)v.n_src )
        {
            atomicOr( v.status, DEV_BAD_INDEX );
            return false;
        }
    if ( T.ci == 0.0 )
    {
        for ( int j = 0; j < T.len; ++j )
            v.put( T.b0 + j, 0.0, 0.0, 0.0 );
        return false;
    }
    T.tx = v.tgt[3 * i];
    T.ty = v.tgt[3 * i + 1];
    T.tz = v.tgt[3 * i + 2];
    auto const dist2 = [&]( int j ) {
        int64_t const sj = v.idx[T.b0 + j];
        return dist2_rn( v.src[3 * sj], v.src[3 * sj + 1], v.src[3 * sj + 2], T.tx, T.ty, T.tz );
    };
    double d2max = 0.0;
    for ( int j = 0; j < T.len; ++j )
        d2max = fmax( d2max, dist2( j ) );
    double const floor_d = 10. * DBL_EPSILON, dmax = sqrt( d2max );
    // the farthest neighbour: the last of largest distance, which is not always
    // one of largest square (two of them can have one root).  Looked for from
    // the end, where a sorted row has it.
    for ( T.far = T.len - 1; T.far > 0; --T.far )
    {
        double const d2 = dist2( T.far );
        if ( d2 >= d2max || ( d2 >= d2max * ( 1.0 - 4.0 * DBL_EPSILON ) && sqrt( d2 ) >= dmax ) )
            break;
    }
    T.radius_live = dmax > floor_d;
    T.inv_r = 1.0 / ( 1.1 * ( T.radius_live ? dmax : floor_d ) );
    return true;
}

// An entry's scaled coordinates, their squares, 1 / |x^| (0 at the target) and
// |x^|, from one reciprocal square root and a Newton step on the root's residual
// (as accurate as a square root; without it, 2.6% faster at 1M x 1M, the 99th
// percentile of the gradients' errors grew by 4% for Wendland<0>).
struct AdjEntry
{
    int64_t sj;
    double x, y, z, xx, yy, zz, inv_rho, rho;
};
__device__ __forceinline__ AdjEntry adjoint_entry( AdjTarget const &T, AdjointView const &v, int j )
{
    AdjEntry a;
    a.sj = v.idx[T.b0 + j];
    a.x = ( v.src[3 * a.sj] - T.tx ) * T.inv_r;
    a.y = ( v.src[3 * a.sj + 1] - T.ty ) * T.inv_r;
    a.z = ( v.src[3 * a.sj + 2] - T.tz ) * T.inv_r;
    a.xx = a.x * a.x;
    a.yy = a.y * a.y;
    a.zz = a.z * a.z;
    double const d2 = ( a.xx + a.yy ) + a.zz;
    a.inv_rho = d2 > 0.0 ? rsqrt( d2 ) : 0.0;
    double const r = d2 * a.inv_rho;
    a.rho = fma( fma( -r, r, d2 ), 0.5 * a.inv_rho, r );
    return a;
}

// rbf(x) and rbf'(x); the common Wendland functions share their powers.
__device__ __forceinline__ void rbf_with_deriv( int rbf, double x, double &phi, double &deriv )
{
    double const y = 1.0 - x, y2 = y * y, y3 = y2 * y;
    if ( rbf == DTK_WENDLAND2 )
    {
        phi = y2 * y2 * fma( 4.0, x, 1.0 );
        deriv = -20.0 * x * y3;
    }
    else if ( rbf == DTK_WENDLAND4 )
    {
        phi = y3 * y3 * fma( fma( 35.0, x, 18.0 ), x, 3.0 );
        deriv = -56.0 * x * fma( 5.0, x, 1.0 ) * ( y3 * y2 );
    }
    else
    {
        phi = rbf_eval<double>( rbf, x );
        deriv = rbf_deriv( rbf, x );
    }
}

// Scaled moments A^ (upper triangle) and b^ = sum phi v P^ (FP64).  The
// quadratic basis has 35 distinct sums for its 55 entries.
template <int M>
__device__ __forceinline__ void adjoint_moments( AdjTarget const &T, AdjointView const &v, double *A, double *bh )
{
    double S[N_MOMENTS<M>];
#pragma unroll
    for ( int u = 0; u < N_MOMENTS<M>; ++u )
        S[u] = 0.0;
#pragma unroll
    for ( int c = 0; c < M; ++c )
        bh[c] = 0.0;
    for ( int j = 0; j < T.len; ++j )
    {
        AdjEntry const a = adjoint_entry( T, v, j );
        double const phi = rbf_eval<double>( v.rbf, a.rho );
        double P[M];
        basis_eval<M, double>( a.x, a.y, a.z, P );
        double const pv = phi * v.values[a.sj];
#pragma unroll
        for ( int c = 0; c < M; ++c )
            bh[c] = fma( pv, P[c], bh[c] );
        add_moments<M>( a.x, a.y, a.z, a.xx, a.yy, a.zz, phi, S );
    }
#pragma unroll
    for ( int a = 0; a < M; ++a )
#pragma unroll
        for ( int c = a; c < M; ++c )
            A[ut<M>( a, c )] = S[moment_index( a, c )];
}

// P . a
template <int M>
__device__ __forceinline__ double adjoint_dot( double const *a, AdjEntry const &e )
{
    double r = a[0];
    if constexpr ( M >= 4 )
        r = fma( a[3], e.z, fma( a[2], e.y, fma( a[1], e.x, r ) ) );
    if constexpr ( M == 10 )
    {
        r = fma( e.x, fma( a[4], e.x, fma( a[5], e.y, a[6] * e.z ) ), r );
        r = fma( e.y, fma( a[7], e.y, a[8] * e.z ), r );
        r = fma( a[9], e.zz, r );
    }
    return r;
}

// d(P . a) / dx^ : a2 = twice a[4], a[7], a[9]
template <int M>
__device__ __forceinline__ void adjoint_grad( double const *a, double const *a2, AdjEntry const &e, double *g )
{
    if constexpr ( M == 1 )
        g[0] = g[1] = g[2] = 0.0;
    else
    {
        g[0] = a[1];
        g[1] = a[2];
        g[2] = a[3];
    }
    if constexpr ( M == 10 )
    {
        g[0] = fma( a2[0], e.x, fma( a[5], e.y, fma( a[6], e.z, g[0] ) ) );
        g[1] = fma( a[5], e.x, fma( a2[1], e.y, fma( a[8], e.z, g[1] ) ) );
        g[2] = fma( a[6], e.x, fma( a[8], e.y, fma( a2[2], e.z, g[2] ) ) );
    }
}

// Given a^ = A^+ e0 and z^ = A^+ b^: the per-entry contributions cot_i dy/dx_j
// and S = sum g_l rho^_l in one pass, then the radius term of the farthest
// neighbour.
template <int M>
__device__ __forceinline__ void adjoint_passes( AdjTarget const &T, AdjointView const &v, double const *ah,
                                                double const *zh )
{
    double a2[3] = {0.0, 0.0, 0.0}, z2[3] = {0.0, 0.0, 0.0};
    if constexpr ( M == 10 )
    {
        a2[0] = 2.0 * ah[4];
        a2[1] = 2.0 * ah[7];
        a2[2] = 2.0 * ah[9];
        z2[0] = 2.0 * zh[4];
        z2[1] = 2.0 * zh[7];
        z2[2] = 2.0 * zh[9];
    }
    double const scale = T.ci * T.inv_r;
    double S = 0.0, fx = 0.0, fy = 0.0, fz = 0.0, ux = 0.0, uy = 0.0, uz = 0.0;
    for ( int j = 0; j < T.len; ++j )
    {
        AdjEntry const a = adjoint_entry( T, v, j );
        double phi, deriv;
        rbf_with_deriv( v.rbf, a.rho, phi, deriv );
        double const al = adjoint_dot<M>( ah, a ), e = v.values[a.sj] - adjoint_dot<M>( zh, a );
        double ga[3], gz[3];
        adjoint_grad<M>( ah, a2, a, ga );
        adjoint_grad<M>( zh, z2, a, gz );
        double const g = al * e * deriv;
        S = fma( g, a.rho, S );
        // phi (e grad(P . a) - al grad(P . z)) + g u, u = x^ / rho^
        double const pe = phi * e, pa = phi * al, gr = g * a.inv_rho;
        double const cx = scale * fma( gr, a.x, fma( pe, ga[0], -( pa * gz[0] ) ) ),
                     cy = scale * fma( gr, a.y, fma( pe, ga[1], -( pa * gz[1] ) ) ),
                     cz = scale * fma( gr, a.z, fma( pe, ga[2], -( pa * gz[2] ) ) );
        v.put( T.b0 + j, cx, cy, cz );
        if ( j == T.far )
        {
            fx = cx;
            fy = cy;
            fz = cz;
            ux = a.x * a.inv_rho;
            uy = a.y * a.inv_rho;
            uz = a.z * a.inv_rho;
        }
    }
    if ( T.radius_live )
    {
        double const r = -1.1 * S * scale;
        v.put( T.b0 + T.far, fma( r, ux, fx ), fma( r, uy, fy ), fma( r, uz, fz ) );
    }
}

// Fast path, one thread per target: FP64 Cholesky A^ = R^T R and S = R^-1,
// in place in a per-thread shared-memory work area (in registers they spill
// at M = 10); a^ and z^ as S (S^T v) with one refinement step against the
// moments (also kept in shared memory).  Taken when the factorization succeeds
// and trace(A^) ||S||_F^2 <= 2^39, a bound on cond(A^) below the eigen path's
// 2^-40 truncation, so A^+ = A^-1; other targets are listed for the eigen
// path.
constexpr int AF = 32; // threads per block of the fast kernel

template <int M>
__global__ void __launch_bounds__( AF )
    k_adjoint_fast( AdjointView v, uint32_t const *order, int64_t n_tgt, int32_t *list, unsigned *count )
{
    constexpr int NU = M * ( M + 1 ) / 2;
    // per thread, interleaved: NU moments, M of b^, NU of the Cholesky work area
    extern __shared__ double s_mom[];
    auto Wk = [&]( int u ) -> double & { return s_mom[( NU + M + u ) * AF + threadIdx.x]; };
    int64_t const g = blockIdx.x * (int64_t)AF + threadIdx.x;
    if ( g >= n_tgt )
        return;
    int64_t const i = order ? (int64_t)order[g] : g;
    AdjTarget T;
    if ( !adjoint_prologue( i, v, T ) )
        return;
    double A[NU];
    {
        double bh[M];
        adjoint_moments<M>( T, v, A, bh );
#pragma unroll
        for ( int c = 0; c < M; ++c )
            s_mom[( NU + c ) * AF + threadIdx.x] = bh[c];
    }
    double trace = 0.0;
#pragma unroll
    for ( int u = 0; u < NU; ++u )
    {
        s_mom[u * AF + threadIdx.x] = A[u];
        Wk( u ) = A[u];
    }
#pragma unroll
    for ( int k = 0; k < M; ++k )
        trace += A[ut<M>( k, k )];
    // Cholesky in place (R upper, row-major packed), then S = R^-1 in place
    bool ok = trace > 0.0;
    {
        double rinv[M];
#pragma unroll
        for ( int j = 0; j < M; ++j )
        {
            double d = Wk( ut<M>( j, j ) );
#pragma unroll
            for ( int k = 0; k < j; ++k )
                d = fma( -Wk( ut<M>( k, j ) ), Wk( ut<M>( k, j ) ), d );
            ok = ok && d > 0.0;
            rinv[j] = d > 0.0 ? rsqrt( d ) : 1.0;
            Wk( ut<M>( j, j ) ) = d > 0.0 ? d * rinv[j] : 1.0;
#pragma unroll
            for ( int c = j + 1; c < M; ++c )
            {
                double v = Wk( ut<M>( j, c ) );
#pragma unroll
                for ( int k = 0; k < j; ++k )
                    v = fma( -Wk( ut<M>( k, j ) ), Wk( ut<M>( k, c ) ), v );
                Wk( ut<M>( j, c ) ) = v * rinv[j];
            }
        }
#pragma unroll
        for ( int j = 0; j < M; ++j )
        {
#pragma unroll
            for ( int r = 0; r < j; ++r )
            {
                double v = 0.0;
#pragma unroll
                for ( int k = r; k < j; ++k )
                    v = fma( Wk( ut<M>( r, k ) ), Wk( ut<M>( k, j ) ), v );
                Wk( ut<M>( r, j ) ) = -v * rinv[j];
            }
            Wk( ut<M>( j, j ) ) = rinv[j];
        }
    }
    double fro = 0.0;
#pragma unroll
    for ( int u = 0; u < NU; ++u )
        fro = fma( Wk( u ), Wk( u ), fro );
    if ( !ok || !( trace * fro <= 549755813888.0 ) ) // 2^39; false for NaN
    {
        list[atomicAdd( count, 1u )] = (int32_t)i;
        return;
    }
    // x = S (S^T v)
    auto apply_inv = [&]( double const *v, double *x ) {
        double w[M];
#pragma unroll
        for ( int k = 0; k < M; ++k )
        {
            double acc = 0.0;
#pragma unroll
            for ( int r = 0; r <= k; ++r )
                acc = fma( Wk( ut<M>( r, k ) ), v[r], acc );
            w[k] = acc;
        }
#pragma unroll
        for ( int r = 0; r < M; ++r )
        {
            double acc = 0.0;
#pragma unroll
            for ( int k = r; k < M; ++k )
                acc = fma( Wk( ut<M>( r, k ) ), w[k], acc );
            x[r] = acc;
        }
    };
    // right-hand side rhs_r = (r == 0) for e0, else b^ from shared memory
    auto solve = [&]( bool unit, double *x ) {
        double v[M];
#pragma unroll
        for ( int r = 0; r < M; ++r )
            v[r] = unit ? ( r == 0 ? 1.0 : 0.0 ) : s_mom[( NU + r ) * AF + threadIdx.x];
        apply_inv( v, x );
#pragma unroll
        for ( int r = 0; r < M; ++r )
        {
            double acc = unit ? ( r == 0 ? 1.0 : 0.0 ) : s_mom[( NU + r ) * AF + threadIdx.x];
#pragma unroll
            for ( int c = 0; c < M; ++c )
                acc = fma( -s_mom[ut<M>( r, c ) * AF + threadIdx.x], x[c], acc );
            v[r] = acc;
        }
        double d[M];
        apply_inv( v, d );
#pragma unroll
        for ( int r = 0; r < M; ++r )
            x[r] += d[r];
    };
    double ah[M], zh[M];
    solve( true, ah );
    solve( false, zh );
    adjoint_passes<M>( T, v, ah, zh );
}

// Eigen path over the targets the fast path listed (list[0 .. *count),
// persistent blocks): FP32 Jacobi, B = V32^T A V32, one FP64 sweep,
// truncation at 2^-40 of the largest eigenvalue, one FP64 refinement step.
template <int M>
__global__ void __launch_bounds__( AB )
    k_adjoint_entries( AdjointView v, int32_t const *list, unsigned const *count )
{
    constexpr int NU = M * ( M + 1 ) / 2;
    extern __shared__ unsigned char smem_raw[];
    // per thread, interleaved: A64 (NU doubles), B (NU doubles; A32 first),
    // W (M*M doubles), V32 (M*M floats)
    double *sa = reinterpret_cast<double *>( smem_raw );
    double *sb = sa + NU * AB;
    double *sw = sb + NU * AB;
    float *sv = reinterpret_cast<float *>( sw + M * M * AB );
    int const t = threadIdx.x;
    auto A64 = [&]( int u ) -> double & { return sa[u * AB + t]; };
    auto B = [&]( int u ) -> double & { return sb[u * AB + t]; };
    auto A32 = [&]( int u ) -> float & { return reinterpret_cast<float *>( sb )[u * AB + t]; };
    auto W = [&]( int r, int c ) -> double & { return sw[( r * M + c ) * AB + t]; };
    auto V32 = [&]( int r, int c ) -> float & { return sv[( r * M + c ) * AB + t]; };

    int64_t const n_list = *count;
    for ( int64_t g = blockIdx.x * (int64_t)AB + threadIdx.x; g < n_list; g += (int64_t)gridDim.x * AB )
    {
        AdjTarget T;
        if ( !adjoint_prologue( list[g], v, T ) )
            continue;
        double bh[M];
        {
            double A[NU];
            adjoint_moments<M>( T, v, A, bh );
#pragma unroll
            for ( int u = 0; u < NU; ++u )
            {
                A64( u ) = A[u];
                A32( u ) = (float)A[u];
            }
        }
#pragma unroll
        for ( int r = 0; r < M; ++r )
#pragma unroll
            for ( int c = 0; c < M; ++c )
                V32( r, c ) = r == c ? 1.f : 0.f;
        for ( int sweep = 0; sweep < 12; ++sweep )
            if ( jacobi_sweep<M, float>( A32, V32, 1e-7f ) == 0 )
                break;
        for ( int k = 0; k < M; ++k )
        {
            double ck[M];
#pragma unroll
            for ( int r = 0; r < M; ++r )
            {
                double acc = 0.0;
#pragma unroll
                for ( int c = 0; c < M; ++c )
                    acc = fma( A64( ut<M>( r, c ) ), (double)V32( c, k ), acc );
                ck[r] = acc;
            }
            for ( int jj = 0; jj <= k; ++jj )
            {
                double acc = 0.0;
#pragma unroll
                for ( int r = 0; r < M; ++r )
                    acc = fma( (double)V32( r, jj ), ck[r], acc );
                B( ut<M>( jj, k ) ) = acc;
            }
        }
#pragma unroll
        for ( int r = 0; r < M; ++r )
#pragma unroll
            for ( int c = 0; c < M; ++c )
                W( r, c ) = (double)V32( r, c );
        jacobi_sweep<M, double>( B, W, 1e-15 );
        double lmax = 0.0;
        for ( int k = 0; k < M; ++k )
            lmax = fmax( lmax, fabs( B( ut<M>( k, k ) ) ) );
        double const cut = lmax * 9.094947017729282e-13; // 2^-40
        for ( int k = 0; k < M; ++k )
        {
            double const lk = B( ut<M>( k, k ) );
            B( ut<M>( k, k ) ) = ( fabs( lk ) > cut && lk != 0.0 ) ? 1.0 / lk : 0.0;
        }
        // y += A^+ v, then one refinement step against the FP64 moments
        auto pinv_add = [&]( double const *v, double *y ) {
            for ( int k = 0; k < M; ++k )
            {
                double acc = 0.0;
#pragma unroll
                for ( int r = 0; r < M; ++r )
                    acc = fma( W( r, k ), v[r], acc );
                acc *= B( ut<M>( k, k ) );
#pragma unroll
                for ( int r = 0; r < M; ++r )
                    y[r] = fma( W( r, k ), acc, y[r] );
            }
        };
        auto solve = [&]( double const *rhs, double *x ) {
#pragma unroll
            for ( int r = 0; r < M; ++r )
                x[r] = 0.0;
            pinv_add( rhs, x );
            double res[M];
#pragma unroll
            for ( int r = 0; r < M; ++r )
            {
                double acc = rhs[r];
#pragma unroll
                for ( int c = 0; c < M; ++c )
                    acc = fma( -A64( ut<M>( r, c ) ), x[c], acc );
                res[r] = acc;
            }
            pinv_add( res, x );
        };
        double e0[M], ah[M], zh[M];
#pragma unroll
        for ( int r = 0; r < M; ++r )
            e0[r] = r == 0 ? 1.0 : 0.0;
        solve( e0, ah );
        solve( bh, zh );
        adjoint_passes<M>( T, v, ah, zh );
    }
}

template <int M>
void launch_adjoint_entries( dtk_mls_s const *h, AdjointView const &v, cudaStream_t s )
{
    constexpr int NU = M * ( M + 1 ) / 2;
    DeviceBuffer<int32_t> list( std::max<int64_t>( 1, h->n_tgt ), s );
    DeviceBuffer<unsigned> count( 1, s );
    DTK_CUDA_OR_THROW( cudaMemsetAsync( count.get(), 0, sizeof( unsigned ), s ) );
    k_adjoint_fast<M><<<(unsigned)( ( h->n_tgt + AF - 1 ) / AF ), AF, ( 2 * NU + M ) * sizeof( double ) * AF, s>>>(
        v, h->order.get(), h->n_tgt, list.get(), count.get() );
    check_launch( "k_adjoint_fast" );
    size_t const smem = ( 2 * NU * sizeof( double ) + M * M * sizeof( double ) +
                          M * M * sizeof( float ) ) * AB;
    ensure_dynamic_smem( k_adjoint_entries<M>, smem );
    int64_t const want = ( h->n_tgt + AB - 1 ) / AB;
    unsigned const blocks = (unsigned)std::max<int64_t>( 1, std::min<int64_t>( want, 4 * num_sms() ) );
    k_adjoint_entries<M><<<blocks, AB, smem, s>>>( v, list.get(), count.get() );
    check_launch( "k_adjoint_entries" );
}

// (the handle takes the buffers once all of them are there: a call that runs
// out of memory on the way can be made again)
void build_transpose_for( dtk_mls_s *h, cudaStream_t s )
{
    if ( h->t_offset.get() )
        return;
    int64_t const nnz = h->nnz, n_src = h->n_src;
    DeviceBuffer<uint32_t> keys( std::max<int64_t>( 1, nnz ), s );
    DeviceBuffer<int32_t> t_entry( std::max<int64_t>( 1, nnz ), s ), t_offset( n_src + 1, s );
    unsigned const blocks = (unsigned)std::max<int64_t>( 1, ( nnz + 255 ) / 256 );
    if ( nnz )
    {
        k_entry_pairs<<<blocks, 256, 0, s>>>( h->idx.get(), nnz, keys.get(),
                                              reinterpret_cast<uint32_t *>( t_entry.get() ) );
        check_launch( "k_entry_pairs" );
        int bits = 1;
        while ( ( int64_t( 1 ) << bits ) < n_src )
            ++bits;
        radix_sort_pairs( keys.get(), reinterpret_cast<uint32_t *>( t_entry.get() ), nnz, ( bits + 7 ) / 8 * 8, s );
    }
    DeviceBuffer<int64_t> counts( n_src, s ), offs( n_src + 1, s );
    DTK_CUDA_OR_THROW( cudaMemsetAsync( counts.get(), 0, n_src * sizeof( int64_t ), s ) );
    if ( nnz )
    {
        k_source_counts<<<blocks, 256, 0, s>>>( keys.get(), nnz, counts.get() );
        check_launch( "k_source_counts" );
    }
    exclusive_scan_i64( counts.get(), offs.get(), n_src, s );
    k_narrow<<<(unsigned)( ( n_src + 256 ) / 256 ), 256, 0, s>>>( offs.get(), t_offset.get(), n_src );
    check_launch( "k_narrow" );
    h->t_entry = std::move( t_entry );
    h->t_offset = std::move( t_offset );
}

// The entries' places in the transpose, for the coordinate adjoint.
void build_places_for( dtk_mls_s *h, cudaStream_t s )
{
    if ( h->t_place.get() || h->nnz == 0 )
        return;
    DeviceBuffer<int32_t> t_place( h->nnz, s );
    k_entry_places<<<(unsigned)( ( h->nnz + 255 ) / 256 ), 256, 0, s>>>( h->t_entry.get(), h->nnz, t_place.get() );
    check_launch( "k_entry_places" );
    h->t_place = std::move( t_place );
}

} // namespace
} // namespace dtk

using namespace dtk;

extern "C" dtk_status dtk_mls_apply_adjoint( dtk_mls_handle h, const double *cot, int64_t n_cot,
                                             const double *source_values, double *grad_values,
                                             double *grad_coords, dtk_stream_t stream_ )
{
    try
    {
        NvtxRange const nvtx_range( "DTK_apply_adjoint" );
        DTK_REQUIRE_OR_THROW( h != nullptr, "handle is null" );
        DTK_REQUIRE_OR_THROW( n_cot == h->n_tgt, "cot.extent(0) == n_target_points" );
        DTK_REQUIRE_OR_THROW( h->n_tgt == 0 || cot != nullptr, "cot is null" );
        DTK_REQUIRE_OR_THROW( grad_values != nullptr, "grad_values is null" );
        if ( grad_coords )
        {
            DTK_REQUIRE_OR_THROW( source_values != nullptr,
                                  "the coordinate adjoint needs the source values" );
            DTK_REQUIRE_OR_THROW( h->src_copy.get() != nullptr,
                                  "the coordinate adjoint needs a handle created with keep_points" );
        }
        require_device_memory( h->n_tgt ? cot : nullptr, "cot" );
        require_device_memory( grad_values, "grad_values" );
        require_device_memory( source_values, "source_values" );
        require_device_memory( grad_coords, "grad_coords" );
        cudaStream_t s = reinterpret_cast<cudaStream_t>( stream_ );
        TouchOnExit const touch{&h->life, s};
        build_transpose_for( h, s );
        DeviceBuffer<unsigned> status( 1, s );
        DTK_CUDA_OR_THROW( cudaMemsetAsync( status.get(), 0, sizeof( unsigned ), s ) );
        DeviceBuffer<int32_t> row_of;
        if ( h->uniform_row <= 0 && h->nnz )
        {
            row_of.allocate( h->nnz, s );
            k_entry_rows<<<(unsigned)( ( h->n_tgt + 255 ) / 256 ), 256, 0, s>>>( h->offset.get(), h->n_tgt,
                                                                                 row_of.get() );
            check_launch( "k_entry_rows" );
        }
        if ( grad_coords && h->nnz )
        {
            build_places_for( h, s );
            DeviceBuffer<double> contrib( 4 * h->nnz, s );
            AdjointView const v{h->src_copy.get(), h->tgt_copy.get(), h->offset.get(),  h->idx.get(),
                                h->t_place.get(),  h->n_src,          h->opts.rbf,      source_values,
                                cot,               h->coeff64.get(),  h->coeff32.get(), contrib.get(),
                                status.get()};
            switch ( h->opts.basis )
            {
            case DTK_CONSTANT3:
                launch_adjoint_entries<1>( h, v, s );
                break;
            case DTK_LINEAR3:
                launch_adjoint_entries<4>( h, v, s );
                break;
            default:
                launch_adjoint_entries<10>( h, v, s );
                break;
            }
            k_transpose_sum<<<(unsigned)( ( 4 * h->n_src + 255 ) / 256 ), 256, 0, s>>>(
                h->n_src, h->t_offset.get(), h->t_entry.get(), h->uniform_row, row_of.get(), cot, contrib.get(),
                grad_values, grad_coords );
            check_launch( "k_transpose_sum" );
        }
        else if ( h->n_src )
        {
            if ( grad_coords )
                DTK_CUDA_OR_THROW( cudaMemsetAsync( grad_coords, 0, 3 * h->n_src * sizeof( double ), s ) );
            int const threads = h->n_src >= 2 * GATHER_THREADS * (int64_t)num_sms() ? GATHER_THREADS : 256;
            unsigned const blocks = (unsigned)( ( h->n_src + threads - 1 ) / threads );
            bool const f32 = h->coeff32.get() != nullptr;
            void const *coeff = f32 ? (void const *)h->coeff32.get() : (void const *)h->coeff64.get();
            if ( f32 )
                k_transpose_gather<true><<<blocks, threads, 0, s>>>( h->n_src, h->t_offset.get(), h->t_entry.get(),
                                                                 h->uniform_row, row_of.get(), coeff, cot,
                                                                 grad_values );
            else
                k_transpose_gather<false><<<blocks, threads, 0, s>>>( h->n_src, h->t_offset.get(), h->t_entry.get(),
                                                                  h->uniform_row, row_of.get(), coeff, cot,
                                                                  grad_values );
            check_launch( "k_transpose_gather" );
        }
        unsigned st = 0;
        DTK_CUDA_OR_THROW( cudaMemcpyAsync( &st, status.get(), sizeof( st ), cudaMemcpyDeviceToHost, s ) );
        DTK_CUDA_OR_THROW( cudaStreamSynchronize( s ) );
        if ( st )
            throw Error{DTK_ERR_INTERNAL, "adjoint found a bad neighbour index"};
        return DTK_OK;
    }
    catch ( Error const &e )
    {
        set_error( e.msg );
        return e.status;
    }
    catch ( std::bad_alloc const & )
    {
        set_error( "host allocation failed" );
        return DTK_ERR_OOM;
    }
    catch ( std::exception const &e )
    {
        set_error( e.what() );
        return DTK_ERR_INTERNAL;
    }
}
