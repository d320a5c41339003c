// The fixed-point Jacobi of the FP64 setup (datatransferkit_gb300/csrc/
// dtk_fixed.cuh), built for the host: row 0 of the pseudo-inverse of each
// target's moment matrix, and the coefficients from it, for given rows.
// Built and driven by tests/test_fixed_jacobi_cpu.py against the oracle.
#define __host__
#define __device__
#define __forceinline__ inline
#define __noinline__ __attribute__( ( noinline ) )
#include "dtk_fixed.cuh"

#include <cmath>
#include <cstring>
#include <vector>

using namespace dtk;

namespace
{

// one lane runs both parts of the matrix
template <int M>
struct State
{
    using Lay = FxLayout<M>;
    mutable double n[Lay::OFF + M], vw[M];
    mutable int32_t last[Lay::OFF];
    mutable int e[M];
    mutable double c[600], sn[600];
    mutable int ls[600];
    double &a( int u ) const { return n[u]; }
    FxNum<3> f( int u ) const
    {
        FxNum<3> x;
        std::memcpy( x.d, &n[u], 8 );
        x.d[2] = last[u];
        return x;
    }
    void set_f( int u, FxNum<3> const &x ) const
    {
        std::memcpy( &n[u], x.d, 8 );
        last[u] = x.d[2];
    }
    int64_t diag( int k ) const
    {
        int64_t x;
        std::memcpy( &x, &n[Lay::diag( k )], 8 );
        return x;
    }
    void set_diag( int k, int64_t x ) const { std::memcpy( &n[Lay::diag( k )], &x, 8 ); }
    FxNum<2> v( int k ) const
    {
        FxNum<2> x;
        std::memcpy( x.d, &vw[k], 8 );
        return x;
    }
    void set_v( int k, FxNum<2> const &x ) const { std::memcpy( &vw[k], x.d, 8 ); }
    double &w( int k ) const { return vw[k]; }
    void column( int, int p, int q, int t, int &up, int &uq ) const { Lay::column( p, q, t, up, uq ); }
    int exp( int k ) const { return e[k]; }
    void set_exp( int k, int d ) const { e[k] = d; }
    void log( int r, double c_, double s_, int l ) const
    {
        c[r] = c_;
        sn[r] = s_;
        ls[r] = l;
    }
    template <class Fn>
    void for_parts( Fn const &fn ) const
    {
        fn( 0 );
        fn( 1 );
    }
    void merge( int &, int &, float & ) const {}
    void sync() const {}
    bool any( bool x ) const { return x; }
    bool both( bool x ) const { return x; }
};

template <int M>
bool row0( double const *moments, int cap, double *z )
{
    using Lay = FxLayout<M>;
    static State<M> st;
    for ( int i = 0, o = 0; i < M; ++i )
        for ( int j = i; j < M; ++j, ++o )
            st.a( i == j ? Lay::diag( i ) : Lay::pair( i, j ) ) = moments[o];
    // (fx_jacobi hands back what fx_load refuses)
    int const n = fx_jacobi<M>( st, cap, fx_load<M>( st, true ) );
    if ( n < 0 )
        return false;
    for ( int k = 0; k < M; ++k )
        z[k] = st.w( k );
    for ( int r = n - 1; r >= 0; --r )
    {
        int const l = st.ls[r] >> 4, s = st.ls[r] & 15;
        double const X = z[l < s ? l : s], Y = z[l < s ? s : l];
        z[l] = st.c[r] * X - st.sn[r] * Y;
        z[s] = st.sn[r] * X + st.c[r] * Y;
    }
    return true;
}

} // namespace

// moments: count x m (m + 1) / 2 (upper triangle, row-major); out: count x m;
// handed_back[i] = 1 where the form does not take the matrix.
extern "C" void fixed_row0( int m, long count, double const *moments, int cap, double *out, int *handed_back )
{
    for ( long i = 0; i < count; ++i )
    {
        double const *a = moments + i * ( m * ( m + 1 ) / 2 );
        double *z = out + i * m;
        handed_back[i] = ( m == 10 ? row0<10>( a, cap, z ) : row0<4>( a, cap, z ) ) ? 0 : 1;
    }
}
