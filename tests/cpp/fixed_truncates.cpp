// The early truncation test of the fixed-point Jacobi (datatransferkit_gb300/
// csrc/dtk_fixed.cuh), built for the host.  Built and driven by
// tests/test_fixed_truncation_cpu.py.
#define __host__
#define __device__
#define __forceinline__ inline
#define __noinline__ __attribute__( ( noinline ) )
#include "dtk_fixed.cuh"

#include <cmath>
#include <cstring>

using namespace dtk;

namespace
{

template <int M>
struct State
{
    using Lay = FxLayout<M>;
    mutable double n[Lay::OFF + M];
    mutable int32_t last[Lay::OFF];
    mutable int e[M];
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
    void set_v( int, FxNum<2> const & ) const {}
    int exp( int k ) const { return e[k]; }
    void set_exp( int k, int d ) const { e[k] = d; }
    template <class Fn>
    void for_parts( Fn const &fn ) const
    {
        fn( 0 );
        fn( 1 );
    }
    void sync() const {}
    bool both( bool x ) const { return x; }
};

template <int M>
int truncates( double const *moments )
{
    using Lay = FxLayout<M>;
    static State<M> st;
    for ( int i = 0, o = 0; i < M; ++i )
        for ( int j = i; j < M; ++j, ++o )
            st.a( i == j ? Lay::diag( i ) : Lay::pair( i, j ) ) = moments[o];
    return fx_load<M>( st, true ) ? (int)fx_truncates<M>( st ) : -1;
}

} // namespace

// out[i]: -1 the form does not load the matrix, else the test's answer
extern "C" void fixed_truncates( int m, long count, double const *moments, int *out )
{
    for ( long i = 0; i < count; ++i )
    {
        double const *a = moments + i * ( m * ( m + 1 ) / 2 );
        out[i] = m == 10 ? truncates<10>( a ) : truncates<4>( a );
    }
}
