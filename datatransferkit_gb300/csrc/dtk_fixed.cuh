// The reference's two-sided Jacobi (largest off-diagonal pivot, absolute
// DBL_EPSILON stop, packages/Meshfree/src/DTK_DetailsSVDImpl.hpp:197-302) of
// a positive definite moment matrix on the integer pipes.
//
// GB300 issues one FP64 warp instruction per 64 cycles per SM sub-partition,
// a 32 x 32 -> 64 bit integer multiply-add in 4 to 5, and other integer
// instructions in 2, so 89-bit fixed point is several times faster than FP64.
// The matrix is kept as
//     E(i, j) = F(i, j) 2^(d_i + d_j),  |F(i, j)| < 1,
// F in three digits (a signed leading one of 31 bits, two of 29; the diagonal
// and column 0 of V in two), with a power of two 2^d_i >= sqrt(E(i, i)) per row
// (|E(i, j)|^2 <= E(i, i) E(j, j)): moments of a fine cloud span 2^40 between
// the constant and the quadratic terms, and every row keeps its own 89 bits.
// A rotation multiplies the two rows by four factors of two digits (58 bits
// after the point, below 4) that carry the change of scale; the product of the
// lowest digits is left out.  An FP64 rotation rounds at 2^-53 of its operands;
// this one at 2^-58 of them and at a unit, 2^-89 2^(d_i + d_j), of the result.
// Cosine and sine come from the same angle to 2^-58 whatever the pivot block is
// (the doubles kept of them have c^2 + s^2 = 1 to 3.2e-16 over 7.6M blocks, nearly
// equal diagonal entries and pivots down to the last unit among them).
// (Two digits throughout were a fifth faster, but their unit can be within 2^-12
// of the absolute stop for the entries of the constant term: a few of them on the
// wrong side make one rotation more or less, which moved 1 in 1000 targets by up
// to 1e-8, and running the doubtful ones again, up to 13 in 100, took the gain
// back.)
//
// A matrix whose form does not hold is handed back to the FP64 loop, whose
// truncation decisions rest on its own rounding: a diagonal entry that is not
// positive, scales out of range, a pivot block singular to 2^-22, an eigenvalue
// at the absolute truncation threshold (found before the first rotation for most
// such matrices, at the end for the others), or more rotations than the log
// takes.  Host builds of the same code are tested against the oracle.
#ifndef DTK_FIXED_CUH
#define DTK_FIXED_CUH

#include "dtk_ieee.cuh"

#include <cmath>
#include <cstdint>

namespace dtk
{

constexpr int FX_DIGIT = 29;
constexpr int FX_MASK = ( 1 << FX_DIGIT ) - 1, FX_HALF = 1 << ( FX_DIGIT - 1 );
constexpr int FX_ONE = 60;  // the two leading digits as an integer: 2^60 is 1
constexpr int FX_COEF = 58; // rotation factors: 2^58 is 1
constexpr int FX_V = 54;    // column 0 of V (two digits): 2^54 is 1 at row 0's scale (headroom 64, eight times that after each fx_shrink_v)
constexpr int FX_V_SHRINK = 18; // by how much the unit may grow (rows 2^-18 of row 0's scale)
constexpr int FX_LOG = 224;    // rotations (a quadratic basis takes 113 on a fine cloud, up to 183 at unit spacing)
constexpr int FX_NOISE = 16;   // off-diagonal entries up to 16 units of the last digit count as zero
constexpr int FX_MAX_EXP = 40; // scales 2^-40 .. 2^40, so that FP32 holds every squared magnitude that decides

// The high 64 bits of a b, at most 2 too small (without the carries of the
// low words): three IMAD.WIDE.
__host__ __device__ __forceinline__ uint64_t fx_mulhi( uint64_t a, uint64_t b )
{
    uint32_t const a0 = (uint32_t)a, a1 = (uint32_t)( a >> 32 ), b0 = (uint32_t)b, b1 = (uint32_t)( b >> 32 );
    return (uint64_t)a1 * b1 + ( (uint64_t)a1 * b0 >> 32 ) + ( (uint64_t)a0 * b1 >> 32 );
}
__host__ __device__ __forceinline__ int fx_clz( uint64_t a )
{
#ifdef __CUDA_ARCH__
    return __clzll( (long long)a );
#else
    return a ? __builtin_clzll( a ) : 64;
#endif
}
__host__ __device__ __forceinline__ float fx_rsqrt( float x )
{
#ifdef __CUDA_ARCH__
    return rsqrtf( x );
#else
    return 1.0f / std::sqrt( x );
#endif
}
__host__ __device__ __forceinline__ float fx_fma( float a, float b, float c )
{
#ifdef __CUDA_ARCH__
    return __fmaf_rn( a, b, c );
#else
    return std::fma( a, b, c );
#endif
}
__host__ __device__ __forceinline__ int fx_float_bits( float x )
{
#ifdef __CUDA_ARCH__
    return __float_as_int( x );
#else
    int b;
    std::memcpy( &b, &x, sizeof b );
    return b;
#endif
}
__host__ __device__ __forceinline__ float fx_bits_float( int b )
{
#ifdef __CUDA_ARCH__
    return __int_as_float( b );
#else
    float x;
    std::memcpy( &x, &b, sizeof x );
    return x;
#endif
}
// a * b + c, one IMAD.WIDE
__host__ __device__ __forceinline__ int64_t fx_mad( int32_t a, int32_t b, int64_t c )
{
    return (int64_t)a * b + c;
}
// 2^e for |e| <= 126
__host__ __device__ __forceinline__ float fx_pow2( int e )
{
    return fx_bits_float( ( e + 127 ) << 23 );
}
// x >> n, 0 for n >= 64 (n >= 0)
__host__ __device__ __forceinline__ uint64_t fx_shr( uint64_t x, int n )
{
#ifdef __CUDA_ARCH__
    uint64_t r; // PTX clamps the shift amount
    asm( "shr.u64 %0, %1, %2;" : "=l"( r ) : "l"( x ), "r"( n ) );
    return r;
#else
    return n < 64 ? x >> n : 0;
#endif
}
// x >> n rounded to nearest (n >= 1)
__host__ __device__ __forceinline__ uint64_t fx_shr_round( uint64_t x, int n )
{
    return ( fx_shr( x, n - 1 ) + 1 ) >> 1;
}

// sign * m 2^e as a double (m > 0, truncated to 53 bits; the result normal)
__host__ __device__ __forceinline__ double fx_double( uint64_t m, int e, bool negative )
{
    int const z = fx_clz( m );
    uint64_t const t = ( m << z ) >> 11; // 2^52 <= t < 2^53
    return of_bits( ( negative ? SIGN_BIT : 0 ) + ( (uint64_t)( e + 63 - z + 1022 ) << 52 ) + t );
}

// 1 / sqrt(r) of r = rho / 2^64, rho in [2^62, 2^64): in (1, 2], 2^62 is 1.
// An FP32 seed (relative error below 2^-20) and one step of the third-order
// iteration g (1 + e/2 + 3 e^2 / 8), e = 1 - r g^2 (error 5 e^3 / 16).
__host__ __device__ __forceinline__ uint64_t fx_inv_sqrt( uint64_t rho )
{
    float const f = (float)(uint32_t)( rho >> 32 );       // in [2^30, 2^32]
    uint32_t const g = (uint32_t)( fx_rsqrt( f ) * 70368744177664.f ); // 2^46: g / 2^30 in (1, 2]
    uint64_t const g2 = (uint64_t)g * g;                  // 2^60 is 1
    int64_t const e = (int64_t)( 1ull << 60 ) - (int64_t)fx_mulhi( rho, g2 );
    int32_t const e50 = (int32_t)( e >> 10 );
    int64_t const q = (int64_t)e50 * e50 >> 40;           // e^2, 2^60 is 1
    int64_t const c = ( e >> 1 ) + ( 3 * q >> 3 );        // 2^60 is 1, |c| < 2^40
    // g c: 32 x 41 bits, 2^90 is 1
    uint32_t const c0 = (uint32_t)c;
    int32_t const c1 = (int32_t)( c >> 32 );
    int64_t const gc = (int64_t)( ( (uint64_t)g * c0 ) >> 28 ) + (int64_t)c1 * (int64_t)(uint64_t)g * 16;
    return (uint64_t)( ( (int64_t)g << 32 ) + gc );
}

// A number of D = 2 or 3 digits: d[0] signed, the others balanced, in [-2^28,
// 2^28), so that a small value of either sign has small digits (its magnitude
// as a float needs no sign handling).
template <int D>
struct FxNum
{
    int32_t d[D];
};
// the balanced low digit of v, and v without it
__host__ __device__ __forceinline__ int32_t fx_low( int64_t v )
{
    return (int32_t)( (uint32_t)v << ( 32 - FX_DIGIT ) ) >> ( 32 - FX_DIGIT );
}
__host__ __device__ __forceinline__ int32_t fx_high( int64_t v )
{
    return (int32_t)( ( v + FX_HALF ) >> FX_DIGIT );
}
// A rotation factor.
struct FxCoef
{
    int32_t hi, lo;
};
__host__ __device__ __forceinline__ FxCoef fx_coef( int64_t v )
{
    return FxCoef{fx_high( v ), fx_low( v )};
}
// the leading 60 bits as an integer (2^60 is 1)
template <int D>
__host__ __device__ __forceinline__ int64_t fx_lead( FxNum<D> const &x )
{
    return ( (int64_t)x.d[0] << FX_DIGIT ) + x.d[1];
}
template <int D>
__host__ __device__ __forceinline__ int32_t fx_last( FxNum<D> const &x )
{
    return D == 3 ? x.d[D - 1] : 0; // the digit below the lead
}
template <int D>
__host__ __device__ __forceinline__ FxNum<D> fx_num( int64_t lead, int32_t last = 0 )
{
    FxNum<D> x;
    x.d[0] = fx_high( lead );
    x.d[1] = fx_low( lead );
    if constexpr ( D == 3 )
        x.d[2] = last;
    return x;
}
// a x + b y, rounded (without the product of the lowest digits, below half a
// unit each): six (D = 2) or ten IMAD.WIDE.  Each column carries FX_HALF into
// the next, so that a digit is its low 29 bits less FX_HALF; the constant 2^57
// in a column is that carry.  fits: the result is within the leading digit.
template <int D>
__host__ __device__ __forceinline__ FxNum<D> fx_dot( FxCoef a, FxNum<D> const &x, FxCoef b, FxNum<D> const &y,
                                                     bool &fits )
{
    constexpr int64_t HALF = FX_HALF, CARRY = (int64_t)FX_HALF << FX_DIGIT;
    int64_t low = HALF + CARRY;
    if constexpr ( D == 3 )
        low = ( fx_mad( b.lo, y.d[1],
                        fx_mad( b.hi, y.d[2], fx_mad( a.lo, x.d[1], fx_mad( a.hi, x.d[2], low ) ) ) ) >>
                FX_DIGIT ) +
              CARRY;
    int64_t const m =
        fx_mad( b.lo, y.d[0], fx_mad( b.hi, y.d[1], fx_mad( a.lo, x.d[0], fx_mad( a.hi, x.d[1], low ) ) ) );
    int64_t const h = fx_mad( b.hi, y.d[0], fx_mad( a.hi, x.d[0], m >> FX_DIGIT ) );
    fits = ( h >> FX_ONE ) == ( h >> 63 );
    FxNum<D> r;
    r.d[0] = (int32_t)( h >> FX_DIGIT );
    r.d[1] = ( (int32_t)h & FX_MASK ) - FX_HALF;
    if constexpr ( D == 3 )
        r.d[2] = ( (int32_t)m & FX_MASK ) - FX_HALF;
    return r;
}
// x as a float in units of its last digit (relative error below 2^-22)
template <int D>
__host__ __device__ __forceinline__ float fx_float( FxNum<D> const &x )
{
    float f = (float)x.d[0];
#pragma unroll
    for ( int k = 1; k < D; ++k )
        f = fx_fma( f, 536870912.f, (float)x.d[k] ); // 2^29
    return f;
}
template <int D>
__host__ __device__ __forceinline__ bool fx_zero( FxNum<D> const &x )
{
    return ( x.d[0] | x.d[1] | fx_last( x ) ) == 0;
}
// x's magnitude is at most FX_NOISE units of its last digit
__host__ __device__ __forceinline__ bool fx_noise( FxNum<3> const &x )
{
    return ( x.d[0] | x.d[1] ) == 0 && (uint32_t)( x.d[2] + FX_NOISE ) <= 2u * FX_NOISE;
}
// |x| = m 2^(-e - 60) with 2^62 <= m < 2^63 (x not zero; m truncated)
template <int D>
__host__ __device__ __forceinline__ uint64_t fx_normal( FxNum<D> const &x, int &e, bool &negative )
{
    int64_t lead = fx_lead( x );
    int32_t last = fx_last( x );
    negative = lead < 0 || ( lead == 0 && last < 0 );
    if ( negative )
    {
        lead = -lead;
        last = -last;
    }
    if ( D == 3 && lead <= 1 )
    {
        // the last digit leads, or decides whether the 1 above it stays
        uint64_t const v = ( (uint64_t)lead << FX_DIGIT ) + (int64_t)last;
        int const z = fx_clz( v ) - 1;
        e = z + FX_DIGIT;
        return v << ( z & 63 );
    }
    // (a negative last digit below a power of two takes one from its bits)
    lead -= D == 3 && last < 0;
    int const z = fx_clz( (uint64_t)lead ) - 1;
    e = z;
    uint64_t const m = (uint64_t)lead << ( z & 63 );
    if constexpr ( D == 2 )
        return m;
    last &= FX_MASK;
    // as many of the last digit's bits as fit below the lead's
    return m + ( z >= FX_DIGIT ? (uint64_t)last << ( ( z - FX_DIGIT ) & 63 )
                               : (uint64_t)( last >> ( ( FX_DIGIT - z ) & 31 ) ) );
}

// The rotation of one pivot block: the row with the larger diagonal entry is
// "L", the other "S".  In the rows' scales the new rows are
//     X = cx F(L, .) + sx F(S, .)   (the larger eigenvalue, at exponent dl)
//     Y = cy F(S, .) - sy F(L, .)   (the smaller, at exponent ds)
// and c, s the rotation itself as doubles (s with the sign of the pivot).
struct FxRotation
{
    FxCoef cx, sx, cy, sy_neg;
    int64_t fl, fs; // the new diagonal entries
    int dl, ds;     // the new exponents
    double c, s;
    bool ok;
};

// fl, fs: diagonal entries of L and S (exponents dl, ds); the pivot is +-bm
// 2^(-zb - 60), 2^62 <= bm < 2^63.  E(L, L) >= E(S, S) > 0.
//
// cos 2t = (a - d) / r, sin 2t = 2 b / r, r^2 = (a - d)^2 + 4 b^2, the angle
// of the reference's 2x2 SVD of a positive definite block (atan2(2b(a + d),
// a^2 - d^2) / 2); c = sqrt((1 + cos 2t) / 2), s = sin 2t / (2 c), tan t = s /
// c, and the eigenvalues a + b tan t, d - b tan t.
__host__ __device__ __forceinline__ FxRotation fx_rotation( int64_t fl, int64_t fs, uint64_t bm, int zb, bool negative,
                                                           int dl, int ds )
{
    FxRotation r;
    int const u = dl > ds ? dl : ds; // common unit 2^(2u - 60)
    int const hl = u - dl, hs = u - ds;
    uint64_t const x0 = fx_shr( (uint64_t)fl, 2 * hl ) - fx_shr( (uint64_t)fs, 2 * hs );
    int const sh = zb + hl + hs; // 2 |b| = (bm << 1) 2^-sh
    // x0 and 2 |b| scaled by 2^z, below 2^63 with the larger one's leading bit
    // there.  2 |b| comes from bm, not from its whole units: with a difference
    // of a few units (nearly equal diagonal entries, as grids give them) what
    // is cut off there is the angle, and c and s no longer belong together.
    int const zx = fx_clz( x0 ) - 1;
    int const z = x0 && zx < sh - 1 ? zx : sh - 1;
    uint64_t const x = x0 ? x0 << ( z & 63 ) : 0, y = fx_shr( bm << 1, sh - z );
    uint64_t const r2 = fx_mulhi( x, x ) + fx_mulhi( y, y ); // about [2^60, 2^63)
    int const h = r2 < ( 1ull << 62 ) ? 1 : 0;               // sqrt of the scaling
    uint64_t const g = fx_inv_sqrt( r2 << ( 2 * h ) );       // 2^64 / r = g 2^h / 2^62
    uint64_t cos2 = fx_mulhi( x, g ) << h;                   // 2^62 is 1
    cos2 = cos2 > ( 1ull << 62 ) - 1 ? ( 1ull << 62 ) - 1 : cos2;
    uint64_t const half = ( ( 1ull << 62 ) + cos2 ) << 1; // (1 + cos 2t) / 2, 2^64 is 1
    uint64_t const t = fx_inv_sqrt( half );               // 1 / c, 2^62 is 1
    uint64_t c = fx_mulhi( half, t );                     // 2^62 is 1
    c = c > ( 1ull << 62 ) - 8 ? ( 1ull << 62 ) - 8 : c;
    // s with its own exponent: |s| = q 2^es
    uint64_t const q = fx_mulhi( fx_mulhi( bm, g ) << 1, t ); // [2^59, 2^62)
    int const es = z + 1 - hl - hs - zb + h - 62;
    // tan t = s / c = s t = w 2^(es + 1); |b| tan t = bm 2^-zb w 2^(es + 1) in
    // units of 2^(dl + ds): 2^(dl - ds) more of S's unit, as much less of L's
    uint64_t const w = fx_mulhi( q << 1, t );
    uint64_t const v = fx_mulhi( bm, w ) << 4; // [2^60, 2^64)
    int const kk = dl - ds, nv = zb - es - 61;
    int64_t ns = fs - (int64_t)fx_shr( v, nv - kk ), nl = fl + (int64_t)fx_shr( v, nv + kk );
    bool ok = z >= 0 && nv >= kk && nv >= -kk && ns > ( fs >> 22 ) && ns > ( int64_t( 1 ) << 30 );
    // the scales follow the new diagonal
    int const dl0 = dl, ds0 = ds;
    if ( nl >= ( int64_t( 1 ) << FX_ONE ) )
    {
        nl >>= 2;
        ++dl;
    }
    if ( dl < ds - 1 )
    {
        nl = (int64_t)fx_shr( (uint64_t)nl, 2 * ( ds - 1 - dl ) );
        dl = ds - 1;
    }
    // |s| 2^(dl0 - ds) must stay below 4 (2^58 is 1; q < 2^62)
    int ny = ds - dl0 - es - FX_COEF + 2;
    ok = ok && ny >= 1;
    if ( ns <= ( int64_t( 1 ) << ( FX_ONE - 2 ) ) && fx_shr( q << 2, ny ) < ( 3ull << ( FX_COEF - 1 ) ) && ny >= 2 )
    {
        ns <<= 2;
        --ds;
        --ny;
    }
    int const nx = dl - ds0 - es - FX_COEF + 2;
    int64_t const sy = (int64_t)fx_shr_round( q << 2, ny );
    int64_t const sx = (int64_t)fx_shr_round( q << 2, nx );
    r.ok = ok && nx >= 1 && sy < ( int64_t( 1 ) << 60 ) && sx < ( int64_t( 1 ) << 60 ) && dl <= FX_MAX_EXP &&
           ds >= -FX_MAX_EXP;
    r.cx = fx_coef( (int64_t)fx_shr_round( c, 62 - FX_COEF - dl0 + dl ) );
    r.cy = fx_coef( (int64_t)fx_shr_round( c, 62 - FX_COEF - ds0 + ds ) );
    r.sx = fx_coef( negative ? -sx : sx );
    r.sy_neg = fx_coef( negative ? sy : -sy );
    r.fl = nl;
    r.fs = ns;
    r.dl = dl;
    r.ds = ds;
    r.c = fx_double( c, -62, false );
    r.s = fx_double( q, es, negative );
    return r;
}

// Where the entries lie: pair {i, i + d mod M} with d = 1 .. M/2 in slot
// (d - 1) M + i (d = M/2: i < M/2 only), so that the two halves of a scan (part
// h: the rows i = M/2 h + r) run the same code, on one lane after the other or
// on two lanes; as doubles, before fx_load, the diagonal follows.
template <int M>
struct FxLayout
{
    static_assert( M % 2 == 0, "two halves of the rows" );
    static constexpr int HALF = M / 2;
    static constexpr int OFF = M * ( M - 1 ) / 2; // off-diagonal slots
    static constexpr int MID = ( HALF + 1 ) / 2;  // a part's share of the last distance
    __host__ __device__ __forceinline__ static int diag( int i ) { return OFF + i; }
    __host__ __device__ __forceinline__ static int pair( int i, int j )
    {
        int d = j - i;
        d += d < 0 ? M : 0;
        bool const flip = d > HALF || ( d == HALF && i >= HALF );
        return ( ( flip ? M - d : d ) - 1 ) * M + ( flip ? j : i );
    }
    // the slots of {p, j} and {q, j}, j the t-th index past p and q
    __host__ __device__ __forceinline__ static void column( int p, int q, int t, int &up, int &uq )
    {
        int j = t;
        j += j >= p;
        j += j >= q;
        up = pair( p, j );
        uq = pair( q, j );
    }
    // the pair of a slot, p < q
    __host__ __device__ __forceinline__ static void of_slot( int u, int &p, int &q )
    {
        int const d = u / M, i = u - d * M;
        int j = i + d + 1;
        j -= j >= M ? M : 0;
        p = i < j ? i : j;
        q = i < j ? j : i;
    }
};

// The state of one matrix behind accessors: a(u) an entry as a double (before
// fx_load); then f(u) / set_f(u, x) the off-diagonal numbers, diag(k) /
// set_diag(k, x) the diagonal's leads, v(k) / set_v(k, x) column 0 of V and, at
// the end and in its place, w(k) = V(k) / E(k, k); exp(k) / set_exp(k, d) the
// rows' exponents; column(u, p, q, t, up, uq) is FxLayout's, u being the slot of
// {p, q}; log(r, c, s, ls) rotation r: ls = 16 L + S, the rows before
// it (the new rows are min(L, S) = X, max(L, S) = Y).  for_parts(fn) runs fn(h)
// for the parts of this lane; merge(k1, k2, sum) combines a scan with the
// other lane's; both(x) is x of all the matrix's lanes; sync() orders their
// accesses.

// the scale of row exponent d as a float: fx_float( F(i, j) ) fx_scale( d_i )
// fx_scale( d_j ) is E(i, j) times 2^29
__host__ __device__ __forceinline__ float fx_scale( int d )
{
    return fx_pow2( d - 30 );
}
constexpr float FX_UNIT = 536870912.f;

// Converts E to F, in place, and sets the exponents and V; false when a
// diagonal entry is not positive or out of range, or an entry is above its
// bound.  (Loops kept rolled: this runs once a matrix, and the kernels' loops
// compete for the instruction cache.)  All lanes of the warp together.
template <int M, class State>
__host__ __device__ __forceinline__ bool fx_load( State const &st, bool live )
{
    using Lay = FxLayout<M>;
    bool ok = live;
    st.for_parts( [&]( int h ) {
#pragma unroll 1
        for ( int k = h; k < M; k += 2 )
        {
            uint64_t const b = bits_of( st.a( Lay::diag( k ) ) );
            int const e = (int)( b >> 52 ) - 1023; // a negative entry gives e > 1024
            // E(k, k) < 2^(e + 1) <= 2^(2 d)
            int const d = ( e + 2 ) >> 1;
            bool const in = d >= -FX_MAX_EXP && d <= FX_MAX_EXP - 4;
            ok = ok && in;
            st.set_exp( k, in ? d : 0 );
            st.set_v( k, fx_num<2>( k == 0 ? int64_t( 1 ) << FX_V : 0 ) );
        }
    } );
    st.sync();
    st.for_parts( [&]( int h ) {
#pragma unroll 1
        for ( int u = h; u < Lay::OFF + M; u += 2 )
        {
            int p = u - Lay::OFF, q = p;
            if ( u < Lay::OFF )
                Lay::of_slot( u, p, q );
            int const d = st.exp( p ) + st.exp( q );
            uint64_t const bits = bits_of( st.a( u ) );
            int const e = (int)( ( bits >> 52 ) & 0x7ff ) - 1023;
            // |E(i, j)| <= 2^(d_i + d_j) up to its rounding
            ok = ok && e < d;
            // |F| = m 2^(e - 52 - d): the leading 60 bits and the 29 below
            uint64_t const m = e > -1023 && ok ? ( bits & 0xfffffffffffffull ) | 0x10000000000000ull : 0;
            int const n = d - e - 8; // lead = m 2^-n
            int64_t lead = (int64_t)( n >= 0 ? fx_shr( m, n ) : m << ( -n & 63 ) );
            int32_t low = n > 0 ? (int32_t)( n <= FX_DIGIT ? m << ( FX_DIGIT - n ) : fx_shr( m, n - FX_DIGIT ) ) & FX_MASK
                                : 0;
            if ( u >= Lay::OFF )
            {
                st.set_diag( p, lead );
                continue;
            }
            if ( low >= FX_HALF )
            {
                low -= 1 << FX_DIGIT;
                ++lead;
            }
            if ( bits & SIGN_BIT )
            {
                low = -low;
                lead = -lead;
            }
            st.set_f( u, fx_num<3>( lead, low ) );
        }
    } );
    return st.both( ok );
}

constexpr int FX_TRUNCATE = -51; // 2^-51, twice DBL_EPSILON

// Pivots K .. of the LDL^T of a, in units of 2^(d_i + d_j).
template <int M, int K, class State>
__host__ __device__ __forceinline__ void fx_pivots( State const &st, float ( &a )[M][M], bool &truncates )
{
    // (no pivot is taken for smaller than its rounding, 2^-17)
    float const d = a[K][K] > 7.6293945e-6f ? a[K][K] : 7.6293945e-6f;
    // d 2^(2 d_K) < 2^FX_TRUNCATE, with a margin for the FP32 sums
    truncates |= d * 1.125f < fx_pow2( FX_TRUNCATE - 2 * st.exp( K ) );
    if constexpr ( K + 1 < M )
    {
        float const r = 1.0f / d;
#pragma unroll
        for ( int i = K + 1; i < M; ++i )
        {
            float const l = a[K][i] * r;
#pragma unroll
            for ( int j = K + 1; j < M; ++j )
                if ( j >= i )
                    a[i][j] = fx_fma( -l, a[K][j], a[i][j] );
        }
        fx_pivots<M, K + 1>( st, a, truncates );
    }
}

// The smallest eigenvalue is at most the truncation threshold, so that the
// matrix would be handed back at the end: one of the pivots of an LDL^T of F in
// FP32 is (each bounds it from above, as the smallest eigenvalue of a leading
// block does).  Without it clouds of so small a scale paid for both forms: 300k
// quadratic targets in a cube of edge 0.01 took 9.8 ms, now 8.6 (FP64 alone
// 7.4).
template <int M, class State>
__host__ __device__ __forceinline__ bool fx_truncates( State const &st )
{
    using Lay = FxLayout<M>;
    // (a pivot is 2^-17 2^(2 d) at least: most clouds end here)
    bool small = false;
#pragma unroll
    for ( int k = 0; k < M; ++k )
        small |= 2 * st.exp( k ) - 17 < FX_TRUNCATE;
    if ( !small )
        return false;
    float a[M][M]; // the upper triangle, in units of 2^(d_i + d_j)
    bool truncates = false;
#pragma unroll
    for ( int i = 0; i < M; ++i )
    {
        a[i][i] = (float)(int32_t)( st.diag( i ) >> 30 ) * 9.3132257e-10f; // 2^-30
#pragma unroll
        for ( int j = 1; j < M; ++j )
            if ( j > i )
                a[i][j] = fx_float( st.f( Lay::pair( i, j ) ) ) * 1.6155871e-27f; // 2^-89
    }
    fx_pivots<M, 0>( st, a, truncates );
    return truncates;
}

// The slot of the largest |E(i, j)|, first in row-major order, compared
// exactly.
template <int M, class State>
__host__ __device__ __noinline__ int fx_exact_pivot( State const st )
{
    int be = -10000, best = 0;
    uint64_t bm = 0;
#pragma unroll 1
    for ( int i = 0; i < M; ++i )
#pragma unroll 1
        for ( int j = i + 1; j < M; ++j )
        {
            int const u = FxLayout<M>::pair( i, j );
            auto const f = st.f( u );
            if ( fx_zero( f ) )
                continue;
            int z;
            bool negative;
            uint64_t const m = fx_normal( f, z, negative );
            int const e = st.exp( i ) + st.exp( j ) - z;
            if ( e > be || ( e == be && m > bm ) )
            {
                be = e;
                bm = m;
                best = u;
            }
        }
    return best;
}

// sqrt(sum over i != j of E(i, j)^2) > DBL_EPSILON in FP64
template <int M, class State>
__host__ __device__ __noinline__ bool fx_exact_go( State const st )
{
    double acc = 0.0;
#pragma unroll 1
    for ( int u = 0; u < FxLayout<M>::OFF; ++u )
    {
        auto const f = st.f( u );
        if ( fx_zero( f ) )
            continue;
        int z, p, q;
        bool negative;
        FxLayout<M>::of_slot( u, p, q );
        uint64_t const m = fx_normal( f, z, negative );
        double const e = fx_double( m, st.exp( p ) + st.exp( q ) - z - FX_ONE, false );
        acc += e * e;
    }
    return sqrt( 2.0 * acc ) > 2.220446049250313e-16;
}

// V in units eight times as large (an entry outgrew its leading digit: rows
// whose scale is far below row 0's; 10 of 600k matrices of 20 neighbours, 58
// of 100k of 15, and one matrix left to the FP64 kernel takes its 1 ms).
template <int M, class State>
__host__ __device__ __forceinline__ void fx_shrink_v( State const &st )
{
#pragma unroll 1
    for ( int k = 0; k < M; ++k )
    {
        FxNum<2> const v = st.v( k );
        int64_t const x = ( (int64_t)v.d[0] * ( int64_t( 1 ) << FX_DIGIT ) ) + v.d[1];
        st.set_v( k, fx_num<2>( ( x + 4 ) >> 3 ) );
    }
}

// Runs the Jacobi on the state (live: this lane's matrix takes part), all
// lanes of the warp together; returns the rotations made, or -1 when the
// matrix is handed back.
template <int M, class State>
__host__ __device__ __forceinline__ int fx_jacobi( State const &st, int cap, bool live )
{
    using Lay = FxLayout<M>;
    live = live && !fx_truncates<M>( st );
    int const d0 = live ? st.exp( 0 ) : 0; // V's unit
    int fv = FX_V;                         // 2^fv is 1 in it
    int it = 0;
    bool ok = live;
    while ( st.any( live ) )
    {
        // the two largest |E(i, j)| and the sum of the squares: FP32
        // magnitudes with the slot in their low bits
        int k1 = 0, k2 = 0;
        float sum = 0.f;
        if ( live )
            st.for_parts( [&]( int h ) {
                auto visit = [&]( int u, float si, float sj, bool mine ) {
                    float const m = mine ? fx_float( st.f( u ) ) * si * sj : 0.f;
                    sum = fx_fma( m, m, sum );
                    int const key = ( fx_float_bits( m ) & 0x7fffffc0 ) | u;
                    int const lo = k1 < key ? k1 : key;
                    k2 = k2 > lo ? k2 : lo;
                    k1 = k1 > key ? k1 : key;
                };
                float sc[M - 1];
                int const i0 = Lay::HALF * h;
#pragma unroll
                for ( int r = 0; r < M - 1; ++r )
                {
                    int const i = i0 + r;
                    sc[r] = fx_scale( st.exp( i >= M ? i - M : i ) );
                }
#pragma unroll
                for ( int d = 1; d < Lay::HALF; ++d )
#pragma unroll
                    for ( int r = 0; r < Lay::HALF; ++r )
                        visit( ( d - 1 ) * M + i0 + r, sc[r], sc[r + d], true );
#pragma unroll
                for ( int r = 0; r < Lay::MID; ++r )
                {
                    int const i = Lay::MID * h + r;
                    bool const mine = i < Lay::HALF;
                    visit( ( Lay::HALF - 1 ) * M + i, fx_scale( st.exp( i ) ),
                           fx_scale( st.exp( mine ? i + Lay::HALF : i ) ), mine );
                }
            } );
        st.merge( k1, k2, sum );
        // sqrt(sum over i != j) > DBL_EPSILON: 2 sum against 2^-104, in m's
        // unit; within the FP32 error of the threshold, in FP64
        constexpr float tol2 = 2.465190328815662e-32f * FX_UNIT * FX_UNIT; // 2^-105
        bool go = live && sum > tol2;
        if ( live && sum > tol2 * 0.9990234375f && sum < tol2 * 1.0009765625f )
            go = fx_exact_go<M>( st );
        // two magnitudes within the FP32 error: the exact order
        int u = k1 & 63;
        if ( go && ( k1 >> 6 ) - ( k2 >> 6 ) <= 4 )
            u = fx_exact_pivot<M>( st );
        int p, q;
        Lay::of_slot( u, p, q );
        FxNum<3> const fpq = st.f( u );
        // (the largest entry is this form's rounding: made zero below)
        bool const noise = go && fx_noise( fpq );
        if ( live && !noise && ( !go || it == cap ) )
        {
            ok = !go;
            live = go = false;
        }
        bool const turn = go && !noise;
        it += turn;
        int const dp = st.exp( p ), dq = st.exp( q );
        int64_t const fpp = st.diag( p ), fqq = st.diag( q );
        st.sync(); // both lanes have read what the rotation writes
        if ( turn )
        {
            // L: the row of the larger diagonal entry (p on ties); it becomes row p
            int const k = dp - dq;
            bool const swap = k >= 0 ? (uint64_t)fpp < fx_shr( (uint64_t)fqq, 2 * k )
                                     : fx_shr( (uint64_t)fpp, -2 * k ) < (uint64_t)fqq;
            int zb;
            bool negative;
            uint64_t const bm = fx_normal( fpq, zb, negative );
            FxRotation const r = fx_rotation( swap ? fqq : fpp, swap ? fpp : fqq, bm, zb, negative, swap ? dq : dp,
                                              swap ? dp : dq );
            bool fits = true;
            st.for_parts( [&]( int h ) {
                // the rows' other columns, every second one: all loads first
                constexpr int N = Lay::HALF - 1;
                FxNum<3> fl[N], fs[N];
                int up[N], uq[N];
#pragma unroll
                for ( int t = 0; t < N; ++t )
                {
                    st.column( u, p, q, 2 * t + h, up[t], uq[t] );
                    fl[t] = st.f( swap ? uq[t] : up[t] );
                    fs[t] = st.f( swap ? up[t] : uq[t] );
                }
#pragma unroll
                for ( int t = 0; t < N; ++t )
                {
                    // (the entries of F are bounded by the diagonal)
                    bool fx, fy;
                    st.set_f( up[t], fx_dot( r.cx, fl[t], r.sx, fs[t], fx ) );
                    st.set_f( uq[t], fx_dot( r.cy, fs[t], r.sy_neg, fl[t], fy ) );
                }
                if ( h == 0 )
                {
                    // column 0 of V
                    FxNum<2> a = st.v( swap ? q : p ), b = st.v( swap ? p : q );
                    bool fx, fy;
                    FxNum<2> vp = fx_dot( r.cx, a, r.sx, b, fx ), vq = fx_dot( r.cy, b, r.sy_neg, a, fy );
                    while ( !( fx && fy ) && fv > FX_V - FX_V_SHRINK )
                    {
                        fx_shrink_v<M>( st );
                        fv -= 3;
                        a = st.v( swap ? q : p );
                        b = st.v( swap ? p : q );
                        vp = fx_dot( r.cx, a, r.sx, b, fx );
                        vq = fx_dot( r.cy, b, r.sy_neg, a, fy );
                    }
                    st.set_v( p, vp );
                    st.set_v( q, vq );
                    fits = fx && fy;
                }
                else
                {
                    st.set_diag( p, r.fl );
                    st.set_diag( q, r.fs );
                    st.set_f( u, fx_num<3>( 0 ) );
                    st.set_exp( p, r.dl );
                    st.set_exp( q, r.ds );
                    st.log( it - 1, r.c, r.s, swap ? q * 16 + p : p * 16 + q );
                }
            } );
            live = ok = r.ok && fits;
        }
        else if ( noise )
        {
            // nothing is left when the whole matrix is rounding
            live = !fx_zero( fpq );
            st.set_f( u, fx_num<3>( 0 ) );
        }
        live = st.both( live || !turn ) && live;
        ok = turn ? live : ok;
        st.sync();
    }
    {
        // (the lane that turned V knows its unit)
        int shrunk = FX_V - fv, none = 0;
        float zero = 0.f;
        st.merge( shrunk, none, zero );
        fv = FX_V - shrunk;
    }
    // w_k = v_k / E(k, k)
    st.for_parts( [&]( int h ) {
#pragma unroll 1
        for ( int k = h; ok && k < M; k += 2 )
        {
            int const d = st.exp( k );
            int64_t const f = st.diag( k );
            FxNum<2> const v = st.v( k );
            // E(k, k) at least twice the truncation threshold
            ok = f > 0 && 63 - fx_clz( (uint64_t)f ) + 2 * d - FX_ONE >= FX_TRUNCATE;
            double w = 0.0;
            if ( ok && !fx_zero( v ) )
            {
                int z;
                bool negative;
                uint64_t const m = fx_normal( v, z, negative );
                w = fx_double( m, d - d0 - z - fv, negative ) / fx_double( (uint64_t)f, 2 * d - FX_ONE, false );
            }
            st.w( k ) = w;
        }
    } );
    return st.both( ok ) ? it : -1;
}

} // namespace dtk

#endif
