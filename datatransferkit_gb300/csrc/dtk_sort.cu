// Device-wide exclusive scan and stable LSD radix sort (no CUB).
//
// Radix sort: 8-bit digits.  What bounds it below a few million points is the
// chain of short kernels and, inside them, of barriers, not the bytes:
//  * up to 16k pairs one block sorts everything in shared memory, one launch
//    for all digits (a create at 1k points 563 -> 417 us, at 10k 1228 -> 1043
//    us against five launches a digit; 16 pairs a thread is what the block's
//    registers and 160 KB of shared memory hold), with as many pairs a thread
//    as n needs, two at a time (10k pairs, 30 bits: 16 pairs 56 us, 10 47);
//  * beyond, a pass is a per-tile histogram and a stable scatter.  Every warp
//    ranks its own run of the tile against its own counts (__match_any_sync
//    for the lanes, a shared-memory count per digit and warp for the rounds),
//    so a tile takes a handful of barriers in place of four a round; the tile
//    is then reordered by digit in shared memory and written out in digit runs;
//  * up to 128 tiles the scatter sums the tiles' histograms itself (each block
//    reads up to 128 KB of them from L2, under the 13 us of the three scan
//    launches; a create at 100k points 1.25 -> 1.13 ms), beyond that a
//    device-wide scan of the (digit, tile) table runs in between.
#include "dtk_common.cuh"

#include <algorithm>
#include <utility>

namespace dtk
{
namespace
{

constexpr int SCAN_THREADS = 256;
constexpr int SCAN_ITEMS = 8;
constexpr int SCAN_TILE = SCAN_THREADS * SCAN_ITEMS;

template <class T>
__device__ T block_exclusive_scan( T v, T *s_warp, T &total )
{
    int const lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    T incl = v;
#pragma unroll
    for ( int o = 1; o < 32; o <<= 1 )
    {
        T n = __shfl_up_sync( 0xffffffffu, incl, o );
        if ( lane >= o )
            incl += n;
    }
    if ( lane == 31 )
        s_warp[warp] = incl;
    __syncthreads();
    if ( warp == 0 )
    {
        T w = lane < ( SCAN_THREADS / 32 ) ? s_warp[lane] : T( 0 );
        T wi = w;
#pragma unroll
        for ( int o = 1; o < 32; o <<= 1 )
        {
            T n = __shfl_up_sync( 0xffffffffu, wi, o );
            if ( lane >= o )
                wi += n;
        }
        if ( lane < ( SCAN_THREADS / 32 ) )
            s_warp[lane] = wi - w;
        if ( lane == ( SCAN_THREADS / 32 ) - 1 )
            s_warp[SCAN_THREADS / 32] = wi;
    }
    __syncthreads();
    T const res = s_warp[warp] + incl - v;
    total = s_warp[SCAN_THREADS / 32];
    __syncthreads();
    return res;
}

__global__ void __launch_bounds__( SCAN_THREADS )
    k_tile_reduce( int64_t const *in, int64_t n, int64_t *tile_sums )
{
    __shared__ int64_t s_warp[SCAN_THREADS / 32 + 1];
    int64_t const base = (int64_t)blockIdx.x * SCAN_TILE + threadIdx.x * SCAN_ITEMS;
    int64_t acc = 0;
#pragma unroll
    for ( int i = 0; i < SCAN_ITEMS; ++i )
        if ( base + i < n )
            acc += in[base + i];
    int64_t total;
    block_exclusive_scan<int64_t>( acc, s_warp, total );
    if ( threadIdx.x == 0 )
        tile_sums[blockIdx.x] = total;
}

// Single block: exclusive scan of the tile sums in place, with carry.
__global__ void __launch_bounds__( SCAN_THREADS )
    k_scan_tile_sums( int64_t *sums, int64_t n_tiles, int64_t *grand_total )
{
    __shared__ int64_t s_warp[SCAN_THREADS / 32 + 1];
    int64_t carry = 0;
    for ( int64_t b = 0; b < n_tiles; b += SCAN_THREADS )
    {
        int64_t const i = b + threadIdx.x;
        int64_t const v = i < n_tiles ? sums[i] : 0;
        int64_t total;
        int64_t const ex = block_exclusive_scan<int64_t>( v, s_warp, total );
        if ( i < n_tiles )
            sums[i] = carry + ex;
        carry += total;
    }
    if ( threadIdx.x == 0 )
        *grand_total = carry;
}

__global__ void __launch_bounds__( SCAN_THREADS )
    k_tile_scan( int64_t const *in, int64_t *out, int64_t n, int64_t const *tile_offsets )
{
    __shared__ int64_t s_warp[SCAN_THREADS / 32 + 1];
    int64_t const base = (int64_t)blockIdx.x * SCAN_TILE + threadIdx.x * SCAN_ITEMS;
    int64_t vals[SCAN_ITEMS];
    int64_t acc = 0;
#pragma unroll
    for ( int i = 0; i < SCAN_ITEMS; ++i )
    {
        vals[i] = base + i < n ? in[base + i] : 0;
        acc += vals[i];
    }
    int64_t total;
    int64_t run = block_exclusive_scan<int64_t>( acc, s_warp, total ) + tile_offsets[blockIdx.x];
#pragma unroll
    for ( int i = 0; i < SCAN_ITEMS; ++i )
    {
        if ( base + i < n )
            out[base + i] = run;
        run += vals[i];
    }
}

// One block: the whole scan of a short array, SCAN_ONE_TILE values a round
// (three launches of about 4 us each are mostly their latency: 12 -> 4 us at 1k
// values, 13 -> 11 at 10k, two scans a tree).
constexpr int SCAN_ONE_THREADS = 1024;
constexpr int SCAN_ONE_TILE = SCAN_ONE_THREADS * SCAN_ITEMS;
constexpr int64_t SCAN_ONE_MAX = 2 * SCAN_ONE_TILE;

__global__ void __launch_bounds__( SCAN_ONE_THREADS )
    k_scan_one( int64_t const *in, int64_t *out, int64_t n )
{
    __shared__ int64_t s_warp[SCAN_ONE_THREADS / 32];
    int const lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    int64_t carry = 0;
    for ( int64_t t = 0; t < n; t += SCAN_ONE_TILE )
    {
        int64_t const base = t + (int64_t)threadIdx.x * SCAN_ITEMS;
        int64_t v[SCAN_ITEMS], sum = 0;
#pragma unroll
        for ( int i = 0; i < SCAN_ITEMS; ++i )
        {
            v[i] = base + i < n ? in[base + i] : 0;
            sum += v[i];
        }
        int64_t incl = sum;
#pragma unroll
        for ( int o = 1; o < 32; o <<= 1 )
        {
            int64_t const x = __shfl_up_sync( 0xffffffffu, incl, o );
            if ( lane >= o )
                incl += x;
        }
        if ( lane == 31 )
            s_warp[warp] = incl;
        __syncthreads();
        // every warp scans the warps' sums for itself
        int64_t w = s_warp[lane];
#pragma unroll
        for ( int o = 1; o < 32; o <<= 1 )
        {
            int64_t const x = __shfl_up_sync( 0xffffffffu, w, o );
            if ( lane >= o )
                w += x;
        }
        int64_t const total = __shfl_sync( 0xffffffffu, w, 31 );
        int64_t const before = __shfl_sync( 0xffffffffu, w, warp ? warp - 1 : 0 );
        int64_t run = carry + ( warp ? before : 0 ) + incl - sum;
#pragma unroll
        for ( int i = 0; i < SCAN_ITEMS; ++i )
        {
            if ( base + i < n )
                out[base + i] = run;
            run += v[i];
        }
        carry += total;
        __syncthreads();
    }
    if ( threadIdx.x == 0 )
        out[n] = carry;
}

// ---------------------------------------------------------------------------
// Radix sort
// ---------------------------------------------------------------------------
constexpr int RS_THREADS = 256;
constexpr int RS_ROUNDS = 16;
constexpr int RS_TILE = RS_THREADS * RS_ROUNDS;
constexpr int RS_WARPS = RS_THREADS / 32;
constexpr int RS_DIRECT_TILES = 128; // tiles whose histograms the scatter sums itself

// Exclusive scan over 256 values, one a thread of the first 8 warps (s_warp:
// 8 words; two barriers; all threads of the block call it).
__device__ __forceinline__ unsigned scan_digits( unsigned v, unsigned *s_warp )
{
    int const lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    unsigned incl = v;
#pragma unroll
    for ( int o = 1; o < 32; o <<= 1 )
    {
        unsigned const n = __shfl_up_sync( 0xffffffffu, incl, o );
        if ( lane >= o )
            incl += n;
    }
    if ( lane == 31 && warp < 8 )
        s_warp[warp] = incl;
    __syncthreads();
    unsigned pre = incl - v;
    for ( int w = 0; w < warp && w < 8; ++w )
        pre += s_warp[w];
    __syncthreads();
    return pre;
}

// Ranks of a warp's ROUNDS x 32 keys among the equal digits before them in the
// warp, in order (round by round, lane by lane); counts (256 words of the warp,
// zeroed) ends with the warp's digit counts.  Digit 256 marks no key.
template <int ROUNDS>
__device__ __forceinline__ void warp_ranks( unsigned const *digit, unsigned short *rank, unsigned *counts )
{
    unsigned const lt_mask = ( 1u << ( threadIdx.x & 31 ) ) - 1u;
#pragma unroll
    for ( int r = 0; r < ROUNDS; ++r )
    {
        unsigned const peers = __match_any_sync( 0xffffffffu, digit[r] );
        unsigned const before = __popc( peers & lt_mask );
        unsigned const base = digit[r] < 256u ? counts[digit[r]] : 0u;
        __syncwarp();
        if ( before == 0 && digit[r] < 256u )
            counts[digit[r]] = base + __popc( peers );
        __syncwarp();
        rank[r] = (unsigned short)( base + before );
    }
}

// hist: digit-major (digit, tile) as int64 for the scan, or tile-major words
// for the scatter to sum (DIRECT).
template <bool DIRECT>
__global__ void __launch_bounds__( RS_THREADS )
    k_radix_hist( uint32_t const *keys, int64_t n, int shift, int64_t n_tiles,
                  int64_t *hist )
{
    __shared__ unsigned s_hist[256];
    s_hist[threadIdx.x] = 0;
    int64_t const base = (int64_t)blockIdx.x * RS_TILE + threadIdx.x;
    uint32_t key[RS_ROUNDS];
#pragma unroll
    for ( int r = 0; r < RS_ROUNDS; ++r )
        key[r] = base + r * RS_THREADS < n ? keys[base + r * RS_THREADS] : 0u;
    __syncthreads();
#pragma unroll
    for ( int r = 0; r < RS_ROUNDS; ++r )
        if ( base + r * RS_THREADS < n )
            atomicAdd( &s_hist[( key[r] >> shift ) & 255u], 1u );
    __syncthreads();
    if ( DIRECT )
        reinterpret_cast<unsigned *>( hist )[(int64_t)blockIdx.x * 256 + threadIdx.x] = s_hist[threadIdx.x];
    else
        hist[(int64_t)threadIdx.x * n_tiles + blockIdx.x] = s_hist[threadIdx.x];
}

// Stable scatter of one tile (offsets: the scanned table, or with DIRECT the
// tiles' histograms).
template <bool DIRECT>
__global__ void __launch_bounds__( RS_THREADS )
    k_radix_scatter( uint32_t const *keys, uint32_t const *vals, uint32_t *keys_out,
                     uint32_t *vals_out, int64_t n, int shift, int64_t n_tiles,
                     int64_t const *offsets )
{
    __shared__ int64_t s_base[256];      // global position of the tile's first element of each digit
    __shared__ unsigned s_start[256];    // tile position of the first element of each digit
    __shared__ unsigned s_wcount[RS_WARPS][256];
    __shared__ unsigned s_warp[RS_WARPS];
    __shared__ uint32_t s_key[RS_TILE], s_val[RS_TILE];
    int const tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    int64_t const base = (int64_t)blockIdx.x * RS_TILE;
    int64_t const rem = n - base;
    int const count = rem < RS_TILE ? (int)rem : RS_TILE;
    // the warp's run: RS_ROUNDS rows of 32 consecutive keys
    int const first = warp * RS_ROUNDS * 32 + lane;
    uint32_t key[RS_ROUNDS], val[RS_ROUNDS];
#pragma unroll
    for ( int r = 0; r < RS_ROUNDS; ++r )
    {
        bool const valid = first + 32 * r < count;
        key[r] = valid ? keys[base + first + 32 * r] : 0u;
        val[r] = valid ? vals[base + first + 32 * r] : 0u;
    }
#pragma unroll
    for ( int w = 0; w < RS_WARPS; ++w )
        s_wcount[w][tid] = 0;
    if ( DIRECT )
    {
        unsigned const *h = reinterpret_cast<unsigned const *>( offsets ) + tid;
        unsigned before = 0, total = 0;
#pragma unroll 8
        for ( int t = 0; t < n_tiles; ++t )
        {
            unsigned const c = h[256 * t];
            total += c;
            before += t < (int)blockIdx.x ? c : 0u;
        }
        s_base[tid] = scan_digits( total, s_warp ) + before;
    }
    else
        s_base[tid] = offsets[(int64_t)tid * n_tiles + blockIdx.x];
    __syncthreads();
    unsigned digit[RS_ROUNDS];
    unsigned short rank[RS_ROUNDS];
#pragma unroll
    for ( int r = 0; r < RS_ROUNDS; ++r )
        digit[r] = first + 32 * r < count ? ( key[r] >> shift ) & 255u : 256u;
    warp_ranks<RS_ROUNDS>( digit, rank, s_wcount[warp] );
    __syncthreads();
    // each warp's first place of each digit in the tile
    unsigned run = 0;
#pragma unroll
    for ( int w = 0; w < RS_WARPS; ++w )
    {
        unsigned const c = s_wcount[w][tid];
        s_wcount[w][tid] = run;
        run += c;
    }
    unsigned const start = scan_digits( run, s_warp );
    s_start[tid] = start;
#pragma unroll
    for ( int w = 0; w < RS_WARPS; ++w )
        s_wcount[w][tid] += start;
    __syncthreads();
#pragma unroll
    for ( int r = 0; r < RS_ROUNDS; ++r )
        if ( digit[r] < 256u )
        {
            unsigned const pos = s_wcount[warp][digit[r]] + rank[r];
            s_key[pos] = key[r];
            s_val[pos] = val[r];
        }
    __syncthreads();
    for ( int i = tid; i < count; i += RS_THREADS )
    {
        uint32_t const k = s_key[i];
        unsigned const d = ( k >> shift ) & 255u;
        int64_t const pos = s_base[d] + ( i - s_start[d] );
        keys_out[pos] = k;
        vals_out[pos] = s_val[i];
    }
}

// The whole sort of up to RB_THREADS x ROUNDS pairs in one block: the pairs
// stay in registers between the digits and change places through shared
// memory.
constexpr int RB_THREADS = 1024;
constexpr int RB_WARPS = RB_THREADS / 32;
constexpr int RB_MAX_ROUNDS = 16;

template <int ROUNDS>
constexpr size_t block_sort_smem()
{
    return ( (size_t)RB_WARPS * 256 + 8 + 2 * RB_THREADS * ROUNDS ) * sizeof( unsigned );
}

template <int ROUNDS>
__global__ void __launch_bounds__( RB_THREADS )
    k_block_sort( uint32_t *keys, uint32_t *vals, int n, int bits )
{
    extern __shared__ unsigned s_mem[];
    unsigned *const s_count = s_mem, *const s_warp = s_count + RB_WARPS * 256;
    uint32_t *const s_key = s_warp + 8, *const s_val = s_key + RB_THREADS * ROUNDS;
    int const tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    int const first = warp * ROUNDS * 32 + lane;
    unsigned *const mine = s_count + warp * 256;
    for ( int i = tid; i < n; i += RB_THREADS )
    {
        s_key[i] = keys[i];
        s_val[i] = vals[i];
    }
    for ( int shift = 0; shift < bits; shift += 8 )
    {
        __syncthreads();
        uint32_t key[ROUNDS], val[ROUNDS];
        unsigned digit[ROUNDS];
        unsigned short rank[ROUNDS];
#pragma unroll
        for ( int r = 0; r < ROUNDS; ++r )
        {
            int const i = first + 32 * r;
            bool const valid = i < n;
            key[r] = valid ? s_key[i] : 0u;
            val[r] = valid ? s_val[i] : 0u;
            digit[r] = valid ? ( key[r] >> shift ) & 255u : 256u;
        }
#pragma unroll
        for ( int i = 0; i < 8; ++i )
            mine[32 * i + lane] = 0;
        __syncwarp();
        warp_ranks<ROUNDS>( digit, rank, mine );
        __syncthreads();
        unsigned run = 0;
        if ( tid < 256 )
            for ( int w = 0; w < RB_WARPS; ++w )
            {
                unsigned const c = s_count[w * 256 + tid];
                s_count[w * 256 + tid] = run;
                run += c;
            }
        unsigned const start = scan_digits( run, s_warp );
        if ( tid < 256 )
            for ( int w = 0; w < RB_WARPS; ++w )
                s_count[w * 256 + tid] += start;
        __syncthreads();
#pragma unroll
        for ( int r = 0; r < ROUNDS; ++r )
            if ( digit[r] < 256u )
            {
                unsigned const pos = mine[digit[r]] + rank[r];
                s_key[pos] = key[r];
                s_val[pos] = val[r];
            }
    }
    __syncthreads();
    for ( int i = tid; i < n; i += RB_THREADS )
    {
        keys[i] = s_key[i];
        vals[i] = s_val[i];
    }
}

template <int ROUNDS>
void launch_block_sort( uint32_t *keys, uint32_t *values, int64_t n, int bits, cudaStream_t s )
{
    ensure_dynamic_smem( k_block_sort<ROUNDS>, block_sort_smem<ROUNDS>() );
    k_block_sort<ROUNDS><<<1, RB_THREADS, block_sort_smem<ROUNDS>(), s>>>( keys, values, (int)n, bits );
    check_launch( "k_block_sort" );
}

} // namespace

void exclusive_scan_i64( int64_t const *in, int64_t *out, int64_t n, cudaStream_t s )
{
    if ( n <= SCAN_ONE_MAX )
    {
        k_scan_one<<<1, SCAN_ONE_THREADS, 0, s>>>( in, out, n );
        check_launch( "k_scan_one" );
        return;
    }
    int64_t const n_tiles = ( n + SCAN_TILE - 1 ) / SCAN_TILE;
    DeviceBuffer<int64_t> sums( n_tiles + 1, s );
    k_tile_reduce<<<(unsigned)n_tiles, SCAN_THREADS, 0, s>>>( in, n, sums.get() );
    check_launch( "k_tile_reduce" );
    k_scan_tile_sums<<<1, SCAN_THREADS, 0, s>>>( sums.get(), n_tiles, out + n );
    check_launch( "k_scan_tile_sums" );
    k_tile_scan<<<(unsigned)n_tiles, SCAN_THREADS, 0, s>>>( in, out, n, sums.get() );
    check_launch( "k_tile_scan" );
}

void radix_sort_pairs( uint32_t *keys, uint32_t *values, int64_t n, int bits,
                       cudaStream_t s )
{
    if ( n <= 1 || bits <= 0 )
        return;
    if ( n <= RB_THREADS * RB_MAX_ROUNDS )
    {
        switch ( ( n + 2 * RB_THREADS - 1 ) / ( 2 * RB_THREADS ) )
        {
        case 1: launch_block_sort<2>( keys, values, n, bits, s ); break;
        case 2: launch_block_sort<4>( keys, values, n, bits, s ); break;
        case 3: launch_block_sort<6>( keys, values, n, bits, s ); break;
        case 4: launch_block_sort<8>( keys, values, n, bits, s ); break;
        case 5: launch_block_sort<10>( keys, values, n, bits, s ); break;
        case 6: launch_block_sort<12>( keys, values, n, bits, s ); break;
        case 7: launch_block_sort<14>( keys, values, n, bits, s ); break;
        default: launch_block_sort<RB_MAX_ROUNDS>( keys, values, n, bits, s ); break;
        }
        return;
    }
    int64_t const n_tiles = ( n + RS_TILE - 1 ) / RS_TILE;
    bool const direct = n_tiles <= RS_DIRECT_TILES;
    DeviceBuffer<uint32_t> k2( n, s ), v2( n, s );
    DeviceBuffer<int64_t> hist( 256 * n_tiles, s ), offs;
    if ( !direct )
        offs.allocate( 256 * n_tiles + 1, s );
    uint32_t *ka = keys, *va = values, *kb = k2.get(), *vb = v2.get();
    for ( int shift = 0; shift < bits; shift += 8 )
    {
        if ( direct )
        {
            k_radix_hist<true><<<(unsigned)n_tiles, RS_THREADS, 0, s>>>( ka, n, shift, n_tiles, hist.get() );
            check_launch( "k_radix_hist" );
            k_radix_scatter<true><<<(unsigned)n_tiles, RS_THREADS, 0, s>>>( ka, va, kb, vb, n, shift, n_tiles,
                                                                            hist.get() );
        }
        else
        {
            k_radix_hist<false><<<(unsigned)n_tiles, RS_THREADS, 0, s>>>( ka, n, shift, n_tiles, hist.get() );
            check_launch( "k_radix_hist" );
            exclusive_scan_i64( hist.get(), offs.get(), 256 * n_tiles, s );
            k_radix_scatter<false><<<(unsigned)n_tiles, RS_THREADS, 0, s>>>( ka, va, kb, vb, n, shift, n_tiles,
                                                                             offs.get() );
        }
        check_launch( "k_radix_scatter" );
        std::swap( ka, kb );
        std::swap( va, vb );
    }
    if ( ka != keys )
    {
        DTK_CUDA_OR_THROW( cudaMemcpyAsync( keys, ka, n * sizeof( uint32_t ),
                                            cudaMemcpyDeviceToDevice, s ) );
        DTK_CUDA_OR_THROW( cudaMemcpyAsync( values, va, n * sizeof( uint32_t ),
                                            cudaMemcpyDeviceToDevice, s ) );
    }
}

} // namespace dtk
