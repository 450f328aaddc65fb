// ng_owned.cuh -- the min_delay-slice cycle with the targets owned by SMs:
// the ring buffers live in shared memory and a slice costs one exchange of
// its spikes.
//
// The scatter form (k_deliver, k_run_slices) adds every synaptic event to a
// ring cell in global memory: random 64-bit atomics at the L2, about 5e10 a
// second on a B200, and a grid barrier on either side of them.  Here one CTA
// per SM owns every G-th neuron of a network: its threads keep the neurons'
// state in registers and their pending input in shared memory for the whole
// launch, and a copy of the CTA's in-edges, grouped by source, lies in HBM.
// In each slice a CTA
//   1. runs its neurons over the slice's lags (one thread per neuron),
//   2. publishes their spikes to the other CTAs of the network,
//   3. draws the next slice's Poisson drive while they travel,
//   4. collects the network's spikes of the slice and adds the CTA's edges of
//      those sources to its own ring cells (shared-memory atomics).
// No ring cell is written by two SMs, so nothing else has to be ordered and
// step 4 needs no barrier behind it.  Arithmetic and operation order of the
// neuron update are the other kernels'; the ring sums are the same wherever
// they do not depend on the order of the adds.
//
// Ring cells, W slots per neuron (the arrival times of the next W steps):
//   OW_COUNT  all edges of an input class have one weight: a cell counts the
//             class-0 events (low 16 bits) and class-1 events (high 16 bits),
//             one native 32-bit shared atomic per event, and the edge is its
//             4-byte word alone.  The cell's value is count x weight (fixed
//             point), or the weight added count times in FP64 -- bit for bit
//             what count separate adds of equal weights give.
//   OW_I64    fixed point: 32 low bits per channel and one word with 16 high
//             bits of either channel; a carry or a negative weight (rare: one
//             add in several) costs a second atomic.  12 bytes per slot and
//             neuron instead of the 16 of two 64-bit cells, and native 32-bit
//             atomics instead of the 64-bit compare-and-swap loop that
//             shared-memory 64-bit adds compile to.
//   OW_F64    FP64 cells, shared-memory FP64 adds.
// An event that arrives after the window (or, at the first steps of a
// launch, was delivered by an earlier launch) goes through the neuron's
// global ring cell, which the update adds in.  The edges whose delay can
// exceed the window are segments of their own, so that the others are added
// without a look at it.
//
// What bounds it.  Small and middle networks: a slice is one chain (inputs
// 1.4k cycles, recurrence beside the drive 2-3.5k, exchange 3.5-4k, delivery
// 2k: 10-12k cycles on 9,000 to 12,500 neurons).  Large ones: the segments'
// random reads (77,169 neurons: 72k of 112k cycles a step, 1,580 spikes of
// some 40 edges per SM; 1,569 segments of 320 B alone take 37k cycles, 3.8
// TB/s) beside the adds (32-bit shared atomics: 2.5 cycles per random warp
// instruction; 64-bit ones 18).  One call, the scatter or graph form before
// and this kernel [us]: 10,000 steps of 12,500 neurons in FP64 9,283 -> 6,234,
// of 9,377 in FP32 8,773 -> 5,610; 5,000 steps of 8 x 7,001 neurons 16,085 ->
// 8,471; 300 steps of the layered network at 1/4 size in FP64 8,626 -> 3,741,
// at full size in FP32 30,113 -> 17,636.
#pragma once

#include "ng_persistent.cuh"

namespace ng
{

enum
{
  OW_COUNT = 0,
  OW_I64 = 1,
  OW_F64 = 2
};

constexpr int OW_LIST = 4096;        // spikes staged in shared memory at a time
constexpr int OW_TAB = 64;           // OW_COUNT: inputs of up to OW_TAB - 1 events of a class, tabulated
constexpr int OW_TPB = 512;          // threads per CTA: 16 warps of up to 128 registers (1024 spilled 350-800 B a thread)
constexpr int OW_DVT = 32;           // drive inputs tabulated where a CTA's neurons share one weight
constexpr int OW_MAX_G = 256;        // CTAs of a network, at most
constexpr int OW_CDF = 512;          // drive thresholds staged in shared memory (more: read through L1)
constexpr int OW_SBITS = 18;         // published spike: source within the network; above: lag

// One CTA's share: every G-th neuron of the n neurons from a on, starting
// at a + (blockIdx.x - c0).
struct OwnCta
{
  int a, n, c0, G;
};

struct OwnNet
{
  const OwnCta* cta;
  const long long* rp_base;   // per CTA: its row table's start in rp
  const uint32_t* rp;         // per CTA: n + 1 segment starts, by source [quads of edges]
  const long long* e_base;    // per CTA: its edges' start [quads]
  const uint32_t* rp_far;     // the same for the edges that can arrive after the window (far only)
  const long long* e_far;
  // edge word: delay x nl + local target, bit 31: input class.  A segment's
  // last quad is padded with edges to the column nl - 1, which is no neuron's.
  const uint4* word;          // OW_COUNT, OW_F64: the edge words of a quad
  const uint4* word_w;        // OW_I64: two (edge word, fixed-point weight) pairs; a quad is two of them
  const double2* weight;      // OW_F64: two weights; a quad is two of them
  unsigned long long* xchg;   // [2][grid][x_cap]: (tag, count), then (tag, spike) words of every CTA
  long long x_cap;
  unsigned seq0;              // tag of the launch's first slice
  int nl;                     // columns of a ring slot: the most neurons of a CTA, and one
  int W;                      // ring window [slots]
  int gw_log2;                // lanes per segment
  int w16;                    // OW_COUNT: 2-byte edge words (bit 15: input class), where all distances fit
  int far;                    // W < L: the far segments exist
  int kc;                     // lags whose inputs are staged at a time
  int rp_smem;                // the row table is staged in shared memory
  int n_cdf;                  // drive thresholds staged in shared memory (0: not)
  double cw[ 2 ];             // OW_COUNT: the class weights
  int cwi[ 2 ];
  long long origin0;
  PkCtl* pk;
};

// Bytes of dynamic shared memory, and the offsets of its parts.
struct OwnSmem
{
  size_t tab, dvt, cdf, list, dref, ddw, dpd, drv, stage, state, rp, ring, total;
};

__host__ __device__ inline size_t
own_cell_bytes( int cell, bool two )
{
  return cell == OW_COUNT ? 4 : cell == OW_I64 ? ( two ? 12 : 8 ) : ( two ? 16 : 8 );
}

__host__ __device__ inline OwnSmem
own_smem( int cell, bool two, bool held, int nl, int W, int md, int rsz, int kc, int n_rp )
{
  OwnSmem s;
  size_t at = 0;
  s.tab = at;
  at += 2 * OW_TAB * 8;
  s.dvt = at;
  at += OW_DVT * 8;
  s.cdf = at;
  at += OW_CDF * 8;
  s.list = at;
  at += OW_LIST * 4;
  s.dref = at;
  at += ( size_t ) nl * 8;
  s.ddw = at;
  at += ( size_t ) nl * 8;
  s.dpd = at;
  at += ( ( size_t ) nl * 4 + 15 ) / 16 * 16;
  s.drv = at;
  at += ( ( size_t ) nl * md + 15 ) / 16 * 16;
  s.stage = at;
  at += ( ( size_t ) nl * kc * rsz * ( two ? 2 : 1 ) + 15 ) / 16 * 16;
  s.state = at;
  at += held ? 0 : ( ( size_t ) nl * ( ( two ? 6 : 3 ) * rsz + 20 ) + 15 ) / 16 * 16;
  s.rp = at;
  at += ( ( size_t ) n_rp * 4 + 15 ) / 16 * 16;
  s.ring = at;
  at += ( size_t ) W * nl * own_cell_bytes( cell, two );
  s.total = at;
  return s;
}

// A ring cell's value g and k events of one weight: in FP64 g + w + w + ...
// in this order, as separate adds of equal weights give it.
template < bool FIX >
__device__ __forceinline__ typename RingVal< FIX >::type
own_sum( typename RingVal< FIX >::type g, unsigned k, double w, int wi )
{
  if constexpr ( FIX )
    return g + ( long long ) k * wi;
  else
  {
    for ( unsigned j = 0; j < k; ++j )
      g += w;
    return g;
  }
}

// Exchange words: (tag, payload) in one 8-byte word, written and read as a
// whole, so a word with the expected tag carries its payload and no fence or
// flag has to order the words.
__device__ __forceinline__ unsigned long long
own_ld( const unsigned long long* p )
{
  unsigned long long v;
  asm volatile( "ld.relaxed.gpu.global.u64 %0, [%1];" : "=l"( v ) : "l"( p ) : "memory" );
  return v;
}

__device__ __forceinline__ void
own_st( unsigned long long* p, unsigned tag, unsigned v )
{
  const unsigned long long x = ( ( unsigned long long ) tag << 32 ) | v;
  asm volatile( "st.relaxed.gpu.global.u64 [%0], %1;" ::"l"( p ), "l"( x ) : "memory" );
}

// Index of the first threshold of the table, from the fifth on, that m does
// not exceed (the last one at most): drive_at's inversion; long tables are
// bisected.
__device__ __noinline__ unsigned
own_invert_rest( const uint64_t* cdf, int n, uint64_t m )
{
  int lo = 4, hi = n - 1;
  if ( n <= 24 )
  {
    while ( lo < hi && m > cdf[ lo ] )
      ++lo;
    return ( unsigned ) lo;
  }
  while ( lo < hi )
  {
    const int mid = ( lo + hi ) >> 1;
    if ( m > cdf[ mid ] )
      lo = mid + 1;
    else
      hi = mid;
  }
  return ( unsigned ) lo;
}

// Four edges of a segment, as edge words.
template < int CELL >
struct OwnQuad
{
  uint32_t t[ 4 ];
  typename std::conditional< CELL == OW_F64, double, int >::type w[ CELL == OW_COUNT ? 1 : 4 ];
};

template < int CELL >
__device__ __forceinline__ void
own_load( const OwnNet& o, long long q, OwnQuad< CELL >& x )
{
  if constexpr ( CELL == OW_I64 )
  {
    const uint4 a = __ldg( o.word_w + 2 * q ), b = __ldg( o.word_w + 2 * q + 1 );
    x.t[ 0 ] = a.x;
    x.w[ 0 ] = ( int ) a.y;
    x.t[ 1 ] = a.z;
    x.w[ 1 ] = ( int ) a.w;
    x.t[ 2 ] = b.x;
    x.w[ 2 ] = ( int ) b.y;
    x.t[ 3 ] = b.z;
    x.w[ 3 ] = ( int ) b.w;
  }
  else if ( CELL == OW_COUNT && o.w16 )
  {
    const uint2 a = __ldg( reinterpret_cast< const uint2* >( o.word ) + q );
    x.t[ 0 ] = a.x & 0xffffu;
    x.t[ 1 ] = a.x >> 16;
    x.t[ 2 ] = a.y & 0xffffu;
    x.t[ 3 ] = a.y >> 16;
  }
  else
  {
    const uint4 a = __ldg( o.word + q );
    x.t[ 0 ] = a.x;
    x.t[ 1 ] = a.y;
    x.t[ 2 ] = a.z;
    x.t[ 3 ] = a.w;
    if constexpr ( CELL == OW_F64 )
    {
      const double2 u = __ldg( o.weight + 2 * q ), v = __ldg( o.weight + 2 * q + 1 );
      x.w[ 0 ] = u.x;
      x.w[ 1 ] = u.y;
      x.w[ 2 ] = v.x;
      x.w[ 3 ] = v.y;
    }
  }
}

// A neuron's state and coefficients, and one step of it
// (iaf_psc_delta:272-329, iaf_psc_exp:288-348, iaf_psc_alpha update): the
// reference's operations in its order, its branches as selections (the lanes
// of a warp never part).
template < typename Real, int MODEL >
struct OwnNeuron
{
  static constexpr bool ALPHA = MODEL == NG_IAF_PSC_ALPHA_ID;
  static constexpr bool EXP = MODEL == NG_IAF_PSC_EXP_ID || ALPHA;
  static constexpr int NS = EXP ? 6 : 3;  // state arrays: V, x1, x2, i0, i1, I_e or V, y0, I_e
  Real V, x1, x2, i0, i1, Ie;
  Real c0, c1, c2, c3, c4, c5, c9, Vth, Vreset;
  AlphaCoef< Real > ac;
  int r, refr;

  __device__ __forceinline__ void
  coef( const double* ct )
  {
    if constexpr ( ALPHA )
    {
      alpha_coef< Real >( ct, ac );
      Vth = ac.Vth;
      Vreset = ac.Vreset;
      refr = ac.refr;
    }
    else if constexpr ( EXP )
    {
      c0 = ( Real ) ct[ 0 ];
      c1 = ( Real ) ct[ 1 ];
      c2 = ( Real ) ct[ 2 ];
      c3 = ( Real ) ct[ 3 ];
      c4 = ( Real ) ct[ 4 ];
      c5 = ( Real ) ct[ 5 ];
      Vth = ( Real ) ct[ 6 ];
      Vreset = ( Real ) ct[ 7 ];
      refr = ( int ) ct[ 8 ];
      c9 = ( Real ) ct[ 9 ];
    }
    else
    {
      c0 = ( Real ) ct[ 0 ];
      c1 = ( Real ) ct[ 1 ];
      Vth = ( Real ) ct[ 2 ];
      Vreset = ( Real ) ct[ 3 ];
      c2 = ( Real ) ct[ 4 ];
      refr = ( int ) ct[ 5 ];
    }
  }

  // array k of the state
  __device__ __forceinline__ Real&
  var( int k )
  {
    if constexpr ( EXP )
      return k == 0 ? V : k == 1 ? x1 : k == 2 ? x2 : k == 3 ? i0 : k == 4 ? i1 : Ie;
    else
      return k == 0 ? V : k == 1 ? x1 : Ie;
  }

  __device__ __forceinline__ bool
  step( const Real ex, const Real inh )
  {
    Real Vn;
    if constexpr ( ALPHA )
    {
      const Real y0 = Real( 0 );
      Vn = ac.P30 * ( y0 + Ie ) + ac.P31e * i0 + ac.P32e * x1 + ac.P31i * i1 + ac.P32i * x2 + ac.em1 * V + V;
      Vn = ( Vn < ac.Vmin ? ac.Vmin : Vn );
    }
    else if constexpr ( EXP )
      Vn = V * c0 + x1 * c1 + x2 * c2 + ( Ie + i0 ) * c3;
    else
    {
      Vn = c1 * ( x1 + Ie ) + c0 * V + ex;
      Vn = ( Vn < c2 ? c2 : Vn );
    }
    V = r == 0 ? Vn : V;
    r = r == 0 ? 0 : r - 1;
    if constexpr ( ALPHA )
    {
      x1 = ac.P21e * i0 + ac.P11e * x1;
      i0 *= ac.P11e;
      i0 += ac.Ee * ex;
      x2 = ac.P21i * i1 + ac.P11i * x2;
      i1 *= ac.P11i;
      i1 += ac.Ei * inh;
    }
    else if constexpr ( EXP )
    {
      x1 *= c4;
      x2 *= c5;
      x1 += c9 * i1;
      x1 += ex;
      x2 += inh;
      i0 = Real( 0 );
      i1 = Real( 0 );
    }
    else
      x1 = Real( 0 );
    const bool spk = V >= Vth;
    r = spk ? refr : r;
    V = spk ? Vreset : V;
    return spk;
  }
};

// 512 threads, up to 1024 neurons.  HOLD (at most one neuron per thread): a
// neuron's state stays in registers for the launch; else the states lie in
// shared memory between the slices and a thread takes its neurons in turn.
// (1024 threads of 64 registers spilled 300 to 500 bytes each, which 228 KB of
// shared memory leave no L1 for: a delivery of the layered network took
// 300,000 cycles.)
template < typename Real, bool FIX, int MODEL, int CELL, bool HOLD >
__global__ void __launch_bounds__( OW_TPB, 1 )
k_run_owned( Net d, Block b, OwnNet o, int n_slices )
{
  constexpr int TPB = OW_TPB;
  using Neuron = OwnNeuron< Real, MODEL >;
  using Raw = typename RingVal< FIX >::type;
  constexpr bool EXP = Neuron::EXP;
  constexpr int NW = TPB / 32;
  constexpr int XJ = 3;                        // exchange polls a warp has in flight
  constexpr int R = CELL == OW_COUNT ? 2 : 1;  // quads of a segment in flight per lane
  extern __shared__ __align__( 16 ) unsigned char o_smem[];
  __shared__ int s_cnt, s_rec, s_total, s_fail;
  __shared__ int s_base[ OW_MAX_G ], s_num[ OW_MAX_G ];  // a region's place in the list, its spikes
  __shared__ unsigned long long s_lb, s_ev, s_drive;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const OwnCta oc = o.cta[ blockIdx.x ];
  const int G = oc.G, rank = ( int ) blockIdx.x - oc.c0;
  const int nloc = ( oc.n - rank + G - 1 ) / G;
  const int md = d.min_delay, W = o.W, nl = o.nl, L = d.L;
  const OwnSmem sm = own_smem( CELL, EXP, HOLD, nl, W, md, sizeof( Real ), o.kc, o.rp_smem ? oc.n + 1 : 0 );
  Real* const tab = reinterpret_cast< Real* >( o_smem + sm.tab );
  Real* const dvt = reinterpret_cast< Real* >( o_smem + sm.dvt );
  uint32_t* const list = reinterpret_cast< uint32_t* >( o_smem + sm.list );
  int2* const dref = reinterpret_cast< int2* >( o_smem + sm.dref );
  double* const ddw = reinterpret_cast< double* >( o_smem + sm.ddw );  // drive weights
  int* const dpd = reinterpret_cast< int* >( o_smem + sm.dpd );
  Real* const st_ex = reinterpret_cast< Real* >( o_smem + sm.stage );  // [kc][nl] inputs of the staged lags
  Real* const st_in = st_ex + ( size_t ) o.kc * nl;
  uint8_t* const drv = o_smem + sm.drv;
  Real* const held = reinterpret_cast< Real* >( o_smem + sm.state );       // !HOLD: [NS][nl] state
  int* const held_r = reinterpret_cast< int* >( held + Neuron::NS * nl );  // ... refractory counts
  unsigned* const held_c = reinterpret_cast< unsigned* >( held_r + nl );   // ... class, bit 31: recorded
  unsigned* const held_m = held_c + nl;                                    // ... spikes of the window
  int* const held_p = reinterpret_cast< int* >( held_m + nl );             // ... place in the CTA's log entries
  unsigned* const held_n = reinterpret_cast< unsigned* >( held_p + nl );   // ... spikes of the launch
  uint64_t* const s_cdf = reinterpret_cast< uint64_t* >( o_smem + sm.cdf );
  // ring: [W][nl] words (OW_COUNT), [channel][W][nl] cells and, OW_I64, [W][nl] high words
  const int WN = W * nl;
  uint32_t* const r32 = reinterpret_cast< uint32_t* >( o_smem + sm.ring );
  uint32_t* const rhi = r32 + ( size_t ) WN * ( EXP ? 2 : 1 );
  double* const r64 = reinterpret_cast< double* >( o_smem + sm.ring );
  const uint32_t* rp = o.rp + o.rp_base[ blockIdx.x ];
  const long long eb = o.e_base[ blockIdx.x ];
  const long long lb0 = ld_volatile( &d.ctl->log_base );

  // ---- the CTA's neurons: q is neuron oc.a + q G + rank
  const bool act = HOLD && tid < nloc;
  auto global_of = [ & ]( int q ) { return ( int64_t ) oc.a + ( int64_t ) q * G + rank; };
  auto local_of = [ & ]( int q ) { return ( uint32_t ) ( q * G + rank ); };  // within the network
  uint2* const log_buf = log_half( d );
  long long t_off = 0;
  uint32_t il0 = ( uint32_t ) oc.a, key0 = d.key0, key1 = d.key1;  // drive counters: first neuron, key
  uint32_t log_id = 0u;
  if ( d.nid )
  {
    // a serving engine: the CTA's neurons are of one network
    const int id = d.nid[ oc.a ];
    const uint2 kk = d.net_key[ id ];
    t_off = d.net_step0[ id ];
    il0 = ( uint32_t ) ( oc.a - d.net_off[ id ] );
    key0 = kk.x;
    key1 = kk.y;
    log_id = ( uint32_t ) id << LOG_ID_SHIFT;
  }
  Neuron nr {};
  unsigned smask = 0;  // HOLD: the neuron's spikes of the window, ...
  int rpos = 0;        // ... its place in the CTA's log entries
  unsigned n_spk = 0;  // ... its spikes of the launch
  bool rec = false;
  auto load_state = [ & ]( Neuron& n, int q ) {
    const int64_t li = global_of( q ) - b.off;
    n.coef( b.ctab + ( int64_t ) b.cls[ li ] * CT_STRIDE );
#pragma unroll
    for ( int k = 0; k < Neuron::NS; ++k )
      n.var( k ) = ( ( const Real* ) b.s[ k ] )[ li ];
    n.r = b.r[ li ];
  };
  auto store_state = [ & ]( Neuron& n, int q ) {
    const int64_t li = global_of( q ) - b.off;
#pragma unroll
    for ( int k = 0; k + 1 < Neuron::NS; ++k )  // (the last one, I_e, is a parameter)
      ( ( Real* ) b.s[ k ] )[ li ] = n.var( k );
    b.r[ li ] = n.r;
  };
  auto put_held = [ & ]( Neuron& n, int q ) {
#pragma unroll
    for ( int k = 0; k < Neuron::NS; ++k )
      held[ k * nl + q ] = n.var( k );
    held_r[ q ] = n.r;
  };
  auto get_held = [ & ]( Neuron& n, int q ) {
    n.coef( b.ctab + ( int64_t ) ( held_c[ q ] & 0x7fffffffu ) * CT_STRIDE );
#pragma unroll
    for ( int k = 0; k < Neuron::NS; ++k )
      n.var( k ) = held[ k * nl + q ];
    n.r = held_r[ q ];
  };
  if constexpr ( HOLD )
  {
    if ( act )
    {
      load_state( nr, tid );
      rec = d.rec == nullptr || d.rec[ global_of( tid ) ] != 0;
    }
  }
  else
    for ( int q = tid; q < nloc; q += TPB )
    {
      Neuron n {};
      load_state( n, q );
      put_held( n, q );
      held_n[ q ] = 0u;
      const int64_t i = global_of( q );
      held_c[ q ] = ( unsigned ) b.cls[ i - b.off ] | ( d.rec == nullptr || d.rec[ i ] ? 0x80000000u : 0u );
    }
  // drive: table references, weights, delays; uniform weights are tabulated
  double w_first = 0.0;
  if ( d.has_pois && d.pois_cdf_ref[ global_of( 0 ) ].y > 0 )
    w_first = d.pois_w[ global_of( 0 ) ];
  bool same_w = true;
  for ( int q = tid; q < nloc; q += TPB )
  {
    const int64_t i = global_of( q );
    int2 rf = make_int2( 0, 0 );
    int pd = 0;
    double dw = w_first;
    if ( d.has_pois )
    {
      rf = d.pois_cdf_ref[ i ];
      if ( rf.y > 0 )
      {
        pd = d.pois_d[ i ];
        dw = d.pois_w[ i ];
      }
    }
    dref[ q ] = rf;
    dpd[ q ] = pd;
    ddw[ q ] = dw;
    same_w = same_w && dw == w_first;
  }
  same_w = __syncthreads_and( same_w );
  if ( tid < OW_DVT )
    dvt[ tid ] = ( Real ) ( w_first * u32_to_f64( tid ) );
  // ---- shared memory
  for ( size_t q = tid; q < ( size_t ) WN * own_cell_bytes( CELL, EXP ) / 4; q += TPB )
    r32[ q ] = 0u;
  if ( o.n_cdf > 0 )
  {
    for ( int q = tid; q < o.n_cdf; q += TPB )
      s_cdf[ q ] = d.pois_cdf[ q ];
  }
  if ( o.rp_smem )
  {
    uint32_t* const s_rp = reinterpret_cast< uint32_t* >( o_smem + sm.rp );
    for ( int q = tid; q <= oc.n; q += TPB )
      s_rp[ q ] = rp[ q ];
    rp = s_rp;
  }
  if ( CELL == OW_COUNT && tid < 2 )
  {
    // the input of k events of a class
    double x = 0.0;
    for ( int k = 0; k < OW_TAB; ++k )
    {
      if constexpr ( FIX )
        tab[ tid * OW_TAB + k ] = ring_real< Real, FIX >( d, ( long long ) k * o.cwi[ tid ] );
      else
        tab[ tid * OW_TAB + k ] = x;
      x += o.cw[ tid ];
    }
  }
  if ( tid == 0 )
  {
    s_cnt = s_rec = s_total = s_fail = 0;
    s_lb = s_ev = s_drive = 0ull;
  }
  __syncthreads();

  // work items (k, q), k a lag or a pair of lags, of the CTA's neurons q: an
  // item thread's first one and the step to the next
  struct Items
  {
    int k0, q0, dk, dq, nq;
    __device__ __forceinline__
    Items( int first, int stride, int n )
      : k0( first / n )
      , q0( first - k0 * n )
      , dk( stride / n )
      , dq( stride - dk * n )
      , nq( n )
    {
    }
    __device__ __forceinline__ void
    next( int& k, int& q ) const
    {
      k += dk;
      q += dq;
      if ( q >= nq )
      {
        q -= nq;
        ++k;
      }
    }
  };
  const Items all( tid, TPB, nloc );
  // The drive depends on no spike.  Where half of the warps or more have no
  // neuron and a slice's inputs are staged at once (its drive counts are then
  // free), those warps draw the next slice's drive beside the recurrence;
  // else every thread does while the spikes travel.
  const int busy = ( nloc + 31 ) & ~31;
  const bool beside = HOLD && o.kc >= md && 2 * busy <= TPB;
  const bool drawer = !beside || tid >= busy;
  const Items dit( beside ? max( tid - busy, 0 ) : tid, beside ? TPB - busy : TPB, nloc );
  const int np = md / 2 + 1;
  unsigned long long dcnt = 0;
  // the drive counts of the slice from t0 on: one Philox block serves the
  // two steps of a pair (drive_at); work item: (pair, neuron)
  auto draw = [ & ]( long long t0 ) {
    if ( !drawer )
      return;
    const long long ts = t0 - t_off;
    // every step of the slice lies inside the drive's window for every delay
    const bool inside = ts - L > ( d.pois_start > 0 ? ( long long ) d.pois_start : 0ll ) && ts + md <= d.pois_stop;
    auto items = [ & ]( auto count, int& pr, int& q ) {
      constexpr int U = decltype( count )::value;
      int prs[ U ], qs[ U ], ka[ U ];
      bool in[ U ];
      int2 rf[ U ];
      long long tp[ U ];
      uint32_t x[ U ][ 4 ];
#pragma unroll
      for ( int u = 0; u < U; ++u )
      {
        prs[ u ] = pr;
        qs[ u ] = q;
        dit.next( pr, q );
      }
#pragma unroll
      for ( int u = 0; u < U; ++u )
      {
        in[ u ] = prs[ u ] < np;
        rf[ u ] = dref[ qs[ u ] ];
        const long long tg0 = ts - dpd[ qs[ u ] ];
        tp[ u ] = ( tg0 >> 1 ) + prs[ u ];
        ka[ u ] = 2 * prs[ u ] - ( int ) ( tg0 & 1 );  // lags of the pair's two steps: ka, ka + 1
      }
#pragma unroll
      for ( int u = 0; u < U; ++u )
        philox4x32_10( il0 + local_of( qs[ u ] ), ( uint32_t ) tp[ u ], ( uint32_t ) ( ( unsigned long long ) tp[ u ] >> 32 ),
          DRIVE_STREAM, key0, key1, x[ u ] );
#pragma unroll
      for ( int u = 0; u < U; ++u )
      {
        bool wa = in[ u ] && rf[ u ].y > 0, wb = wa;
        if ( !inside )
        {
          const long long ta = 2 * tp[ u ], tb = ta + 1;
          wa = wa && ta >= 0 && d.pois_start < ta && ta <= d.pois_stop;
          wb = wb && tb >= 0 && d.pois_start < tb && tb <= d.pois_stop;
        }
        const bool la = in[ u ] && ka[ u ] >= 0 && ka[ u ] < md, lb = in[ u ] && ka[ u ] + 1 < md;
        wa = wa && la;
        wb = wb && lb;
        const uint64_t ma = u53_bits( x[ u ][ 0 ], x[ u ][ 1 ] ), mb = u53_bits( x[ u ][ 2 ], x[ u ][ 3 ] );
        unsigned na = 0, nb = 0;
        uint64_t c[ 4 ];
#pragma unroll
        for ( int e = 0; e < 4; ++e )
        {
          c[ e ] = ~0ull;
          if ( e < rf[ u ].y - 1 )
            c[ e ] = o.n_cdf > 0 ? s_cdf[ rf[ u ].x + e ] : __ldg( d.pois_cdf + rf[ u ].x + e );
        }
        // thresholds do not decrease: the number of them below m is the index
#pragma unroll
        for ( int e = 0; e < 4; ++e )
        {
          na += ma > c[ e ] ? 1u : 0u;
          nb += mb > c[ e ] ? 1u : 0u;
        }
        if ( na == 4 && wa )
          na = own_invert_rest( o.n_cdf > 0 ? s_cdf + rf[ u ].x : d.pois_cdf + rf[ u ].x, rf[ u ].y, ma );
        if ( nb == 4 && wb )
          nb = own_invert_rest( o.n_cdf > 0 ? s_cdf + rf[ u ].x : d.pois_cdf + rf[ u ].x, rf[ u ].y, mb );
        na = wa ? na : 0u;
        nb = wb ? nb : 0u;
        dcnt += na + nb;
        if ( la )
          drv[ ka[ u ] * nl + qs[ u ] ] = ( uint8_t ) na;
        if ( lb )
          drv[ ( ka[ u ] + 1 ) * nl + qs[ u ] ] = ( uint8_t ) nb;
      }
    };
    // two items at a time where a thread has several: their Philox rounds are
    // chains of dependent multiplies that 16 warps alone do not hide
    int pr = dit.k0, q = dit.q0;
    while ( pr + dit.dk < np )
      items( std::integral_constant< int, 2 >(), pr, q );
    while ( pr < np )
      items( std::integral_constant< int, 1 >(), pr, q );
  };

  // The edges of a quad of a spike of lag k: base = ( k - min_delay + the next
  // slice's first window position ) x nl, so that edge word + base is the
  // cell, up to the window's wrap.
  const bool w16 = CELL == OW_COUNT && o.w16;
  const uint32_t w_mask = w16 ? 0x7fffu : 0x7fffffffu;
  const int w_class = w16 ? 15 : 31;
  auto add_quad = [ & ]( const OwnQuad< CELL >& x, int base ) {
    int at[ 4 ];
    uint32_t old[ 4 ];
#pragma unroll
    for ( int e = 0; e < 4; ++e )
    {
      at[ e ] = ( int ) ( x.t[ e ] & w_mask ) + base;
      if ( at[ e ] >= WN )
        at[ e ] -= WN;
      const unsigned cl = x.t[ e ] >> w_class;
      if constexpr ( CELL == OW_COUNT )
        atomicAdd( r32 + at[ e ], cl ? 65536u : 1u );
      else if constexpr ( CELL == OW_I64 )
        old[ e ] = atomicAdd( r32 + ( EXP && cl ? WN : 0 ) + at[ e ], ( uint32_t ) x.w[ e ] );
      else
        atomicAdd( r64 + ( EXP && cl ? WN : 0 ) + at[ e ], x.w[ e ] );
    }
    if constexpr ( CELL == OW_I64 )
    {
#pragma unroll
      for ( int e = 0; e < 4; ++e )
      {
        const int w = x.w[ e ];
        const int up = ( w >> 31 ) + ( old[ e ] + ( uint32_t ) w < old[ e ] ? 1 : 0 );
        if ( up != 0 )
          atomicAdd( rhi + at[ e ], EXP && x.t[ e ] >> 31 ? ( uint32_t ) up << 16 : ( uint32_t ) up );
      }
    }
  };
  // The edges of a far quad: off = ( k - min_delay ) x nl, gs: the next
  // slice's first slot in the global ring.
  auto add_far = [ & ]( const OwnQuad< CELL >& x, int off, int wbn, int gs ) {
#pragma unroll 1
    for ( int e = 0; e < 4; ++e )
    {
      const uint32_t t = e == 0 ? x.t[ 0 ] : e == 1 ? x.t[ 1 ] : e == 2 ? x.t[ 2 ] : x.t[ 3 ];
      const int rel = ( int ) ( t & w_mask ) + off, dist = rel / nl, l = rel - dist * nl;
      const unsigned cl = t >> w_class;
      if ( l == nl - 1 )
        continue;  // padding
      typename std::conditional< CELL == OW_F64, double, int >::type w = 0;
      if constexpr ( CELL != OW_COUNT )
        w = e == 0 ? x.w[ 0 ] : e == 1 ? x.w[ 1 ] : e == 2 ? x.w[ 2 ] : x.w[ 3 ];
      if ( rel < WN )
      {
        int at = rel + wbn;
        if ( at >= WN )
          at -= WN;
        if constexpr ( CELL == OW_COUNT )
          atomicAdd( r32 + at, cl ? 65536u : 1u );
        else if constexpr ( CELL == OW_I64 )
        {
          const uint32_t old = atomicAdd( r32 + ( EXP && cl ? WN : 0 ) + at, ( uint32_t ) w );
          const int up = ( w >> 31 ) + ( old + ( uint32_t ) w < old ? 1 : 0 );
          if ( up != 0 )
            atomicAdd( rhi + at, EXP && cl ? ( uint32_t ) up << 16 : ( uint32_t ) up );
        }
        else
          atomicAdd( r64 + ( EXP && cl ? WN : 0 ) + at, w );
        continue;
      }
      int slot = gs + dist;
      if ( slot >= L )
        slot -= L;
      const int64_t g = ( ( int64_t ) slot * d.C + ( EXP ? cl : 0u ) ) * d.N + oc.a + ( int64_t ) l * G + rank;
      if constexpr ( CELL == OW_F64 )
        atomicAdd( ( double* ) d.ring + g, w );
      else if constexpr ( !FIX )
        atomicAdd( ( double* ) d.ring + g, o.cw[ cl ] );
      else if constexpr ( CELL == OW_I64 )
        atomicAdd( ( unsigned long long* ) d.ring + g, ( unsigned long long ) ( long long ) w );
      else
        atomicAdd( ( unsigned long long* ) d.ring + g, ( unsigned long long ) ( long long ) o.cwi[ cl ] );
    }
  };

  auto ring_p = [ & ]( int slot, int ch, int q ) {
    return ( Raw* ) d.ring + ( ( int64_t ) slot * d.C + ch ) * d.N + oc.a + ( int64_t ) q * G + rank;
  };
  // inputs (ex, inh) of neuron q at one lag: its window cell at position wp
  // (cleared), its global ring cell's value (vex, vin), its drive
  auto inputs = [ & ]( int q, int lag, int wp, Raw vex, Raw vin, Real& ex, Real& inh ) {
    inh = Real( 0 );
    if constexpr ( CELL == OW_COUNT )
    {
      uint32_t* const p = r32 + wp * nl + q;
      const uint32_t v = *p;
      *p = 0u;
      const unsigned n0 = v & 0xffffu, n1 = v >> 16;
      if ( vex == 0 && vin == 0 && n0 < OW_TAB && n1 < OW_TAB && ( EXP || n1 == 0 ) )
      {
        ex = tab[ n0 ];
        if constexpr ( EXP )
          inh = tab[ OW_TAB + n1 ];
      }
      else if constexpr ( EXP )
      {
        ex = ring_real< Real, FIX >( d, own_sum< FIX >( vex, n0, o.cw[ 0 ], o.cwi[ 0 ] ) );
        inh = ring_real< Real, FIX >( d, own_sum< FIX >( vin, n1, o.cw[ 1 ], o.cwi[ 1 ] ) );
      }
      else
        ex = ring_real< Real, FIX >( d,
          own_sum< FIX >( own_sum< FIX >( vex, n0, o.cw[ 0 ], o.cwi[ 0 ] ), n1, o.cw[ 1 ], o.cwi[ 1 ] ) );
    }
    else if constexpr ( CELL == OW_I64 )
    {
      uint32_t* const ph = rhi + wp * nl + q;
      uint32_t* const p0 = r32 + wp * nl + q;
      const uint32_t h = *ph, l0 = *p0;
      const int h0 = ( int ) ( int16_t ) ( h & 0xffffu );
      vex += ( long long ) ( ( ( unsigned long long ) ( long long ) h0 << 32 ) + l0 );
      *p0 = 0u;
      if constexpr ( EXP )
      {
        const uint32_t l1 = p0[ WN ];
        const int h1 = ( int ) ( int16_t ) ( ( h - ( uint32_t ) h0 ) >> 16 );
        vin += ( long long ) ( ( ( unsigned long long ) ( long long ) h1 << 32 ) + l1 );
        p0[ WN ] = 0u;
        inh = ring_real< Real, FIX >( d, vin );
      }
      *ph = 0u;
      ex = ring_real< Real, FIX >( d, vex );
    }
    else
    {
      double* const p0 = r64 + wp * nl + q;
      ex = ( Real ) ( vex + p0[ 0 ] );
      p0[ 0 ] = 0.0;
      if constexpr ( EXP )
      {
        inh = ( Real ) ( vin + p0[ WN ] );
        p0[ WN ] = 0.0;
      }
    }
    const unsigned dk = drv[ lag * nl + q ];
    Real dv;
    if ( same_w )
      dv = dvt[ min( dk, ( unsigned ) OW_DVT - 1u ) ];
    if ( !same_w || dk >= OW_DVT )
      dv = ( Real ) ( ddw[ q ] * u32_to_f64( dk ) );
    if constexpr ( EXP )
    {
      ex = dv > Real( 0 ) ? ex + dv : ex;
      inh = dv < Real( 0 ) ? inh + dv : inh;
    }
    else
      ex = dv != Real( 0 ) ? ex + dv : ex;
  };
  auto trace = [ & ]( Neuron& n, int q, long long stamp ) {
    if constexpr ( EXP )
    {
      const double vals[ 6 ] = { ( double ) n.V, ( double ) n.x1, ( double ) n.x2, ( double ) n.i0, ( double ) n.i1,
        ( double ) n.Ie };
      trace_put( d, global_of( q ), stamp, vals );
    }
    else
    {
      const double vals[ 3 ] = { ( double ) n.V, ( double ) n.x1, ( double ) n.Ie };
      trace_put( d, global_of( q ), stamp, vals );
    }
  };

  unsigned long long spk_acc = 0;  // (thread 0's)
  draw( o.origin0 );
  // slices of one step with far edges: the next step's global ring cells, read
  // ahead (W >= min_delay: no far arrival is still to come there)
  const bool ahead = o.far && md == 1;
  Raw g_ex[ 2 ] = { 0, 0 }, g_in[ 2 ] = { 0, 0 };
  auto read_ahead = [ & ]( int slot ) {
#pragma unroll
    for ( int u = 0; u < ( HOLD ? 1 : 2 ); ++u )
      if ( tid + u * TPB < nloc )
      {
        g_ex[ u ] = __ldcg( ring_p( slot, 0, tid + u * TPB ) );
        if constexpr ( EXP )
          g_in[ u ] = __ldcg( ring_p( slot, 1, tid + u * TPB ) );
      }
  };
  if ( ahead )
    read_ahead( ( int ) ( o.origin0 % L ) );
  __syncthreads();
  const int gw = 1 << o.gw_log2, gl = tid & ( gw - 1 ), gi = tid >> o.gw_log2, ng = TPB >> o.gw_log2;
  int wpos = ( int ) ( o.origin0 % W );  // window position and global slot of the open slice's first step
  int gpos = ( int ) ( o.origin0 % L );
  int xg = 3;  // log2 of the words of an exchange region read at once
  int sl = 0;
  for ( ; sl < n_slices; ++sl )
  {
    const long long origin = o.origin0 + ( long long ) sl * md;
    const unsigned tag = o.seq0 + ( unsigned ) sl;
    unsigned long long* const xbuf = o.xchg + ( size_t ) ( tag & 1u ) * gridDim.x * o.x_cap;
    unsigned long long* const mine = xbuf + ( size_t ) blockIdx.x * o.x_cap;
    // ---- 1. node update, 2. publish
    const int wb = wpos + md >= W ? wpos + md - W : wpos + md;  // the next slice's first window position, global slot
    const int gb = gpos + md >= L ? gpos + md - L : gpos + md;
    for ( int c32 = 0; c32 < md; c32 += 32 )
    {
      const int hi = min( md, c32 + 32 );
      for ( int cb = c32; cb < hi; )
      {
        const int nk = min( o.kc, hi - cb );
        // the staged lags' inputs, by all threads (the cells, counts and
        // conversions of different lags do not wait for one another)
        if ( ahead )
        {
#pragma unroll
          for ( int u = 0; u < ( HOLD ? 1 : 2 ); ++u )
          {
            const int q = tid + u * TPB;
            if ( q < nloc )
            {
              if ( g_ex[ u ] != Raw( 0 ) )
                *ring_p( gpos, 0, q ) = Raw( 0 );
              if constexpr ( EXP )
                if ( g_in[ u ] != Raw( 0 ) )
                  *ring_p( gpos, 1, q ) = Raw( 0 );
              Real ex, inh;
              inputs( q, 0, wpos, g_ex[ u ], g_in[ u ], ex, inh );
              st_ex[ q ] = ex;
              if constexpr ( EXP )
                st_in[ q ] = inh;
            }
          }
        }
        else if ( o.far || origin + cb < o.origin0 + L )
        {
          // the global ring takes part while it can hold anything
          for ( int k = all.k0, q = all.q0; k < nk; all.next( k, q ) )
          {
            const int lag = cb + k;
            int wp = wpos + lag, gs = gpos + lag;
            if ( wp >= W )
              wp -= W;
            if ( gs >= L )
              gs -= L;
            Raw vex = 0, vin = 0;
            if ( o.far || origin + lag < o.origin0 + L )
            {
              Raw* const ge = ring_p( gs, 0, q );
              vex = __ldcg( ge );
              if constexpr ( EXP )
                vin = __ldcg( ge + d.N );
              if ( vex != Raw( 0 ) )
                *ge = Raw( 0 );
              if constexpr ( EXP )
                if ( vin != Raw( 0 ) )
                  ge[ d.N ] = Raw( 0 );
            }
            Real ex, inh;
            inputs( q, lag, wp, vex, vin, ex, inh );
            st_ex[ k * nl + q ] = ex;
            if constexpr ( EXP )
              st_in[ k * nl + q ] = inh;
          }
        }
        else
        {
#pragma unroll 4
          for ( int k = all.k0, q = all.q0; k < nk; all.next( k, q ) )
          {
            int wp = wpos + cb + k;
            if ( wp >= W )
              wp -= W;
            Real ex, inh;
            inputs( q, cb + k, wp, Raw( 0 ), Raw( 0 ), ex, inh );
            st_ex[ k * nl + q ] = ex;
            if constexpr ( EXP )
              st_in[ k * nl + q ] = inh;
          }
        }
        __syncthreads();
        auto steps = [ & ]( Neuron& n, int q, unsigned m ) -> unsigned {
          if ( d.trace_col )
          {
            for ( int k = 0; k < nk; ++k )
            {
              if ( n.step( st_ex[ k * nl + q ], EXP ? st_in[ k * nl + q ] : Real( 0 ) ) )
                m |= 1u << ( cb + k - c32 );
              trace( n, q, origin + cb + k + 1 );
            }
          }
          else
          {
#pragma unroll 4
            for ( int k = 0; k < nk; ++k )
              m |= ( n.step( st_ex[ k * nl + q ], EXP ? st_in[ k * nl + q ] : Real( 0 ) ) ? 1u : 0u ) << ( cb + k - c32 );
          }
          return m;
        };
        if constexpr ( HOLD )
        {
          if ( act )
            smask = steps( nr, tid, cb == c32 ? 0u : smask );
          else if ( beside && tid >= busy && sl + 1 < n_slices )
            draw( origin + md );
        }
        else
          for ( int q = tid; q < nloc; q += TPB )
          {
            Neuron n;
            get_held( n, q );
            held_m[ q ] = steps( n, q, cb == c32 ? 0u : held_m[ q ] );
            put_held( n, q );
          }
        cb += nk;
        if ( cb < md )
          __syncthreads();  // the stage is refilled
      }
      auto publish = [ & ]( int q, unsigned mask, bool log, int& place ) {
        const int cnt = __popc( mask );
        int at = 1 + atomicAdd( &s_cnt, cnt );
        for ( unsigned m = mask; m; m &= m - 1 )
          own_st( mine + at++, tag, local_of( q ) | ( ( uint32_t ) ( c32 + __ffs( m ) - 1 ) << OW_SBITS ) );
        if ( log )
        {
          if ( hi < md )
          {
            // a slice of more than 32 lags: this window's log entries at once
            unsigned long long at_log = atomicAdd( &d.ctl->log_count, ( unsigned long long ) cnt );
            for ( unsigned m = mask; m; m &= m - 1, ++at_log )
              if ( ( long long ) at_log < d.log_cap )
                log_buf[ at_log ] =
                  make_uint2( ( il0 + local_of( q ) ) | log_id, ( uint32_t ) ( origin + c32 + __ffs( m ) - lb0 ) | ( 1u << 24 ) );
              else
                atomicOr( &d.ctl->err, ERR_LOG );
          }
          else
            place = atomicAdd( &s_rec, cnt );
        }
        if constexpr ( HOLD )
          n_spk += ( unsigned ) cnt;
        else
          held_n[ q ] += ( unsigned ) cnt;
      };
      if constexpr ( HOLD )
      {
        if ( smask )
          publish( tid, smask, rec, rpos );
      }
      else
        for ( int q = tid; q < nloc; q += TPB )
          if ( held_m[ q ] )
            publish( q, held_m[ q ], ( held_c[ q ] >> 31 ) != 0, held_p[ q ] );
    }
    __syncthreads();
    if ( tid == 0 )
    {
      own_st( mine, tag, ( unsigned ) s_cnt );
      spk_acc += ( unsigned ) s_cnt;
      if ( s_rec > 0 )
        s_lb = atomicAdd( &d.ctl->log_count, ( unsigned long long ) s_rec );
      s_cnt = s_rec = 0;  // next added to behind the exchange's barrier
    }
    // ---- 3. what depends on no spike
    if ( !beside && sl + 1 < n_slices )
      draw( origin + md );
    if ( ahead && sl + 1 < n_slices )
      read_ahead( gb );
    // ---- 4. the network's spikes of the slice
    // (1 << xg lanes read a region's first words; a warp has XJ such reads in flight)
    const int xn = 1 << xg, xl = lane & ( xn - 1 ), xper = 32 >> xg;
    for ( int cbase = warp * xper + ( lane >> xg ); __any_sync( FULL, cbase < G ); cbase += NW * xper * XJ )
    {
      unsigned long long v[ XJ ];
      int cnt[ XJ ];
      const unsigned long long* const reg0 = xbuf + ( size_t ) ( oc.c0 + cbase ) * o.x_cap + xl;
      const size_t reg_step = ( size_t ) NW * xper * o.x_cap;
#pragma unroll
      for ( int j = 0; j < XJ; ++j )
      {
        v[ j ] = 0ull;
        if ( cbase + j * NW * xper < G )
          v[ j ] = own_ld( reg0 + j * reg_step );
      }
      unsigned polls = 0;
      for ( ;; )
      {
        bool good = true;
#pragma unroll
        for ( int j = 0; j < XJ; ++j )
        {
          const bool in = cbase + j * NW * xper < G;
          const unsigned long long hd = __shfl_sync( FULL, v[ j ], lane & ~( xn - 1 ) );
          const bool ok = ( unsigned ) ( hd >> 32 ) == tag;
          cnt[ j ] = in && ok ? ( int ) ( unsigned ) hd : 0;
          if ( in && !( ok && ( xl > cnt[ j ] || ( unsigned ) ( v[ j ] >> 32 ) == tag ) ) )
          {
            good = false;
            v[ j ] = own_ld( reg0 + j * reg_step );
          }
        }
        if ( __all_sync( FULL, good ) )
          break;
        ++polls;
        const bool quit = polls > PK_POLL_LIMIT || ( ( polls & 255u ) == 0 && ld_volatile( &o.pk->err ) != 0 );
        if ( __any_sync( FULL, quit ) )
        {
          if ( lane == 0 )
          {
            atomicOr( &o.pk->err, 1 );
            s_fail = 1;
          }
#pragma unroll
          for ( int j = 0; j < XJ; ++j )
            cnt[ j ] = 0;
          break;
        }
      }
      // places in the list: one reservation per warp
      int at[ XJ ], sum = 0;
#pragma unroll
      for ( int j = 0; j < XJ; ++j )
      {
        int x = cnt[ j ];  // (the same in all lanes of a region)
        for ( int w = xn; w < 32; w <<= 1 )
        {
          const int y = __shfl_up_sync( FULL, x, w );
          if ( lane >= w )
            x += y;
        }
        at[ j ] = sum + x - cnt[ j ];
        sum += __shfl_sync( FULL, x, 31 );
      }
      int base0 = 0;
      if ( lane == 0 && sum > 0 )
        base0 = atomicAdd( &s_total, sum );
      base0 = __shfl_sync( FULL, base0, 0 );
#pragma unroll
      for ( int j = 0; j < XJ; ++j )
      {
        const int c = cbase + j * NW * xper, base = base0 + at[ j ];
        if ( xl == 0 && c < G )
        {
          s_num[ c ] = cnt[ j ];
          s_base[ c ] = base;
        }
        if ( __reduce_max_sync( FULL, cnt[ j ] ) == 0 )
          continue;
        const unsigned long long* const reg = reg0 - xl + j * reg_step;
        if ( xl >= 1 && xl <= cnt[ j ] && base + xl - 1 < OW_LIST )
          list[ base + xl - 1 ] = ( uint32_t ) v[ j ];
        // the words beyond the first ones
        for ( int w = xn + xl; w <= cnt[ j ]; w += xn )
        {
          unsigned long long x = own_ld( reg + w );
          for ( unsigned p = 0; ( unsigned ) ( x >> 32 ) != tag && p < PK_POLL_LIMIT; ++p )
            x = own_ld( reg + w );
          if ( ( unsigned ) ( x >> 32 ) != tag )
          {
            atomicOr( &o.pk->err, 1 );
            s_fail = 1;
            break;
          }
          if ( base + w - 1 < OW_LIST )
            list[ base + w - 1 ] = ( uint32_t ) x;
        }
        __syncwarp();
      }
    }
    __syncthreads();
    if ( s_fail )
      break;
    const int total = s_total;
    // next slice: read as many words per region as this one's mean spikes ask for
    xg = s_total > 12 * G ? 5 : s_total > 4 * G ? 4 : 3;
    // the recorder log of this CTA's spikes (room reserved at the publication)
    auto log_put = [ & ]( int q, unsigned mask, int place ) {
      unsigned long long at = s_lb + ( unsigned ) place;
      for ( unsigned m = mask; m; m &= m - 1, ++at )
        if ( ( long long ) at < d.log_cap )
          log_buf[ at ] = make_uint2( ( il0 + local_of( q ) ) | log_id,
            ( uint32_t ) ( origin + ( ( md - 1 ) & ~31 ) + __ffs( m ) - lb0 ) | ( 1u << 24 ) );
        else
          atomicOr( &d.ctl->err, ERR_LOG );
    };
    if constexpr ( HOLD )
    {
      if ( smask && rec )
        log_put( tid, smask, rpos );
    }
    else
      for ( int q = tid; q < nloc; q += TPB )
        if ( held_m[ q ] && held_c[ q ] >> 31 )
          log_put( q, held_m[ q ], held_p[ q ] );
    // segments of the staged spikes, gw lanes and R quads per lane each, two
    // segments of a group in flight and the next two's row entries behind them
    for ( int first = 0; first < total; first += OW_LIST )
    {
      const int nlist = min( total - first, OW_LIST );
      if ( first > 0 )
      {
        // more spikes than the list holds (all their words have arrived)
        __syncthreads();
        for ( int c = warp; c < G; c += NW )
        {
          const unsigned long long* const reg = xbuf + ( size_t ) ( oc.c0 + c ) * o.x_cap + 1;
          const int n = s_num[ c ], at = n > 0 ? s_base[ c ] - first : 0;
          for ( int w = max( 0, -at ) + lane; w < n && at + w < nlist; w += 32 )
            list[ at + w ] = ( uint32_t ) own_ld( reg + w );
        }
        __syncthreads();
      }
      uint32_t a[ 2 ], z[ 2 ];
      int of[ 2 ];
      const int wbn = wb * nl;
      auto row = [ & ]( int k, uint32_t& from, uint32_t& to, int& base ) {
        from = to = 0u;
        base = 0;
        if ( k < nlist )
        {
          const uint32_t en = list[ k ], src = en & ( ( 1u << OW_SBITS ) - 1u );
          from = rp[ src ] + gl;
          to = rp[ src + 1 ];
          base = ( ( int ) ( en >> OW_SBITS ) - md ) * nl + wbn;
        }
      };
      row( gi, a[ 0 ], z[ 0 ], of[ 0 ] );
      row( gi + ng, a[ 1 ], z[ 1 ], of[ 1 ] );
      for ( int k = gi; k < nlist; k += 2 * ng )
      {
        OwnQuad< CELL > x[ 2 ][ R ];
#pragma unroll
        for ( int u = 0; u < 2; ++u )
#pragma unroll
          for ( int v = 0; v < R; ++v )
            if ( a[ u ] + v * gw < z[ u ] )
              own_load< CELL >( o, eb + a[ u ] + v * gw, x[ u ][ v ] );
        uint32_t an[ 2 ], zn[ 2 ];
        int ofn[ 2 ];
        row( k + 2 * ng, an[ 0 ], zn[ 0 ], ofn[ 0 ] );
        row( k + 3 * ng, an[ 1 ], zn[ 1 ], ofn[ 1 ] );
#pragma unroll
        for ( int u = 0; u < 2; ++u )
        {
#pragma unroll
          for ( int v = 0; v < R; ++v )
            if ( a[ u ] + v * gw < z[ u ] )
              add_quad( x[ u ][ v ], of[ u ] );
          for ( uint32_t q = a[ u ] + R * gw; q < z[ u ]; q += gw )
          {
            OwnQuad< CELL > y;
            own_load< CELL >( o, eb + q, y );
            add_quad( y, of[ u ] );
          }
          a[ u ] = an[ u ];
          z[ u ] = zn[ u ];
          of[ u ] = ofn[ u ];
        }
      }
      if ( o.far )
      {
        // far segments (a few edges each): two lanes per spike
        const uint32_t* const rf = o.rp_far + o.rp_base[ blockIdx.x ];
        const long long ef = o.e_far[ blockIdx.x ];
        for ( int k = tid >> 1; k < nlist; k += TPB / 2 )
        {
          const uint32_t en = list[ k ], src = en & ( ( 1u << OW_SBITS ) - 1u );
          const int off = ( ( int ) ( en >> OW_SBITS ) - md ) * nl;
          for ( uint32_t q = rf[ src ] + ( tid & 1 ), end = rf[ src + 1 ]; q < end; q += 2 )
          {
            OwnQuad< CELL > y;
            own_load< CELL >( o, ef + q, y );
            add_far( y, off, wbn, gb );
          }
        }
      }
    }
    __syncthreads();
    if ( tid == 0 )
      s_total = 0;  // next added to behind the update's barrier
    wpos = wb;
    gpos = gb;
  }

  // ---- what is still to arrive goes back to the global ring, where the
  // next launch (of whatever form) finds it
  __syncthreads();
  for ( int q = tid; q < WN; q += TPB )
  {
    const int pos = q / nl, l = q - pos * nl;
    if ( l >= nloc )
      continue;
    int rel = pos - wpos;
    if ( rel < 0 )
      rel += W;
    int slot = gpos + rel;
    if ( slot >= L )
      slot -= L;
    Raw* const gr = ( Raw* ) d.ring + ( int64_t ) slot * d.C * d.N + oc.a + ( int64_t ) l * G + rank;
    if constexpr ( CELL == OW_COUNT )
    {
      const uint32_t v = r32[ q ];
      const unsigned n0 = v & 0xffffu, n1 = v >> 16;
      Raw* const g1 = gr + ( EXP ? d.N : 0 );
      if ( n0 )
        *gr = own_sum< FIX >( __ldcg( gr ), n0, o.cw[ 0 ], o.cwi[ 0 ] );
      if ( n1 )
        *g1 = own_sum< FIX >( __ldcg( g1 ), n1, o.cw[ 1 ], o.cwi[ 1 ] );
    }
    else if constexpr ( CELL == OW_I64 )
    {
      const uint32_t h = rhi[ q ];
      const int h0 = ( int ) ( int16_t ) ( h & 0xffffu );
      const long long v0 = ( long long ) ( ( ( unsigned long long ) ( long long ) h0 << 32 ) + r32[ q ] );
      if ( v0 )
        gr[ 0 ] = __ldcg( gr ) + v0;
      if constexpr ( EXP )
      {
        const int h1 = ( int ) ( int16_t ) ( ( h - ( uint32_t ) h0 ) >> 16 );
        const long long v1 = ( long long ) ( ( ( unsigned long long ) ( long long ) h1 << 32 ) + r32[ WN + q ] );
        if ( v1 )
          gr[ d.N ] = __ldcg( gr + d.N ) + v1;
      }
    }
    else
    {
      if ( r64[ q ] != 0.0 )
        gr[ 0 ] = __ldcg( gr ) + r64[ q ];
      if constexpr ( EXP )
        if ( r64[ WN + q ] != 0.0 )
          gr[ d.N ] = __ldcg( gr + d.N ) + r64[ WN + q ];
    }
  }
  if constexpr ( HOLD )
  {
    if ( act )
      store_state( nr, tid );
  }
  else
    for ( int q = tid; q < nloc; q += TPB )
    {
      Neuron n;
      get_held( n, q );
      store_state( n, q );
    }
  unsigned long long ev = 0;
  if constexpr ( HOLD )
  {
    if ( act )
      ev = ( unsigned long long ) n_spk * ( unsigned ) d.real_deg[ global_of( tid ) ];
  }
  else
    for ( int q = tid; q < nloc; q += TPB )
      ev += ( unsigned long long ) held_n[ q ] * ( unsigned ) d.real_deg[ global_of( q ) ];
  if ( ev )
    atomicAdd( &s_ev, ev );
  if ( dcnt )
    atomicAdd( &s_drive, dcnt );
  __syncthreads();
  if ( tid == 0 )
  {
    if ( spk_acc )
    {
      atomicAdd( &d.ctl->syn_events, s_ev );
      atomicAdd( &d.ctl->n_spikes, spk_acc );
    }
    if ( s_drive )
      atomicAdd( &d.ctl->drive_events, s_drive );
    if ( s_fail )
      atomicOr( &d.ctl->err, ERR_BARRIER );
    // the clock at a slice boundary, as the graph form leaves it (the host
    // passes the origin: no CTA of this launch reads it)
    if ( blockIdx.x == 0 )
      d.ctl->origin = o.origin0 + ( long long ) sl * md;
  }
}

// ---------------------------------------------------------------------
// The owners' edge copies, built on the device from the engine's rows.
// ---------------------------------------------------------------------
// Smallest and largest target of every row (an empty row: itself).
__global__ void
k_own_span( long long n, const int64_t* row_beg, const int32_t* real_deg, const uint32_t* tdc, uint32_t tmask, int2* span )
{
  const long long s = ( ( long long ) blockIdx.x * blockDim.x + threadIdx.x ) >> 5;
  const int lane = threadIdx.x & 31;
  if ( s >= n )
    return;
  int lo = ( int ) s, hi = ( int ) s;
  const long long r0 = row_beg[ s ];
  for ( int j = lane; j < real_deg[ s ]; j += 32 )
  {
    const int t = ( int ) ( tdc[ r0 + j ] & tmask );
    lo = min( lo, t );
    hi = max( hi, t );
  }
  lo = __reduce_min_sync( FULL, lo );
  hi = __reduce_max_sync( FULL, hi );
  if ( lane == 0 )
    span[ s ] = make_int2( lo, hi );
}

// What the builder works on: rows a .. a + n of one network, owned by the
// CTAs c0 .. c0 + G.  An edge is near (the segments rp) up to a delay of
// d_near steps, far (rp_far) beyond.
struct OwnBuild
{
  int a, n, c0, G;
  const int64_t* row_beg;
  const int32_t* real_deg;
  const uint32_t* tdc;
  const void* w;
  uint32_t tmask, dmask;
  int tbits;
  const long long* rp_base;
  uint32_t* rp;
  uint32_t* rp_far;
  int d_near;
  int split;  // a weight's class is its sign instead of its channel (iaf_psc_delta has one channel)
};

// FP64 and int32 weights mapped to unsigned order.
template < typename T >
__device__ __forceinline__ unsigned long long
own_order( T w )
{
  if constexpr ( sizeof( T ) == 8 )
  {
    const unsigned long long u = ( unsigned long long ) __double_as_longlong( w );
    return ( u >> 63 ) ? ~u : ( u | ( 1ull << 63 ) );
  }
  else
    return ( unsigned long long ) ( ( long long ) w + ( 1ll << 40 ) );
}

// The smallest and largest weight of each class, from the weights alone (the
// channel of a non-zero weight is its sign, set where the edge was packed).
template < typename T >
__global__ void __launch_bounds__( 256 )
k_own_bounds( OwnBuild q, unsigned long long* wmin, unsigned long long* wmax )
{
  __shared__ unsigned long long s_min[ 2 ], s_max[ 2 ];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  if ( threadIdx.x < 2 )
  {
    s_min[ threadIdx.x ] = ~0ull;
    s_max[ threadIdx.x ] = 0ull;
  }
  __syncthreads();
  unsigned long long mn[ 2 ] = { ~0ull, ~0ull }, mx[ 2 ] = { 0ull, 0ull };
  for ( long long s = ( long long ) blockIdx.x * 8 + warp; s < q.n; s += ( long long ) gridDim.x * 8 )
  {
    const T* const w = ( const T* ) q.w + q.row_beg[ q.a + s ];
    const int deg = q.real_deg[ q.a + s ];
#pragma unroll 4
    for ( int j = lane; j < deg; j += 32 )
    {
      const T x = w[ j ];
      const unsigned long long u = own_order< T >( x );
      const bool second = q.split ? x < T( 0 ) : !( x > T( 0 ) );
      if ( x == T( 0 ) )
        continue;
      // (selections: an array indexed by the class would be in local memory)
      mn[ 0 ] = second ? mn[ 0 ] : min( mn[ 0 ], u );
      mx[ 0 ] = second ? mx[ 0 ] : max( mx[ 0 ], u );
      mn[ 1 ] = second ? min( mn[ 1 ], u ) : mn[ 1 ];
      mx[ 1 ] = second ? max( mx[ 1 ], u ) : mx[ 1 ];
    }
  }
#pragma unroll
  for ( int c = 0; c < 2; ++c )
    if ( mx[ c ] )
    {
      atomicMin( &s_min[ c ], mn[ c ] );
      atomicMax( &s_max[ c ], mx[ c ] );
    }
  __syncthreads();
  if ( threadIdx.x < 2 && s_max[ threadIdx.x ] )
  {
    atomicMin( wmin + threadIdx.x, s_min[ threadIdx.x ] );
    atomicMax( wmax + threadIdx.x, s_max[ threadIdx.x ] );
  }
}

// Near and far edges of every (owner, source), in one pass over the rows.
template < typename T >
__global__ void __launch_bounds__( 256 )
k_own_count( OwnBuild q )
{
  __shared__ unsigned s_h[ 8 ][ 2 * OW_MAX_G ];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int G2 = q.rp_far ? 2 * q.G : q.G;
  for ( long long s = ( long long ) blockIdx.x * 8 + warp; s < q.n; s += ( long long ) gridDim.x * 8 )
  {
    for ( int k = lane; k < G2; k += 32 )
      s_h[ warp ][ k ] = 0u;
    __syncwarp();
    const long long r0 = q.row_beg[ q.a + s ];
    const int deg = q.real_deg[ q.a + s ];
#pragma unroll 4
    for ( int j = lane; j < deg; j += 32 )
    {
      const T w = ( ( const T* ) q.w )[ r0 + j ];
      const uint32_t t = q.tdc[ r0 + j ];
      if ( w == T( 0 ) )
        continue;
      const int dl = ( int ) ( ( t >> q.tbits ) & q.dmask );
      const unsigned l = ( t & q.tmask ) - ( unsigned ) q.a;
      atomicAdd( &s_h[ warp ][ l % ( unsigned ) q.G + ( dl > q.d_near ? q.G : 0 ) ], 1u );
    }
    __syncwarp();
    for ( int k = lane; k < q.G; k += 32 )
    {
      q.rp[ q.rp_base[ q.c0 + k ] + s ] = s_h[ warp ][ k ];
      if ( q.rp_far )
        q.rp_far[ q.rp_base[ q.c0 + k ] + s ] = s_h[ warp ][ q.G + k ];
    }
    __syncwarp();
  }
}

// One CTA per owner (and, blockIdx.y, near or far): its counts become segment
// starts in quads of edges (entry n: its total).
__global__ void __launch_bounds__( 1024 )
k_own_scan( const OwnCta* cta, const long long* rp_base, uint32_t* rp_near, uint32_t* rp_far, unsigned long long* total )
{
  uint32_t* const rp = blockIdx.y ? rp_far : rp_near;
  __shared__ unsigned s_w[ 32 ];
  __shared__ unsigned s_carry;
  const int n = cta[ blockIdx.x ].n;
  uint32_t* const p = rp + rp_base[ blockIdx.x ];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  if ( threadIdx.x == 0 )
    s_carry = 0u;
  __syncthreads();
  for ( int k0 = 0; k0 < n; k0 += 1024 )
  {
    const int k = k0 + ( int ) threadIdx.x;
    const unsigned v = k < n ? ( p[ k ] + 3u ) >> 2 : 0u;
    unsigned x = v;
#pragma unroll
    for ( int s = 1; s < 32; s <<= 1 )
    {
      const unsigned y = __shfl_up_sync( FULL, x, s );
      if ( lane >= s )
        x += y;
    }
    if ( lane == 31 )
      s_w[ warp ] = x;
    __syncthreads();
    unsigned before = s_carry;
    for ( int w = 0; w < warp; ++w )
      before += s_w[ w ];
    if ( k < n )
      p[ k ] = before + x - v;
    __syncthreads();
    if ( threadIdx.x == 1023 )
      s_carry = before + x;
    __syncthreads();
  }
  if ( threadIdx.x == 0 )
  {
    p[ n ] = s_carry;
    total[ blockIdx.y * gridDim.x + blockIdx.x ] = s_carry;
  }
}

// The words that pad the segments, everywhere before the edges are written.
__global__ void
k_own_pad( int w16, int pair, size_t n, uint32_t v, uint32_t* word )
{
  for ( size_t k = ( size_t ) blockIdx.x * blockDim.x + threadIdx.x; k < n; k += ( size_t ) gridDim.x * blockDim.x )
    if ( w16 )
      reinterpret_cast< uint16_t* >( word )[ k ] = ( uint16_t ) v;
    else if ( pair )
      reinterpret_cast< uint2* >( word )[ k ] = make_uint2( v, 0u );
    else
      word[ k ] = v;
}

// An edge's owner segment (near: owner, far: G + owner) and its word.
template < typename T >
__device__ __forceinline__ unsigned
own_place( const OwnBuild& q, uint32_t t, T w, bool by_sign, int nl, uint32_t& x )
{
  const int dl = ( int ) ( ( t >> q.tbits ) & q.dmask );
  const unsigned l = ( t & q.tmask ) - ( unsigned ) q.a, c = l / ( unsigned ) q.G, own = l - c * ( unsigned ) q.G;
  const unsigned cl = by_sign ? ( w < T( 0 ) ? 1u : 0u ) : t >> 31;
  x = ( ( uint32_t ) dl * ( uint32_t ) nl + c ) | ( cl << 31 );
  return own + ( dl > q.d_near ? q.G : 0 );
}

__device__ __forceinline__ uint16_t
own_word16( uint32_t x )
{
  return ( uint16_t ) ( ( x & 0x7fffu ) | ( x >> 16 & 0x8000u ) );
}

// Edges into the owners' segments (any order within a segment), a row per
// warp: rows of a few edges per segment.
template < typename T, int CELL >
__global__ void __launch_bounds__( 256 )
k_own_fill( OwnBuild q, int w16, int nl, const long long* e_near, const long long* e_far, uint32_t* word, double* weight )
{
  __shared__ unsigned s_at[ 8 ][ 2 * OW_MAX_G ];
  __shared__ long long s_base[ 2 * OW_MAX_G ];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int G2 = q.rp_far ? 2 * q.G : q.G;
  for ( int k = threadIdx.x; k < G2; k += blockDim.x )
    s_base[ k ] = 4 * ( k < q.G ? e_near[ q.c0 + k ] : e_far[ q.c0 + k - q.G ] );
  __syncthreads();
  for ( long long s = ( long long ) blockIdx.x * 8 + warp; s < q.n; s += ( long long ) gridDim.x * 8 )
  {
    for ( int k = lane; k < G2; k += 32 )
      s_at[ warp ][ k ] = 4u
        * ( k < q.G ? q.rp[ q.rp_base[ q.c0 + k ] + s ] : q.rp_far[ q.rp_base[ q.c0 + k - q.G ] + s ] );
    __syncwarp();
    const long long r0 = q.row_beg[ q.a + s ];
    const int deg = q.real_deg[ q.a + s ];
    for ( int j = lane; j < deg; j += 32 )
    {
      const T w = ( ( const T* ) q.w )[ r0 + j ];
      if ( w == T( 0 ) )
        continue;
      uint32_t x;
      const unsigned seg = own_place( q, q.tdc[ r0 + j ], w, q.split && CELL == OW_COUNT, nl, x );
      const long long e = s_base[ seg ] + atomicAdd( &s_at[ warp ][ seg ], 1u );
      if ( CELL == OW_I64 )
        reinterpret_cast< uint2* >( word )[ e ] = make_uint2( x, ( uint32_t ) ( int ) w );
      else if ( CELL == OW_COUNT && w16 )
        reinterpret_cast< uint16_t* >( word )[ e ] = own_word16( x );
      else
      {
        word[ e ] = x;
        if ( CELL == OW_F64 )
          weight[ e ] = ( double ) w;
      }
    }
    __syncwarp();
  }
}

// Bytes of a quad of edges in the staging buffer: words, and FP64 weights.
__host__ __device__ inline int
own_quad_bytes( int cell, int w16 )
{
  return cell == OW_I64 ? 32 : cell == OW_F64 ? 48 : w16 ? 8 : 16;
}

constexpr int OW_FILL_SMEM = 73728;  // three CTAs' staging buffers fit an SM

// The same for long rows, a row per CTA: the row's segments are put together
// in shared memory, padding included, and written out whole.  (Written edge by
// edge, each to a sector of its own, 4.6e8 edges took 12.6 ms.)  Segments that
// do not fit the buffer together are taken in rounds over the row, one that
// does not fit it alone edge by edge.
template < typename T, int CELL >
__global__ void __launch_bounds__( 512 )
k_own_fill_rows( OwnBuild q, int w16, int nl, uint32_t pad, const long long* e_near, const long long* e_far, uint32_t* word,
  double* weight )
{
  extern __shared__ __align__( 16 ) unsigned char f_smem[];
  __shared__ long long s_base[ 2 * OW_MAX_G ];   // a segment's first quad
  __shared__ int s_p[ 2 * OW_MAX_G + 1 ];        // ... its place in the row's segments one after the other [quads]
  __shared__ unsigned s_cnt[ 2 * OW_MAX_G ];
  __shared__ int s_w[ 16 ];
  static_assert( 2 * OW_MAX_G == 512, "a thread per segment" );
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int G2 = q.rp_far ? 2 * q.G : q.G, cap = OW_FILL_SMEM / own_quad_bytes( CELL, w16 );
  uint32_t* const b32 = reinterpret_cast< uint32_t* >( f_smem );
  uint2* const b64 = reinterpret_cast< uint2* >( f_smem );
  uint16_t* const b16 = reinterpret_cast< uint16_t* >( f_smem );
  double* const bw = reinterpret_cast< double* >( f_smem + ( size_t ) cap * 16 );  // (OW_F64)
  for ( long long s = blockIdx.x; s < q.n; s += gridDim.x )
  {
    int len = 0;
    if ( tid < G2 )
    {
      const bool far = tid >= q.G;
      const int c = q.c0 + ( far ? tid - q.G : tid );
      const uint32_t* const rp = ( far ? q.rp_far : q.rp ) + q.rp_base[ c ] + s;
      len = ( int ) ( rp[ 1 ] - rp[ 0 ] );
      s_base[ tid ] = ( far ? e_far[ c ] : e_near[ c ] ) + rp[ 0 ];
    }
    int x = len;
#pragma unroll
    for ( int d = 1; d < 32; d <<= 1 )
    {
      const int y = __shfl_up_sync( FULL, x, d );
      if ( lane >= d )
        x += y;
    }
    if ( lane == 31 )
      s_w[ warp ] = x;
    __syncthreads();
    for ( int k = 0; k < warp; ++k )
      x += s_w[ k ];
    s_p[ tid + 1 ] = x;
    if ( tid == 0 )
      s_p[ 0 ] = 0;
    __syncthreads();
    const long long r0 = q.row_beg[ q.a + s ];
    const int deg = q.real_deg[ q.a + s ];
    for ( int k0 = 0; k0 < G2; )
    {
      // segments k0 .. k1 - 1 fit the buffer together
      int k1 = k0, hi = G2;
      while ( k1 < hi )
      {
        const int mid = ( k1 + hi + 1 ) >> 1;
        if ( s_p[ mid ] - s_p[ k0 ] <= cap )
          k1 = mid;
        else
          hi = mid - 1;
      }
      const bool staged = k1 > k0;
      if ( !staged )
        k1 = k0 + 1;
      const int p0 = s_p[ k0 ], nq = s_p[ k1 ] - p0;
      if ( tid >= k0 && tid < k1 )
        s_cnt[ tid ] = 0u;
      if ( staged )
      {
        for ( int k = tid; k < 4 * nq; k += 512 )
          if ( CELL == OW_I64 )
            b64[ k ] = make_uint2( pad, 0u );
          else if ( CELL == OW_COUNT && w16 )
            b16[ k ] = ( uint16_t ) pad;
          else
          {
            b32[ k ] = pad;
            if ( CELL == OW_F64 )
              bw[ k ] = 0.0;
          }
      }
      __syncthreads();
#pragma unroll 4
      for ( int j = tid; j < deg; j += 512 )
      {
        const T w = ( ( const T* ) q.w )[ r0 + j ];
        const uint32_t t = q.tdc[ r0 + j ];
        if ( w == T( 0 ) )
          continue;
        uint32_t v;
        const int seg = ( int ) own_place( q, t, w, q.split && CELL == OW_COUNT, nl, v );
        if ( seg < k0 || seg >= k1 )
          continue;
        const unsigned at = atomicAdd( &s_cnt[ seg ], 1u );
        if ( staged )
        {
          const unsigned e = 4u * ( unsigned ) ( s_p[ seg ] - p0 ) + at;
          if ( CELL == OW_I64 )
            b64[ e ] = make_uint2( v, ( uint32_t ) ( int ) w );
          else if ( CELL == OW_COUNT && w16 )
            b16[ e ] = own_word16( v );
          else
          {
            b32[ e ] = v;
            if ( CELL == OW_F64 )
              bw[ e ] = ( double ) w;
          }
        }
        else
        {
          const long long e = 4 * s_base[ seg ] + at;
          if ( CELL == OW_I64 )
            reinterpret_cast< uint2* >( word )[ e ] = make_uint2( v, ( uint32_t ) ( int ) w );
          else if ( CELL == OW_COUNT && w16 )
            reinterpret_cast< uint16_t* >( word )[ e ] = own_word16( v );
          else
          {
            word[ e ] = v;
            if ( CELL == OW_F64 )
              weight[ e ] = ( double ) w;
          }
        }
      }
      __syncthreads();
      if ( staged )
      {
        for ( int k = k0 + warp; k < k1; k += 16 )
        {
          const int l0 = s_p[ k ] - p0, n = s_p[ k + 1 ] - s_p[ k ];
          const long long g0 = s_base[ k ];
          if ( CELL == OW_COUNT && w16 )
          {
            for ( int u = lane; u < n; u += 32 )
              reinterpret_cast< uint2* >( word )[ g0 + u ] = reinterpret_cast< const uint2* >( f_smem )[ l0 + u ];
          }
          else
          {
            constexpr int V = CELL == OW_I64 ? 2 : 1;  // 16-byte pieces of a quad's words
            for ( int u = lane; u < V * n; u += 32 )
              reinterpret_cast< uint4* >( word )[ V * g0 + u ] = reinterpret_cast< const uint4* >( f_smem )[ V * l0 + u ];
            if ( CELL == OW_F64 )
              for ( int u = lane; u < 2 * n; u += 32 )
                reinterpret_cast< double2* >( weight )[ 2 * g0 + u ] = reinterpret_cast< const double2* >( bw )[ 2 * l0 + u ];
          }
        }
      }
      else
        for ( long long e = 4 * s_base[ k0 ] + s_cnt[ k0 ] + tid; e < 4 * ( s_base[ k0 ] + nq ); e += 512 )
        {
          // the padding of a segment written edge by edge
          if ( CELL == OW_I64 )
            reinterpret_cast< uint2* >( word )[ e ] = make_uint2( pad, 0u );
          else if ( CELL == OW_COUNT && w16 )
            reinterpret_cast< uint16_t* >( word )[ e ] = ( uint16_t ) pad;
          else
          {
            word[ e ] = pad;
            if ( CELL == OW_F64 )
              weight[ e ] = 0.0;
          }
        }
      __syncthreads();  // (the buffer and counters are used again)
      k0 = k1;
    }
  }
}

// The largest in-degree of a neuron and input class, from the owners' copies:
// one CTA per owner counts its columns in shared memory (an L2 atomic per edge
// as the rows are read took as long again as the reading).
template < int CELL >
__global__ void __launch_bounds__( 1024 )
k_own_indeg( OwnNet o, const unsigned long long* total, unsigned* most )
{
  __shared__ unsigned s_h[ 2 ][ 2 * OW_TPB + 1 ];
  for ( int k = threadIdx.x; k < 2 * OW_TPB + 1; k += blockDim.x )
    s_h[ 0 ][ k ] = s_h[ 1 ][ k ] = 0u;
  __syncthreads();
  const bool w16 = CELL == OW_COUNT && o.w16;
  for ( int f = 0; f <= o.far; ++f )
  {
    const long long base = f ? o.e_far[ blockIdx.x ] : o.e_base[ blockIdx.x ];
    const long long n = ( long long ) total[ f * gridDim.x + blockIdx.x ];
    for ( long long k = threadIdx.x; k < n; k += blockDim.x )
    {
      OwnQuad< CELL > x;
      own_load< CELL >( o, base + k, x );
#pragma unroll
      for ( int e = 0; e < 4; ++e )
        atomicAdd( &s_h[ w16 ? x.t[ e ] >> 15 : x.t[ e ] >> 31 ][ ( x.t[ e ] & ( w16 ? 0x7fffu : 0x7fffffffu ) ) % ( unsigned ) o.nl ],
          1u );
    }
  }
  __syncthreads();
  unsigned m = 0;
  for ( int k = threadIdx.x; k < o.nl - 1; k += blockDim.x )  // (column nl - 1: the segments' padding)
    m = max( m, max( s_h[ 0 ][ k ], s_h[ 1 ][ k ] ) );
  m = __reduce_max_sync( FULL, m );
  if ( ( threadIdx.x & 31 ) == 0 && m )
    atomicMax( most, m );
}

}  // namespace ng
