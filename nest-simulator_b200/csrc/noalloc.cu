// noalloc.cu -- ng_simulate_noalloc: the slice cycle of a small iaf_psc_delta
// network (plain FP64 form) that allocates no memory at all.
//
// Who needs it: callers that may not allocate device memory on the path
// that steps the network -- e.g. a host framework that owns all device
// memory through its own allocator or memory pool and forbids foreign
// cudaMalloc calls, or a closed-loop controller that steps a small network
// every control tick, where an allocation's implicit device synchronisation
// and latency jitter are not acceptable.  The caller passes every input and
// output as device memory it owns; the ring buffer, the per-slice spike list
// and the control counters live in one file-scope device array
// (g_noalloc_scratch, NG_NOALLOC_SCRATCH_BYTES = 16 MiB) that every GPU
// which loads the library holds until the process exits.
//
// The kernels are variants of the engine's node-update and delivery kernels
// (ng_kernels.cuh) for unpadded CSR input: same arithmetic in the same order,
// so a run matches ng_simulate on the same network.  A controller that steps
// the network a few steps per tick sets continue_run: the ring buffer and
// the open slice's spikes stay in the scratch array between its calls, and
// a chain of calls equals one call over the same steps.  The edges come from
// caller memory and are range-checked on the device before they index the
// ring.
#include <cstddef>
#include <cstdint>
#include <algorithm>
#include <mutex>

#include <cuda_runtime.h>

#include "../../include/nestgpu.h"

namespace
{

constexpr int NA_MAX_DEVICES = 64;

__device__ __align__( 256 ) unsigned char g_noalloc_scratch[ NG_NOALLOC_SCRATCH_BYTES ];

// counters at the start of the scratch array
struct NaCtl
{
  unsigned long long n_spk;   // spikes of the open slice
  unsigned long long n_out;   // spikes of this call (written to the caller's output up to out_cap)
  unsigned long long n_skip;  // edges of this call skipped for an out-of-range target or delay
};

// Where the previous call on a device stopped, for continue_run: the
// scratch array holds that run's ring and open-slice spike list.
struct NaRun
{
  bool valid = false;
  int64_t n = 0;
  int32_t min_delay = 0, max_delay = 0;
  int64_t next_step = 0;
};

struct NaNet
{
  int64_t n;
  int32_t L, min_delay, max_delay;
  const double *P33, *P30, *V_th, *V_reset, *V_min, *I_e;
  const int32_t* refr_counts;
  double* V;
  int32_t* r;
  const int64_t* row_ptr;
  const int32_t* target;
  const double* weight;
  const int32_t* delay;
  int32_t* out_src;
  int64_t* out_stamp;
  int64_t out_cap;
  unsigned long long* out_count;
  unsigned long long* out_skipped;
  // scratch
  NaCtl* ctl;
  double* ring;     // [L][n]
  int2* spk;       // (source, emission slot)
  int64_t spk_cap;
};

// iaf_psc_delta::update (models/iaf_psc_delta.cpp:272-329), one thread per
// neuron over the lags [from, to) of the slice at `origin`.
__global__ void
k_na_update( NaNet d, long long origin, int from, int to )
{
  const int64_t i = ( int64_t ) blockIdx.x * blockDim.x + threadIdx.x;
  if ( i >= d.n )
    return;
  double V = d.V[ i ];
  int r = d.r[ i ];
  const double P33 = d.P33[ i ], P30 = d.P30[ i ], Vth = d.V_th[ i ], Vreset = d.V_reset[ i ], Vmin = d.V_min[ i ];
  const double Ie = d.I_e[ i ];
  const int refr = d.refr_counts[ i ];
  const double y0 = 0.0;
  for ( int lag = from; lag < to; ++lag )
  {
    const long long t = origin + lag;
    const int slot = ( int ) ( t % d.L );
    const double in = d.ring[ ( int64_t ) slot * d.n + i ];
    d.ring[ ( int64_t ) slot * d.n + i ] = 0.0;
    if ( r == 0 )
    {
      V = P30 * ( y0 + Ie ) + P33 * V + in;
      V = ( V < Vmin ? Vmin : V );
    }
    else
    {
      --r;
    }
    if ( V >= Vth )
    {
      r = refr;
      V = Vreset;
      const unsigned long long k = atomicAdd( &d.ctl->n_spk, 1ull );
      if ( ( int64_t ) k < d.spk_cap )
        d.spk[ k ] = make_int2( ( int ) i, slot );
      const unsigned long long o = atomicAdd( &d.ctl->n_out, 1ull );
      if ( ( int64_t ) o < d.out_cap )
      {
        d.out_src[ o ] = ( int32_t ) i;
        d.out_stamp[ o ] = t + 1;
      }
    }
  }
  d.V[ i ] = V;
  d.r[ i ] = r;
}

// Delivery of the closing slice: one warp per spike walks its CSR row and
// adds the weights into ring[(t_emit + d) mod L][target].  The edges come
// from caller memory: one whose target or delay is out of range would index
// outside the ring, so it is skipped and counted instead.
__global__ void
k_na_deliver( NaNet d )
{
  const unsigned long long nspk = *( volatile unsigned long long* ) &d.ctl->n_spk;
  const int64_t warp = ( ( int64_t ) blockIdx.x * blockDim.x + threadIdx.x ) >> 5;
  const int lane = threadIdx.x & 31;
  const int64_t nw = ( ( int64_t ) gridDim.x * blockDim.x ) >> 5;
  const int64_t ns = ( int64_t ) nspk < d.spk_cap ? ( int64_t ) nspk : d.spk_cap;
  for ( int64_t s = warp; s < ns; s += nw )
  {
    const int2 sp = d.spk[ s ];
    const int64_t e0 = d.row_ptr[ sp.x ], e1 = d.row_ptr[ sp.x + 1 ];
    for ( int64_t e = e0 + lane; e < e1; e += 32 )
    {
      const int32_t tg = d.target[ e ];
      const int32_t dl = d.delay[ e ];
      if ( tg < 0 || ( int64_t ) tg >= d.n || dl < d.min_delay || dl > d.max_delay )
      {
        atomicAdd( &d.ctl->n_skip, 1ull );
        continue;
      }
      int slot = sp.y + dl;  // sp.y < L and dl <= max_delay < L
      if ( slot >= d.L )
        slot -= d.L;
      atomicAdd( d.ring + ( int64_t ) slot * d.n + tg, d.weight[ e ] );
    }
  }
}

// ---------------------------------------------------------------------
// A call on a network of up to NA_CL_CTAS x NA_CL_TPB neurons in one launch: one
// cluster of CTAs, one thread per neuron.  A CTA keeps its neurons' state in
// registers and its own spikes of the open slice in shared memory, delivers
// them itself when the slice closes (the ring holds min_delay + max_delay
// slots, so a delivery meets no cell that another CTA still has to read), and
// one cluster barrier per slice orders the deliveries before the next update.
// The launches of the kernels above, three per slice, each with its fixed
// cost, were the time of a controller's call.  The ring cells of up to NA_LAGS
// lags are read ahead of the recurrence, whose lags would else wait for one L2
// round trip each.
// Why 16 CTAs: the adds of a busy network are issued by the cluster's SMs
// alone, where the per-slice launches have 64 CTAs on as many SMs.  Ten slices
// by 8 CTAs, by 16, by launches [us]: 1,000 neurons x 100 inputs at 68 Hz 80,
// 75, 237; 4,000 x 600 at 116 Hz 470, 292, 399; 8,192 x 600 at 188 Hz 1,255,
// 753, 963; 8,192 x 2,000 at 300 Hz 5,992, 3,419, 5,446.  With 16 the one launch
// was the faster form at every size from 100 neurons and every rate up to what
// refractoriness allows (25 to 2,000 inputs); with 8 it was the slower one above
// some 1e6 edges at 70 to 200 Hz.  Networks of up to NA_CL_SMALL neurons have so
// few adds that the dearer barrier of 16 CTAs is what remains (257 neurons, 285
// steps: 127.0 us with 8, 128.5 with 16; 319, 164 steps: 75.8 and 77.5; 587 and
// more: 16 no slower).
// ---------------------------------------------------------------------
constexpr int NA_CL_CTAS = 16;  // (above the portable 8: a device that cannot place it takes the launches per slice)
constexpr int NA_CL_SMALL = 512;
constexpr int NA_CL_TPB = 512;  // threads per CTA: the neurons, and warps to share the deliveries
constexpr int NA_LAGS = 8;
constexpr int NA_LIST = NA_CL_TPB * NA_LAGS;  // a CTA's spikes held at a time

__device__ __forceinline__ void
na_cluster_sync()
{
  asm volatile( "barrier.cluster.arrive.release.aligned;" ::: "memory" );
  asm volatile( "barrier.cluster.wait.acquire.aligned;" ::: "memory" );
}

// one warp: the edges of a spike (source, emission slot)
__device__ __forceinline__ void
na_deliver_spike( const NaNet& d, int src, int slot0, unsigned long long& skipped )
{
  const int64_t e1 = d.row_ptr[ src + 1 ];
  for ( int64_t e0 = d.row_ptr[ src ] + ( threadIdx.x & 31 ); e0 < e1; e0 += 128 )
  {
    // four edges per lane in flight
    int32_t tg[ 4 ], dl[ 4 ];
    double w[ 4 ];
#pragma unroll
    for ( int u = 0; u < 4; ++u )
    {
      const int64_t e = e0 + 32 * u;
      tg[ u ] = e < e1 ? d.target[ e ] : 0;
      dl[ u ] = e < e1 ? d.delay[ e ] : 0;
      w[ u ] = e < e1 ? d.weight[ e ] : 0.0;
    }
#pragma unroll
    for ( int u = 0; u < 4; ++u )
    {
      if ( e0 + 32 * u >= e1 )
        continue;
      if ( tg[ u ] < 0 || ( int64_t ) tg[ u ] >= d.n || dl[ u ] < d.min_delay || dl[ u ] > d.max_delay )
      {
        ++skipped;
        continue;
      }
      int slot = slot0 + dl[ u ];  // slot0 < L and dl <= max_delay < L
      if ( slot >= d.L )
        slot -= d.L;
      atomicAdd( d.ring + ( int64_t ) slot * d.n + tg[ u ], w[ u ] );
    }
  }
}

__global__ void __launch_bounds__( NA_CL_TPB )
k_na_run( NaNet d, int per, long long start, long long n_steps, int fresh )
{
  __shared__ uint32_t s_list[ NA_LIST ];  // local neuron, lag of the chunk << 16
  __shared__ int s_n;
  __shared__ unsigned long long s_out;
  const int tid = threadIdx.x, warp = tid >> 5, nw = blockDim.x >> 5;
  const int64_t i0 = ( int64_t ) blockIdx.x * per, i = i0 + tid;  // `per` neurons per CTA
  const bool act = tid < per && i < d.n;
  const bool first = blockIdx.x == 0 && tid == 0;
  if ( fresh )
  {
    // counters and ring of a new run
    for ( int64_t k = ( int64_t ) blockIdx.x * blockDim.x + tid; k < ( int64_t ) d.L * d.n;
          k += ( int64_t ) gridDim.x * blockDim.x )
      d.ring[ k ] = 0.0;
    if ( first )
      d.ctl->n_spk = 0ull;
  }
  if ( first )
    d.ctl->n_out = d.ctl->n_skip = 0ull;
  if ( tid == 0 )
    s_n = 0;
  double V = 0, P33 = 0, Vth = 0, Vreset = 0, Vmin = 0, drive = 0;
  int r = 0, refr = 0;
  if ( act )
  {
    const double y0 = 0.0;
    V = d.V[ i ];
    r = d.r[ i ];
    P33 = d.P33[ i ];
    Vth = d.V_th[ i ];
    Vreset = d.V_reset[ i ];
    Vmin = d.V_min[ i ];
    refr = d.refr_counts[ i ];
    drive = d.P30[ i ] * ( y0 + d.I_e[ i ] );
  }
  unsigned long long skipped = 0;
  long long t = start;
  const long long end = start + n_steps;
  // spikes of the open slice that earlier calls left; where it closes in this
  // call the list is emptied once every CTA has read its length (a slice left
  // open at the end adds to it behind the first close's barrier)
  const unsigned long long n_old = fresh ? 0ull : __ldcg( &d.ctl->n_spk );
  const int64_t old = ( int64_t ) n_old < d.spk_cap ? ( int64_t ) n_old : d.spk_cap;
  bool old_open = old > 0;
  int slot_t = ( int ) ( t % d.L );
  long long close = t - t % d.min_delay + d.min_delay;  // the open slice's end
  na_cluster_sync();
  if ( first && close <= end )
    d.ctl->n_spk = 0ull;
  while ( t < end )
  {
    const long long to = close < end ? close : end;
    while ( t < to )
    {
      const int nk = ( int ) ( to - t < NA_LAGS ? to - t : NA_LAGS );
      const int slot0 = slot_t;
      double in[ NA_LAGS ];
#pragma unroll
      for ( int k = 0; k < NA_LAGS; ++k )
      {
        int slot = slot0 + k;
        if ( slot >= d.L )
          slot -= d.L;
        in[ k ] = act && k < nk ? __ldcg( d.ring + ( int64_t ) slot * d.n + i ) : 0.0;
      }
      unsigned mask = 0;
#pragma unroll
      for ( int k = 0; k < NA_LAGS; ++k )
        if ( act && k < nk )
        {
          double Vn = drive + P33 * V + in[ k ];
          Vn = ( Vn < Vmin ? Vmin : Vn );
          V = r == 0 ? Vn : V;
          r = r == 0 ? 0 : r - 1;
          const bool spk = V >= Vth;
          r = spk ? refr : r;
          V = spk ? Vreset : V;
          mask |= ( spk ? 1u : 0u ) << k;
        }
#pragma unroll
      for ( int k = 0; k < NA_LAGS; ++k )
        if ( in[ k ] != 0.0 )
        {
          int slot = slot0 + k;
          if ( slot >= d.L )
            slot -= d.L;
          d.ring[ ( int64_t ) slot * d.n + i ] = 0.0;
        }
      // the chunk's spikes: the CTA's list, the caller's output
      int at = 0;
      if ( mask )
        at = atomicAdd( &s_n, __popc( mask ) );
      __syncthreads();
      const int n_list = s_n;
      if ( n_list > 0 )
      {
        unsigned long long out0 = 0ull;
        if ( tid == 0 )
          out0 = atomicAdd( &d.ctl->n_out, ( unsigned long long ) n_list );
        int q = at;
        for ( unsigned m = mask; m; m &= m - 1 )
          s_list[ q++ ] = ( uint32_t ) tid | ( uint32_t ) ( __ffs( m ) - 1 ) << 16;
        __syncthreads();
        if ( close <= end )
        {
          // the slice closes in this call: deliver (arrivals lie past its end)
          for ( int k = warp; k < n_list; k += nw )
          {
            int slot = slot0 + ( int ) ( s_list[ k ] >> 16 );
            if ( slot >= d.L )
              slot -= d.L;
            na_deliver_spike( d, ( int ) ( i0 + ( s_list[ k ] & 0xffffu ) ), slot, skipped );
          }
        }
        else
        {
          // it stays open: a later call delivers them
          for ( int k = tid; k < n_list; k += blockDim.x )
          {
            int slot = slot0 + ( int ) ( s_list[ k ] >> 16 );
            if ( slot >= d.L )
              slot -= d.L;
            const unsigned long long p = atomicAdd( &d.ctl->n_spk, 1ull );
            if ( ( int64_t ) p < d.spk_cap )
              d.spk[ p ] = make_int2( ( int ) ( i0 + ( s_list[ k ] & 0xffffu ) ), slot );
          }
        }
        if ( tid == 0 )
          s_out = out0;
        __syncthreads();  // (the list's last readers, too)
        int64_t o = ( int64_t ) s_out + at;
        for ( unsigned m = mask; m; m &= m - 1, ++o )
          if ( o < d.out_cap )
          {
            d.out_src[ o ] = ( int32_t ) i;
            d.out_stamp[ o ] = t + __ffs( m );
          }
        if ( tid == 0 )
          s_n = 0;
      }
      __syncthreads();
      t += nk;
      slot_t += nk;
      if ( slot_t >= d.L )
        slot_t -= d.L;
    }
    if ( t == close )
    {
      if ( old_open )
      {
        for ( int64_t k = ( int64_t ) blockIdx.x * nw + warp; k < old; k += ( int64_t ) gridDim.x * nw )
        {
          const int2 sp = d.spk[ k ];
          na_deliver_spike( d, sp.x, sp.y, skipped );
        }
        old_open = false;
      }
      close += d.min_delay;
      na_cluster_sync();
    }
  }
  if ( act )
  {
    d.V[ i ] = V;
    d.r[ i ] = r;
  }
  if ( skipped )
    atomicAdd( &d.ctl->n_skip, skipped );
  na_cluster_sync();
  if ( first )
  {
    *d.out_count = __ldcg( &d.ctl->n_out );
    if ( d.out_skipped )
      *d.out_skipped = __ldcg( &d.ctl->n_skip );
  }
}

__global__ void
k_na_close_slice( NaNet d )
{
  d.ctl->n_spk = 0ull;
}

// A continued run keeps the ring and the open slice's spikes; only the
// per-call counters start from zero.
__global__ void
k_na_begin_call( NaNet d )
{
  d.ctl->n_out = 0ull;
  d.ctl->n_skip = 0ull;
}

__global__ void
k_na_finish( NaNet d )
{
  *d.out_count = d.ctl->n_out;
  if ( d.out_skipped )
    *d.out_skipped = d.ctl->n_skip;
}

std::mutex g_na_mutex;
void* g_na_addr[ NA_MAX_DEVICES ] = {};
NaRun g_na_run[ NA_MAX_DEVICES ];
int g_na_cluster[ NA_MAX_DEVICES ] = {};  // 0: not asked yet, 1: the device places k_na_run's cluster, -1: not

}  // namespace

void ng_internal_set_error( const char* msg );

extern "C" {

int
ng_simulate_noalloc( const ng_noalloc_net* net, int64_t n_steps, void* cuda_stream )
{
  if ( !net || n_steps < 0 )
  {
    ng_internal_set_error( "ng_simulate_noalloc: null network or negative step count" );
    return NG_ERR_ARG;
  }
  if ( net->n < 1 || net->n > INT32_MAX || net->min_delay < 1 || net->max_delay < net->min_delay
    || net->start_step < 0 || net->out_cap < 0 || ( net->continue_run != 0 && net->continue_run != 1 )
    || net->reserved != 0 )
  {
    ng_internal_set_error( "ng_simulate_noalloc: need 1 <= n < 2^31, 1 <= min_delay <= max_delay, start_step >= 0, "
                           "out_cap >= 0, continue_run 0 or 1, reserved 0" );
    return NG_ERR_ARG;
  }
  if ( !net->continue_run && net->start_step % net->min_delay != 0 )
  {
    ng_internal_set_error( "ng_simulate_noalloc: a fresh run starts at a slice boundary (start_step a multiple of "
                           "min_delay)" );
    return NG_ERR_ARG;
  }
  if ( !net->P33 || !net->P30 || !net->V_th_rel || !net->V_reset_rel || !net->V_min_rel || !net->I_e
    || !net->refr_counts || !net->V_m_rel || !net->r || !net->row_ptr || !net->target || !net->weight || !net->delay
    || !net->out_src || !net->out_stamp || !net->out_count )
  {
    ng_internal_set_error( "ng_simulate_noalloc: a required device pointer is null" );
    return NG_ERR_ARG;
  }
  int dev = 0;
  if ( cudaGetDevice( &dev ) != cudaSuccess || dev < 0 || dev >= NA_MAX_DEVICES )
  {
    ng_internal_set_error( "ng_simulate_noalloc: no current CUDA device" );
    return NG_ERR_CUDA;
  }
  const int64_t L = ( int64_t ) net->min_delay + net->max_delay;
  // scratch layout: [NaCtl | pad to 256][ring L*n doubles][spike list n*min_delay int2]
  const size_t ctl_bytes = 256;
  const size_t ring_bytes = ( size_t ) L * ( size_t ) net->n * sizeof( double );
  const size_t spk_cap = ( size_t ) net->n * ( size_t ) net->min_delay;
  const size_t need = ctl_bytes + ( ( ring_bytes + 255 ) & ~( size_t ) 255 ) + spk_cap * sizeof( int2 );
  if ( L > INT32_MAX / 2 || need > NG_NOALLOC_SCRATCH_BYTES )
  {
    ng_internal_set_error( "ng_simulate_noalloc: the network's ring buffer and spike list need more than the "
                           "16 MiB static scratch array (NG_NOALLOC_SCRATCH_BYTES)" );
    return NG_ERR_CAPACITY;
  }
  std::lock_guard< std::mutex > lock( g_na_mutex );
  // once per device, with that device current: the scratch array's device
  // address (the symbol itself names a host-side stand-in)
  if ( !g_na_addr[ dev ] )
  {
    if ( cudaGetSymbolAddress( &g_na_addr[ dev ], g_noalloc_scratch ) != cudaSuccess )
    {
      g_na_addr[ dev ] = nullptr;
      ng_internal_set_error( "ng_simulate_noalloc: cudaGetSymbolAddress of the scratch array failed" );
      return NG_ERR_CUDA;
    }
  }
  void* const base = g_na_addr[ dev ];
  NaRun& run = g_na_run[ dev ];
  if ( net->continue_run
    && !( run.valid && run.n == net->n && run.min_delay == net->min_delay && run.max_delay == net->max_delay
      && run.next_step == net->start_step ) )
  {
    ng_internal_set_error( "ng_simulate_noalloc: continue_run needs the previous call on this device to have run the "
                           "same network (n, min_delay, max_delay) up to start_step" );
    return NG_ERR_STATE;
  }
  cudaStream_t st = ( cudaStream_t ) cuda_stream;
  NaNet d {};
  d.n = net->n;
  d.L = ( int32_t ) L;
  d.min_delay = net->min_delay;
  d.max_delay = net->max_delay;
  d.P33 = net->P33;
  d.P30 = net->P30;
  d.V_th = net->V_th_rel;
  d.V_reset = net->V_reset_rel;
  d.V_min = net->V_min_rel;
  d.I_e = net->I_e;
  d.refr_counts = net->refr_counts;
  d.V = net->V_m_rel;
  d.r = net->r;
  d.row_ptr = net->row_ptr;
  d.target = net->target;
  d.weight = net->weight;
  d.delay = net->delay;
  d.out_src = net->out_src;
  d.out_stamp = net->out_stamp;
  d.out_cap = net->out_cap;
  d.out_count = net->out_count;
  d.out_skipped = net->out_skipped;
  d.ctl = ( NaCtl* ) base;
  d.ring = ( double* ) ( ( unsigned char* ) base + ctl_bytes );
  d.spk = ( int2* ) ( ( unsigned char* ) base + ctl_bytes + ( ( ring_bytes + 255 ) & ~( size_t ) 255 ) );
  d.spk_cap = ( int64_t ) spk_cap;
  // until this call has been enqueued, no later call may continue its run
  run.valid = false;
  cudaError_t ce;
  const int ctas = net->n <= NA_CL_SMALL ? NA_CL_CTAS / 2 : NA_CL_CTAS;
  cudaLaunchConfig_t lc = {};
  lc.gridDim = dim3( NA_CL_CTAS );
  lc.blockDim = dim3( NA_CL_TPB );
  lc.stream = st;
  cudaLaunchAttribute at[ 1 ];
  at[ 0 ].id = cudaLaunchAttributeClusterDimension;
  at[ 0 ].val.clusterDim.x = NA_CL_CTAS;
  at[ 0 ].val.clusterDim.y = 1;
  at[ 0 ].val.clusterDim.z = 1;
  lc.attrs = at;
  lc.numAttrs = 1;
  if ( !g_na_cluster[ dev ] )
  {
    // once per device: can it place the cluster?
    int clusters = 0;
    const bool ok = cudaFuncSetAttribute( k_na_run, cudaFuncAttributeNonPortableClusterSizeAllowed, 1 ) == cudaSuccess
      && cudaOccupancyMaxActiveClusters( &clusters, k_na_run, &lc ) == cudaSuccess && clusters > 0;
    if ( !ok )
      cudaGetLastError();  // (a refusal leaves no error behind)
    g_na_cluster[ dev ] = ok ? 1 : -1;
  }
  if ( net->n <= NA_CL_CTAS * NA_CL_TPB && g_na_cluster[ dev ] > 0 )
  {
    const int per = ( int ) ( ( net->n + ctas - 1 ) / ctas );
    lc.gridDim.x = at[ 0 ].val.clusterDim.x = ( unsigned ) ctas;
    if ( cudaLaunchKernelEx( &lc, k_na_run, d, per, ( long long ) net->start_step, ( long long ) n_steps,
           net->continue_run ? 0 : 1 )
      != cudaSuccess )
    {
      cudaGetLastError();
      ng_internal_set_error( "ng_simulate_noalloc: kernel launch failed" );
      return NG_ERR_CUDA;
    }
    run.valid = true;
    run.n = net->n;
    run.min_delay = net->min_delay;
    run.max_delay = net->max_delay;
    run.next_step = net->start_step + n_steps;
    return NG_OK;
  }
  if ( net->continue_run )
  {
    k_na_begin_call<<< 1, 1, 0, st >>>( d );
    ce = cudaGetLastError();
  }
  else
  {
    // a fresh run: counters and ring buffer to zero
    ce = cudaMemsetAsync( base, 0, ctl_bytes + ring_bytes, st );
  }
  if ( ce != cudaSuccess )
  {
    ng_internal_set_error( "ng_simulate_noalloc: clearing the scratch array failed" );
    return NG_ERR_CUDA;
  }
  const unsigned ugrid = ( unsigned ) ( ( net->n + 255 ) / 256 );
  const unsigned dgrid = 64;
  // slice origin and the lag the run stands at (a continued run may stop
  // and resume inside a slice; fresh runs start at a slice boundary)
  const int64_t lag0 = net->start_step % net->min_delay;
  long long origin = net->start_step - lag0;
  int from = ( int ) lag0;
  int64_t left = n_steps;
  while ( left > 0 )
  {
    const int to = ( int ) std::min< int64_t >( ( int64_t ) from + left, net->min_delay );
    k_na_update<<< ugrid, 256, 0, st >>>( d, origin, from, to );
    left -= to - from;
    if ( to == net->min_delay )
    {
      k_na_deliver<<< dgrid, 256, 0, st >>>( d );
      k_na_close_slice<<< 1, 1, 0, st >>>( d );
      origin += net->min_delay;
      from = 0;
    }
    else
    {
      from = to;
    }
  }
  k_na_finish<<< 1, 1, 0, st >>>( d );
  if ( cudaGetLastError() != cudaSuccess )
  {
    ng_internal_set_error( "ng_simulate_noalloc: kernel launch failed" );
    return NG_ERR_CUDA;
  }
  run.valid = true;
  run.n = net->n;
  run.min_delay = net->min_delay;
  run.max_delay = net->max_delay;
  run.next_step = net->start_step + n_steps;
  return NG_OK;
}

}  // extern "C"
