// Checks of caller arrays on the device, one read of each array: event offsets
// (order, ends) with their uint32 copy, event times (range), counts (largest).
// The findings come back in one block of int64 words, so that a call waits for
// the GPU once.  Bound by bandwidth, and by the waits that it saves: 108 million
// events, 20,000 frames, 1 Mpx 2.86 ms per call with separate reductions
// (0.16 ms of kernels, 8.7 MB copied as int64, four waits), 2.64 here.  A CSR
// stack's columns are read by the count pass anyway, which checks them: 445
// million elements 14.41 ms with a minimum and maximum first (0.28 ms, and 0.20
// of largest count against bandwidth), 13.87 without.
#include "g2_host.h"

namespace g2 {
namespace check {

constexpr int THREADS = 256;

// stats[0], stats[1]: first and last offset; stats[2]: a later offset is smaller.
template <typename To>
__global__ void __launch_bounds__(THREADS)
    offsets_kernel(const To* __restrict__ offsets, int64_t n, uint32_t* __restrict__ out,
                   unsigned long long* __restrict__ stats) {
  bool bad = false;
  for (int64_t i = static_cast<int64_t>(blockIdx.x) * THREADS + threadIdx.x; i < n;
       i += static_cast<int64_t>(gridDim.x) * THREADS) {
    const To v = offsets[i];
    out[i] = static_cast<uint32_t>(v);
    if (i + 1 < n) bad |= offsets[i + 1] < v;
    if (i == 0) stats[0] = static_cast<unsigned long long>(static_cast<long long>(v));
    if (i + 1 == n) stats[1] = static_cast<unsigned long long>(static_cast<long long>(v));
  }
  if (bad) stats[2] = 1;  // one value from any thread
}

// stats[3]: a time outside [0, T) (times given); stats[4]: the largest count;
// over the first min(n, *limit) elements (limit may be null).
template <typename Tv, bool TIMES>
__global__ void __launch_bounds__(THREADS)
    events_kernel(const int32_t* __restrict__ times, const Tv* __restrict__ data, int64_t n,
                  const long long* __restrict__ limit, int32_t T, unsigned long long* __restrict__ stats) {
  if (limit) {
    const long long m = *limit;
    if (m < n) n = m > 0 ? m : 0;
  }
  constexpr int PER = 16 / sizeof(Tv);  // counts of a 16-byte word
  const int64_t first = static_cast<int64_t>(blockIdx.x) * THREADS + threadIdx.x;
  const int64_t step = static_cast<int64_t>(gridDim.x) * THREADS;
  uint32_t most = 0;
  bool bad = false;
  auto one = [&](int64_t i) {
    most = max(most, static_cast<uint32_t>(data[i]));
    if (TIMES) bad |= static_cast<uint32_t>(times[i]) >= static_cast<uint32_t>(T);
  };
  // whole words where both arrays start on 16 bytes, single elements elsewhere
  const bool wide = ((reinterpret_cast<uintptr_t>(data) | (TIMES ? reinterpret_cast<uintptr_t>(times) : 0)) & 15) == 0;
  const int64_t words = wide ? n / PER : 0;
  for (int64_t w = first; w < words; w += step) {
    const uint4 q = reinterpret_cast<const uint4*>(data)[w];
    const uint32_t x[4] = {q.x, q.y, q.z, q.w};
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      if (sizeof(Tv) == 1) {
        most = max(most, max(max(x[k] & 255u, (x[k] >> 8) & 255u), max((x[k] >> 16) & 255u, x[k] >> 24)));
      } else {
        most = max(most, max(x[k] & 0xFFFFu, x[k] >> 16));
      }
    }
    if (TIMES) {
#pragma unroll
      for (int k = 0; k < PER / 4; ++k) {
        const uint4 t = reinterpret_cast<const uint4*>(times)[w * (PER / 4) + k];
        bad |= max(max(t.x, t.y), max(t.z, t.w)) >= static_cast<uint32_t>(T);  // negative: above 2^31
      }
    }
  }
  for (int64_t i = words * PER + first; i < n; i += step) one(i);
  most = __reduce_max_sync(0xffffffffu, most);
  __shared__ uint32_t s_most[THREADS / 32];
  if ((threadIdx.x & 31) == 0) s_most[threadIdx.x >> 5] = most;
  __syncthreads();
  if (threadIdx.x == 0) {
    for (int w = 1; w < THREADS / 32; ++w) most = max(most, s_most[w]);
    if (most) atomicMax(&stats[4], static_cast<unsigned long long>(most));
  }
  if (bad) stats[3] = 1;
}

}  // namespace check
}  // namespace g2

namespace {
int grid_for(int64_t n, int64_t per, unsigned* out) {
  const int sms = g2::sm_count_current();
  if (sms <= 0) return G2_ERR_CUDA;
  const int64_t want = (n + per - 1) / per, most = sms * 8ll;
  *out = static_cast<unsigned>(want < 1 ? 1 : want < most ? want : most);
  return G2_OK;
}
}  // namespace

extern "C" int g2_check_offsets(const void* offsets_dev, int32_t offset_bytes, int64_t n, uint32_t* out_dev,
                                int64_t* stats_dev, void* stream) {
  using namespace g2;
  if (!offsets_dev || !out_dev || !stats_dev || n <= 0 || (offset_bytes != 4 && offset_bytes != 8)) return G2_ERR_ARG;
  unsigned grid = 0;
  const int st = grid_for(n, check::THREADS, &grid);
  if (st != G2_OK) return st;
  auto* s = reinterpret_cast<unsigned long long*>(stats_dev);
  if (offset_bytes == 4)
    check::offsets_kernel<<<grid, check::THREADS, 0, as_stream(stream)>>>(reinterpret_cast<const int32_t*>(offsets_dev),
                                                                          n, out_dev, s);
  else
    check::offsets_kernel<<<grid, check::THREADS, 0, as_stream(stream)>>>(reinterpret_cast<const int64_t*>(offsets_dev),
                                                                          n, out_dev, s);
  return launch_status();
}

extern "C" int g2_check_events(const int32_t* times_dev, const void* data_dev, int32_t elem_bytes, int64_t n,
                               const int64_t* limit_dev, int32_t nframes, int64_t* stats_dev, void* stream) {
  using namespace g2;
  if (!data_dev || !stats_dev || n < 0 || (elem_bytes != 1 && elem_bytes != 2) || nframes <= 0 ||
      !aligned(data_dev, elem_bytes))
    return G2_ERR_ARG;
  if (n == 0) return G2_OK;
  unsigned grid = 0;
  const int st = grid_for(n, check::THREADS * 16, &grid);
  if (st != G2_OK) return st;
  auto* s = reinterpret_cast<unsigned long long*>(stats_dev);
  auto* lim = reinterpret_cast<const long long*>(limit_dev);
#define G2_EVENTS_CHECK(TV, TIMES)                                                                                   \
  check::events_kernel<TV, TIMES><<<grid, check::THREADS, 0, as_stream(stream)>>>(                                   \
      times_dev, reinterpret_cast<const TV*>(data_dev), n, lim, nframes, s)
  if (elem_bytes == 1 && times_dev) G2_EVENTS_CHECK(uint8_t, true);
  else if (elem_bytes == 1) G2_EVENTS_CHECK(uint8_t, false);
  else if (times_dev) G2_EVENTS_CHECK(uint16_t, true);
  else G2_EVENTS_CHECK(uint16_t, false);
#undef G2_EVENTS_CHECK
  return launch_status();
}
