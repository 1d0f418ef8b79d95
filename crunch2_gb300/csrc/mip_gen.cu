// Mip generation on the GPU: crnlib's mipmapped_texture::generate_mipmaps
// (crnlib/crn_mipmapped_texture.cpp:2140-2215) with its resampler, image_utils::
// resample_multithreaded (crnlib/crn_image_utils.cpp:662-874) over threaded_resampler
// (crnlib/crn_threaded_resampler.cpp:66-357). Every level is resampled from the level-0 image, in
// two launches for the whole chain:
//
//   k_mip_rows      level 0 RGBA8 (the sRGB-to-linear table for R, G, B when gamma filtering,
//                   v / 255 otherwise and for alpha) -> every level's row-filtered image: per source
//                   row and destination column the weighted sum of the column's contributors;
//   k_mip_columns   per destination texel the weighted sum over its row contributors, clamped to
//                   [0, 1], then back to 8 bits (255 v + 0.5 truncated, or the 8192-entry
//                   linear-to-sRGB table).
//
// The contributor lists (Resampler::make_clist, crnlib/crn_resampler.cpp:119-412: filter support
// stretched by the scale factor and the filter scale, weights normalised, the rounding residue
// added to the largest weight, clamp or wrap addressing) and the two gamma tables are built on the
// host with the reference's float expressions; the kernels add in the reference's order with
// round-to-nearest multiplies and adds (no contraction), so every level matches the reference.
//
// A destination sample's contributors are consecutive source positions ("virtual": before clamping
// or wrapping), so a list is kept as a dense window of weights, its ends rounded out to multiples
// of four positions with zero weights. A zero weight adds +0 to the sum (texels are >= 0 and
// finite), which changes nothing, so the sums are the lists' sums.
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <cstdint>
#include <cstring>
#include <list>
#include <map>
#include <memory>
#include <mutex>
#include <tuple>
#include <vector>

#include "crngpu_internal.h"

namespace crngpu {
namespace mip {
namespace {

// ---- the mip filters of crn_mip_filter (crnlib/crn_resample_filters.cpp), published kernels:
// box, tent (triangle), Lanczos (sinc windowed by sinc, 4 lobes), Mitchell-Netravali (B = C = 1/3),
// Kaiser-windowed sinc (40 dB attenuation, half-width 3)
constexpr double kPi = 3.14159265358979323846;

float f_box(float t) { return (t >= -0.5f && t < 0.5f) ? 1.0f : 0.0f; }

float f_tent(float t) {
  if (t < 0.0f) t = -t;
  return t < 1.0f ? 1.0f - t : 0.0f;
}

double sinc(double x) {
  x = x * kPi;
  if (x < 0.01f && x > -0.01f) return 1.0f + x * x * (-1.0f / 6.0f + x * x * 1.0f / 120.0f);
  return std::sin(x) / x;
}

float clean(double t) {
  const float eps = .0000125f;
  if (std::fabs(t) < eps) return 0.0f;
  return (float)t;
}

float f_lanczos4(float t) {
  if (t < 0.0f) t = -t;
  return t < 4.0f ? clean(sinc(t) * sinc(t / 4.0f)) : 0.0f;
}

float mitchell(float t, const float B, const float C) {
  const float tt = t * t;
  if (t < 0.0f) t = -t;
  if (t < 1.0f) {
    t = (((12.0f - 9.0f * B - 6.0f * C) * (t * tt)) + ((-18.0f + 12.0f * B + 6.0f * C) * tt) + (6.0f - 2.0f * B));
    return t / 6.0f;
  }
  if (t < 2.0f) {
    t = (((-1.0f * B - 6.0f * C) * (t * tt)) + ((6.0f * B + 30.0f * C) * tt) + ((-12.0f * B - 48.0f * C) * t) +
         (8.0f * B + 24.0f * C));
    return t / 6.0f;
  }
  return 0.0f;
}
float f_mitchell(float t) { return mitchell(t, 1.0f / 3.0f, 1.0f / 3.0f); }

// modified Bessel function of the first kind, order 0, by its power series
double bessel0(double x) {
  const double eps_ratio = 1E-16;
  const double xh = 0.5 * x;
  double sum = 1.0, pw = 1.0, ds = 1.0;
  int k = 0;
  while (ds > sum * eps_ratio) {
    ++k;
    pw = pw * (xh / k);
    ds = pw * pw;
    sum = sum + ds;
  }
  return sum;
}

double kaiser(double alpha, double half_width, double x) {
  const double ratio = x / half_width;
  return bessel0(alpha * std::sqrt(1 - ratio * ratio)) / bessel0(alpha);
}

float f_kaiser(float t) {
  if (t < 0.0f) t = -t;
  if (t < 3) {
    const float att = 40.0f;
    const float alpha = (float)(std::exp(std::log((double)0.58417 * (att - 20.96)) * 0.4) + 0.07886 * (att - 20.96));
    return (float)clean(sinc(t) * kaiser(alpha, 3, t));
  }
  return 0.0f;
}

struct Filter {
  float (*fn)(float);
  float support;
};
const Filter kFilters[5] = {{f_box, 0.5f}, {f_tent, 1.0f}, {f_lanczos4, 4.0f}, {f_mitchell, 2.0f}, {f_kaiser, 3.0f}};

// The window of one destination sample along one axis: virtual positions [a, b), both multiples of
// four, weights at w + (position - a).
struct Span {
  int a, b;
  uint32_t w;
};

int floor4(int v) { return v & ~3; }

// Values that depend on their keys alone, the most recently used up to `most` bytes of them.
template <class Key, class T>
class Kept {
 public:
  explicit Kept(size_t most) : most_(most) {}
  std::shared_ptr<const T> find(const Key& key) {
    std::lock_guard<std::mutex> lock(mu_);
    const auto it = at_.find(key);
    if (it == at_.end()) return nullptr;
    items_.splice(items_.begin(), items_, it->second);
    return it->second->value;
  }
  // the value kept under the key: `value`, or one that another thread has added meanwhile
  std::shared_ptr<const T> add(const Key& key, std::shared_ptr<const T> value, size_t bytes) {
    std::lock_guard<std::mutex> lock(mu_);
    const auto it = at_.find(key);
    if (it != at_.end()) return it->second->value;
    if (bytes > most_) return value;
    items_.push_front(Item{key, value, bytes});
    at_[key] = items_.begin();
    bytes_ += bytes;
    while (bytes_ > most_) {
      bytes_ -= items_.back().bytes;
      at_.erase(items_.back().key);
      items_.pop_back();
    }
    return value;
  }

 private:
  struct Item {
    Key key;
    std::shared_ptr<const T> value;
    size_t bytes;
  };
  std::mutex mu_;
  std::list<Item> items_;  // most recently used first
  std::map<Key, typename std::list<Item>::iterator> at_;
  size_t most_, bytes_ = 0;
};

// Resampler::make_clist (crnlib/crn_resampler.cpp:119-412) with a zero source offset. The spans'
// weights are appended to `pool`; a sample whose filter arguments equal its predecessor's (every
// sample of a power-of-two scale) shares them, one copy per alignment of the window.
bool make_axis(int src, int dst, const Filter& F, float filter_scale, std::vector<float>& pool, std::vector<Span>& spans) {
  const float oo_filter_scale = 1.0f / filter_scale;
  const float nudge = 0.5f;
  const float xscale = dst / (float)src;
  const bool down = xscale < 1.0f;
  const float half_width = down ? (F.support / xscale) * filter_scale : F.support * filter_scale;
  spans.resize(dst);
  std::vector<float> args, last_args, weight;
  int first = 0;  // first and one-past-last position of the non-zero weights, relative to `left`
  int64_t shared[4] = {-1, -1, -1, -1};
  for (int i = 0; i < dst; i++) {
    float center = ((float)i + nudge) / xscale;
    center -= nudge;
    const int left = (int)(float)std::floor(center - half_width);
    const int right = (int)(float)std::ceil(center + half_width);
    args.clear();
    for (int j = left; j <= right; j++)
      args.push_back(down ? (center - (float)j) * xscale * oo_filter_scale : (center - (float)j) * oo_filter_scale);
    if (i == 0 || args.size() != last_args.size() ||
        std::memcmp(args.data(), last_args.data(), args.size() * sizeof(float)) != 0) {
      float total = 0;
      weight.clear();
      for (float t : args) {
        weight.push_back(F.fn(t));
        total += weight.back();
      }
      const float norm = (float)(1.0f / total);
      total = 0;
      int max_k = -1, used = 0, last = 0;
      float max_w = -1e+20f;
      first = 0;
      for (int k = 0; k < (int)weight.size(); k++) {
        const float w = weight[k] = weight[k] * norm;
        if (w == 0.0f) continue;
        if (!used++) first = k;
        last = k + 1;
        total += w;
        if (w > max_w) { max_w = w; max_k = k; }
      }
      if (max_k < 0 || !used) return false;
      if (total != 1.0f) weight[max_k] += 1.0f - total;
      weight.erase(weight.begin() + last, weight.end());
      weight.erase(weight.begin(), weight.begin() + first);
      last_args = args;
      for (int64_t& k : shared) k = -1;
    }
    const int v0 = left + first, v1 = v0 + (int)weight.size();
    Span& s = spans[i];
    s.a = floor4(v0);
    s.b = floor4(v1 + 3);
    int64_t& at = shared[v0 - s.a];
    if (at < 0) {
      at = (int64_t)pool.size();
      if (pool.size() + (size_t)(s.b - s.a) > 0xFFFFFFF0u) return false;
      pool.resize(pool.size() + (size_t)(s.b - s.a), 0.0f);
      std::memcpy(pool.data() + at + (v0 - s.a), weight.data(), weight.size() * sizeof(float));
    }
    s.w = (uint32_t)at;
  }
  return true;
}

struct Axis {
  std::vector<Span> spans;  // weights in `pool`
  std::vector<float> pool;
};

// Textures of many shapes share their sides' axes, which are most of the work of a plan (4096 x 4096:
// 4.3 ms, 0.3 with the axes at hand), so axes are kept too.
std::shared_ptr<const Axis> cached_axis(int src, int dst, uint32_t filter, float filter_scale) {
  static Kept<std::tuple<int, int, uint32_t, float>, Axis> kept(64u << 20);
  const auto key = std::make_tuple(src, dst, filter, filter_scale);
  std::shared_ptr<const Axis> axis = kept.find(key);
  if (axis) return axis;
  auto made = std::make_shared<Axis>();
  if (!make_axis(src, dst, kFilters[filter], filter_scale, made->pool, made->spans)) return nullptr;
  return kept.add(key, made, made->spans.size() * sizeof(Span) + made->pool.size() * sizeof(float));
}

// One warp's work: one or two neighbouring destination samples (the second window empty, a1 = b1 =
// b0, for one). Rows: sample k of source row y goes to float4 dst + y * stride + k of the row-
// filtered images; columns: sample k of column x to texel dst + k * stride + x of the output.
struct Item {
  uint32_t dst, stride;
  int a0, b0;
  uint32_t w0;
  int a1, b1;
  uint32_t w1;
};
// The items of a run of CTAs (one per group of rows or columns) over virtual positions [v0, v1).
struct Job {
  uint32_t item, items;
  int v0, v1;
  uint32_t src, width;  // columns: float4 offset of the level's row-filtered image, its width
  uint32_t cta;         // first CTA of the job
  uint32_t single;      // at most kSingles items of one sample each
};

constexpr int kThreads = 512, kWarps = kThreads / 32;
constexpr int kRows = 32, kRowChunk = 160;     // k_mip_rows: rows of a CTA, positions staged at a time
constexpr int kCols = 32, kColChunk = 64;      // k_mip_columns: columns of a CTA, rows staged at a time
constexpr int kSingles = kWarps / 2;           // single-sample jobs: half the rows / columns per CTA,
constexpr int kRowChunk1 = 2 * kRowChunk, kColChunk1 = 2 * kColChunk;  // twice the positions
// float4 strides of a staged row: odd, so that 32 (or 8) rows' reads at one position fall in
// different banks
constexpr int kRowStride = kRowChunk + 1, kRowStride1 = kRowChunk1 + 1;
constexpr int kRowStage = kRows * kRowStride;  // float4s; not less than kRows / 2 * kRowStride1
constexpr int kColStage = kCols * kColChunk;   // float4s of one of the two buffers
static_assert(kRows / 2 * kRowStride1 <= kRowStage && kCols / 2 * kColChunk1 == kColStage, "staging buffers");
constexpr int kPairJob = 32;                   // samples of a job (more for the first levels' rows)
constexpr int kMaxPairJob = 128;

// ---- kernels
// A warp takes an item and a lane a row (or column) with its four channels, so the weights are the
// same for the warp (one 16-byte load per four positions), and a staged texel, read once, serves
// two samples' sums, added in the reference's order. Positions are staged chunk by chunk; an item
// whose window goes on in the next chunk leaves its sums in shared memory.
//
// A row pass multiplies and adds, separately rounded, (support x 2 x filter scale) values per source
// texel and channel at every level, and no product is shared between levels: 0.22 ms of FP32 for 4096 x
// 4096. Two samples per lane because a texel's 16-byte reads take 4 shared-memory cycles per warp
// against 8 multiplies and adds per sample, and an SM issues four of those a cycle: with one sample
// per read the reads would be the bound. As it is no pipe is at its limit: the row pass (1.15 ms) issues
// on 47 % of its cycles, the FMA pipe is busy for 25 % and the shared-memory data path for 55 %, 8 % of its
// loads' cycles for bank conflicts; warps wait for the chunks' barriers (5.4 of 16 cycles between two
// issues) and for weights and texels (4.2). Every job stages and converts its
// texels anew, each texel about ten times.

__device__ __forceinline__ int source_index(int j, int n, int wrap) {
  if (j >= 0 && j < n) return j;
  if (!wrap) return j < 0 ? 0 : n - 1;
  if (j >= n) return j % n;
  const int m = (-j) % n;
  return m ? n - m : 0;
}

__device__ __forceinline__ void add1(float4& s, const float4& p, float w) {
  s.x = __fadd_rn(s.x, __fmul_rn(p.x, w));
  s.y = __fadd_rn(s.y, __fmul_rn(p.y, w));
  s.z = __fadd_rn(s.z, __fmul_rn(p.z, w));
  s.w = __fadd_rn(s.w, __fmul_rn(p.w, w));
}

// Adds positions [q, e) (multiples of four); at(q): this lane's texel at position q.
template <class At>
__device__ __forceinline__ void add_one(float4& s, int q, int e, const float* w, At at) {
#pragma unroll 2
  for (; q < e; q += 4) {
    const float4 c = __ldg(reinterpret_cast<const float4*>(w + q));
    add1(s, at(q), c.x);
    add1(s, at(q + 1), c.y);
    add1(s, at(q + 2), c.z);
    add1(s, at(q + 3), c.w);
  }
}

// The part of an item inside the staged positions [c0, c1). acc: this lane's two saved sums of the
// item. done(k, sum): sample k is complete.
template <class At, class Done>
__device__ __forceinline__ void item_chunk(const Item& it, int c0, int c1, const float* __restrict__ weights, float4* acc,
                                           At at, Done done) {
  const bool on0 = it.a0 < c1 && it.b0 > c0, on1 = it.a1 < c1 && it.b1 > c0 && it.b1 > it.a1;
  if (!on0 && !on1) return;
  float4 s0 = make_float4(0.f, 0.f, 0.f, 0.f), s1 = s0;
  if (on0 && it.a0 < c0) s0 = acc[0];
  if (on1 && it.a1 < c0) s1 = acc[32];
  const float* w0 = weights + (ptrdiff_t)it.w0 - it.a0;
  const float* w1 = weights + (ptrdiff_t)it.w1 - it.a1;
  add_one(s0, max(it.a0, c0), min(min(it.a1, it.b0), c1), w0, at);
  const int e = min(it.b0, c1);
#pragma unroll 2
  for (int q = max(it.a1, c0); q < e; q += 4) {
    const float4 u = __ldg(reinterpret_cast<const float4*>(w0 + q)), v = __ldg(reinterpret_cast<const float4*>(w1 + q));
    float4 p = at(q);
    add1(s0, p, u.x);
    add1(s1, p, v.x);
    p = at(q + 1);
    add1(s0, p, u.y);
    add1(s1, p, v.y);
    p = at(q + 2);
    add1(s0, p, u.z);
    add1(s1, p, v.z);
    p = at(q + 3);
    add1(s0, p, u.w);
    add1(s1, p, v.w);
  }
  add_one(s1, max(max(it.b0, it.a1), c0), min(it.b1, c1), w1, at);
  if (on0) {
    if (it.b0 <= c1) done(0, s0); else acc[0] = s0;
  }
  if (on1) {
    if (it.b1 <= c1) done(1, s1); else acc[32] = s1;
  }
}

// A single-sample item: the smallest levels' samples are chains of thousands of additions, and few
// of them, so a lane takes one channel of a row (or column) and keeps its one sum in a register.
// The weights come 128 positions at a time through a buffer of the warp's own, the next 128 on
// their way while the current ones are added; loaded as they were needed, the chain waited for them
// (the 1x1 level of 4096x4096: 22,000 additions took 0.64 ms in the column pass).
struct Single {
  Item it;
  float sum = 0.f;
  float* buf;  // 128 floats of shared memory, 16-byte aligned
  float4 next;
  int cur = -1, nxt = -1;  // blocks of 128 in the buffer and in `next`

  __device__ __forceinline__ float4 load(const float* __restrict__ weights, int block) const {
    const int k = block * 128 + (int)(threadIdx.x & 31) * 4;
    return k < it.b0 - it.a0 ? __ldg(reinterpret_cast<const float4*>(weights + it.w0 + k)) : make_float4(0.f, 0.f, 0.f, 0.f);
  }

  // true when the window ends in [c0, c1)
  template <class At>
  __device__ __forceinline__ bool chunk(int c0, int c1, const float* __restrict__ weights, At at) {
    if (it.a0 >= c1 || it.b0 <= c0) return false;
    const int hi = min(it.b0, c1);
    float s = sum;
    for (int q = max(it.a0, c0); q < hi;) {
      const int block = (q - it.a0) >> 7;
      if (block != cur) {
        if (nxt != block) next = load(weights, block);
        __syncwarp();
        *reinterpret_cast<float4*>(buf + (threadIdx.x & 31) * 4) = next;
        __syncwarp();
        cur = block;
        nxt = block + 1;
        next = load(weights, block + 1);
      }
      const int e = min(hi, it.a0 + (block + 1) * 128);
      const float* wb = buf - block * 128 - it.a0;
#pragma unroll 4
      for (; q < e; q += 4) {
        const float4 w = *reinterpret_cast<const float4*>(wb + q);
        s = __fadd_rn(s, __fmul_rn(at(q), w.x));
        s = __fadd_rn(s, __fmul_rn(at(q + 1), w.y));
        s = __fadd_rn(s, __fmul_rn(at(q + 2), w.z));
        s = __fadd_rn(s, __fmul_rn(at(q + 3), w.w));
      }
    }
    sum = s;
    return it.b0 <= c1;
  }
};

// the last job whose first CTA is at or before this one
__device__ __forceinline__ Job find_job(const Job* __restrict__ jobs, uint32_t njobs) {
  uint32_t lo = 0, hi = njobs;
  while (hi - lo > 1) {
    const uint32_t mid = (lo + hi) >> 1;
    if (__ldg(&jobs[mid].cta) <= blockIdx.x) lo = mid; else hi = mid;
  }
  return jobs[lo];
}

// Stages a job's positions: kR rows of kC positions, each texel converted once, the next chunk's
// texels already on their way in registers.
template <int kR, int kC>
struct RowStage {
  static constexpr int kPer = kR * kC / kThreads, kStride = kC + 1;
  uint32_t raw[kPer];
  __device__ __forceinline__ void fetch(const uint32_t* __restrict__ src, int w, int h, int wrap, int row0, int c0, int v1) {
#pragma unroll
    for (int k = 0; k < kPer; k++) {
      const int idx = (int)threadIdx.x + kThreads * k, r = idx / kC, j = c0 + idx % kC;
      if (j < v1) raw[k] = __ldg(src + (size_t)min(row0 + r, h - 1) * w + source_index(j, w, wrap));
    }
  }
  __device__ __forceinline__ void store(float4* stage, const float* lut, int c0, int v1) const {
#pragma unroll
    for (int k = 0; k < kPer; k++) {
      const int idx = (int)threadIdx.x + kThreads * k, r = idx / kC, px = idx % kC;
      if (c0 + px < v1)
        stage[r * kStride + px] = make_float4(lut[raw[k] & 255u], lut[(raw[k] >> 8) & 255u], lut[(raw[k] >> 16) & 255u],
                                              __fmul_rn((float)(raw[k] >> 24), 1.0f / 255.0f));
    }
  }
};

__global__ void __launch_bounds__(kThreads, 2)
    k_mip_rows(const uint32_t* __restrict__ src, int w, int h, const float* __restrict__ to_linear,
               const Job* __restrict__ jobs, uint32_t njobs, const Item* __restrict__ items,
               const float* __restrict__ weights, int wrap, float4* __restrict__ tmp) {
  extern __shared__ __align__(16) float4 sm[];
  float4* acc = sm + kRowStage + 64;
  float* lut = reinterpret_cast<float*>(sm + kRowStage);
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const Job job = find_job(jobs, njobs);
  if (tid < 256) lut[tid] = __ldg(to_linear + tid);
  if (job.single) {
    const int row0 = (int)(blockIdx.x - job.cta) * (kRows / 2);
    RowStage<kRows / 2, kRowChunk1> st;
    // warps 0-7: the first eight rows, 8-15 the others; channel lane & 3 of row lane >> 2
    const int r = (warp / kSingles) * 8 + (lane >> 2), y = row0 + r, c = lane & 3, mine = warp % kSingles;
    Single one;
    const bool any = mine < (int)job.items;
    if (any) one.it = items[job.item + mine];
    one.buf = reinterpret_cast<float*>(acc) + warp * 128;
    const float* plane = reinterpret_cast<const float*>(sm) + r * kRowStride1 * 4 + c;
    // chunks beyond the image's ends add one texel over and over (clamp): nothing to stage
    auto flat = [&](int c0, int c1) { return !wrap && (c1 <= 0 || c0 >= w); };
    if (!flat(job.v0, min(job.v0 + kRowChunk1, job.v1))) st.fetch(src, w, h, wrap, row0, job.v0, job.v1);
    for (int c0 = job.v0; c0 < job.v1; c0 += kRowChunk1) {
      const int c1 = min(c0 + kRowChunk1, job.v1), c2 = min(c1 + kRowChunk1, job.v1);
      const bool edge = flat(c0, c1);
      __syncthreads();  // the table is there; the chunk before is done with
      if (!edge) st.store(sm, lut, c0, job.v1);
      __syncthreads();
      if (c1 < job.v1 && !flat(c1, c2)) st.fetch(src, w, h, wrap, row0, c1, job.v1);
      if (!any) continue;
      bool end;
      if (edge) {
        const uint32_t px = __ldg(src + (size_t)min(y, h - 1) * w + (c1 <= 0 ? 0 : w - 1)) >> (8 * c) & 255u;
        const float v = c == 3 ? __fmul_rn((float)px, 1.0f / 255.0f) : lut[px];
        end = one.chunk(c0, c1, weights, [&](int) { return v; });
      } else {
        end = one.chunk(c0, c1, weights, [&](int q) { return plane[(q - c0) * 4]; });
      }
      if (end && y < h) reinterpret_cast<float*>(tmp + one.it.dst + (size_t)y * one.it.stride)[c] = one.sum;
    }
    return;
  }
  const int row0 = (int)(blockIdx.x - job.cta) * kRows, y = row0 + lane;
  RowStage<kRows, kRowChunk> st;
  st.fetch(src, w, h, wrap, row0, job.v0, job.v1);
  const float4* row = sm + lane * kRowStride;
  for (int c0 = job.v0; c0 < job.v1; c0 += kRowChunk) {
    const int c1 = min(c0 + kRowChunk, job.v1);
    __syncthreads();
    st.store(sm, lut, c0, job.v1);
    __syncthreads();
    if (c1 < job.v1) st.fetch(src, w, h, wrap, row0, c1, job.v1);
    for (uint32_t i = warp; i < job.items; i += kWarps) {
      const Item it = items[job.item + i];
      item_chunk(it, c0, c1, weights, acc + i * 64 + lane, [&](int q) { return row[q - c0]; },
                 [&](int k, const float4& s) {
                   if (y < h) tmp[(size_t)it.dst + (size_t)y * it.stride + k] = s;
                 });
    }
  }
}

__device__ __forceinline__ uint8_t to_u8_linear(float v) {
  int c = (int)__fadd_rn(__fmul_rn(255.0f, v), .5f);
  return (uint8_t)(c < 0 ? 0 : c > 255 ? 255 : c);
}

__device__ __forceinline__ void copy16(uint32_t dst, const void* src) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dst), "l"(src));
}

__device__ __forceinline__ uint8_t to_u8(float v, int c, const uint8_t* __restrict__ to_srgb, int srgb, int alpha) {
  v = fminf(fmaxf(v, 0.0f), 1.0f);
  if (c == 3) return alpha ? to_u8_linear(v) : (uint8_t)255;
  if (!srgb) return to_u8_linear(v);
  const int j = (int)__fadd_rn(__fmul_rn(8192.0f, v), .5f);
  return __ldg(to_srgb + (j < 0 ? 0 : j > 8191 ? 8191 : j));
}

// Rows of kC columns come through two shared-memory buffers, the next chunk's copies in flight
// while the current one is added. A level's row-filtered image is read once per job (the jobs of a
// level share only their windows' overlap).
template <int kC, int kN, class Chunk>
__device__ __forceinline__ void column_chunks(const float4* __restrict__ tmp, int h, int wrap, const Job& job, int x0,
                                              float4* sm, Chunk chunk) {
  const uint32_t base = (uint32_t)__cvta_generic_to_shared(sm);
  const int tid = threadIdx.x;
  auto fetch = [&](int c0, int buf) {
#pragma unroll
    for (int k = 0; k < kC * kN / kThreads; k++) {
      const int idx = tid + kThreads * k, r = idx / kC, seg = idx % kC;
      if (c0 + r < job.v1)
        copy16(base + (uint32_t)(buf * kColStage + idx) * 16u,
               tmp + job.src + (size_t)source_index(c0 + r, h, wrap) * job.width + min(x0 + seg, (int)job.width - 1));
    }
    asm volatile("cp.async.commit_group;");
  };
  fetch(job.v0, 0);
  int buf = 0;
  for (int c0 = job.v0; c0 < job.v1; c0 += kN, buf ^= 1) {
    const int c1 = min(c0 + kN, job.v1);
    if (c1 < job.v1) fetch(c1, buf ^ 1); else asm volatile("cp.async.commit_group;");
    asm volatile("cp.async.wait_group 1;");
    __syncthreads();
    chunk(c0, c1, sm + buf * kColStage);
    __syncthreads();  // the buffer is refilled by the next iteration's fetch
  }
}

__global__ void __launch_bounds__(kThreads, 2)
    k_mip_columns(const float4* __restrict__ tmp, int h, const Job* __restrict__ jobs, uint32_t njobs,
                  const Item* __restrict__ items, const float* __restrict__ weights, int wrap,
                  const uint8_t* __restrict__ to_srgb, int srgb, int alpha, uint8_t* __restrict__ out) {
  extern __shared__ __align__(16) float4 sm[];
  float4* acc = sm + 2 * kColStage;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const Job job = find_job(jobs, njobs);
  if (job.single) {
    const int x0 = (int)(blockIdx.x - job.cta) * (kCols / 2), col = (warp / kSingles) * 8 + (lane >> 2), c = lane & 3;
    const int mine = warp % kSingles, x = x0 + col;
    Single one;
    const bool any = mine < (int)job.items;
    if (any) one.it = items[job.item + mine];
    one.buf = reinterpret_cast<float*>(acc) + warp * 128;
    column_chunks<kCols / 2, kColChunk1>(tmp, h, wrap, job, x0, sm, [&](int c0, int c1, const float4* buf) {
      const float* p = reinterpret_cast<const float*>(buf + col) + c;
      if (any && one.chunk(c0, c1, weights, [&](int q) { return p[(q - c0) * (kCols / 2) * 4]; }) && x < (int)job.width)
        out[((size_t)one.it.dst + x) * 4 + c] = to_u8(one.sum, c, to_srgb, srgb, alpha);
    });
    return;
  }
  const int x0 = (int)(blockIdx.x - job.cta) * kCols, x = x0 + lane;
  column_chunks<kCols, kColChunk>(tmp, h, wrap, job, x0, sm, [&](int c0, int c1, const float4* buf) {
    for (uint32_t i = warp; i < job.items; i += kWarps) {
      const Item it = items[job.item + i];
      item_chunk(it, c0, c1, weights, acc + i * 64 + lane, [&](int q) { return buf[(q - c0) * kCols + lane]; },
                 [&](int k, const float4& s) {
                   if (x >= (int)job.width) return;
                   reinterpret_cast<uint32_t*>(out)[(size_t)it.dst + (size_t)k * it.stride + x] =
                       (uint32_t)to_u8(s.x, 0, to_srgb, srgb, alpha) | (uint32_t)to_u8(s.y, 1, to_srgb, srgb, alpha) << 8 |
                       (uint32_t)to_u8(s.z, 2, to_srgb, srgb, alpha) << 16 | (uint32_t)to_u8(s.w, 3, to_srgb, srgb, alpha) << 24;
                 });
    }
  });
}

// ---- the plan of a chain: jobs, items and weights in one upload

struct Plan {
  std::vector<uint8_t> blob;  // row jobs, column jobs, items, weights (16-byte aligned parts)
  size_t o_rows, o_cols, o_items, o_weights;
  uint32_t row_jobs, col_jobs, row_ctas, col_ctas;
  uint32_t row_acc, col_acc;  // items whose sums a CTA may have to keep between chunks
  uint64_t tmp;               // float4 entries of the row-filtered images
};

// Samples of a row job: as many as one chunk holds with their windows where that is at least
// kPairJob (the first two levels; nothing is kept between chunks then), else kPairJob, two items to
// a warp's one for 16 warps.
int row_job(const std::vector<Span>& sp) {
  int n = 1;
  while (n < (int)sp.size() && n < kMaxPairJob && sp[n].b - sp[0].a <= kRowChunk - 4) n++;
  return std::max(kPairJob, n & ~1);
}

// Appends the items of samples [d0, d0 + n) and widens the job's range by them. Pairs share their
// loads; in a level of few samples an item is one sample.
void add_items(std::vector<Item>& items, Job& job, const std::vector<Span>& sp, int d0, int n, bool pairs, uint64_t dst,
               uint32_t stride, uint64_t step) {
  for (int i = 0; i < n;) {
    const Span& s = sp[d0 + i];
    Item it = {(uint32_t)(dst + (uint64_t)(d0 + i) * step), stride, s.a, s.b, s.w, s.b, s.b, s.w};
    int got = 1;
    if (pairs && i + 1 < n) {
      const Span& t = sp[d0 + i + 1];
      if (t.a >= s.a && t.b >= s.b) {
        it.a1 = t.a;
        it.b1 = t.b;
        it.w1 = t.w;
        got = 2;
      }
    }
    if (!job.items) { job.v0 = it.a0; job.v1 = it.b1; }
    job.v0 = std::min(job.v0, it.a0);
    job.v1 = std::max(job.v1, std::max(it.b0, it.b1));
    items.push_back(it);
    job.items++;
    i += got;
  }
}

// Levels of at most this many samples go to single-sample jobs. Columns: 16, so that a level's few
// chains run side by side (with pairs of samples at 8 and 16 the column pass of 4096x4096 took 0.30
// ms, with singles 0.21). Rows: 4 (every row has its own chains; both ways take the same time at 8
// and 16).
constexpr int kFewRowSamples = 4, kFewColSamples = 16;
// Few windows of a small level reach a chunk (5.4 scales wide: 8 pairs of samples at a scale of 16, 4 at
// 64, for 16 warps), so three levels at a time share their jobs' chunks: 4096 x 4096 1.88 ms with a job
// for each, 1.51 so (from a scale of 16 on; of 8 1.58, of 4 1.51 and 1000 x 3000 442 us, 471 from 16 on;
// four levels 1.59). Not for images whose jobs do not fill the SMs (512 x 512 107 us, merged 110).
constexpr uint32_t kMergeScale = 4, kMergeLevels = 3;
constexpr uint64_t kMergeTexels = 1u << 21;

bool make_plan(uint32_t width, uint32_t height, uint32_t levels, uint32_t filter, float filter_scale, Plan& plan) {
  std::vector<float> pool;
  std::vector<Item> items;
  std::vector<Job> rows, cols;
  std::map<std::pair<int, int>, std::vector<Span>> axes;
  auto axis = [&](int src, int dst) -> const std::vector<Span>* {
    std::vector<Span>& sp = axes[{src, dst}];
    if (sp.empty()) {
      const std::shared_ptr<const Axis> a = cached_axis(src, dst, filter, filter_scale);
      if (!a || pool.size() + a->pool.size() > 0xFFFFFFF0u) return nullptr;
      sp = a->spans;
      for (Span& s : sp) s.w += (uint32_t)pool.size();
      pool.insert(pool.end(), a->pool.begin(), a->pool.end());
    }
    return &sp;
  };
  uint64_t tmp = 0;
  std::vector<uint64_t> tmp_of(levels, 0);
  for (uint32_t l = 1; l < levels; l++) {
    tmp_of[l] = tmp;
    tmp += (uint64_t)std::max(1u, width >> l) * height;
  }
  for (uint32_t l = 1; l < levels; l++) {
    const int dw = (int)std::max(1u, width >> l);
    const std::vector<Span>* sp = axis((int)width, dw);
    if (!sp) return false;
    const bool single = dw <= kFewRowSamples;
    if (!single && (uint64_t)width * height >= kMergeTexels && (uint32_t)dw * kMergeScale <= width) {
      // the level and up to two after it in common jobs over the same part of the row
      uint32_t end = l + 1;
      while (end < levels && end < l + kMergeLevels && (int)(width >> end) > kFewRowSamples) end++;
      for (int d = 0; d < dw; d += kPairJob) {
        Job j = {};
        j.item = (uint32_t)items.size();
        for (uint32_t k = l; k < end; k++) {
          const int kw = (int)(width >> k), from = (int)((int64_t)d * kw / dw),
                    to = (int)((int64_t)std::min(d + kPairJob, dw) * kw / dw);
          const std::vector<Span>* ks = axis((int)width, kw);
          if (!ks) return false;
          add_items(items, j, *ks, from, to - from, true, tmp_of[k], (uint32_t)kw, 1);
        }
        // by their windows' middles, so that the ones that reach a chunk go to different warps
        std::stable_sort(items.begin() + j.item, items.end(), [](const Item& a, const Item& b) {
          return a.a0 + std::max(a.b0, a.b1) < b.a0 + std::max(b.b0, b.b1);
        });
        rows.push_back(j);
      }
      l = end - 1;
      continue;
    }
    const int per = single ? kSingles : row_job(*sp);
    for (int d = 0; d < dw; d += per) {
      // the last levels' few samples (4 + 2 + 1, and a side's 1s) share a job: the source is the same
      const int n = std::min(per, dw - d);
      const bool join = single && !rows.empty() && rows.back().single && rows.back().items + (uint32_t)n <= (uint32_t)kSingles;
      if (!join) {
        rows.push_back(Job());
        rows.back().item = (uint32_t)items.size();
        rows.back().single = single;
      }
      add_items(items, rows.back(), *sp, d, n, !single, tmp_of[l], (uint32_t)dw, 1);
    }
  }
  uint64_t out = (uint64_t)width * height;
  for (uint32_t l = 1; l < levels; l++) {
    const int dw = (int)std::max(1u, width >> l), dh = (int)std::max(1u, height >> l);
    const std::vector<Span>* sp = axis((int)height, dh);
    if (!sp) return false;
    const bool single = dh <= kFewColSamples;
    const int per = single ? kSingles : kPairJob;
    for (int d = 0; d < dh; d += per) {
      Job j = {};
      j.item = (uint32_t)items.size();
      j.src = (uint32_t)tmp_of[l];
      j.width = (uint32_t)dw;
      j.single = single;
      add_items(items, j, *sp, d, std::min(per, dh - d), !single, out, (uint32_t)dw, (uint32_t)dw);
      cols.push_back(j);
    }
    out += (uint64_t)dw * dh;
  }
  // the longest chains of additions first
  auto longer = [](const Job& a, const Job& b) { return a.v1 - a.v0 > b.v1 - b.v0; };
  std::stable_sort(rows.begin(), rows.end(), longer);
  std::stable_sort(cols.begin(), cols.end(), longer);
  plan.row_acc = plan.col_acc = (uint32_t)kWarps / 2;  // the single items' weight buffers
  uint64_t row_ctas = 0, ctas = 0;
  for (Job& j : rows) {
    const uint32_t per = j.single ? kRows / 2 : kRows;
    j.cta = (uint32_t)row_ctas;
    row_ctas += (height + per - 1) / per;
    if (!j.single && j.v1 - j.v0 > kRowChunk) plan.row_acc = std::max(plan.row_acc, j.items);
  }
  for (Job& j : cols) {
    const uint32_t per = j.single ? kCols / 2 : kCols;
    j.cta = (uint32_t)ctas;
    ctas += (j.width + per - 1) / per;
    if (!j.single && j.v1 - j.v0 > kColChunk) plan.col_acc = std::max(plan.col_acc, j.items);
  }
  if (ctas > 0x7FFFFFFFu || row_ctas > 0x7FFFFFFFu) return false;
  plan.row_ctas = (uint32_t)row_ctas;
  plan.row_jobs = (uint32_t)rows.size();
  plan.col_jobs = (uint32_t)cols.size();
  plan.col_ctas = (uint32_t)ctas;
  plan.tmp = tmp;
  auto put = [&](const void* p, size_t bytes) {
    const size_t o = plan.blob.size();
    plan.blob.resize(o + ((bytes + 15) & ~(size_t)15), 0);
    if (bytes) std::memcpy(plan.blob.data() + o, p, bytes);
    return o;
  };
  plan.o_rows = put(rows.data(), rows.size() * sizeof(Job));
  plan.o_cols = put(cols.data(), cols.size() * sizeof(Job));
  plan.o_items = put(items.data(), items.size() * sizeof(Item));
  plan.o_weights = put(pool.data(), pool.size() * sizeof(float));
  return true;
}

// Plans depend on sizes and parameters alone, and are kept for the process up to 64 MB (about a
// hundred of 2000 x 1500 images, a thousand of 256 x 256); a caller holds its own reference while it uses
// one.
std::shared_ptr<const Plan> cached_plan(uint32_t width, uint32_t height, uint32_t levels, uint32_t filter,
                                        float filter_scale) {
  static Kept<std::tuple<uint32_t, uint32_t, uint32_t, uint32_t, float>, Plan> kept(64u << 20);
  const auto key = std::make_tuple(width, height, levels, filter, filter_scale);
  std::shared_ptr<const Plan> plan = kept.find(key);
  if (plan) return plan;
  auto made = std::make_shared<Plan>();
  if (!make_plan(width, height, levels, filter, filter_scale, *made)) return nullptr;
  return kept.add(key, made, made->blob.size());
}

struct GammaTables {
  float to_linear[256];
  float to_unit[256];  // without gamma: v / 255
  uint8_t to_srgb[8192];
  GammaTables() {
    // resample_multithreaded's tables with the source gamma generate_mipmaps leaves at 2.2
    const float gamma = 2.2f;
    for (int i = 0; i < 256; ++i) to_linear[i] = (float)std::pow(i * 1.0f / 255.0f, gamma);
    const float inv = 1.0f / 255.0f;
    for (int i = 0; i < 256; ++i) to_unit[i] = (float)i * inv;
    const float inv_size = 1.0f / 8192, inv_gamma = 1.0f / gamma;
    for (int i = 0; i < 8192; ++i) {
      const int k = (int)(255.0f * std::pow(i * inv_size, inv_gamma) + .5f);
      to_srgb[i] = (uint8_t)(k < 0 ? 0 : k > 255 ? 255 : k);
    }
  }
};

// Both kernels ask for more than 48 KB: the staged positions and up to kMaxPairJob items' saved
// sums (a job's samples pair up except where one window reaches past the next one's end).
int set_smem() {
  static bool done[64] = {};
  int dev = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e != cudaSuccess) return cuda_check(e, "cudaGetDevice");
  if (dev < 0 || dev >= 64) { set_error("device index out of range"); return CRNGPU_E_DEVICE; }
  std::lock_guard<std::mutex> lock(device_setup_mutex());
  if (!done[dev]) {
    constexpr int most = (kRowStage + 64 + kMaxPairJob * 64) * (int)sizeof(float4);
    static_assert(most <= 227 << 10 && 2 * kColStage <= kRowStage, "mip kernels' shared memory");
    e = cudaFuncSetAttribute(k_mip_rows, cudaFuncAttributeMaxDynamicSharedMemorySize, most);
    if (e == cudaSuccess) e = cudaFuncSetAttribute(k_mip_columns, cudaFuncAttributeMaxDynamicSharedMemorySize, most);
    if (e != cudaSuccess) return cuda_check(e, "set mip kernels' shared memory");
    done[dev] = true;
  }
  return CRNGPU_OK;
}

}  // namespace
}  // namespace mip
}  // namespace crngpu

using namespace crngpu;
using namespace crngpu::mip;

extern "C" int64_t crngpu_generate_mipmaps(const uint8_t* rgba, uint32_t width, uint32_t height, uint32_t levels,
                                           uint32_t filter, float filter_scale, uint32_t flags, uint8_t* out,
                                           uint64_t out_size, int mem, void* stream) try {
  clear_error();
  if (!rgba || !out || !width || !height || width > 16384 || height > 16384 || filter > 4 || !(filter_scale > 0.0f)) {
    set_error("crngpu_generate_mipmaps: bad arguments");
    return CRNGPU_E_PARAM;
  }
  uint32_t full = 1;
  while ((width >> full) || (height >> full)) full++;
  if (!levels) levels = full;
  if (levels > full) { set_error("crngpu_generate_mipmaps: more levels than the mip chain has"); return CRNGPU_E_PARAM; }
  uint64_t need = 0;
  for (uint32_t l = 0; l < levels; l++) need += (uint64_t)std::max(1u, width >> l) * std::max(1u, height >> l) * 4;
  if (out_size < need) { set_error("crngpu_generate_mipmaps: output too small"); return CRNGPU_E_PARAM; }
  const bool srgb = (flags & CRNGPU_MIP_SRGB) != 0, wrap = (flags & CRNGPU_MIP_WRAP) != 0,
             alpha = (flags & CRNGPU_MIP_ALPHA) != 0;
  cudaStream_t s = as_stream(stream);
  static const GammaTables gt;
  std::shared_ptr<const Plan> plan;
  if (levels > 1 && !(plan = cached_plan(width, height, levels, filter, filter_scale))) {
    set_error("crngpu_generate_mipmaps: filter has no contributors");
    return CRNGPU_E_PARAM;
  }
  const uint64_t texels0 = (uint64_t)width * height;
  cudaError_t e;
  int rc;
  Staging staging(s);
  DevBuf& tables = staging[4];
  DevBuf& work = staging[5];
  const size_t blob = plan ? plan->blob.size() : 0, o_lin = blob, o_srgb = o_lin + sizeof(gt.to_linear);
  const size_t tmp_bytes = plan ? plan->tmp * sizeof(float4) : 0;
  uint8_t* d_in = nullptr;
  if (plan) {
    if ((e = tables.ensure(blob + sizeof(gt.to_linear) + sizeof(gt.to_srgb))) != cudaSuccess)
      return cuda_check(e, "alloc mip tables");
    uint8_t* tb = static_cast<uint8_t*>(tables.ptr);
    if ((e = cudaMemcpyAsync(tb, plan->blob.data(), blob, cudaMemcpyHostToDevice, s)) != cudaSuccess)
      return cuda_check(e, "upload mip plan");
    if ((e = cudaMemcpyAsync(tb + o_lin, srgb ? gt.to_linear : gt.to_unit, sizeof(gt.to_linear), cudaMemcpyHostToDevice,
                             s)) != cudaSuccess ||
        (srgb && (e = cudaMemcpyAsync(tb + o_srgb, gt.to_srgb, sizeof(gt.to_srgb), cudaMemcpyHostToDevice, s)) !=
                     cudaSuccess))
      return cuda_check(e, "upload mip tables");
  }
  if ((e = work.ensure(tmp_bytes + (mem != CRNGPU_MEM_DEVICE ? texels0 * 4 : 0) + 16)) != cudaSuccess)
    return cuda_check(e, "alloc mip work");
  d_in = static_cast<uint8_t*>(work.ptr) + tmp_bytes;
  uint8_t* d_out = out;
  // host buffers are staged through device memory
  DevBuf* so = nullptr;
  if (mem != CRNGPU_MEM_DEVICE) {
    if ((e = cudaMemcpyAsync(d_in, rgba, texels0 * 4, cudaMemcpyHostToDevice, s)) != cudaSuccess)
      return cuda_check(e, "copy level 0");
    so = &staging[6];
    if ((e = so->ensure(need)) != cudaSuccess) return cuda_check(e, "alloc mip output");
    d_out = static_cast<uint8_t*>(so->ptr);
  } else {
    if (((uintptr_t)rgba & 3) || ((uintptr_t)out & 3)) { set_error("device buffers must be 4-byte aligned"); return CRNGPU_E_PARAM; }
    d_in = const_cast<uint8_t*>(rgba);
  }
  // level 0 as given
  if ((e = cudaMemcpyAsync(d_out, d_in, texels0 * 4, cudaMemcpyDeviceToDevice, s)) != cudaSuccess)
    return cuda_check(e, "copy level 0 out");
  if (plan) {
    const uint8_t* tb = static_cast<const uint8_t*>(tables.ptr);
    const Item* items = reinterpret_cast<const Item*>(tb + plan->o_items);
    const float* weights = reinterpret_cast<const float*>(tb + plan->o_weights);
    const size_t row_smem = (size_t)(kRowStage + 64 + plan->row_acc * 64) * sizeof(float4);
    const size_t col_smem = (size_t)(2 * kColStage + plan->col_acc * 64) * sizeof(float4);
    if ((rc = set_smem()) != CRNGPU_OK) return rc;
    k_mip_rows<<<plan->row_ctas, kThreads, row_smem, s>>>(
        reinterpret_cast<const uint32_t*>(d_in), (int)width, (int)height, reinterpret_cast<const float*>(tb + o_lin),
        reinterpret_cast<const Job*>(tb + plan->o_rows), plan->row_jobs, items, weights, wrap ? 1 : 0,
        static_cast<float4*>(work.ptr));
    k_mip_columns<<<plan->col_ctas, kThreads, col_smem, s>>>(
        static_cast<const float4*>(work.ptr), (int)height, reinterpret_cast<const Job*>(tb + plan->o_cols),
        plan->col_jobs, items, weights, wrap ? 1 : 0, tb + o_srgb, srgb ? 1 : 0, alpha ? 1 : 0, d_out);
    if ((e = cudaGetLastError()) != cudaSuccess) return cuda_check(e, "launch mip kernels");
  }
  if (so) {
    if ((e = cudaMemcpyAsync(out, so->ptr, need, cudaMemcpyDeviceToHost, s)) != cudaSuccess)
      return cuda_check(e, "copy mips");
    if ((rc = staging.synchronize()) != CRNGPU_OK) return rc;
  }
  return (int64_t)need;
} catch (...) {
  return crngpu::exception_status();
}
