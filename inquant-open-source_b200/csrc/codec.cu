// K4 key encoder (sampled statistics + donor selection + mixed 4/8-bit packing), V2/V4
// group-wise value encoder, their exact inverses and the role-map builder.
//
// Compile this translation unit with -fmad=false: the packed bytes must equal the
// reference's bit for bit, and the reference performs separate IEEE multiplies, adds and
// divisions.  The only fused operations are the explicit fma() calls of the division-by-
// integer below, which is proven to return the correctly rounded quotient.
#include <algorithm>
#include <type_traits>

#include "common.cuh"

namespace inq {

constexpr int kMaxChannels = 1024;
constexpr int kMaxWords = kMaxChannels / 32;
constexpr int kRcpTable = 512;  // tokens per row for which 1/(t+1) is tabulated
struct InverseTable {
  double of[kRcpTable];
};
constexpr InverseTable make_inverse_table() {
  InverseTable table{};
  for (int t = 0; t < kRcpTable; ++t) table.of[t] = 1.0 / (double)(t + 1);   // correctly rounded
  return table;
}
static __device__ const InverseTable kInverse = make_inverse_table();

// ------------------------------------------------------------------------------------------
// Sampled statistics in the summation order of the reference's CPU reduction: samples are
// added one by one into a level-0 accumulator that is folded into level 1 every `step`
// samples (level 1 into level 2 every step^2, ...), a remainder shorter than `step` stays in
// level 0, and the levels are added lowest first at the end.
struct CascadePair {
  float abs_acc[4], sum_acc[4];
  int i, full_end, mask, level_power;
  __device__ void init(int n) {
#pragma unroll
    for (int k = 0; k < 4; ++k) abs_acc[k] = sum_acc[k] = 0.f;
    int ceil_log2 = n <= 1 ? 0 : 32 - __clz(n - 1);
    level_power = max(4, ceil_log2 / 4);
    int step = 1 << level_power;
    mask = step - 1;
    full_end = (n / step) * step;
    i = 0;
  }
  __device__ void add(float v) {
    abs_acc[0] = abs_acc[0] + fabsf(v);
    sum_acc[0] = sum_acc[0] + v;
    ++i;
    if (i <= full_end && (i & mask) == 0) {
#pragma unroll
      for (int level = 1; level < 4; ++level) {
        abs_acc[level] = abs_acc[level] + abs_acc[level - 1];
        sum_acc[level] = sum_acc[level] + sum_acc[level - 1];
        abs_acc[level - 1] = 0.f;
        sum_acc[level - 1] = 0.f;
        if (i & (mask << (level * level_power))) break;
      }
    }
  }
  __device__ void finish(float& abs_total, float& sum_total) {
#pragma unroll
    for (int level = 1; level < 4; ++level) {
      abs_acc[0] = abs_acc[0] + abs_acc[level];
      sum_acc[0] = sum_acc[0] + sum_acc[level];
    }
    abs_total = abs_acc[0];
    sum_total = sum_acc[0];
  }
};

// d / n for a small positive integer n, given y = RN(1/n): one multiply and two fused
// corrections return the correctly rounded IEEE quotient (Markstein's theorem).
__device__ __forceinline__ double divide_by_count(double d, double n, double y) {
  double q0 = d * y;
  double r = fma(-q0, n, d);
  return fma(r, y, q0);
}

struct ChannelStats {
  float saliency, sampled_mean, donor_error, absmax;
  bool finite;
};

// One thread walks one channel over all tokens of a row.
template <typename T>
__device__ ChannelStats channel_statistics(const T* column, long long s_token, int tokens, int sample_stride,
                                           bool want_error, const double* rcp_table) {
  ChannelStats out;
  CascadePair cascade;
  int samples = (tokens + sample_stride - 1) / sample_stride;
  cascade.init(samples);
  float absmax = 0.f;
  bool finite = true;
  double mean = 0.0, m2 = 0.0;
  int next_sample = 0;
  constexpr int kUnroll = 8;
  for (int base = 0; base < tokens; base += kUnroll) {
    float v[kUnroll];
#pragma unroll
    for (int u = 0; u < kUnroll; ++u) {
      int t = base + u;
      v[u] = t < tokens ? to_float<T>(column[(long long)t * s_token]) : 0.f;
    }
#pragma unroll
    for (int u = 0; u < kUnroll; ++u) {
      int t = base + u;
      if (t < tokens) {
        float x = v[u];
        finite = finite && finite_f32(x);
        absmax = fmaxf(absmax, fabsf(x));
        if (t == next_sample) {
          cascade.add(x);
          next_sample += sample_stride;
        }
        if (want_error) {
          // Welford's update in float64, sequential over tokens (torch CPU var_mean).
          double xd = (double)x;
          double delta = xd - mean;
          double q = rcp_table ? divide_by_count(delta, (double)(t + 1), rcp_table[t]) : delta / (double)(t + 1);
          mean = mean + q;
          m2 = m2 + delta * (xd - mean);
        }
      }
    }
  }
  float abs_total, sum_total;
  cascade.finish(abs_total, sum_total);
  out.saliency = abs_total / (float)samples;
  out.sampled_mean = sum_total / (float)samples;
  out.absmax = absmax;
  out.finite = finite;
  out.donor_error = 0.f;
  if (want_error) {
    float variance = (float)(m2 / (double)tokens);
    float diff = (float)mean - out.sampled_mean;
    out.donor_error = variance + diff * diff;
  }
  return out;
}

// ------------------------------------------------------------------------------------------
// Donor selection.  Called by every thread of a CTA whose blockDim.x >= channels.
// Shared inputs: saliency[C], error[C] (if use_error).  Shared scratch: rank_key[C] (u32),
// sel_mask / avail_mask [NW words].  Outputs in shared memory: sources[count] ascending,
// donors[count].
template <int NW>
__device__ int highest_below(const unsigned (&mask)[NW], int pos) {  // largest set index < pos, or -1
  int w = pos >> 5;
  if (w < NW) {
    unsigned m = (pos & 31) ? (mask[w] & ((1u << (pos & 31)) - 1u)) : 0u;
    if (m) return (w << 5) + 31 - __clz(m);
  }
  for (int k = min(w, NW) - 1; k >= 0; --k)
    if (mask[k]) return (k << 5) + 31 - __clz(mask[k]);
  return -1;
}
template <int NW>
__device__ int lowest_above(const unsigned (&mask)[NW], int pos, int limit) {  // smallest set index > pos, or limit
  int start = pos + 1;
  int w = start >> 5;
  if (w < NW) {
    unsigned m = mask[w] & (0xffffffffu << (start & 31));
    if (m) return (w << 5) + __ffs(m) - 1;
    for (int k = w + 1; k < NW; ++k)
      if (mask[k]) return (k << 5) + __ffs(mask[k]) - 1;
  }
  return limit;
}
template <int NW>
__device__ __forceinline__ bool test_bit(const unsigned (&mask)[NW], int pos) {
  return pos >= 0 && (pos >> 5) < NW && ((mask[pos >> 5] >> (pos & 31)) & 1u);
}

template <int NW>
__device__ void assign_donors_serial(const float* saliency, const unsigned* sel_words, const unsigned* avail_words,
                                     int channels, int count, int* sources, int* donors) {
  unsigned selected[NW], available[NW];
#pragma unroll
  for (int k = 0; k < NW; ++k) {
    selected[k] = sel_words[k];
    available[k] = avail_words[k];
  }
  int n = 0;
#pragma unroll
  for (int k = 0; k < NW; ++k) {
    unsigned m = selected[k];
    while (m && n < count) {
      sources[n++] = (k << 5) + __ffs(m) - 1;
      m &= m - 1;
    }
  }
  for (int i = 0; i < count; ++i) {
    int source = sources[i];
    int low = test_bit<NW>(available, source - 1) ? source - 1 : -1;
    int high = (source + 1 < channels && test_bit<NW>(available, source + 1)) ? source + 1 : -1;
    if (low < 0 && high < 0) {
      // Ends of the contiguous salient run that contains the source.
      int left = source, right = source;
      while (test_bit<NW>(selected, left - 1)) --left;
      while (right + 1 < channels && test_bit<NW>(selected, right + 1)) ++right;
      int below = highest_below<NW>(available, left);
      int above = lowest_above<NW>(available, right, channels);
      int d_below = below >= 0 ? left - below : 0x7fffffff;
      int d_above = above < channels ? above - right : 0x7fffffff;
      if (d_below <= d_above) low = below;
      if (d_above <= d_below && above < channels) high = above;
    }
    int donor;
    if (low >= 0 && high >= 0)
      donor = saliency[low] <= saliency[high] ? low : high;  // ties: the lower channel
    else
      donor = low >= 0 ? low : high;
    if (donor < 0) donor = 0;  // unreachable for count <= channels/2
    donors[i] = donor;
    available[donor >> 5] &= ~(1u << (donor & 31));
  }
}

__device__ void select_donors_cta(const float* saliency, const float* error, bool use_error, int channels, int count,
                                  unsigned* rank_key, unsigned* sel_mask, unsigned* avail_mask, int* sources,
                                  int* donors) {
  const int c = threadIdx.x;
  const int words = (channels + 31) >> 5;
  if (c < kMaxWords) {
    sel_mask[c] = 0u;
    avail_mask[c] = 0u;
  }
  __syncthreads();
  bool selected = false;
  if (c < channels && count > 0) {
    // Non-negative floats order like their bit patterns; ties go to the lower channel.
    unsigned mine = __float_as_uint(saliency[c]);
    int rank = 0;
    for (int o = 0; o < channels; ++o) {
      unsigned other = __float_as_uint(saliency[o]);
      rank += (other > mine) || (other == mine && o < c);
    }
    selected = rank < count;
    if (selected) atomicOr(&sel_mask[c >> 5], 1u << (c & 31));
    if (use_error) rank_key[c] = selected ? 0x7f800000u : __float_as_uint(error[c]);
    if (!use_error && !selected) atomicOr(&avail_mask[c >> 5], 1u << (c & 31));
  }
  __syncthreads();
  if (use_error && c < channels && count > 0 && !selected) {
    unsigned mine = rank_key[c];
    int rank = 0;
    for (int o = 0; o < channels; ++o) {
      unsigned other = rank_key[o];
      rank += (other < mine) || (other == mine && o < c);
    }
    if (rank < count) atomicOr(&avail_mask[c >> 5], 1u << (c & 31));
  }
  __syncthreads();
  if (c == 0 && count > 0) {
    if (words <= 4)
      assign_donors_serial<4>(saliency, sel_mask, avail_mask, channels, count, sources, donors);
    else
      assign_donors_serial<kMaxWords>(saliency, sel_mask, avail_mask, channels, count, sources, donors);
  }
  __syncthreads();
}

// ------------------------------------------------------------------------------------------
struct K4Params {
  InputRef in;
  int sample_stride, count, min_error;
  FieldRef payload, scales, salient, donors, padding, roles;
  int descriptor_i32, role_bytes;
  int vector_path;  // 1: rows are 16-byte aligned and channels % 8 == 0
  int* status;
};

struct K4Shared {
  float* saliency;
  float* error;
  float* sampled_mean;
  float* scale;      // divisor per slot (the source's scale for a donor slot)
  int* read_from;    // channel whose value fills this slot
  int* kind;         // 0 normal, 1 salient (high nibble), 2 donor slot (low nibble of its source)
  unsigned* rank_key;
  unsigned* sel_mask;
  unsigned* avail_mask;
  int* sources;
  int* donors;
  double* rcp;
};

__host__ __device__ inline size_t k4_shared_bytes(int channels, int count, int tokens, bool min_error) {
  size_t bytes = 0;
  bytes += (size_t)channels * 4 * 7;          // saliency, error, sampled_mean, scale, read_from, kind, rank_key
  bytes += (size_t)kMaxWords * 4 * 2;         // masks
  bytes += (size_t)(count > 0 ? count : 1) * 4 * 2;
  bytes = (bytes + 7) & ~(size_t)7;
  if (min_error && tokens <= kRcpTable) bytes += (size_t)tokens * 8;
  return bytes;
}

__device__ inline K4Shared carve_k4_shared(unsigned char* raw, int channels, int count, int tokens, bool min_error) {
  K4Shared s;
  float* f = (float*)raw;
  s.saliency = f; f += channels;
  s.error = f; f += channels;
  s.sampled_mean = f; f += channels;
  s.scale = f; f += channels;
  s.read_from = (int*)f; f += channels;
  s.kind = (int*)f; f += channels;
  s.rank_key = (unsigned*)f; f += channels;
  s.sel_mask = (unsigned*)f; f += kMaxWords;
  s.avail_mask = (unsigned*)f; f += kMaxWords;
  s.sources = (int*)f; f += (count > 0 ? count : 1);
  s.donors = (int*)f; f += (count > 0 ? count : 1);
  size_t used = ((size_t)((unsigned char*)f - raw) + 7) & ~(size_t)7;
  s.rcp = (min_error && tokens <= kRcpTable) ? (double*)(raw + used) : nullptr;
  return s;
}

__device__ __forceinline__ unsigned encode_slot(float x, float scale, int kind) {
  float q = rintf(x / scale);
  if (kind == 0) return (unsigned)(int)(fminf(fmaxf(q, -7.f), 7.f) + 8.f);
  unsigned code = (unsigned)(int)(fminf(fmaxf(q, -127.f), 127.f) + 128.f);
  return kind == 1 ? (code >> 4) : (code & 15u);
}

template <typename T, int kMaxThreads>
__global__ void __launch_bounds__(kMaxThreads) k4_encode_kernel(K4Params p) {
  extern __shared__ __align__(16) unsigned char raw[];
  const int C = p.in.channels, tokens = p.in.tokens, count = p.count;
  K4Shared s = carve_k4_shared(raw, C, count, tokens, p.min_error != 0);
  const long long outer = blockIdx.x / p.in.n_inner, inner = blockIdx.x % p.in.n_inner;
  const long long slot = p.in.slot(outer);
  if (!p.in.slot_ok(slot)) {   // uniform over the CTA: nothing of this row is written
    if (threadIdx.x == 0) atomicOr(p.status, INQ_STATUS_BAD_INDEX);
    return;
  }
  const T* row = (const T*)p.in.x + outer * p.in.s_outer + inner * p.in.s_inner;
  const int c = threadIdx.x;

  if (s.rcp)
    for (int t = c; t < tokens; t += blockDim.x) s.rcp[t] = 1.0 / (double)(t + 1);
  __syncthreads();

  float absmax = 0.f;
  if (c < C) {
    ChannelStats st = channel_statistics<T>(row + c, p.in.s_token, tokens, p.sample_stride, p.min_error != 0, s.rcp);
    s.saliency[c] = st.saliency;
    s.sampled_mean[c] = st.sampled_mean;
    s.error[c] = st.donor_error;
    absmax = st.absmax;
    if (!st.finite) atomicOr(p.status, INQ_STATUS_NONFINITE);
    s.kind[c] = 0;
    s.read_from[c] = c;
  }
  __syncthreads();
  select_donors_cta(s.saliency, s.error, p.min_error != 0, C, count, s.rank_key, s.sel_mask, s.avail_mask,
                    s.sources, s.donors);

  if (c < C) {
    bool selected = (s.sel_mask[c >> 5] >> (c & 31)) & 1u;
    float own = fmaxf(absmax / (selected ? 127.0f : 7.0f), 1.17549435e-38f);
    s.scale[c] = own;
    ((float*)p.scales.at(slot, inner))[c] = own;
    if (selected) s.kind[c] = 1;
  }
  __syncthreads();
  if (c < count) {
    int source = s.sources[c], donor = s.donors[c];
    s.kind[donor] = 2;
    s.read_from[donor] = source;
    ((float*)p.padding.at(slot, inner))[c] = s.sampled_mean[donor];
    if (p.salient.base) {
      if (p.descriptor_i32) {
        ((int*)p.salient.at(slot, inner))[c] = source;
        ((int*)p.donors.at(slot, inner))[c] = donor;
      } else {
        ((unsigned char*)p.salient.at(slot, inner))[c] = (unsigned char)source;
        ((unsigned char*)p.donors.at(slot, inner))[c] = (unsigned char)donor;
      }
    }
  }
  __syncthreads();
  if (c < count) s.scale[s.donors[c]] = s.scale[s.sources[c]];  // a donor slot divides by its source's scale
  if (p.roles.base) {
    // role: donor channel of a salient channel, -1 for a normal one, -2-i for the i-th donor
    if (c < C) {
      int role = -1;
      for (int i = 0; i < count; ++i) {
        if (s.sources[i] == c) role = s.donors[i];
        if (s.donors[i] == c) role = -2 - i;
      }
      if (p.role_bytes == 1)
        ((signed char*)p.roles.at(slot, inner))[c] = (signed char)role;
      else
        ((short*)p.roles.at(slot, inner))[c] = (short)role;
    }
  }
  __syncthreads();

  unsigned char* payload = (unsigned char*)p.payload.at(slot, inner);
  const int row_bytes = C / 2;
  if (p.vector_path) {
    // A thread owns 8 fixed channels (4 payload bytes) and strides over tokens.
    const int chunks = C / 8;
    const int lanes = (blockDim.x / chunks) * chunks;
    if (c < lanes) {
      const int chunk = c % chunks, t0 = c / chunks, t_step = lanes / chunks;
      float scale[8];
      int kind[8], from[8];
      bool any_remote = false;
#pragma unroll
      for (int j = 0; j < 8; ++j) {
        int ch = chunk * 8 + j;
        scale[j] = s.scale[ch];
        kind[j] = s.kind[ch];
        from[j] = s.read_from[ch];
        any_remote |= (from[j] != ch);
      }
      for (int t = t0; t < tokens; t += t_step) {
        const T* src = row + (long long)t * p.in.s_token;
        float v[8];
        if (sizeof(T) == 2) {
          uint4 bits = *(const uint4*)(src + chunk * 8);
          const T* h = (const T*)&bits;
#pragma unroll
          for (int j = 0; j < 8; ++j) v[j] = to_float<T>(h[j]);
        } else {
          float4 a = *(const float4*)(src + chunk * 8), b = *(const float4*)(src + chunk * 8 + 4);
          v[0] = a.x; v[1] = a.y; v[2] = a.z; v[3] = a.w; v[4] = b.x; v[5] = b.y; v[6] = b.z; v[7] = b.w;
        }
        if (any_remote) {
#pragma unroll
          for (int j = 0; j < 8; ++j)
            if (kind[j] == 2) v[j] = to_float<T>(src[from[j]]);
        }
        unsigned word = 0;
#pragma unroll
        for (int j = 0; j < 8; ++j) word |= encode_slot(v[j], scale[j], kind[j]) << (4 * j);
        *(unsigned*)(payload + (long long)t * row_bytes + chunk * 4) = word;
      }
    }
  } else {
    for (long long idx = c; idx < (long long)tokens * row_bytes; idx += blockDim.x) {
      int t = (int)(idx / row_bytes), b = (int)(idx % row_bytes);
      const T* src = row + (long long)t * p.in.s_token;
      unsigned lo = encode_slot(to_float<T>(src[s.read_from[2 * b]]), s.scale[2 * b], s.kind[2 * b]);
      unsigned hi = encode_slot(to_float<T>(src[s.read_from[2 * b + 1]]), s.scale[2 * b + 1], s.kind[2 * b + 1]);
      payload[idx] = (unsigned char)(lo | (hi << 4));
    }
  }
}

// ------------------------------------------------------------------------------------------
// 128-channel fast path (every decode-capable layout): same arithmetic as k4_encode_kernel,
// fewer instructions per element.
//   * |x| maximum and the finite check come from one unsigned maximum of the fp32 bit patterns
//     (NaN and Inf sort above every finite value);
//   * x / s uses a correctly rounded reciprocal and two fused corrections, which returns the
//     IEEE quotient (Markstein); scales below 2^-100 keep the plain division;
//   * the sets of channels are masks in registers.
// A launch of few rows lasts as long as one CTA, one of many is bound by issue; us per launch in graphs of 20, with
// the float64 chain walked by every channel, all-pairs ranks, settled donor choices and a branch per slot before,
// with what the comments below describe now: 12 rows of 256 tokens 21.5 -> 13.5, 496 rows 39.9 -> 24.2, 47 x 8
// token-major rows 41.0 -> 23.5, 187 x 8 of 64 tokens 42.2 -> 27.1, 400 of 16 tokens 11.2 -> 8.4.
struct Mask128 {
  unsigned long long lo, hi;
  __device__ __forceinline__ int below(int pos) const {   // largest member < pos, or -1
    if (pos > 64) {
      unsigned long long m = pos >= 128 ? hi : (hi & ((1ull << (pos - 64)) - 1ull));
      if (m) return 127 - __clzll((long long)m);
      pos = 64;
    }
    unsigned long long m = pos >= 64 ? lo : (lo & ((1ull << pos) - 1ull));
    return m ? 63 - __clzll((long long)m) : -1;
  }
  __device__ __forceinline__ int above(int pos) const {   // smallest member > pos, or 128
    int start = pos + 1;
    if (start < 64) {
      unsigned long long m = lo & (~0ull << start);
      if (m) return __ffsll((long long)m) - 1;
      start = 64;
    }
    if (start >= 128) return 128;
    unsigned long long m = hi & (~0ull << (start - 64));
    return m ? 63 + __ffsll((long long)m) : 128;
  }
};

// the n lowest bits, for any n
__device__ __forceinline__ unsigned bits_below(int n) { return n <= 0 ? 0u : n >= 32 ? ~0u : (1u << n) - 1u; }

__device__ __forceinline__ float exact_quotient(float x, float s, float r, bool plain) {
  if (plain) return x / s;
  const float q0 = x * r;
  const float rem = fmaf(-q0, s, x);
  return fmaf(rem, r, q0);
}

template <typename T>
__device__ __forceinline__ unsigned f32_bits_of(T v) { return __float_as_uint(to_float<T>(v)); }

__device__ __forceinline__ void stage_copy16(void* dst, const void* src) {
  const unsigned d = (unsigned)__cvta_generic_to_shared(dst);
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(d), "l"(src) : "memory");
}
__device__ __forceinline__ void stage_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N>
__device__ __forceinline__ void stage_wait() { asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory"); }

// Channels (of 128, one per thread) with a larger key than `mine`, or the same one and a lower number than c.
// Keys are at most 0x7fffffff; `keys` holds those of the thread's own warp at least, `sorted` is scratch for 128.
// The warp's own keys are compared one by one, which sorts them; the other three sorted lists are searched by
// halves.  (Comparing with all 128 keys takes twice the instructions.)  Contains a CTA barrier between the two.
__device__ __forceinline__ int rank_of(const unsigned* keys, unsigned* sorted, unsigned mine, int c) {
  const int warp = c >> 5, lane = c & 31, own = lane >> 2;
  int rank = 0;
#pragma unroll
  for (int o4 = 0; o4 < 8; ++o4) {
    const uint4 k = *(const uint4*)(keys + 32 * warp + 4 * o4);
    const unsigned limit = mine + (o4 < own ? 0u : 1u);
    rank += (k.x >= limit) + (k.y >= limit) + (k.z >= limit) + (k.w >= limit);
  }
#pragma unroll
  for (int e = 0; e < 3; ++e) rank += e < (lane & 3) && keys[32 * warp + 4 * own + e] == mine;
  sorted[32 * warp + rank] = mine;   // descending
  __syncthreads();
  const unsigned* list[3];
  unsigned limit[3];
  int ahead[3] = {0, 0, 0};
#pragma unroll
  for (int d = 0; d < 3; ++d) {
    const int other = (warp + 1 + d) & 3;
    list[d] = sorted + 32 * other;
    limit[d] = mine + (other < warp ? 0u : 1u);
  }
#pragma unroll
  for (int step = 16; step; step >>= 1)
#pragma unroll
    for (int d = 0; d < 3; ++d) ahead[d] += list[d][ahead[d] + step - 1] >= limit[d] ? step : 0;
#pragma unroll
  for (int d = 0; d < 3; ++d) rank += ahead[d] + (list[d][ahead[d]] >= limit[d]);
  return rank;
}

// Welford's update in float64, sequential over tokens (the reference's var_mean), of one channel.
template <typename T>
__device__ __noinline__ void welford(const T* column, long long step, int tokens, const double* inverse, double& mean_out, double& m2_out) {
  double mean = 0.0, m2 = 0.0, n = 0.0;
  for (int t = 0; t < tokens; ++t) {
    const double x = (double)to_float<T>(column[t * step]);
    const double delta = x - mean;
    n = n + 1.0;
    mean = mean + divide_by_count(delta, n, inverse[t]);
    m2 = m2 + delta * (x - mean);
  }
  mean_out = mean;
  m2_out = m2;
}

// What the encoder needs of Welford's chain is one float32 number, the error of the channel as a donor:
// (float)(m2 / tokens) + ((float)mean - sampled mean)^2.  Plain float64 sums S1 of x and S2 of x * x lie close enough
// to the chain that its rounding is nearly always decided: the chain's five dependent operations a token (68 cycles
// of a warp alone, 25 of its issue) become two additions that depend on nothing but their own sums.  Every
// rounding on the way is monotone, so the chain's number lies between those that the ends of intervals give which
// hold the chain's mean and m2.  Where the two differ -- by a unit in the last place -- the chain is walked only if
// that could decide which channels are among the least.
//
// With u = 2^-53, n tokens of at most M, V = sum (x - mean)^2 and S2 = sum x^2, and first-order terms (a margin of a
// tenth stands for the others):
//   chain, mean:   mean_k = mean_{k-1} (1 - 1/k) + x/k + r_k, k |r_k| <= u (2 |x - mean_{k-1}| + k |mean_k|), and the error
//                  of mean_k is at most 1/k times the sum of these.  sum (x_k - mean_{k-1}) (x_k - mean_k) = V with
//                  x_k - mean_k = (x_k - mean_{k-1}) (1 - 1/k), so the first parts add up to 2 (M + sqrt(2 k S2)); |mean_k| <=
//                  sqrt(S2 / k), so the second to 2/3 (k + 1)^1.5 sqrt(S2).  For any k up to n the error is at most
//                  E = u (2 M + sqrt(S2) (4.9 + 0.67 sqrt(n))).
//   chain, m2:     a summand is off by |x - mean_{k-1}| E + |x - mean_k| E + E^2 + 3 u |summand|; the absolute values add
//                  up to sqrt(2 n V) and sqrt(n V) (the first summand is exactly 0), and the additions give
//                  n u V:  2.42 E sqrt(n V) + n E^2 + (n + 3) u V.
//   plain sums:    in four interleaved parts:  S1 is off by u (n/4 + 3) sum |x|, S2 by u (n/4 + 4) S2, and with
//                  sum |x| <= sqrt(n S2):  S2 - S1^2 / n is off by u (n/4 + 4) S2 + 2 u (n/4 + 3) S2 + 4 u S2.
// `inverse` is 1 / (double)n, correctly rounded.
__device__ __forceinline__ void plain_donor_error(double s1, double s2, int tokens, double inverse, float absmax, float sampled_mean,
                                                  float& low, float& high) {
  const double n = (double)tokens;
  const double mean = s1 * inverse, v = s2 - s1 * mean;
  const float nf = (float)tokens, u = 1.110223e-16f;
  const float s2f = (float)s2 * 1.0001f, vf = fmaxf((float)v, 0.f) * 1.0001f + u * (0.75f * nf + 14.f) * s2f;   // no less than V
  const float e = u * (2.f * absmax + sqrtf(s2f) * (4.9f + 0.67f * sqrtf(nf)));
  const float mean_bound = 1.1f * (e + u * (0.25f * nf + 5.f) * absmax);
  const float m2_bound = 1.1f * (2.42f * e * sqrtf(nf * vf) + nf * e * e + (nf + 3.f) * u * vf + (0.75f * nf + 14.f) * u * s2f);
  const float d0 = (float)(mean - (double)mean_bound) - sampled_mean, d1 = (float)(mean + (double)mean_bound) - sampled_mean;
  const float near = d0 * d1 > 0.f ? fminf(fabsf(d0), fabsf(d1)) : 0.f, far = fmaxf(fabsf(d0), fabsf(d1));
  low = fmaxf((float)((v - (double)m2_bound) / n) + near * near, 0.f);
  high = (float)((v + (double)m2_bound) / n) + far * far;
  // (the bounds are computed in float32: a channel whose squares leave its range may be anything)
  if (!(absmax > 1e-12f && absmax < 1e15f)) {
    low = 0.f;
    high = absmax == 0.f ? 0.f : INFINITY;
  }
}

// REGULAR: tokens % 8 == 0 and sample_stride == 8.
// STAGED (16-bit inputs, contiguous rows, tokens % 32 == 0): the row's tokens stream twice -- once
// for the statistics, once for the packing -- through a ring of four 8 KB shared-memory stages
// filled by 16-byte asynchronous copies, three groups of 32 tokens in flight per CTA; every warp
// stages exactly the bytes it reads, so the two passes run without CTA-wide barriers.  A thread
// that fetches its own channel with 2-byte loads keeps only 16 bytes in flight, which left the
// kernel waiting on memory latency at a tenth of the HBM rate.
template <typename T, bool REGULAR, bool STAGED = false>
__global__ void __launch_bounds__(128, STAGED ? 5 : 7) k4_encode128_kernel(K4Params p) {
  constexpr int C = 128;
  constexpr int kGroupTokens = 32, kRing = 4;
  constexpr int kRowBytes = C * (int)sizeof(T);
  constexpr int kGroupBytes = kGroupTokens * kRowBytes;
  constexpr int kWarpStage = kGroupBytes / 4;   // a warp's share of a stage
  // STAGED: the ring; else two pairs of rows per warp
  __shared__ __align__(16) unsigned char s_ring[STAGED ? kRing * kGroupBytes : 4 * 4 * kRowBytes];
  __shared__ __align__(16) float s_sal[C];      // read four at a time, like s_key
  __shared__ float s_mean[C], s_scale[C], s_rcp[C];
  __shared__ __align__(16) unsigned s_key[C];
  __shared__ unsigned s_sorted[C];
  __shared__ unsigned char s_kind[C], s_from[C], s_plain[C];
  __shared__ signed char s_role[C];
  __shared__ int s_src[64], s_don[64];
  __shared__ unsigned s_sel[4], s_avail[4], s_range[2];
  __shared__ uint2 s_pool[32];                  // {channel, saliency bits} of the least-error channels, ascending
  __shared__ __align__(16) uint4 s_seek[32];    // per source: pool entries below it, its run of sources, itself
  const int tokens = p.in.tokens, count = p.count;
  const bool want_error = p.min_error != 0;
  const long long outer = blockIdx.x / p.in.n_inner, inner = blockIdx.x % p.in.n_inner;
  const long long slot = p.in.slot(outer);
  if (!p.in.slot_ok(slot)) {   // uniform over the CTA: nothing of this row is written
    if (threadIdx.x == 0) atomicOr(p.status, INQ_STATUS_BAD_INDEX);
    return;
  }
  const T* row = (const T*)p.in.x + outer * p.in.s_outer + inner * p.in.s_inner;
  const int c = threadIdx.x;
  if (c < 4) s_sel[c] = s_avail[c] = 0u;
  s_role[c] = -1;

  // ---- statistics: one thread per channel
  unsigned top_bits = 0u;
  CascadePair cascade;
  const int samples = (tokens + p.sample_stride - 1) / p.sample_stride;
  cascade.init(samples);
  double s1[4] = {0.0, 0.0, 0.0, 0.0}, s2[4] = {0.0, 0.0, 0.0, 0.0};   // of x and of x * x, see plain_donor_error
  int next_sample = 0;
  {
    const T* column = row + c;
    constexpr int kUnroll = 8;
    const long long step = p.in.s_token;
    // the next batch of tokens is requested before the current one is consumed, so the
    // sequential (Welford) chain never waits on a freshly issued load
    T ahead[kUnroll];
    if constexpr (STAGED) {
      // Every warp stages what it reads itself, so the passes need no CTA-wide barrier: for the
      // statistics the 64 bytes of its 32 channels in each of the group's 32 token rows.
      const int n_groups = tokens / kGroupTokens;
      const int warp_id = c >> 5, lane_id = c & 31;
      unsigned char* const warp_ring = s_ring + warp_id * (kRing * kWarpStage);
      const unsigned char* src_bytes = (const unsigned char*)row;
      auto issue = [&](int step_index) {
        if (step_index < 2 * n_groups) {
          unsigned char* dst = warp_ring + (step_index & (kRing - 1)) * kWarpStage;
          if (step_index < n_groups) {
            const unsigned char* src = src_bytes + (long long)step_index * kGroupBytes + warp_id * 64;
#pragma unroll
            for (int k = 0; k < 4; ++k) {
              const int idx = k * 32 + lane_id, token = idx >> 2, part = idx & 3;
              stage_copy16(dst + token * 64 + part * 16, src + token * kRowBytes + part * 16);
            }
          } else {
            // packing: the thread's own 16 bytes of token rows 2 * warp + lane / 16 + 8k
            const unsigned char* src = src_bytes + (long long)(step_index - n_groups) * kGroupBytes;
#pragma unroll
            for (int k = 0; k < 4; ++k) {
              const int token = 2 * warp_id + (lane_id >> 4) + 8 * k;
              stage_copy16(dst + (2 * k + (lane_id >> 4)) * kRowBytes + (lane_id & 15) * 16,
                           src + token * kRowBytes + (lane_id & 15) * 16);
            }
          }
        }
        stage_commit();
      };
      issue(0);
      issue(1);
      issue(2);
      for (int g = 0; g < n_groups; ++g) {
        stage_wait<kRing - 2>();
        __syncwarp();   // group g has landed for every lane; the stage of group g - 1 is free
        issue(g + 3);
        const T* tile = (const T*)(warp_ring + (g & (kRing - 1)) * kWarpStage) + lane_id;
#pragma unroll
        for (int b = 0; b < kGroupTokens / kUnroll; ++b) {
          float v[kUnroll];
#pragma unroll
          for (int u = 0; u < kUnroll; ++u) v[u] = to_float<T>(tile[(b * kUnroll + u) * 32]);
          cascade.add(v[0]);   // every eighth token is a sample
#pragma unroll
          for (int u = 0; u < kUnroll; ++u) {
            const float x = v[u];
            top_bits = max(top_bits, __float_as_uint(x) & 0x7fffffffu);
            if (want_error) {
              const double xd = (double)x;
              s1[u & 3] = s1[u & 3] + xd;
              s2[u & 3] = fma(xd, xd, s2[u & 3]);
            }
          }
        }
      }
      (void)step;
      (void)ahead;
    } else if (REGULAR) {
      const T* cursor = column;
#pragma unroll
      for (int u = 0; u < kUnroll; ++u) ahead[u] = cursor[u * step];
      for (int base = 0; base < tokens; base += kUnroll) {
        float v[kUnroll];
#pragma unroll
        for (int u = 0; u < kUnroll; ++u) v[u] = to_float<T>(ahead[u]);
        cursor += kUnroll * step;
        if (base + kUnroll < tokens) {
#pragma unroll
          for (int u = 0; u < kUnroll; ++u) ahead[u] = cursor[u * step];
        }
        cascade.add(v[0]);   // every eighth token is a sample
#pragma unroll
        for (int u = 0; u < kUnroll; ++u) {
          const float x = v[u];
          top_bits = max(top_bits, __float_as_uint(x) & 0x7fffffffu);
          if (want_error) {
            const double xd = (double)x;
            s1[u & 3] = s1[u & 3] + xd;
            s2[u & 3] = fma(xd, xd, s2[u & 3]);
          }
        }
      }
    } else {
#pragma unroll
    for (int u = 0; u < kUnroll; ++u) ahead[u] = u < tokens ? column[(long long)u * p.in.s_token] : T();
    for (int base = 0; base < tokens; base += kUnroll) {
      float v[kUnroll];
#pragma unroll
      for (int u = 0; u < kUnroll; ++u) v[u] = to_float<T>(ahead[u]);
#pragma unroll
      for (int u = 0; u < kUnroll; ++u) {
        const int t = base + kUnroll + u;
        if (t < tokens) ahead[u] = column[(long long)t * p.in.s_token];
      }
#pragma unroll
      for (int u = 0; u < kUnroll; ++u) {
        const int t = base + u;
        if (t < tokens) {
          const float x = v[u];
          top_bits = max(top_bits, __float_as_uint(x) & 0x7fffffffu);
          if (t == next_sample) {
            cascade.add(x);
            next_sample += p.sample_stride;
          }
          if (want_error) {
            const double xd = (double)x;
            s1[u & 3] = s1[u & 3] + xd;
            s2[u & 3] = fma(xd, xd, s2[u & 3]);
          }
        }
      }
    }
    }
  }
  float abs_total, sum_total;
  cascade.finish(abs_total, sum_total);
  const float saliency = abs_total / (float)samples, sampled_mean = sum_total / (float)samples;
  if (top_bits >= 0x7f800000u) atomicOr(p.status, INQ_STATUS_NONFINITE);
  const float absmax = __uint_as_float(top_bits);
  float error_low = 0.f, error_high = 0.f;   // hold the channel's error as a donor
  if (want_error)
    plain_donor_error((s1[0] + s1[1]) + (s1[2] + s1[3]), (s2[0] + s2[1]) + (s2[2] + s2[3]), tokens, kInverse.of[tokens - 1], absmax,
                      sampled_mean, error_low, error_high);
  s_sal[c] = saliency;
  s_mean[c] = sampled_mean;
  __syncwarp();

  // ---- top-`count` channels by saliency (ties: lower channel), optional least-error pool
  bool selected = false;
  if (count > 0) {
    selected = rank_of((const unsigned*)s_sal, s_sorted, __float_as_uint(saliency), c) < count;
    if (selected) atomicOr(&s_sel[c >> 5], 1u << (c & 31));
    if (!want_error && !selected) atomicOr(&s_avail[c >> 5], 1u << (c & 31));
  }
  bool open = __syncthreads_or(want_error && !(error_low == error_high));   // a channel's error is not known to the last bit
  // position of this channel in a set of channels
  auto place = [&](const unsigned* set) {
    int position = __popc(set[c >> 5] & ((1u << (c & 31)) - 1u));
    for (int w = 0; w < (c >> 5); ++w) position += __popc(set[w]);
    return position;
  };
  if (selected) s_src[place(s_sel)] = c;   // the ascending list of sources
  if (want_error && count > 0) {
    bool near;
    while (true) {
      // channels with a smaller error, or the same one and a lower number (descending: the smaller the error, the
      // larger the key; a selected channel comes last)
      s_key[c] = 0x7fffffffu - (selected ? 0x7f800000u : __float_as_uint(error_high));
      __syncwarp();
      near = rank_of(s_key, s_sorted, s_key[c], c) < count && !selected;
      if (!open) break;
      // the same channels whatever the open errors are, if the largest taken lies below the smallest left
      if (c == 0) {
        s_range[0] = 0u;
        s_range[1] = 0x7f800000u;
      }
      __syncthreads();
      if (near) atomicMax(&s_range[0], __float_as_uint(error_high));
      else if (!selected) atomicMin(&s_range[1], __float_as_uint(error_low));
      __syncthreads();
      if (s_range[0] < s_range[1]) break;
      double mean, m2;
      welford<T>(row + c, p.in.s_token, tokens, kInverse.of, mean, m2);
      const float variance = (float)(m2 / (double)tokens);
      const float diff = (float)mean - sampled_mean;
      error_high = variance + diff * diff;
      open = false;
      __syncthreads();
    }
    if (near) atomicOr(&s_avail[c >> 5], 1u << (c & 31));
    __syncthreads();
    if (near && count <= 32) s_pool[place(s_avail) & 31] = make_uint2((unsigned)c, __float_as_uint(saliency));
  }
  __syncthreads();
  if (c < 32 && count > 0 && count <= 32 && want_error) {
    // Donors are taken by the sources in ascending order, each from what the earlier ones left.  With least-error
    // donors there are just as many of them as sources, most sources meet a donor that is gone, and one after
    // the other is the order of things: the pool's entries are bits of one word, a source finds its two neighbours
    // by two bit scans and one look-up.  (For 16 sources 3200 to 4500 cycles; settling choices made ahead, as below,
    // 5200 to 8700.)
    const Mask128 others{~((unsigned long long)s_sel[0] | ((unsigned long long)s_sel[1] << 32)),
                         ~((unsigned long long)s_sel[2] | ((unsigned long long)s_sel[3] << 32))};
    if (c < count) {
      const int source = s_src[c];
      int below = 0;
#pragma unroll
      for (int w = 0; w < 4; ++w) below += __popc(s_avail[w] & bits_below(source - 32 * w));
      s_seek[c] = make_uint4(bits_below(below), (unsigned)(others.below(source) + 1), (unsigned)(others.above(source) - 1), (unsigned)source);
    }
    __syncwarp();
    unsigned free_ = bits_below(count);
    uint4 next = s_seek[0];
    for (int i = 0; i < count; ++i) {
      const uint4 seek = next;
      if (i + 1 < count) next = s_seek[i + 1];
      const unsigned b = free_ & seek.x, h = free_ & ~seek.x;
      const int at_low = 31 - __clz(b), at_high = __ffs(h) - 1;      // -1 where there is none
      const uint2 e_low = s_pool[max(at_low, 0)], e_high = s_pool[max(at_high, 0)];
      const int low = (int)e_low.x, high = (int)e_high.x, left = (int)seek.y, right = (int)seek.z, source = (int)seek.w;
      // one next to the source itself wins over any other, else the nearer one; of two the less salient, then the lower
      const bool has_low = b != 0u, has_high = h != 0u;
      const int d_low = has_low ? left - low : C, d_high = has_high ? high - right : C;
      const bool by_low = has_low && low == source - 1, by_high = has_high && high == source + 1, beside = by_low || by_high;
      const bool take_low = beside ? by_low : has_low && d_low <= d_high, take_high = beside ? by_high : has_high && d_high <= d_low;
      const bool lower = __uint_as_float(e_low.y) <= __uint_as_float(e_high.y);
      const bool chosen_low = take_low && (lower || !take_high);
      free_ &= ~(1u << ((chosen_low ? at_low : at_high) & 31));
      if (c == i) s_don[i] = chosen_low ? low : take_high ? high : 0;   // (one is free for every source)
    }
  } else if (c < 32 && count > 0) {
    // Any channel that is not a source may be a donor (or there are more than a word's bits of them).  One lane per
    // source: all choose at once, then the choices are settled one by one (a shuffle, a vote), and only when the
    // donor just taken was the choice of a later source do the later ones choose again -- a donor that is gone
    // but was not a source's choice changes neither which of its candidates is nearer nor the tie between
    // them.  (All of them choosing again from conflict to conflict, with a match and four reductions a round, took
    // 400 rows of 16 tokens 19.3 instead of 11.2 us with least-error donors, 64 rows of 64 19.5 / 11.8, 12 rows of
    // 256 29.0 / 21.8, 496 of 256 46.8 / 39.8; one thread walking the list with branches 18.0, 19.2, 37.1 and
    // 53.7; a walk without branches but with no choice ahead of it 11.4, 12.0, 22.4 and 40.1.)
    const Mask128 others{~((unsigned long long)s_sel[0] | ((unsigned long long)s_sel[1] << 32)),
                         ~((unsigned long long)s_sel[2] | ((unsigned long long)s_sel[3] << 32))};
    unsigned free_[4] = {s_avail[0], s_avail[1], s_avail[2], s_avail[3]};
    for (int first = 0; first < count; first += 32) {
      const int n = min(32, count - first);
      const int source = c < n ? s_src[first + c] : 0;
      const int left = others.below(source) + 1, right = others.above(source) - 1;   // the run of sources around this one
      unsigned below[4], above[4];
#pragma unroll
      for (int w = 0; w < 4; ++w) {
        below[w] = bits_below(left - 32 * w);
        above[w] = ~bits_below(right + 1 - 32 * w);
      }
      int choice = 0, i = 0;
      while (true) {
        // nearest free channel on either side of the run: -1 and 128 where there is none
        int low = -1, high = C;
#pragma unroll
        for (int w = 0; w < 4; ++w) {
          const unsigned b = free_[w] & below[w], h = free_[3 - w] & above[3 - w];
          low = b ? 32 * w + 31 - __clz(b) : low;
          high = h ? 32 * (3 - w) + __ffs(h) - 1 : high;
        }
        // one next to the source itself wins over any other, else the nearer one; of two the less salient, then the lower
        const bool has_low = low >= 0, has_high = high < C;
        const int d_low = has_low ? left - low : C, d_high = has_high ? high - right : C;
        const bool by_low = has_low && low == source - 1, by_high = has_high && high == source + 1, beside = by_low || by_high;
        const bool take_low = beside ? by_low : has_low && d_low <= d_high, take_high = beside ? by_high : has_high && d_high <= d_low;
        const bool lower = s_sal[max(low, 0)] <= s_sal[min(high, C - 1)];
        const int donor = take_low && (lower || !take_high) ? low : take_high ? high : 0;   // (one is free for every source)
        if (c >= i) choice = donor;
        int taken;
        do {
          taken = __shfl_sync(0xffffffffu, choice, i);
#pragma unroll
          for (int w = 0; w < 4; ++w) free_[w] &= (taken >> 5) == w ? ~(1u << (taken & 31)) : ~0u;
          ++i;
        } while (i < n && !__any_sync(0xffffffffu, c >= i && c < n && choice == taken));
        if (i >= n) break;
      }
      if (c < n) s_don[first + c] = choice;
    }
  }
  // ---- scales and per-slot encoding parameters
  const float own_scale = fmaxf(absmax / (selected ? 127.0f : 7.0f), 1.17549435e-38f);
  s_scale[c] = own_scale;
  s_rcp[c] = __frcp_rn(own_scale);
  s_plain[c] = own_scale < 7.8886091e-31f;   // 2^-100: remainders would underflow
  s_kind[c] = selected ? 1 : 0;
  s_from[c] = (unsigned char)c;
  ((float*)p.scales.at(slot, inner))[c] = own_scale;
  __syncthreads();
  if (c < count) {
    const int source = s_src[c], donor = s_don[c];
    s_kind[donor] = 2;
    s_from[donor] = (unsigned char)source;
    s_role[source] = (signed char)donor;
    s_role[donor] = (signed char)(-2 - c);
    ((float*)p.padding.at(slot, inner))[c] = s_mean[donor];
    if (p.salient.base) {
      ((unsigned char*)p.salient.at(slot, inner))[c] = (unsigned char)source;
      ((unsigned char*)p.donors.at(slot, inner))[c] = (unsigned char)donor;
    }
  }
  __syncthreads();
  if (p.roles.base) {
    const int role = s_role[c];
    if (p.role_bytes == 1)
      ((signed char*)p.roles.at(slot, inner))[c] = (signed char)role;
    else
      ((short*)p.roles.at(slot, inner))[c] = (short)role;
  }
  // ---- packing: a thread owns 8 fixed slots (4 payload bytes) and strides over tokens
  unsigned char* payload = (unsigned char*)p.payload.at(slot, inner);
  const int chunk = c & 15, t0 = c >> 4;
  // per slot: divisor, bias and which nibble of the code is stored -- a normal slot keeps q + 8, a salient slot
  // the high nibble of q + 128, a donor slot the low nibble of its source's code; all three are
  // (code >> shift) & 15.  q needs no clamp: a scale is the channel's largest magnitude over 7 (or 127) rounded, or
  // larger, so the quotient is at most that whole number and a few units in its last place and rounds to it.
  // Adding the bias and 1.5 * 2^23 rounds the quotient as rint does (the bias is even, so the sum moves no tie)
  // and leaves the code in the low bits; a rotation brings its nibble to the slot's place.
  float scale[8], rcp[8], bias[8];
  int rotate[8], from[8];
  bool any_plain = false;
#pragma unroll
  for (int j = 0; j < 8; ++j) {
    const int ch = chunk * 8 + j;
    const int kind = s_kind[ch];
    from[j] = s_from[ch];
    const int src_ch = from[j];       // a donor slot divides its source's value by its source's scale
    scale[j] = s_scale[src_ch];
    rcp[j] = s_rcp[src_ch];
    any_plain |= s_plain[src_ch] != 0;
    bias[j] = 12582912.f + (kind ? 128.f : 8.f);
    rotate[j] = 4 * j - (kind == 1 ? 4 : 0);
  }
  // A token's row in shared memory: every slot fetches its value by itself, the donor slots from their sources.
  // (256 tokens of a CTA alone on its SM 7900 cycles; with a 16-byte load of the own channels, a branch per slot
  // for the others and the clamps 12500.)
  auto pack_row = [&](const T* trow, auto plain) {
    unsigned word = 0;
#pragma unroll
    for (int j = 0; j < 8; ++j) {
      const float v = to_float<T>(trow[from[j]]);
      const unsigned code = __float_as_uint(exact_quotient(v, scale[j], rcp[j], decltype(plain)::value) + bias[j]);
      word |= __funnelshift_l(code, code, rotate[j]) & (15u << (4 * j));
    }
    return word;
  };
  any_plain = __any_sync(0xffffffffu, any_plain);
  if constexpr (STAGED) {
    const int n_groups = tokens / kGroupTokens;
    const int warp_id = c >> 5, lane_id = c & 31;
    unsigned char* const warp_ring = s_ring + warp_id * (kRing * kWarpStage);
    const unsigned char* src_bytes = (const unsigned char*)row;
    for (int g = 0; g < n_groups; ++g) {
      const int step_index = n_groups + g;
      stage_wait<kRing - 2>();
      __syncwarp();
      if (step_index + 3 < 2 * n_groups) {
        unsigned char* dst = warp_ring + ((step_index + 3) & (kRing - 1)) * kWarpStage;
        const unsigned char* src = src_bytes + (long long)(g + 3) * kGroupBytes;
#pragma unroll
        for (int k = 0; k < 4; ++k) {
          const int token = 2 * warp_id + (lane_id >> 4) + 8 * k;
          stage_copy16(dst + (2 * k + (lane_id >> 4)) * kRowBytes + (lane_id & 15) * 16,
                       src + token * kRowBytes + (lane_id & 15) * 16);
        }
      }
      stage_commit();
      const unsigned char* tile = warp_ring + (step_index & (kRing - 1)) * kWarpStage;
#pragma unroll
      for (int i = 0; i < kGroupTokens / 8; ++i) {
        const int tl = t0 + 8 * i;   // t0 = 2 * warp + lane / 16
        const T* trow = (const T*)(tile + (2 * i + (lane_id >> 4)) * kRowBytes);
        const unsigned word = any_plain ? pack_row(trow, std::true_type()) : pack_row(trow, std::false_type());
        *(unsigned*)(payload + (long long)(g * kGroupTokens + tl) * 64 + chunk * 4) = word;
      }
    }
    stage_wait<0>();
    return;
  }
  // rows from global memory: a warp passes two tokens at a time through rows of its own in shared memory
  constexpr int kVec = sizeof(T) == 2 ? 1 : 2;   // 16-byte vectors per 8 elements
  T* const lane_row = (T*)s_ring + (c >> 5) * 4 * C + ((c >> 4) & 1) * C;
  uint4 next[kVec];
  if (t0 < tokens) {
#pragma unroll
    for (int q = 0; q < kVec; ++q) next[q] = ((const uint4*)(row + (long long)t0 * p.in.s_token + chunk * 8))[q];
  }
  const long long pack_step = 8 * p.in.s_token;
  const T* src = row + (long long)t0 * p.in.s_token;
  unsigned char* dst = payload + (long long)t0 * 64 + chunk * 4;
  int turn = 0;
  for (int t = t0 & ~1; t < tokens; t += 8) {   // (whole warps walk; the upper half has no token where the last pair is one)
    T* const trow = lane_row + turn;
    turn ^= 2 * C;
#pragma unroll
    for (int q = 0; q < kVec; ++q) ((uint4*)(trow + chunk * 8))[q] = next[q];
    __syncwarp();
    src += pack_step;
    if (t + (t0 & 1) + 8 < tokens) {
#pragma unroll
      for (int q = 0; q < kVec; ++q) next[q] = ((const uint4*)(src + chunk * 8))[q];
    }
    const unsigned word = any_plain ? pack_row(trow, std::true_type()) : pack_row(trow, std::false_type());
    if (t + (t0 & 1) < tokens) *(unsigned*)dst = word;
    dst += 512;
  }
}

template <typename T>
__global__ void __launch_bounds__(1024) k4_statistics_kernel(InputRef in, int sample_stride, float* saliency,
                                                              float* sampled_mean, float* donor_error, float* absmax) {
  extern __shared__ __align__(16) unsigned char raw[];
  double* rcp = (donor_error && in.tokens <= kRcpTable) ? (double*)raw : nullptr;
  const long long outer = blockIdx.x / in.n_inner, inner = blockIdx.x % in.n_inner;
  const T* row = (const T*)in.x + outer * in.s_outer + inner * in.s_inner;
  if (rcp)
    for (int t = threadIdx.x; t < in.tokens; t += blockDim.x) rcp[t] = 1.0 / (double)(t + 1);
  __syncthreads();
  const int c = threadIdx.x;
  if (c >= in.channels) return;
  ChannelStats st = channel_statistics<T>(row + c, in.s_token, in.tokens, sample_stride, donor_error != nullptr, rcp);
  long long o = (long long)blockIdx.x * in.channels + c;
  if (saliency) saliency[o] = st.saliency;
  if (sampled_mean) sampled_mean[o] = st.sampled_mean;
  if (donor_error) donor_error[o] = st.donor_error;
  if (absmax) absmax[o] = st.absmax;
}

__global__ void __launch_bounds__(1024) select_kernel(const float* saliency, const float* error, int channels, int count,
                                                       long long* sources, long long* donors) {
  extern __shared__ __align__(16) unsigned char raw[];
  float* sal = (float*)raw;
  float* err = sal + channels;
  unsigned* rank_key = (unsigned*)(err + channels);
  unsigned* sel_mask = rank_key + channels;
  unsigned* avail_mask = sel_mask + kMaxWords;
  int* src = (int*)(avail_mask + kMaxWords);
  int* don = src + count;
  const long long row = blockIdx.x;
  const int c = threadIdx.x;
  if (c < channels) {
    sal[c] = saliency[row * channels + c];
    err[c] = error ? error[row * channels + c] : 0.f;
  }
  __syncthreads();
  select_donors_cta(sal, err, error != nullptr, channels, count, rank_key, sel_mask, avail_mask, src, don);
  if (c < count) {
    sources[row * count + c] = src[c];
    donors[row * count + c] = don[c];
  }
}

// ------------------------------------------------------------------------------------------
// Eight channels of one token from the thread's word of the payload row.  The row's 16 words lie in 16
// neighbouring lanes, so the low half of a salient code comes from its donor's lane by a shuffle (with a
// load of that byte in a divergent branch per slot the keys of 496 rows of 256 tokens took 30.4 instead of
// 21.6 us); `salient` names the slots where any lane of the warp needs one.  A whole
// number below 2^23 becomes a float by its bits under those of 2^23.  All lanes of the warp call.
template <typename T>
__device__ __forceinline__ uint4 k4_decode8(unsigned word, const int (&role)[8], const float (&scale)[8], const float (&constant)[8],
                                            unsigned salient) {
  uint4 packed;
  T* const vals = (T*)&packed;
#pragma unroll
  for (int k = 0; k < 8; ++k) {
    const unsigned slot = (word >> (4 * k)) & 15u;
    float code = __uint_as_float(0x4B000000u | slot) - 8388616.f;   // slot - 8
    if ((salient >> k) & 1u) {
      const unsigned other = __shfl_sync(0xffffffffu, word, (threadIdx.x & 16) | ((role[k] >> 3) & 15));
      const unsigned both = (slot << 4) | ((other >> (4 * (role[k] & 7))) & 15u);
      if (role[k] >= 0) code = __uint_as_float(0x4B000000u | both) - 8388736.f;   // code - 128
    }
    vals[k] = from_float<T>(role[k] < -1 ? constant[k] : code * scale[k]);
  }
  return packed;
}

// 128-channel rows, 16-bit output: a thread owns 8 consecutive channels of one token (4 payload bytes
// in, 16 bytes out); 16 threads cover a token, a CTA of 256 threads covers 16 tokens per step.
template <typename T>
__global__ void __launch_bounds__(256) k4_dequantize128_kernel(const unsigned char* payload, const float* scales, const void* salient,
                                                               const void* donors, const float* padding, int tokens, int count, T* out,
                                                               int rows_inner, long long out_so, long long out_si) {
  __shared__ int role[128];
  __shared__ float scale[128], pad[128];
  const long long row = blockIdx.x;
  if (threadIdx.x < 128) {
    role[threadIdx.x] = -1;
    scale[threadIdx.x] = scales[row * 128 + threadIdx.x];
    pad[threadIdx.x] = 0.f;
  }
  __syncthreads();
  if ((int)threadIdx.x < count) {
    const int i = threadIdx.x;
    const int s = ((const unsigned char*)salient)[row * count + i], d = ((const unsigned char*)donors)[row * count + i];
    role[s] = d;
    role[d] = -2 - i;
    pad[d] = padding[row * count + i];
  }
  __syncthreads();
  const unsigned char* bytes = payload + row * (long long)tokens * 64;
  T* dst = out + (row / rows_inner) * out_so + (row % rows_inner) * out_si;
  const int c0 = (threadIdx.x & 15) * 8;
  int r[8];
  float sc[8], pd[8];
#pragma unroll
  for (int k = 0; k < 8; ++k) {
    r[k] = role[c0 + k];
    sc[k] = scale[c0 + k];
    pd[k] = pad[c0 + k];
  }
  unsigned any_salient = 0u;
#pragma unroll
  for (int k = 0; k < 8; ++k) any_salient |= __any_sync(0xffffffffu, r[k] >= 0) ? 1u << k : 0u;
  const int per_cta = (tokens + gridDim.y - 1) / gridDim.y;
  const int t_begin = blockIdx.y * per_cta, t_end = min(tokens, t_begin + per_cta);
  // (whole warps walk the tokens; a lane past the end decodes the last token again and stores nothing)
  const int mine = (threadIdx.x >> 4) & 1;
  auto fetch = [&](int t) { return __ldg((const unsigned*)(bytes + (long long)min(t, t_end - 1) * 64 + (c0 >> 1))); };
  int t = t_begin + 2 * (int)(threadIdx.x >> 5);
  unsigned next = t < t_end ? fetch(t + mine) : 0u;
  for (; t < t_end; t += 16) {
    const unsigned word = next;
    if (t + 16 < t_end) next = fetch(t + 16 + mine);
    const uint4 vals = k4_decode8<T>(word, r, sc, pd, any_salient);
    if (t + mine < t_end) *(uint4*)(dst + (long long)(t + mine) * 128 + c0) = vals;
  }
}

template <typename T>
__global__ void k4_dequantize_kernel(const unsigned char* payload, const float* scales, const void* salient,
                                     const void* donors, int descriptor_i32, const float* padding, int tokens,
                                     int channels, int count, T* out, int rows_inner, long long out_so, long long out_si) {
  extern __shared__ __align__(16) unsigned char raw[];
  int* role = (int*)raw;  // >=0 partner slot of a salient channel, -1 normal, <=-2 donor
  float* scale = (float*)(role + channels);
  float* pad = scale + channels;
  const long long row = blockIdx.x;
  for (int c = threadIdx.x; c < channels; c += blockDim.x) {
    role[c] = -1;
    scale[c] = scales[row * channels + c];
    pad[c] = 0.f;
  }
  __syncthreads();
  for (int i = threadIdx.x; i < count; i += blockDim.x) {
    int s = descriptor_i32 ? ((const int*)salient)[row * count + i] : ((const unsigned char*)salient)[row * count + i];
    int d = descriptor_i32 ? ((const int*)donors)[row * count + i] : ((const unsigned char*)donors)[row * count + i];
    role[s] = d;
    role[d] = -2 - i;
    pad[d] = padding[row * count + i];
  }
  __syncthreads();
  const unsigned char* bytes = payload + row * (long long)tokens * (channels / 2);
  // row (outer, inner) lands at out + outer * out_so + inner * out_si (elements); its tokens are contiguous
  T* dst = out + (row / rows_inner) * out_so + (row % rows_inner) * out_si;
  const int t_begin = blockIdx.y * 16, t_end = min(tokens, t_begin + 16);
  for (int idx = t_begin * channels + threadIdx.x; idx < t_end * channels; idx += blockDim.x) {
    int t = idx / channels, c = idx % channels;
    const unsigned char* line = bytes + (long long)t * (channels / 2);
    int slot = (line[c >> 1] >> ((c & 1) * 4)) & 15;
    int r = role[c];
    float value;
    if (r >= 0) {
      int partner = (line[r >> 1] >> ((r & 1) * 4)) & 15;
      value = (float)(((slot << 4) | partner) - 128) * scale[c];
    } else if (r == -1) {
      value = (float)(slot - 8) * scale[c];
    } else {
      value = pad[c];
    }
    dst[idx] = from_float<T>(value);
  }
}

// ------------------------------------------------------------------------------------------
struct VParams {
  InputRef in;
  int bits, group;
  FieldRef payload, scales, offsets;
  int* status;
};

// One warp per token row; a lane owns channels / 32 consecutive channels.
template <typename T, int CPL>
__global__ void __launch_bounds__(256) v_encode_kernel(VParams p) {
  const int warps_per_block = blockDim.x / 32, warp = threadIdx.x / 32, lane = threadIdx.x % 32;
  const long long outer = blockIdx.x / p.in.n_inner, inner = blockIdx.x % p.in.n_inner;
  const long long slot = p.in.slot(outer);
  if (!p.in.slot_ok(slot)) {   // uniform over the CTA: nothing of this row is written
    if (threadIdx.x == 0) atomicOr(p.status, INQ_STATUS_BAD_INDEX);
    return;
  }
  const int t = blockIdx.y * warps_per_block + warp;
  if (t >= p.in.tokens) return;
  const int C = p.in.channels, groups = C / p.group;
  const T* src = (const T*)p.in.x + outer * p.in.s_outer + inner * p.in.s_inner + (long long)t * p.in.s_token + lane * CPL;
  float v[CPL];
#pragma unroll
  for (int j = 0; j < CPL; ++j) v[j] = to_float<T>(src[j]);
  float lo = v[0], hi = v[0];
  bool finite = true;
#pragma unroll
  for (int j = 0; j < CPL; ++j) {
    lo = fminf(lo, v[j]);
    hi = fmaxf(hi, v[j]);
    finite = finite && finite_f32(v[j]);
  }
  const int lanes_per_group = p.group / CPL;
  for (int off = 1; off < lanes_per_group; off <<= 1) {
    lo = fminf(lo, __shfl_xor_sync(0xffffffffu, lo, off));
    hi = fmaxf(hi, __shfl_xor_sync(0xffffffffu, hi, off));
  }
  const float levels = (float)((1 << p.bits) - 1);
  __half offset16 = __float2half_rn(lo);
  __half scale16 = __float2half_rn(fmaxf((hi - lo) / levels, 6.103515625e-05f));
  float offset = __half2float(offset16), scale = __half2float(scale16);
  finite = finite && finite_f32(offset) && finite_f32(scale);
  if (!finite) atomicOr(p.status, INQ_STATUS_NONFINITE);
  const int g = lane / lanes_per_group;
  if (lane % lanes_per_group == 0) {
    ((__half*)p.scales.at(slot, inner))[(long long)t * groups + g] = scale16;
    ((__half*)p.offsets.at(slot, inner))[(long long)t * groups + g] = offset16;
  }
  // Pack this lane's codes, then OR together the lanes that share a 32-bit word.
  const int bits = p.bits, lane_bits = CPL * bits;
  unsigned char* dst = (unsigned char*)p.payload.at(slot, inner) + (long long)t * (C * bits / 8);
  if (lane_bits >= 32) {
    constexpr int kWords = (CPL * 4 + 31) / 32;  // upper bound for bits = 4
    unsigned words[kWords];
#pragma unroll
    for (int w = 0; w < kWords; ++w) words[w] = 0u;
#pragma unroll
    for (int j = 0; j < CPL; ++j) {
      unsigned code = (unsigned)(int)fminf(fmaxf(rintf((v[j] - offset) / scale), 0.f), levels);
      words[(j * bits) >> 5] |= code << ((j * bits) & 31);
    }
    const int n_words = lane_bits / 32;
    for (int w = 0; w < n_words; ++w) ((unsigned*)dst)[lane * n_words + w] = words[w];
  } else {
    unsigned word = 0u;
    const int lanes_per_word = 32 / lane_bits;
#pragma unroll
    for (int j = 0; j < CPL; ++j) {
      unsigned code = (unsigned)(int)fminf(fmaxf(rintf((v[j] - offset) / scale), 0.f), levels);
      word |= code << (((lane % lanes_per_word) * CPL + j) * bits);
    }
    for (int off = 1; off < lanes_per_word; off <<= 1) word |= __shfl_xor_sync(0xffffffffu, word, off);
    if (lane % lanes_per_word == 0) ((unsigned*)dst)[lane / lanes_per_word] = word;
  }
}

// 128-channel fast path of the value encoder: a warp owns 8 consecutive tokens, issues all its
// loads first (2 KB in flight per warp), then quantises two tokens at a time.  A lane owns 8 channels, so
// a group of 64 is reduced in registers and by three shuffles per bound, for two tokens at once.  The kernel
// is bound by issue: with 4 channels per lane and one token per warp 496 rows of 256 tokens took 25.4
// instead of 18.5 us (37.6 MB moved: 5.7 us at the measured 6557 GB/s).
template <typename T, int BITS, int GROUP>
__global__ void __launch_bounds__(256) v_encode128_kernel(VParams p) {
  constexpr int kRows = 8;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, i = lane & 15;
  const long long outer = blockIdx.x / p.in.n_inner, inner = blockIdx.x % p.in.n_inner;
  const long long slot = p.in.slot(outer);
  if (!p.in.slot_ok(slot)) {   // uniform over the CTA: nothing of this row is written
    if (threadIdx.x == 0) atomicOr(p.status, INQ_STATUS_BAD_INDEX);
    return;
  }
  const int t0 = (blockIdx.y * 8 + warp) * kRows;
  if (t0 >= p.in.tokens) return;
  const T* base = (const T*)p.in.x + outer * p.in.s_outer + inner * p.in.s_inner + i * 8;
  constexpr int kVec = sizeof(T) == 2 ? 1 : 2;   // 16-byte vectors per 8 channels
  uint4 raw[kRows / 2][kVec];
#pragma unroll
  for (int k = 0; k < kRows / 2; ++k) {
    const int t = min(t0 + 2 * k + (lane >> 4), p.in.tokens - 1);
#pragma unroll
    for (int q = 0; q < kVec; ++q) raw[k][q] = ((const uint4*)(base + (long long)t * p.in.s_token))[q];
  }
  constexpr int lanes_per_group = GROUP / 8, groups = 128 / GROUP, bits = BITS;
  constexpr float levels = (float)((1 << BITS) - 1);
  unsigned nonfinite = 0u;
  unsigned char* payload = (unsigned char*)p.payload.at(slot, inner);
  __half* scales = (__half*)p.scales.at(slot, inner);
  __half* offsets = (__half*)p.offsets.at(slot, inner);
#pragma unroll
  for (int k = 0; k < kRows / 2; ++k) {
    const int t = t0 + 2 * k + (lane >> 4);
    const bool live = t < p.in.tokens;   // (a lane past the end repeats the last token and stores nothing)
    const T* hv = (const T*)raw[k];
    float v[8];
    unsigned top = 0u;
#pragma unroll
    for (int j = 0; j < 8; ++j) {
      v[j] = to_float<T>(hv[j]);
      top = max(top, __float_as_uint(v[j]) & 0x7fffffffu);
    }
    float lo = fminf(fminf(fminf(v[0], v[1]), fminf(v[2], v[3])), fminf(fminf(v[4], v[5]), fminf(v[6], v[7])));
    float hi = fmaxf(fmaxf(fmaxf(v[0], v[1]), fmaxf(v[2], v[3])), fmaxf(fmaxf(v[4], v[5]), fmaxf(v[6], v[7])));
#pragma unroll
    for (int off = 1; off < lanes_per_group; off <<= 1) {
      lo = fminf(lo, __shfl_xor_sync(0xffffffffu, lo, off));
      hi = fmaxf(hi, __shfl_xor_sync(0xffffffffu, hi, off));
    }
    const __half offset16 = __float2half_rn(lo);
    const __half scale16 = __float2half_rn(fmaxf((hi - lo) / levels, 6.103515625e-05f));
    const float offset = __half2float(offset16), scale = __half2float(scale16);
    top = max(top, max(__float_as_uint(offset) & 0x7fffffffu, __float_as_uint(scale) & 0x7fffffffu));
    nonfinite |= top >= 0x7f800000u;
    if (live && i % lanes_per_group == 0) {
      const int g = i / lanes_per_group;
      scales[(long long)t * groups + g] = scale16;
      offsets[(long long)t * groups + g] = offset16;
    }
    // stored scales are >= 2^-14, so the fused-correction quotient is the IEEE quotient
    const float rcp = __frcp_rn(scale);
    unsigned word = 0u;
#pragma unroll
    for (int j = 0; j < 8; ++j) {
      const float q = exact_quotient(v[j] - offset, scale, rcp, false);
      // rounded to a whole code by the addition (1.5 * 2^23), which leaves it in the low bits
      const unsigned code = __float_as_uint(fminf(fmaxf(q, 0.f), levels) + 12582912.f);
      word |= (code & ((1u << bits) - 1u)) << (j * bits);
    }
    if (bits == 2) {
      // 16 bits per lane, two lanes per 32-bit word
      word |= __shfl_xor_sync(0xffffffffu, word, 1) << 16;
      if (live && (lane & 1) == 0) ((unsigned*)(payload + (long long)t * 32))[i >> 1] = word;
    } else if (live) {
      ((unsigned*)(payload + (long long)t * 64))[i] = word;
    }
  }
  if (nonfinite) atomicOr(p.status, INQ_STATUS_NONFINITE);
}

template <typename T>
__global__ void v_dequantize_kernel(const unsigned char* payload, const __half* scales, const __half* offsets,
                                    long long total, int channels, int bits, int group, T* out, int tokens, int rows_inner,
                                    long long out_so, long long out_si) {
  long long idx = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (idx >= total) return;
  long long token = idx / channels;
  int c = (int)(idx % channels);
  int per_byte = 8 / bits;
  unsigned byte = payload[token * (channels / per_byte) + c / per_byte];
  float code = (float)((byte >> ((c % per_byte) * bits)) & ((1u << bits) - 1u));
  long long param = token * (channels / group) + c / group;
  float value = code * __half2float(scales[param]);
  value = value + __half2float(offsets[param]);
  // row (outer, inner) lands at out + outer * out_so + inner * out_si (elements); its tokens are contiguous
  const long long row = token / tokens;
  out[(row / rows_inner) * out_so + (row % rows_inner) * out_si + (token % tokens) * channels + c] = from_float<T>(value);
}

// 128 channels, 16-bit output: a thread owns 8 consecutive channels of one token (they share a group)
template <typename T, int BITS>
__global__ void __launch_bounds__(256) v_dequantize128_kernel(const unsigned char* payload, const __half* scales, const __half* offsets,
                                                              long long total_tokens, int tokens, int group, T* out, int rows_inner,
                                                              long long out_so, long long out_si) {
  const long long item = (long long)blockIdx.x * blockDim.x + threadIdx.x;   // (token, chunk of 8 channels)
  const long long token = item >> 4;
  if (token >= total_tokens) return;
  const int c0 = (int)(item & 15) * 8;
  constexpr int kBytes = BITS;   // 8 channels x BITS bits
  const unsigned char* src = payload + token * (128 * BITS / 8) + (c0 * BITS / 8);
  unsigned word = 0;
#pragma unroll
  for (int b = 0; b < kBytes; ++b) word |= (unsigned)src[b] << (8 * b);
  const int groups = 128 / group;
  const long long param = token * groups + c0 / group;
  const float sc = __half2float(scales[param]), of = __half2float(offsets[param]);
  T vals[8];
#pragma unroll
  for (int k = 0; k < 8; ++k) {
    const float code = (float)((word >> (BITS * k)) & ((1u << BITS) - 1u));
    float value = code * sc;
    value = value + of;
    vals[k] = from_float<T>(value);
  }
  const long long row = token / tokens;
  T* dst = out + (row / rows_inner) * out_so + (row % rows_inner) * out_si + (token % tokens) * 128 + c0;
  *(uint4*)dst = *(const uint4*)vals;
}

// ------------------------------------------------------------------------------------------
// A cached layer back into its dense history in ONE launch: every sealed block's keys and values, and the rows
// that are dense already (sink, tail, the new states of an update).  A CTA takes one (block, head) row and up to
// kRestoreTokens of its tokens, or a piece of the dense copies.
//
// Coded rows: 16 lanes own a token, 8 channels each.  All channels are first decoded as regular ones and laid as
// a row into shared memory; then one lane per salient channel fetches its two nibbles from the lanes that hold
// them, writes the exact value over its source channel and the donor's constant over the donor slot, and the row
// leaves in 16-byte stores -- instead of every slot of every lane testing for a salient channel, with a shuffle
// and a selection each.  The words of four steps are requested before the first is used: with one step ahead a
// warp waited for memory sixteen times per 256-token row.  In place of two dequantisers, four or six dense copies
// and the concatenation with the new states: 32000 tokens and 700 more through the cache 497 -> 330 us, a prompt
// of 32768 tokens in chunks of 2048 on one layer 9.82 -> 8.68 ms.
constexpr int kRestoreTokens = 64;
constexpr int kRestoreRuns = 8;     // runs of one launch
constexpr long long kRestoreCtas = 1ll << 30;   // fewer of one launch decode

// the blocks of one encoder launch: contiguous fields [block][head]...
struct RestoreRun {
  const unsigned char* key_payload;
  const float* key_scales;
  const unsigned char* key_salient;
  const unsigned char* key_donors;
  const float* key_padding;
  const unsigned char* value_payload;
  const void* value_scales;           // fp16 per token and group, or fp32 per channel (coded values)
  const __half* value_offsets;
  const unsigned char* value_salient;
  const unsigned char* value_donors;
  const float* value_padding;
  long long n_blocks;
};

struct RestoreParams {
  RestoreRun run[kRestoreRuns];
  long long run_end[kRestoreRuns];    // blocks of this run and the ones before it
  const long long* table;             // instead of runs: 6 pointers per block and an int8 role map
  const signed char* roles;
  int n_runs, heads, tokens, parts;   // parts: CTAs per (block, head) row
  int count, value_count, value_group;
  void* out_k;
  void* out_v;
  long long stride_h, position, row_ctas;   // strides in elements; row_ctas: CTAs that decode
  const uint4* copy_src[6];
  uint4* copy_dst[6];
  long long copy_src_h[6], copy_src_t[6], copy_dst_h[6], copy_dst_t[6], copy_end[6];   // 16-byte units; copy_end: vectors up to here
  int copy_tokens[6];
  int n_copies;
};

// One side (keys, or values coded like them) of a (block, head) row as a lane sees it.
struct CodedRow {
  const unsigned char* payload;
  float scale[8];                     // of the lane's channels
  int source, donor;                  // the lane's own salient channel (the first 16; further ones are looked up)
  float source_scale, constant;
  const float* scales;
  const unsigned char* salient;
  const unsigned char* donors;
  const float* padding;
  int count;

  __device__ __forceinline__ void entry(int i, int& s, int& d, float& sc, float& pad) const {
    s = d = 0;
    sc = pad = 0.f;
    if (i < count) {
      s = salient[i] & 127;
      d = donors[i] & 127;
      sc = scales[s];
      pad = padding[i];
    }
  }
  __device__ __forceinline__ void load(int lane) {
    const int c0 = (lane & 15) * 8;
    if (((unsigned long long)scales & 15ull) == 0) {
      const float4 a = *(const float4*)(scales + c0), b = *(const float4*)(scales + c0 + 4);
      scale[0] = a.x; scale[1] = a.y; scale[2] = a.z; scale[3] = a.w;
      scale[4] = b.x; scale[5] = b.y; scale[6] = b.z; scale[7] = b.w;
    } else {
#pragma unroll
      for (int k = 0; k < 8; ++k) scale[k] = scales[c0 + k];
    }
    entry(lane & 15, source, donor, source_scale, constant);
  }
  template <typename T>
  __device__ __forceinline__ uint4 decode(unsigned word, T* row, int lane) const {
    uint4 packed;
    T* const vals = (T*)&packed;
#pragma unroll
    for (int k = 0; k < 8; ++k) {
      // a whole number below 2^23 becomes a float by its bits under those of 2^23: nibble - 8
      const float code = __uint_as_float(0x4B000000u | ((word >> (4 * k)) & 15u)) - 8388616.f;
      vals[k] = from_float<T>(code * scale[k]);
    }
    if (count == 0) return packed;
    row += (lane & 16) * 8;             // the lower 16 lanes' token, the upper ones'
    *(uint4*)(row + (lane & 15) * 8) = packed;
    __syncwarp();
    for (int first = 0; first < count; first += 16) {
      int s = source, d = donor;
      float sc = source_scale, pad = constant;
      if (first) entry(first + (lane & 15), s, d, sc, pad);
      const unsigned hi = __shfl_sync(0xffffffffu, word, (lane & 16) | (s >> 3)), lo = __shfl_sync(0xffffffffu, word, (lane & 16) | (d >> 3));
      const unsigned both = ((hi >> (4 * (s & 7))) & 15u) << 4 | ((lo >> (4 * (d & 7))) & 15u);
      if (first + (lane & 15) < count) {
        row[s] = from_float<T>((__uint_as_float(0x4B000000u | both) - 8388736.f) * sc);   // code - 128
        row[d] = from_float<T>(pad);
      }
    }
    __syncwarp();
    return *(const uint4*)(row + (lane & 15) * 8);
  }
};

// VK: 0 values of 2 bits, 1 coded like the keys, 2 of 4 bits; TABLE: blocks addressed through the decode descriptors
template <typename T, int VK, bool TABLE>
__global__ void __launch_bounds__(256) restore_kernel(const RestoreParams p) {
  if ((long long)blockIdx.x >= p.row_ctas) {
    // dense rows
    const long long total = p.copy_end[p.n_copies - 1];
    long long i = ((long long)blockIdx.x - p.row_ctas) * 1024 + threadIdx.x;
#pragma unroll
    for (int u = 0; u < 4; ++u, i += 256) {
      if (i >= total) break;
      int which = 0;
      while (i >= p.copy_end[which]) ++which;
      const long long at = i - (which ? p.copy_end[which - 1] : 0);
      const int v = (int)(at & 15);
      const int t = (int)((at >> 4) % p.copy_tokens[which]), h = (int)((at >> 4) / p.copy_tokens[which]);
      p.copy_dst[which][h * p.copy_dst_h[which] + t * p.copy_dst_t[which] + v] = p.copy_src[which][h * p.copy_src_h[which] + t * p.copy_src_t[which] + v];
    }
    return;
  }
  __shared__ __align__(16) T rows[8][2][2 * 128];     // per warp, in turn: two tokens
  __shared__ unsigned char s_salient[TABLE ? 64 : 1], s_donors[TABLE ? 64 : 1];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int part = (int)(blockIdx.x % p.parts);
  const long long row = blockIdx.x / p.parts, block = row / p.heads;
  const int h = (int)(row % p.heads), tokens = p.tokens;
  constexpr int kValueRow = VK == 0 ? 32 : 64;
  CodedRow key, coded;
  const unsigned char* values;
  const __half* vs = nullptr;
  const __half* vo = nullptr;
  const int groups = VK == 1 ? 1 : 128 / p.value_group;
  if constexpr (TABLE) {
    const long long* entry = p.table + block * 6;
    key.payload = (const unsigned char*)entry[0] + (long long)h * tokens * 64;
    key.scales = (const float*)entry[1] + h * 128;
    key.padding = (const float*)entry[2] + h * p.count;
    values = (const unsigned char*)entry[3] + (long long)h * tokens * kValueRow;
    vs = (const __half*)entry[4] + (long long)h * tokens * groups;
    vo = (const __half*)entry[5] + (long long)h * tokens * groups;
    const signed char* roles = p.roles + (block * p.heads + h) * 128;
    if (threadIdx.x < 64) s_salient[threadIdx.x] = s_donors[threadIdx.x] = 0;
    __syncthreads();
    if (threadIdx.x < 128) {
      const int d = roles[threadIdx.x];
      if (d >= 0) {
        const int i = -(int)roles[d] - 2;
        if (i >= 0 && i < p.count) {
          s_salient[i] = (unsigned char)threadIdx.x;
          s_donors[i] = (unsigned char)d;
        }
      }
    }
    __syncthreads();
    key.salient = s_salient;
    key.donors = s_donors;
  } else {
    int r = 0;
    while (block >= p.run_end[r]) ++r;
    const RestoreRun& run = p.run[r];
    const long long at = (block - (r ? p.run_end[r - 1] : 0)) * p.heads + h;
    key.payload = run.key_payload + at * tokens * 64;
    key.scales = run.key_scales + at * 128;
    key.salient = run.key_salient + at * p.count;
    key.donors = run.key_donors + at * p.count;
    key.padding = run.key_padding + at * p.count;
    values = run.value_payload + at * tokens * kValueRow;
    if constexpr (VK == 1) {
      coded.payload = values;
      coded.scales = (const float*)run.value_scales + at * 128;
      coded.salient = run.value_salient + at * p.value_count;
      coded.donors = run.value_donors + at * p.value_count;
      coded.padding = run.value_padding + at * p.value_count;
      coded.count = p.value_count;
    } else {
      vs = (const __half*)run.value_scales + at * tokens * groups;
      vo = run.value_offsets + at * tokens * groups;
    }
  }
  key.count = p.count;
  constexpr int kSteps = 4;                       // steps requested at once
  const int c0 = (lane & 15) * 8, group = VK == 1 ? 0 : c0 / p.value_group;
  const int t_end = min(tokens, (part + 1) * kRestoreTokens);
  const int first = part * kRestoreTokens + 2 * warp + (lane >> 4);   // this lane's token of step u: first + 16 u
  unsigned kw[kSteps], vw[kSteps];
  __half sc[kSteps], of[kSteps];
#pragma unroll
  for (int u = 0; u < kSteps; ++u) {
    const int t = min(first + 16 * u, t_end - 1);   // (whole warps walk; past the end the last token is decoded again and not stored)
    kw[u] = __ldg((const unsigned*)(key.payload + (long long)t * 64 + (c0 >> 1)));
    if constexpr (VK == 0) vw[u] = __ldg((const unsigned short*)(values + (long long)t * 32 + (c0 >> 2)));
    else vw[u] = __ldg((const unsigned*)(values + (long long)t * 64 + (c0 >> 1)));
    if constexpr (VK != 1) {
      sc[u] = __ldg(vs + t * groups + group);
      of[u] = __ldg(vo + t * groups + group);
    }
  }
  key.load(lane);
  if constexpr (VK == 1) coded.load(lane);
  const long long base = (long long)h * p.stride_h + (p.position + block * tokens) * 128 + c0;
#pragma unroll
  for (int u = 0; u < kSteps; ++u) {
    if (part * kRestoreTokens + 2 * warp + 16 * u >= t_end) break;   // uniform in the warp
    const int t = first + 16 * u;
    const uint4 k = key.decode<T>(kw[u], rows[warp][0], lane);
    uint4 v;
    if constexpr (VK == 1) {
      v = coded.decode<T>(vw[u], rows[warp][1], lane);
    } else {
      const float vsc = __half2float(sc[u]), vof = __half2float(of[u]);
      constexpr int kBits = VK == 0 ? 2 : 4;
#pragma unroll
      for (int c = 0; c < 8; ++c) {
        float value = (__uint_as_float(0x4B000000u | ((vw[u] >> (kBits * c)) & ((1u << kBits) - 1u))) - 8388608.f) * vsc;
        value = value + vof;
        ((T*)&v)[c] = from_float<T>(value);
      }
    }
    if (t < t_end) {
      *(uint4*)((T*)p.out_k + base + (long long)t * 128) = k;
      *(uint4*)((T*)p.out_v + base + (long long)t * 128) = v;
    }
    __syncwarp();   // the rows are free again
  }
}

template <bool TABLE>
static void launch_restore(const RestoreParams& p, int value_kind, bool half, long long copy_vectors, cudaStream_t stream) {
  const unsigned grid = (unsigned)(p.row_ctas + (copy_vectors + 1023) / 1024);
  if (value_kind == 0) {
    if (half) restore_kernel<__half, 0, TABLE><<<grid, 256, 0, stream>>>(p);
    else restore_kernel<__nv_bfloat16, 0, TABLE><<<grid, 256, 0, stream>>>(p);
  }
  if constexpr (!TABLE) {
    if (value_kind == 1) {
      if (half) restore_kernel<__half, 1, false><<<grid, 256, 0, stream>>>(p);
      else restore_kernel<__nv_bfloat16, 1, false><<<grid, 256, 0, stream>>>(p);
    } else if (value_kind == 2) {
      if (half) restore_kernel<__half, 2, false><<<grid, 256, 0, stream>>>(p);
      else restore_kernel<__nv_bfloat16, 2, false><<<grid, 256, 0, stream>>>(p);
    }
  }
}

__global__ void build_roles_kernel(const void* salient, const void* donors, int descriptor_i32, int channels, int count,
                                   void* roles, int role_bytes) {
  const long long row = blockIdx.x;
  for (int c = threadIdx.x; c < channels; c += blockDim.x) {
    int role = -1;
    for (int i = 0; i < count; ++i) {
      int s = descriptor_i32 ? ((const int*)salient)[row * count + i] : ((const unsigned char*)salient)[row * count + i];
      int d = descriptor_i32 ? ((const int*)donors)[row * count + i] : ((const unsigned char*)donors)[row * count + i];
      if (s == c) role = d;
      if (d == c) role = -2 - i;
    }
    if (role_bytes == 1)
      ((signed char*)roles)[row * channels + c] = (signed char)role;
    else
      ((short*)roles)[row * channels + c] = (short)role;
  }
}

// ------------------------------------------------------------------------------------------
static bool input_ok(const inq_input_t& in) {
  return in.x && valid_dtype(in.dtype) && in.n_outer >= 1 && in.n_inner >= 1 && in.tokens >= 1 && in.channels >= 1 &&
         in.n_outer * in.n_inner < (1ll << 31);
}

static bool rows_vectorizable(const inq_input_t& in) {
  long long es = dtype_size(in.dtype);
  return in.channels % 8 == 0 && ((uintptr_t)in.x % 16 == 0) && (in.stride_outer * es) % 16 == 0 &&
         (in.stride_inner * es) % 16 == 0 && (in.stride_token * es) % 16 == 0;
}

}  // namespace inq

using namespace inq;

extern "C" int inq_k4_encode(const inq_k4_encode_args_t* a, int32_t* status, inq_stream_t stream_) {
  if (!a || !status || !input_ok(a->in)) return INQ_ERR_ARGUMENT;
  const int C = a->in.channels;
  if (C % 2 || a->count < 0 || a->count > C / 2 || a->sample_stride < 1) return INQ_ERR_ARGUMENT;
  if (C > kMaxChannels) return INQ_ERR_UNSUPPORTED;
  if (!a->payload.base || !a->scales.base || (a->count && !a->padding.base)) return INQ_ERR_ARGUMENT;
  if ((a->salient.base == nullptr) != (a->donors.base == nullptr)) return INQ_ERR_ARGUMENT;
  if (a->roles.base && a->role_bytes != 1 && a->role_bytes != 2) return INQ_ERR_ARGUMENT;
  if (!a->descriptor_i32 && C > 256 && a->salient.base) return INQ_ERR_ARGUMENT;
  K4Params p;
  p.in = make_input(a->in);
  p.sample_stride = a->sample_stride;
  p.count = a->count;
  p.min_error = a->min_error;
  p.payload = make_field(a->payload);
  p.scales = make_field(a->scales);
  p.salient = make_field(a->salient);
  p.donors = make_field(a->donors);
  p.padding = make_field(a->padding);
  p.roles = make_field(a->roles);
  p.descriptor_i32 = a->descriptor_i32;
  p.role_bytes = a->role_bytes;
  p.status = status;
  // 4-byte payload stores need 4-byte aligned rows; the payload row is C/2 bytes.
  p.vector_path = rows_vectorizable(a->in) && ((uintptr_t)a->payload.base % 4 == 0) && a->payload.outer_stride % 4 == 0 &&
                  a->payload.inner_stride % 4 == 0;
  cudaStream_t stream = (cudaStream_t)stream_;
  int threads = ((C + 31) / 32) * 32;
  if (threads < 128 && C % 8 == 0) threads = 128;  // more tokens in flight while packing narrow rows
  size_t shared = k4_shared_bytes(C, a->count, a->in.tokens, a->min_error != 0);
  unsigned grid = (unsigned)(a->in.n_outer * a->in.n_inner);
  if (C == 128 && p.vector_path && a->in.tokens <= kRcpTable && !a->descriptor_i32) {
    const bool regular = a->in.tokens % 8 == 0 && a->sample_stride == 8;
    // whole rows contiguous in memory, in groups of 32 tokens: the shared-memory ring variant
    const bool staged = regular && a->in.tokens % 32 == 0 && a->in.stride_token == C;
    switch (a->in.dtype) {
      case INQ_F32:
        if (regular) k4_encode128_kernel<float, true><<<grid, 128, 0, stream>>>(p);
        else k4_encode128_kernel<float, false><<<grid, 128, 0, stream>>>(p);
        break;
      case INQ_F16:
        if (staged) k4_encode128_kernel<__half, true, true><<<grid, 128, 0, stream>>>(p);
        else if (regular) k4_encode128_kernel<__half, true><<<grid, 128, 0, stream>>>(p);
        else k4_encode128_kernel<__half, false><<<grid, 128, 0, stream>>>(p);
        break;
      default:
        if (staged) k4_encode128_kernel<__nv_bfloat16, true, true><<<grid, 128, 0, stream>>>(p);
        else if (regular) k4_encode128_kernel<__nv_bfloat16, true><<<grid, 128, 0, stream>>>(p);
        else k4_encode128_kernel<__nv_bfloat16, false><<<grid, 128, 0, stream>>>(p);
        break;
    }
  } else if (threads <= 256) {
    switch (a->in.dtype) {
      case INQ_F32: k4_encode_kernel<float, 256><<<grid, threads, shared, stream>>>(p); break;
      case INQ_F16: k4_encode_kernel<__half, 256><<<grid, threads, shared, stream>>>(p); break;
      default: k4_encode_kernel<__nv_bfloat16, 256><<<grid, threads, shared, stream>>>(p); break;
    }
  } else {
    switch (a->in.dtype) {
      case INQ_F32: k4_encode_kernel<float, 1024><<<grid, threads, shared, stream>>>(p); break;
      case INQ_F16: k4_encode_kernel<__half, 1024><<<grid, threads, shared, stream>>>(p); break;
      default: k4_encode_kernel<__nv_bfloat16, 1024><<<grid, threads, shared, stream>>>(p); break;
    }
  }
  INQ_CUDA_CHECK(cudaGetLastError());
  return INQ_OK;
}

extern "C" int inq_k4_statistics(const inq_input_t* in, int32_t sample_stride, float* saliency, float* sampled_mean,
                                 float* donor_error, float* absmax, inq_stream_t stream_) {
  if (!in || !input_ok(*in) || sample_stride < 1) return INQ_ERR_ARGUMENT;
  if (in->channels > kMaxChannels) return INQ_ERR_UNSUPPORTED;
  InputRef ref = make_input(*in);
  cudaStream_t stream = (cudaStream_t)stream_;
  int threads = ((in->channels + 31) / 32) * 32;
  size_t shared = (donor_error && in->tokens <= kRcpTable) ? (size_t)in->tokens * 8 : 0;
  unsigned grid = (unsigned)(in->n_outer * in->n_inner);
  switch (in->dtype) {
    case INQ_F32:
      k4_statistics_kernel<float><<<grid, threads, shared, stream>>>(ref, sample_stride, saliency, sampled_mean, donor_error, absmax);
      break;
    case INQ_F16:
      k4_statistics_kernel<__half><<<grid, threads, shared, stream>>>(ref, sample_stride, saliency, sampled_mean, donor_error, absmax);
      break;
    default:
      k4_statistics_kernel<__nv_bfloat16><<<grid, threads, shared, stream>>>(ref, sample_stride, saliency, sampled_mean, donor_error, absmax);
      break;
  }
  INQ_CUDA_CHECK(cudaGetLastError());
  return INQ_OK;
}

extern "C" int inq_select_donors(const float* saliency, const float* donor_error, int64_t rows, int32_t channels,
                                 int32_t count, int64_t* sources, int64_t* donors, inq_stream_t stream_) {
  if (!saliency || rows < 0 || channels < 1 || count < 0 || count > channels / 2 || rows >= (1ll << 31)) return INQ_ERR_ARGUMENT;
  if (channels > kMaxChannels) return INQ_ERR_UNSUPPORTED;
  if (rows == 0 || count == 0) return INQ_OK;
  if (!sources || !donors) return INQ_ERR_ARGUMENT;
  int threads = ((channels + 31) / 32) * 32;
  size_t shared = (size_t)channels * 12 + kMaxWords * 8 + (size_t)count * 8;
  select_kernel<<<(unsigned)rows, threads, shared, (cudaStream_t)stream_>>>(saliency, donor_error, channels, count,
                                                                             (long long*)sources, (long long*)donors);
  INQ_CUDA_CHECK(cudaGetLastError());
  return INQ_OK;
}

extern "C" int inq_k4_dequantize_strided(const uint8_t* payload, const float* scales, const void* salient, const void* donors,
                                         int32_t descriptor_i32, const float* padding, int64_t rows_outer, int32_t rows_inner,
                                         int32_t tokens, int32_t channels, int32_t count, void* out, int64_t out_stride_outer,
                                         int64_t out_stride_inner, int32_t out_dtype, inq_stream_t stream_) {
  const long long rows = rows_outer * (long long)rows_inner;
  if (!payload || !scales || !out || rows_outer < 1 || rows_inner < 1 || tokens < 1 || channels < 2 || channels % 2 || count < 0 ||
      !valid_dtype(out_dtype) || rows >= (1ll << 31) || out_stride_outer < 0 || out_stride_inner < 0)
    return INQ_ERR_ARGUMENT;
  if (count && (!salient || !donors || !padding)) return INQ_ERR_ARGUMENT;
  if (channels > 4096) return INQ_ERR_UNSUPPORTED;
  cudaStream_t stream = (cudaStream_t)stream_;
  if (channels == 128 && !descriptor_i32 && count <= 64 && out_dtype != INQ_F32 && ((uintptr_t)out % 16) == 0 &&
      out_stride_outer % 8 == 0 && out_stride_inner % 8 == 0 && ((uintptr_t)payload % 4) == 0) {
    // enough CTAs per row to fill the device, at least 64 tokens each
    int split = (int)std::min<long long>((tokens + 63) / 64, std::max<long long>(1, 2048 / rows));
    dim3 fast((unsigned)rows, (unsigned)split);
    if (out_dtype == INQ_F16)
      k4_dequantize128_kernel<__half><<<fast, 256, 0, stream>>>(payload, scales, salient, donors, padding, tokens, count, (__half*)out, rows_inner, out_stride_outer, out_stride_inner);
    else
      k4_dequantize128_kernel<__nv_bfloat16><<<fast, 256, 0, stream>>>(payload, scales, salient, donors, padding, tokens, count, (__nv_bfloat16*)out, rows_inner, out_stride_outer, out_stride_inner);
    INQ_CUDA_CHECK(cudaGetLastError());
    return INQ_OK;
  }
  dim3 grid((unsigned)rows, (unsigned)((tokens + 15) / 16));
  size_t shared = (size_t)channels * 12;
  switch (out_dtype) {
    case INQ_F32:
      k4_dequantize_kernel<float><<<grid, 256, shared, stream>>>(payload, scales, salient, donors, descriptor_i32, padding, tokens, channels, count, (float*)out, rows_inner, out_stride_outer, out_stride_inner);
      break;
    case INQ_F16:
      k4_dequantize_kernel<__half><<<grid, 256, shared, stream>>>(payload, scales, salient, donors, descriptor_i32, padding, tokens, channels, count, (__half*)out, rows_inner, out_stride_outer, out_stride_inner);
      break;
    default:
      k4_dequantize_kernel<__nv_bfloat16><<<grid, 256, shared, stream>>>(payload, scales, salient, donors, descriptor_i32, padding, tokens, channels, count, (__nv_bfloat16*)out, rows_inner, out_stride_outer, out_stride_inner);
      break;
  }
  INQ_CUDA_CHECK(cudaGetLastError());
  return INQ_OK;
}

extern "C" int inq_k4_dequantize(const uint8_t* payload, const float* scales, const void* salient, const void* donors,
                                 int32_t descriptor_i32, const float* padding, int64_t rows, int32_t tokens,
                                 int32_t channels, int32_t count, void* out, int32_t out_dtype, inq_stream_t stream_) {
  return inq_k4_dequantize_strided(payload, scales, salient, donors, descriptor_i32, padding, rows, 1, tokens, channels, count, out,
                                   (int64_t)tokens * channels, 0, out_dtype, stream_);
}

template <typename T>
static int launch_v_encode(const VParams& p, int cpl, dim3 grid, cudaStream_t stream) {
  switch (cpl) {
    case 1: v_encode_kernel<T, 1><<<grid, 256, 0, stream>>>(p); break;
    case 2: v_encode_kernel<T, 2><<<grid, 256, 0, stream>>>(p); break;
    case 4: v_encode_kernel<T, 4><<<grid, 256, 0, stream>>>(p); break;
    case 8: v_encode_kernel<T, 8><<<grid, 256, 0, stream>>>(p); break;
    default: return INQ_ERR_UNSUPPORTED;
  }
  return INQ_OK;
}

extern "C" int inq_v_encode(const inq_v_encode_args_t* a, int32_t* status, inq_stream_t stream_) {
  if (!a || !status || !input_ok(a->in)) return INQ_ERR_ARGUMENT;
  if ((a->bits != 2 && a->bits != 4) || (a->group != 32 && a->group != 64 && a->group != 128)) return INQ_ERR_ARGUMENT;
  const int C = a->in.channels;
  if (C % a->group) return INQ_ERR_ARGUMENT;
  if (!a->payload.base || !a->scales.base || !a->offsets.base) return INQ_ERR_ARGUMENT;
  if (C % 32 || C > 256) return INQ_ERR_UNSUPPORTED;
  VParams p;
  p.in = make_input(a->in);
  p.bits = a->bits;
  p.group = a->group;
  p.payload = make_field(a->payload);
  p.scales = make_field(a->scales);
  p.offsets = make_field(a->offsets);
  p.status = status;
  dim3 grid((unsigned)(a->in.n_outer * a->in.n_inner), (unsigned)((a->in.tokens + 7) / 8));
  cudaStream_t stream = (cudaStream_t)stream_;
  const long long es = dtype_size(a->in.dtype);
  const bool aligned8 = ((uintptr_t)a->in.x % 16 == 0) && (a->in.stride_outer * es) % 16 == 0 &&
                        (a->in.stride_inner * es) % 16 == 0 && (a->in.stride_token * es) % 16 == 0 &&
                        ((uintptr_t)a->payload.base % 4 == 0) && a->payload.outer_stride % 4 == 0 && a->payload.inner_stride % 4 == 0;
  if (C == 128 && aligned8) {
    dim3 fast((unsigned)(a->in.n_outer * a->in.n_inner), (unsigned)((a->in.tokens + 63) / 64));
#define INQ_V128(T)                                                                         \
  if (a->bits == 2) {                                                                       \
    if (a->group == 32) v_encode128_kernel<T, 2, 32><<<fast, 256, 0, stream>>>(p);          \
    else if (a->group == 64) v_encode128_kernel<T, 2, 64><<<fast, 256, 0, stream>>>(p);     \
    else v_encode128_kernel<T, 2, 128><<<fast, 256, 0, stream>>>(p);                        \
  } else {                                                                                  \
    if (a->group == 32) v_encode128_kernel<T, 4, 32><<<fast, 256, 0, stream>>>(p);          \
    else if (a->group == 64) v_encode128_kernel<T, 4, 64><<<fast, 256, 0, stream>>>(p);     \
    else v_encode128_kernel<T, 4, 128><<<fast, 256, 0, stream>>>(p);                        \
  }
    switch (a->in.dtype) {
      case INQ_F32: INQ_V128(float) break;
      case INQ_F16: INQ_V128(__half) break;
      default: INQ_V128(__nv_bfloat16) break;
    }
#undef INQ_V128
    INQ_CUDA_CHECK(cudaGetLastError());
    return INQ_OK;
  }
  int rc;
  switch (a->in.dtype) {
    case INQ_F32: rc = launch_v_encode<float>(p, C / 32, grid, stream); break;
    case INQ_F16: rc = launch_v_encode<__half>(p, C / 32, grid, stream); break;
    default: rc = launch_v_encode<__nv_bfloat16>(p, C / 32, grid, stream); break;
  }
  if (rc != INQ_OK) return rc;
  INQ_CUDA_CHECK(cudaGetLastError());
  return INQ_OK;
}

extern "C" int inq_v_dequantize_strided(const uint8_t* payload, const void* scales, const void* offsets, int64_t rows_outer,
                                        int32_t rows_inner, int32_t tokens, int32_t channels, int32_t bits, int32_t group, void* out,
                                        int64_t out_stride_outer, int64_t out_stride_inner, int32_t out_dtype, inq_stream_t stream_) {
  if (!payload || !scales || !offsets || !out || rows_outer < 1 || rows_inner < 1 || tokens < 1 || (bits != 2 && bits != 4) ||
      (group != 32 && group != 64 && group != 128) || channels % group || !valid_dtype(out_dtype) || out_stride_outer < 0 ||
      out_stride_inner < 0)
    return INQ_ERR_ARGUMENT;
  long long total = rows_outer * (long long)rows_inner * tokens * channels;
  unsigned blocks = (unsigned)((total + 255) / 256);
  cudaStream_t stream = (cudaStream_t)stream_;
  if (channels == 128 && out_dtype != INQ_F32 && ((uintptr_t)out % 16) == 0 && out_stride_outer % 8 == 0 && out_stride_inner % 8 == 0) {
    const long long total_tokens = rows_outer * (long long)rows_inner * tokens;
    const unsigned fast = (unsigned)((total_tokens * 16 + 255) / 256);
    const __half* sc = (const __half*)scales;
    const __half* of = (const __half*)offsets;
    if (out_dtype == INQ_F16 && bits == 2)
      v_dequantize128_kernel<__half, 2><<<fast, 256, 0, stream>>>(payload, sc, of, total_tokens, tokens, group, (__half*)out, rows_inner, out_stride_outer, out_stride_inner);
    else if (out_dtype == INQ_F16)
      v_dequantize128_kernel<__half, 4><<<fast, 256, 0, stream>>>(payload, sc, of, total_tokens, tokens, group, (__half*)out, rows_inner, out_stride_outer, out_stride_inner);
    else if (bits == 2)
      v_dequantize128_kernel<__nv_bfloat16, 2><<<fast, 256, 0, stream>>>(payload, sc, of, total_tokens, tokens, group, (__nv_bfloat16*)out, rows_inner, out_stride_outer, out_stride_inner);
    else
      v_dequantize128_kernel<__nv_bfloat16, 4><<<fast, 256, 0, stream>>>(payload, sc, of, total_tokens, tokens, group, (__nv_bfloat16*)out, rows_inner, out_stride_outer, out_stride_inner);
    INQ_CUDA_CHECK(cudaGetLastError());
    return INQ_OK;
  }
  switch (out_dtype) {
    case INQ_F32:
      v_dequantize_kernel<float><<<blocks, 256, 0, stream>>>(payload, (const __half*)scales, (const __half*)offsets, total, channels, bits, group, (float*)out, tokens, rows_inner, out_stride_outer, out_stride_inner);
      break;
    case INQ_F16:
      v_dequantize_kernel<__half><<<blocks, 256, 0, stream>>>(payload, (const __half*)scales, (const __half*)offsets, total, channels, bits, group, (__half*)out, tokens, rows_inner, out_stride_outer, out_stride_inner);
      break;
    default:
      v_dequantize_kernel<__nv_bfloat16><<<blocks, 256, 0, stream>>>(payload, (const __half*)scales, (const __half*)offsets, total, channels, bits, group, (__nv_bfloat16*)out, tokens, rows_inner, out_stride_outer, out_stride_inner);
      break;
  }
  INQ_CUDA_CHECK(cudaGetLastError());
  return INQ_OK;
}

extern "C" int inq_v_dequantize(const uint8_t* payload, const void* scales, const void* offsets, int64_t rows,
                                int32_t tokens, int32_t channels, int32_t bits, int32_t group, void* out,
                                int32_t out_dtype, inq_stream_t stream_) {
  return inq_v_dequantize_strided(payload, scales, offsets, rows, 1, tokens, channels, bits, group, out,
                                  (int64_t)tokens * channels, 0, out_dtype, stream_);
}

extern "C" int inq_build_roles(const void* salient, const void* donors, int32_t descriptor_i32, int64_t rows,
                               int32_t channels, int32_t count, void* roles, int32_t role_bytes, inq_stream_t stream_) {
  if (!roles || rows < 0 || channels < 1 || count < 0 || (role_bytes != 1 && role_bytes != 2) || rows >= (1ll << 31))
    return INQ_ERR_ARGUMENT;
  if (count && (!salient || !donors)) return INQ_ERR_ARGUMENT;
  if (rows == 0) return INQ_OK;
  build_roles_kernel<<<(unsigned)rows, 128, 0, (cudaStream_t)stream_>>>(salient, donors, descriptor_i32, channels, count, roles, role_bytes);
  INQ_CUDA_CHECK(cudaGetLastError());
  return INQ_OK;
}

extern "C" int inq_restore_blocks_table(const int64_t* table, const int8_t* roles, int32_t n_blocks, int32_t heads, int32_t tokens,
                                        int32_t count, void* out_key, void* out_value, int64_t stride_h, int64_t position,
                                        int32_t out_dtype, inq_stream_t stream_) {
  if (!table || !roles || !out_key || !out_value || n_blocks < 0 || heads < 1 || tokens < 1 || count < 0 || count > 64)
    return INQ_ERR_ARGUMENT;
  if (out_dtype != INQ_F16 && out_dtype != INQ_BF16) return INQ_ERR_UNSUPPORTED;
  if ((((uintptr_t)out_key | (uintptr_t)out_value) & 15) != 0 || stride_h % 8 != 0 || position < 0) return INQ_ERR_ARGUMENT;
  if (n_blocks == 0) return INQ_OK;
  RestoreParams p = {};
  p.table = (const long long*)table;
  p.roles = (const signed char*)roles;
  p.heads = heads;
  p.tokens = tokens;
  p.parts = (tokens + kRestoreTokens - 1) / kRestoreTokens;
  p.count = count;
  p.value_group = 64;
  p.out_k = out_key;
  p.out_v = out_value;
  p.stride_h = stride_h;
  p.position = position;
  p.row_ctas = (long long)n_blocks * heads * p.parts;
  if (p.row_ctas >= (1ll << 31)) return INQ_ERR_UNSUPPORTED;
  launch_restore<true>(p, 0, out_dtype == INQ_F16, 0, (cudaStream_t)stream_);
  INQ_CUDA_CHECK(cudaGetLastError());
  return INQ_OK;
}

extern "C" int inq_restore_history(const inq_restore_args_t* a, inq_stream_t stream_) {
  if (!a || a->n_runs < 0 || (a->n_runs && !a->runs) || a->n_copies < 0 || a->n_copies > 6) return INQ_ERR_ARGUMENT;
  if (a->out_dtype != INQ_F16 && a->out_dtype != INQ_BF16) return INQ_ERR_UNSUPPORTED;
  RestoreParams p = {};
  long long vectors = 0;
  for (int i = 0; i < a->n_copies; ++i) {
    const inq_row_copy_t& r = a->copies[i];
    if (r.tokens < 0) return INQ_ERR_ARGUMENT;
    if (!r.tokens) continue;
    if (a->heads < 1 || !r.src || !r.dst || (uintptr_t)r.src % 16 || (uintptr_t)r.dst % 16) return INQ_ERR_ARGUMENT;
    if (r.src_stride_h % 16 || r.src_stride_t % 16 || r.dst_stride_h % 16 || r.dst_stride_t % 16) return INQ_ERR_ARGUMENT;
    const int n = p.n_copies++;
    p.copy_src[n] = (const uint4*)r.src;
    p.copy_dst[n] = (uint4*)r.dst;
    p.copy_src_h[n] = r.src_stride_h / 16;
    p.copy_src_t[n] = r.src_stride_t / 16;
    p.copy_dst_h[n] = r.dst_stride_h / 16;
    p.copy_dst_t[n] = r.dst_stride_t / 16;
    p.copy_tokens[n] = r.tokens;
    vectors += (long long)a->heads * r.tokens * 16;
    p.copy_end[n] = vectors;
  }
  p.heads = a->heads;
  if (a->n_runs) {
    if (a->heads < 1 || a->block_tokens < 1 || a->count < 0 || a->count > 64 || a->value_count < 0 || a->value_count > 64) return INQ_ERR_ARGUMENT;
    if (!a->out_key || !a->out_value || (((uintptr_t)a->out_key | (uintptr_t)a->out_value) & 15) != 0) return INQ_ERR_ARGUMENT;
    if (a->stride_h % 8 != 0 || a->position < 0) return INQ_ERR_ARGUMENT;
    if (a->value_kind == 0 ? (a->value_bits != 2 && a->value_bits != 4) || (a->value_group != 32 && a->value_group != 64 && a->value_group != 128)
                           : a->value_kind != 1)
      return INQ_ERR_ARGUMENT;
    p.parts = (a->block_tokens + kRestoreTokens - 1) / kRestoreTokens;
    for (int r = 0; r < a->n_runs; ++r) {
      const inq_restore_run_t& run = a->runs[r];
      if (run.n_blocks < 1 || run.n_blocks >= (1ll << 31) || !run.key_payload || !run.key_scales || !run.value_payload || !run.value_scales) return INQ_ERR_ARGUMENT;
      if (a->count && (!run.key_salient || !run.key_donors || !run.key_padding)) return INQ_ERR_ARGUMENT;
      if (a->value_kind == 0 ? !run.value_offsets : a->value_count && (!run.value_salient || !run.value_donors || !run.value_padding)) return INQ_ERR_ARGUMENT;
      if (((uintptr_t)run.key_payload | (uintptr_t)run.value_payload) % 4) return INQ_ERR_ARGUMENT;   // words of 8 nibbles or 2-bit codes
      if (run.n_blocks > (kRestoreCtas - 1) / ((long long)a->heads * p.parts)) return INQ_ERR_UNSUPPORTED;   // a run is part of one launch
    }
    p.tokens = a->block_tokens;
    p.count = a->count;
    p.value_count = a->value_count;
    p.value_group = a->value_group;
    p.out_k = a->out_key;
    p.out_v = a->out_value;
    p.stride_h = a->stride_h;
  } else {
    p.parts = 1;
  }
  cudaStream_t stream = (cudaStream_t)stream_;
  const int kind = a->value_kind == 1 ? 1 : a->value_bits == 4 ? 2 : 0;
  long long position = a->position;
  int next = 0;
  do {   // the runs of a launch travel as kernel parameters; the copies go with the first
    p.n_runs = 0;
    long long blocks = 0;
    while (next < a->n_runs && p.n_runs < kRestoreRuns) {
      const inq_restore_run_t& run = a->runs[next];
      if (p.n_runs && (blocks + run.n_blocks) * a->heads * p.parts >= kRestoreCtas) break;
      RestoreRun& out = p.run[p.n_runs];
      out.key_payload = (const unsigned char*)run.key_payload;
      out.key_scales = (const float*)run.key_scales;
      out.key_salient = (const unsigned char*)run.key_salient;
      out.key_donors = (const unsigned char*)run.key_donors;
      out.key_padding = (const float*)run.key_padding;
      out.value_payload = (const unsigned char*)run.value_payload;
      out.value_scales = run.value_scales;
      out.value_offsets = (const __half*)run.value_offsets;
      out.value_salient = (const unsigned char*)run.value_salient;
      out.value_donors = (const unsigned char*)run.value_donors;
      out.value_padding = (const float*)run.value_padding;
      out.n_blocks = run.n_blocks;
      blocks += run.n_blocks;
      p.run_end[p.n_runs++] = blocks;
      ++next;
    }
    p.position = position;
    p.row_ctas = blocks * a->heads * p.parts;
    if (p.row_ctas + vectors) {
      launch_restore<false>(p, kind, a->out_dtype == INQ_F16, vectors, stream);
      INQ_CUDA_CHECK(cudaGetLastError());
    }
    position += blocks * p.tokens;
    vectors = 0;
    p.n_copies = 0;
  } while (next < a->n_runs);
  return INQ_OK;
}
