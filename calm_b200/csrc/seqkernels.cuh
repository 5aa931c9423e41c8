// seqkernels.cuh -- device code of the layer-list models (include/calm_b200_seq.h): packed batches of tokens from many
// sequences, a paged cache for what is indexed by position and per-slot buffers for what is recurrent.
//
// Precision: the residual stream, every norm, softmax, the convolution state, the recurrent state and everything that
// feeds the recurrence after the projections are fp32.  Products read activations of type AT: float (exact mode, SIMT
// FMA) or bf16 (tensor cores, fp32 accumulation).  Weights are bf16 as stored.
#pragma once

#include <cuda_bf16.h>
#include <type_traits>

#include "common.cuh"
#include "tc05.cuh"

typedef __nv_bfloat16 bf16;

// per-step description of the packed batch (device arrays)
struct SeqBatch {
	const int* tok;      // [N] token ids
	const int* tslot;    // [N] slot of the token's sequence
	const int* tpos;     // [N] position of the token in its sequence
	const int* tfirst;   // [N] packed index of the first token its sequence has in this step
	const int* sstart;   // [B] first packed index of sequence b
	const int* scount;   // [B]
	const int* spos0;    // [B] position of its first new token
	const int* sslot;    // [B]
	const int* pages;    // [slots][max_pages] page table
	int N, B, max_pages, page;
};

__device__ __forceinline__ long cache_row(const SeqBatch& sb, int slot, int pos) {
	return (long)sb.pages[(long)slot * sb.max_pages + pos / sb.page] * sb.page + pos % sb.page;
}

template <typename T>
__device__ __forceinline__ T to_act(float v);
template <>
__device__ __forceinline__ float to_act<float>(float v) {
	return v;
}
template <>
__device__ __forceinline__ bf16 to_act<bf16>(float v) {
	return __float2bfloat16_rn(v);
}
__device__ __forceinline__ float ldf(const bf16* p) { return __bfloat162float(*p); }
__device__ __forceinline__ float ldf(const float* p) { return *p; }

__device__ __forceinline__ float sigmoidf_(float z) { return 1.f / (1.f + expf(-z)); }
__device__ __forceinline__ float softplusf_(float z) { return z > 20.f ? z : log1pf(expf(z)); }
// warp_sum / warp_max: common.cuh

// ---------------------------------------------------------------- embedding, norms, small element-wise kernels

// x[n] = E[tok[n]] * scale (+ P[position of n], a learned position row, not scaled), written to every one of `streams` copies
// (and a second copy when a looped span re-adds the embedding).  With a bigram table, row (previous token * mul_prev + token * mul_cur)
// mod buckets of it is added as well; a sequence's first token (tprev < 0) takes row `buckets`, the table's last.  act given: the row also
// leaves in the activation type (post-norm blocks: the first sublayer's input).
struct EmbedBigram {
	const bf16* table; // (buckets + 1, width) or null
	const int* tprev;  // [N] the token before each packed token in its sequence, -1 for a first token
	int buckets, mul_prev, mul_cur;
};
// V columns per thread and pass (8 where rows allow 16-byte accesses, else 1): a thread's loads are all out before its first store.  One column at a time,
// a pass waited for the one before: 16 rows of 2048 took 12.9 us, now 3.1.
template <typename AT, int V>
__global__ void k_seq_embed(float* x, float* x0, AT* act, const bf16* table, const int* tok, int N, int width, float scale, const bf16* pos_table, const int* tpos, int streams, EmbedBigram bg) {
	pdl_enter(); // programmatic dependent launch: let the next kernel's launch overlap this one, then wait for the previous one
	const int n = blockIdx.x;
	const bf16* e = table + (size_t)tok[n] * width;
	const bf16* pr = pos_table ? pos_table + (size_t)tpos[n] * width : nullptr;
	const bf16* br = nullptr;
	if (bg.table) {
		const int prev = bg.tprev[n];
		const long long row = prev < 0 ? bg.buckets : ((long long)prev * bg.mul_prev + (long long)tok[n] * bg.mul_cur) % bg.buckets;
		br = bg.table + (size_t)row * width;
	}
	for (int i = threadIdx.x * V; i < width; i += blockDim.x * V) {
		float v[V];
		auto read = [&](const bf16* from, auto&& use) {
			if constexpr (V == 8) {
				const uint4 q = __ldg(reinterpret_cast<const uint4*>(from + i));
				const uint32_t w[4] = {q.x, q.y, q.z, q.w};
#pragma unroll
				for (int k = 0; k < 4; ++k) use(2 * k, __uint_as_float(w[k] << 16)), use(2 * k + 1, __uint_as_float(w[k] & 0xffff0000u));
			} else use(0, ldf(from + i));
		};
		read(e, [&](int k, float z) { v[k] = z * scale; });
		if (pr) read(pr, [&](int k, float z) { v[k] += z; });
		if (br) read(br, [&](int k, float z) { v[k] += z; });
		auto write = [&](float* to) {
			if constexpr (V == 8) reinterpret_cast<float4*>(to)[0] = make_float4(v[0], v[1], v[2], v[3]), reinterpret_cast<float4*>(to)[1] = make_float4(v[4], v[5], v[6], v[7]);
			else *to = v[0];
		};
		for (int s = 0; s < streams; ++s) write(x + ((size_t)n * streams + s) * width + i);
		if (x0) write(x0 + (size_t)n * width + i);
		if (act) {
#pragma unroll
			for (int k = 0; k < V; ++k) act[(size_t)n * width + i + k] = to_act<AT>(v[k]);
		}
	}
}

__global__ void k_seq_add(float* x, const float* y, size_t n) {
	pdl_enter(); // programmatic dependent launch: let the next kernel's launch overlap this one, then wait for the previous one
	const size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
	if (i < n) x[i] += y[i];
}

// Dynamic Tanh: out[r][i] = tanh(alpha * x[rows ? rows[r] : r][i]) * w[i] + b[i]
template <typename AT>
__global__ void k_seq_dyt(AT* out, const float* x, const int* rows, const bf16* w, const bf16* b, const bf16* alpha, int R, int width) {
	pdl_enter(); // programmatic dependent launch: let the next kernel's launch overlap this one, then wait for the previous one
	const size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
	if (i >= (size_t)R * width) return;
	const int r = (int)(i / width), c = (int)(i % width);
	const float a = ldf(alpha);
	const size_t src = (size_t)(rows ? rows[r] : r) * width + c;
	out[i] = to_act<AT>(tanhf(a * x[src]) * ldf(w + c) + ldf(b + c));
}

// sum over the CTA (whole warps, at most 8 of them); every thread adds the warps' sums in the same order
__device__ __forceinline__ float cta_sum(float v, float* red) {
	v = warp_sum(v);
	if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = v;
	__syncthreads();
	v = 0.f;
	for (int i = 0; i < (int)(blockDim.x >> 5); ++i) v += red[i];
	return v;
}
// RMS norm of whole rows: out[r][i] = x[row][i] / sqrt(mean(x[row]^2) + eps) * (w[i] + offset); one CTA per row (a single decoded
// token of a wide model is one row: a warp alone would walk it in a hundred dependent steps), the row is read once (up to
// blockDim * RMS_KEEP columns stay in registers, wider rows are read again).  LN: a layer norm without bias, the row's mean is taken
// off first and the mean square is that of the deviations.
#define RMS_KEEP 16
template <typename AT, bool LN = false>
__global__ void __launch_bounds__(256) k_seq_rms(AT* out, const float* x, const int* rows, const bf16* w, float offset, float eps, int R, int width) {
	pdl_launch_next();
	__shared__ float red[8], redm[8];
	const int tid = threadIdx.x, nt = blockDim.x, r = blockIdx.x;
	bf16 wk[RMS_KEEP]; // the weights are there before the previous kernel has ended
#pragma unroll
	for (int i = 0; i < RMS_KEEP; ++i)
		if (i * nt + tid < width) wk[i] = w[i * nt + tid];
	pdl_wait_prev();
	const float* src = x + (size_t)(rows ? rows[r] : r) * width;
	float keep[RMS_KEEP];
	float ss = 0.f, mean = 0.f;
	if constexpr (LN) {
		float sum = 0.f;
#pragma unroll
		for (int i = 0; i < RMS_KEEP; ++i) {
			const int c = i * nt + tid;
			keep[i] = c < width ? src[c] : 0.f;
			sum += keep[i];
		}
		for (int c = RMS_KEEP * nt + tid; c < width; c += nt) sum += src[c];
		mean = cta_sum(sum, redm) / (float)width;
	}
#pragma unroll
	for (int i = 0; i < RMS_KEEP; ++i) {
		const int c = i * nt + tid;
		if constexpr (LN) keep[i] = c < width ? keep[i] - mean : 0.f;
		else keep[i] = c < width ? src[c] : 0.f;
		ss = fmaf(keep[i], keep[i], ss);
	}
	for (int c = RMS_KEEP * nt + tid; c < width; c += nt) ss = fmaf(src[c] - mean, src[c] - mean, ss);
	ss = warp_sum(ss);
	if ((tid & 31) == 0) red[tid >> 5] = ss;
	__syncthreads();
	ss = 0.f;
	for (int i = 0; i < (nt >> 5); ++i) ss += red[i]; // every thread adds the warps' sums in the same order
	const float rinv = 1.f / sqrtf(ss / (float)width + eps);
	AT* d = out + (size_t)r * width;
#pragma unroll
	for (int i = 0; i < RMS_KEEP; ++i) {
		const int c = i * nt + tid;
		if (c < width) d[c] = to_act<AT>(keep[i] * rinv * (__bfloat162float(wk[i]) + offset));
	}
	for (int c = RMS_KEEP * nt + tid; c < width; c += nt) d[c] = to_act<AT>((src[c] - mean) * rinv * (ldf(w + c) + offset));
}

// RMS norm with a weight over `len` columns of src rows: segment s of blockIdx.y.  Segment 0 goes to an activation
// matrix, segment 1 (the cached latent) to its cache row; behind the latent the cache row holds the key part that all heads
// share, `rope.dims` channels of the projection turned by the token's position (not normed).
struct RmsSeg {
	int col, len;
	const bf16* w;
};
// rotation of channels 2i and 2i + 1 by position * freq[i] (angles in double, cos and sin times `mag`)
struct PairRope {
	int dims;           // even; 0: none
	const double* freq; // [dims / 2]
	float mag;
};
__device__ __forceinline__ float2 rope_angle(const PairRope& r, int pos, int i) { // (cos, sin) of pair i
	double s, c;
	sincos((double)pos * r.freq[i], &s, &c);
	return make_float2((float)c * r.mag, (float)s * r.mag);
}
__device__ __forceinline__ float2 rope_turn(float2 cs, float u, float v) { return make_float2(u * cs.x - v * cs.y, v * cs.x + u * cs.y); }
template <typename AT>
__global__ void k_seq_latent_norm(const float* proj, int ldp, RmsSeg sq, RmsSeg sc, AT* cq, float* cache, PairRope rope, float2* cs, SeqBatch sb, float eps) {
	pdl_enter(); // programmatic dependent launch: let the next kernel's launch overlap this one, then wait for the previous one
	const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
	const int n = blockIdx.x * (blockDim.x >> 5) + warp;
	if (n >= sb.N) return;
	const RmsSeg s = blockIdx.y ? sc : sq;
	const float* src = proj + (size_t)n * ldp + s.col;
	float ss = 0.f;
	for (int i = lane; i < s.len; i += 32) ss += src[i] * src[i];
	ss = warp_sum(ss);
	const float r = 1.f / sqrtf(ss / (float)max(s.len, 1) + eps);
	if (blockIdx.y == 0) { // (len 0: queries without a latent of their own, only the angles are formed)
		AT* d = cq + (size_t)n * s.len;
		for (int i = lane; i < s.len; i += 32) d[i] = to_act<AT>(src[i] * r * ldf(s.w + i));
		for (int i = lane; i < rope.dims / 2; i += 32) cs[(size_t)n * (rope.dims / 2) + i] = rope_angle(rope, sb.tpos[n], i); // for the queries of this layer
	} else {
		const int pos = sb.tpos[n];
		float* d = cache + cache_row(sb, sb.tslot[n], pos) * (s.len + rope.dims);
		for (int i = lane; i < s.len; i += 32) d[i] = src[i] * r * ldf(s.w + i);
		for (int i = lane; i < rope.dims / 2; i += 32) {
			const float2 t = rope_turn(rope_angle(rope, pos, i), src[s.len + 2 * i], src[s.len + 2 * i + 1]);
			d[s.len + 2 * i] = t.x, d[s.len + 2 * i + 1] = t.y;
		}
	}
}
// the rotated query channels of every head: q[n][h * ldh + col + d] from src[n * lds + h * dims + d], cs [N][dims / 2] the angles k_seq_latent_norm
// formed.  qb given: the queries leave in the activation type instead (split3 = 0), or as [hi | hi | lo] rows of split3 columns each (see
// k_seq_split_q).  One thread per pair.
__global__ void __launch_bounds__(256) k_seq_rope_heads(float* q, bf16* qb, int split3, const float* src, long lds, const float2* cs, int heads, int dims, long ldq, int ldh, int col, int N) {
	pdl_enter(); // programmatic dependent launch: let the next kernel's launch overlap this one, then wait for the previous one
	const int half = dims / 2;
	const size_t e = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
	if (e >= (size_t)N * heads * half) return;
	const size_t n = e / (heads * half);
	const int h = (int)(e % (heads * half)) / half, i = (int)(e % half);
	const float* p = src + n * lds + (size_t)h * dims + 2 * i;
	const float2 r = rope_turn(cs[n * half + i], p[0], p[1]);
	const size_t o = n * ldq + (size_t)h * ldh + col + 2 * i;
	if (!qb) {
		q[o] = r.x, q[o + 1] = r.y;
		return;
	}
	const bf16 h0 = __float2bfloat16_rn(r.x), h1 = __float2bfloat16_rn(r.y);
	bf16* d = qb + o;
	d[0] = h0, d[1] = h1;
	if (split3 > 0) {
		d[split3] = h0, d[split3 + 1] = h1;
		d[2 * split3] = __float2bfloat16_rn(r.x - __bfloat162float(h0)), d[2 * split3 + 1] = __float2bfloat16_rn(r.y - __bfloat162float(h1));
	}
}

// copy `len` columns of fp32 rows into an activation matrix
template <typename AT>
__global__ void k_seq_cast_cols(AT* out, const float* src, int lds, int col, int len, int N) {
	pdl_enter(); // programmatic dependent launch: let the next kernel's launch overlap this one, then wait for the previous one
	const size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
	if (i >= (size_t)N * len) return;
	out[i] = to_act<AT>(src[(i / len) * lds + col + i % len]);
}

// queries for the product path with fp32-accurate scores: per (token, head) the row [hi | hi | lo] of bf16 values, hi = bf16(q), lo = bf16(q - hi);
// against key rows [hi | lo | hi] one product of depth 3 kd sums q_hi k_hi + q_hi k_lo + q_lo k_hi in fp32
__global__ void k_seq_split_q(bf16* out, const float* q, int kd, size_t units) {
	pdl_enter(); // programmatic dependent launch: let the next kernel's launch overlap this one, then wait for the previous one
	const size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
	if (i >= units * kd) return;
	const size_t u = i / kd, d = i % kd;
	const float v = q[i];
	const bf16 hi = __float2bfloat16_rn(v);
	bf16* r = out + u * 3 * kd;
	r[d] = hi, r[kd + d] = hi, r[2 * kd + d] = __float2bfloat16_rn(v - __bfloat162float(hi));
}

// feed-forward unit on the stacked [gate | up] product.  mode 0: g = min(gate, L), u = clamp(up, -L, L), y = g sigmoid(1.702 g) (u + 1);
// mode 1: y = silu(gate) up; mode 2: y = gelu(gate) up, gelu(z) = z/2 (1 + tanh(sqrt(2/pi) (z + 0.044715 z^3)))
// (ld: row stride of gu, 2 * ff when the product holds nothing else)
__device__ __forceinline__ float glu_unit(float g, float u, float limit, int mode) {
	if (mode == 1) return g * sigmoidf_(g) * u;
	if (mode == 2) return 0.5f * g * (1.f + tanhf(0.7978845608028654f * (g + 0.044715f * g * g * g))) * u;
	g = fminf(g, limit), u = fminf(fmaxf(u, -limit), limit);
	return g * sigmoidf_(1.702f * g) * (u + 1.f);
}
template <typename AT>
__global__ void k_seq_ff_act(AT* out, const float* gu, int ff, int N, float limit, int mode, int ld) {
	pdl_enter(); // programmatic dependent launch: let the next kernel's launch overlap this one, then wait for the previous one
	const size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
	if (i >= (size_t)N * ff) return;
	const size_t n = i / ff, c = i % ff;
	out[i] = to_act<AT>(glu_unit(gu[n * ld + c], gu[n * ld + ff + c], limit, mode));
}

// y = silu(gate) up on TWO stacked products in one launch (the routed experts' rows and the shared unit's rows of one feed-forward)
struct FfPair {
	const float* gu[2];
	void* out[2];
	int ff[2], rows[2], ld[2];
};
template <typename AT>
__global__ void k_seq_ff_act2(FfPair a) {
	pdl_enter(); // programmatic dependent launch: let the next kernel's launch overlap this one, then wait for the previous one
	size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
	const size_t n0 = (size_t)a.rows[0] * a.ff[0];
	const int k = i < n0 ? 0 : 1;
	if (k) i -= n0;
	if (i >= (size_t)a.rows[k] * a.ff[k]) return;
	const size_t n = i / a.ff[k], c = i % a.ff[k];
	const float g = a.gu[k][n * a.ld[k] + c];
	((AT*)a.out[k])[i] = to_act<AT>(g * sigmoidf_(g) * a.gu[k][n * a.ld[k] + a.ff[k] + c]);
}

// ---------------------------------------------------------------- short convolution + activation + per-head norm (+ cache append)

// One of q / k / v: `heads` vectors of `hd` channels starting at column `col` of the projection.
struct ConvSeg {
	int col, heads, hd;
	int act;     // 1: SiLU after the convolution
	int norm;    // 0 none, 1 unit vector (sum of squares + 1e-6), 2 RMS (mean of squares + eps)
	float mul;   // factor after the norm
	int to_cache;
	float* dst;  // [N][heads*hd], or the cache [rows][heads*hd]
};
struct ConvArgs {
	ConvSeg seg[3];
	const float* proj;
	int ldp;
	const bf16* w;      // [channels][taps]
	const bf16* bias = nullptr; // [channels] added after the taps, or null
	int pcol = 0;       // column of channel 0 in the projection (segment columns, weights and state count channels from 0)
	int taps, channels; // channels = all of q|k|v
	const float* state; // [slots][taps-1][channels]: the projected values of the taps-1 positions before the step
	float eps;
};
// one warp per (token, head vector)
__global__ void k_seq_conv_heads(ConvArgs a, SeqBatch sb) {
	pdl_enter(); // programmatic dependent launch: let the next kernel's launch overlap this one, then wait for the previous one
	const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
	const int n = blockIdx.x;
	int u = blockIdx.y * (blockDim.x >> 5) + warp, s = 0;
	while (s < 3 && u >= a.seg[s].heads) u -= a.seg[s].heads, ++s;
	if (s == 3) return;
	const ConvSeg sg = a.seg[s];
	const int slot = sb.tslot[n], pos = sb.tpos[n];
	const int back = n - sb.tfirst[n]; // tokens of this step before this one
	const int T1 = a.taps - 1;
	const float* st = a.state + (size_t)slot * T1 * a.channels;
	float* d = sg.dst + (sg.to_cache ? cache_row(sb, slot, pos) : (long)n) * (sg.heads * sg.hd) + u * sg.hd;
	float ss = 0.f;
	for (int i = lane; i < sg.hd; i += 32) {
		const int ch = sg.col + u * sg.hd + i;
		float y = 0.f;
		for (int j = 0; j < a.taps; ++j) {
			const int ago = T1 - j; // tap j multiplies the value `ago` positions back
			const float v = ago <= back ? a.proj[(size_t)(n - ago) * a.ldp + a.pcol + ch] : st[(size_t)(T1 - (ago - back)) * a.channels + ch];
			y += ldf(a.w + (size_t)ch * a.taps + j) * v;
		}
		if (a.bias) y += ldf(a.bias + ch);
		if (sg.act) y = y * sigmoidf_(y);
		d[i] = y;
		ss += y * y;
	}
	if (sg.norm) {
		ss = warp_sum(ss);
		const float r = (sg.norm == 1 ? 1.f / sqrtf(ss + 1e-6f) : 1.f / sqrtf(ss / (float)sg.hd + a.eps)) * sg.mul;
		for (int i = lane; i < sg.hd; i += 32) d[i] *= r;
	}
}
// after the convolution: the state becomes the last taps-1 projected values of each sequence
__global__ void k_seq_conv_state(float* state, const float* proj, int ldp, int taps, int channels, SeqBatch sb, int pcol) {
	pdl_enter(); // programmatic dependent launch: let the next kernel's launch overlap this one, then wait for the previous one
	const int b = blockIdx.y, ch = blockIdx.x * blockDim.x + threadIdx.x;
	if (ch >= channels) return;
	const int T1 = taps - 1, cnt = sb.scount[b], start = sb.sstart[b];
	float* st = state + (size_t)sb.sslot[b] * T1 * channels;
	for (int i = 0; i < T1; ++i) { // new[i] = value T1 - i positions before the end; ascending i only reads old[i + cnt] with cnt >= 1
		const int ago = T1 - i;
		st[(size_t)i * channels + ch] = ago <= cnt ? proj[(size_t)(start + cnt - ago) * ldp + pcol + ch] : st[(size_t)(i + cnt) * channels + ch];
	}
}

// One token per sequence (decode): both at once.  A channel's state is read by one warp only, which puts the new one in its place; the taps' weights are requested before
// the previous kernel has ended, all values of a head vector at a time, and stay in registers (the two kernels above: 9.0 and 4.7 us for 768 and 1536 channels of one
// token, mostly one load waiting for another).  Vectors of up to 32 C channels, two to four taps.
template <int C>
__global__ void __launch_bounds__(128) k_seq_conv_step(ConvArgs a, SeqBatch sb, float* state) {
	pdl_launch_next();
	const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, n = blockIdx.x, T1 = a.taps - 1;
	int u = blockIdx.y * (blockDim.x >> 5) + warp, s = 0;
	while (s < 3 && u >= a.seg[s].heads) u -= a.seg[s].heads, ++s;
	if (s == 3) return;
	const ConvSeg sg = a.seg[s];
	const int ch0 = sg.col + u * sg.hd;
	float w[C][4], b[C];
#pragma unroll
	for (int i = 0; i < C; ++i) {
		const int e = lane + 32 * i;
#pragma unroll
		for (int j = 0; j < 4; ++j) w[i][j] = e < sg.hd && j < a.taps ? ldf(a.w + (size_t)(ch0 + e) * a.taps + j) : 0.f;
		b[i] = e < sg.hd && a.bias ? ldf(a.bias + ch0 + e) : 0.f;
	}
	pdl_wait_prev();
	const int slot = sb.tslot[n], pos = sb.tpos[n];
	float* st = state + (size_t)slot * T1 * a.channels + ch0;
	const float* pr = a.proj + (size_t)n * a.ldp + a.pcol + ch0;
	float* d = sg.dst + (sg.to_cache ? cache_row(sb, slot, pos) : (long)n) * (sg.heads * sg.hd) + u * sg.hd;
	float v[C][4]; // the values of the taps, oldest first
#pragma unroll
	for (int i = 0; i < C; ++i) {
		const int e = lane + 32 * i;
#pragma unroll
		for (int j = 0; j < 4; ++j) v[i][j] = e < sg.hd && j < a.taps ? (j < T1 ? st[(size_t)j * a.channels + e] : pr[e]) : 0.f;
	}
	float y[C], ss = 0.f;
#pragma unroll
	for (int i = 0; i < C; ++i) {
		const int e = lane + 32 * i;
		y[i] = 0.f;
#pragma unroll
		for (int j = 0; j < 4; ++j) {
			if (j < a.taps) y[i] += w[i][j] * v[i][j];
			if (j > 0 && j < a.taps && e < sg.hd) st[(size_t)(j - 1) * a.channels + e] = v[i][j];
		}
		if (a.bias) y[i] += b[i];
		if (sg.act) y[i] = y[i] * sigmoidf_(y[i]);
		if (e < sg.hd) ss += y[i] * y[i];
	}
	float r = 1.f;
	if (sg.norm) {
		ss = warp_sum(ss);
		r = (sg.norm == 1 ? 1.f / sqrtf(ss + 1e-6f) : 1.f / sqrtf(ss / (float)sg.hd + a.eps)) * sg.mul;
	}
#pragma unroll
	for (int i = 0; i < C; ++i)
		if (lane + 32 * i < sg.hd) d[lane + 32 * i] = sg.norm ? y[i] * r : y[i];
}

// ---------------------------------------------------------------- attention over the paged cache
// One CTA per (token, tile of query heads that share one key/value head).  Keys: `kd` floats at column kcol of the K cache
// rows, values: `vd` floats at column vcol of the V cache rows (latent attention: both are the cached latent).  Softmax in
// fp32, online over chunks of ATT_KC keys; `sink` joins the denominator only; `gate` (raw, per token and head) multiplies
// the output through a sigmoid.
#define ATT_KC 64
#define ATT_THREADS 256
#define ATT_MAXI 32 // output elements per thread: heads of the tile x value columns per thread
#define ATT_KPL 18  // key channels per lane held in registers (keys up to 576 wide: a 512-wide latent with its 64 rotated channels)
struct AttArgs {
	const float* q;   // [N][heads][kd]
	const float* kc;  // cache rows of width kld
	const float* vc;
	int kld, vld;
	int heads, group; // query heads per key/value head
	int tile;         // query heads per CTA (divides group)
	int kd, vd;
	int window;       // <= 0: all earlier positions
	int keep_first;   // with a window: positions below this stay visible to every later query
	int chunk = 0;    // > 0: only keys from floor(position / chunk) * chunk on are visible
	const float* slopes = nullptr; // [heads] or null: score -= slopes[h] * (query position - key position)
	int add_one = 0;  // 1: a sink of score zero (one added to the denominator); `sink` is then unused
	float scale;
	const bf16* sink; // [heads] or null
	const float* gate;
	int ldg, ghs, ges; // gate[n * ldg + h * ghs + d * ges]: one value per head (ghs 1, ges 0) or per output channel (ghs vd, ges 1)
	const int* skip;  // [N] or null: 1 = this token's attention is computed by the product path (k_seq_attn_*), the CTA leaves
	int nsplit;       // CTAs that share one (token, head tile)'s keys; > 1: partial results go to `part`, k_seq_attention_merge finishes
	float* part;      // [N][heads][nsplit][vd + 2]: unnormalised output, running maximum, denominator
	const float* qr = nullptr;  // the last `rot` query channels of every head come from here instead, qr[n * ldqr + h * rot + ..], and are turned by the angles in cs
	long ldqr = 0;
	const float2* cs = nullptr; // [N][rot / 2]
	int rot = 0;
	int split = 0;    // 1: on the product path queries, keys and probabilities travel as bf16 pairs (value + remainder), so scores and weights keep fp32 accuracy
	float softcap = 0.f; // > 0: score = softcap tanh(score / softcap), after the scale
	int vshare = 1;      // neighbouring key heads that read one value head
	int parts = 0;       // 1: results go to `part` whatever nsplit is (k_seq_attn_diff_merge finishes)
	int merge_skipped = 0; // 1: k_seq_attention_merge takes the tokens that `skip` names, not the others
	int cluster = 0;     // k_seq_attn_mma: the shares are a thread-block cluster, which folds them itself
};
__device__ __forceinline__ float att_cap(float s, float cap) { return cap > 0.f ? cap * tanhf(s / cap) : s; }
// channel c of the query of (token, head)
__device__ __forceinline__ float att_query(const AttArgs& a, int n, int h, int c) {
	const int e = c - (a.kd - a.rot);
	if (!a.qr || e < 0) return a.q[((size_t)n * a.heads + h) * a.kd + c];
	const float* p = a.qr + (size_t)n * a.ldqr + (size_t)h * a.rot + (e & ~1);
	const float2 r = rope_turn(a.cs[(size_t)n * (a.rot / 2) + e / 2], p[0], p[1]);
	return e & 1 ? r.y : r.x;
}
template <typename AT>
__global__ void __launch_bounds__(ATT_THREADS) k_seq_attention(AttArgs a, AT* out, SeqBatch sb) {
	pdl_enter(); // programmatic dependent launch: let the next kernel's launch overlap this one, then wait for the previous one
	extern __shared__ float sm[];
	const int n = blockIdx.x, h0 = blockIdx.y * a.tile, R = a.tile;
	if (a.skip && a.skip[n]) return;
	const int kvh = h0 / a.group, vh = kvh / a.vshare;
	float* qs = sm;                  // [R][kd]
	float* sc = qs + ((R * a.kd + 3) & ~3); // [R][ATT_KC], 16-byte aligned
	float* mrow = sc + R * ATT_KC;   // [R] running maximum
	float* lrow = mrow + R;          // [R] running denominator
	float* frow = lrow + R;          // [R] rescale factor of this chunk
	__shared__ long rows[ATT_KC];    // cache rows of this chunk's keys
	__shared__ int dist[ATT_KC];     // distance of each key of the chunk from the query
	const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, nwarp = ATT_THREADS / 32;
	const int slot = sb.tslot[n], pos = sb.tpos[n];
	int lo = a.window > 0 ? max(0, pos - a.window + 1) : 0;
	if (a.chunk > 0) lo = max(lo, pos / a.chunk * a.chunk);
	// visible keys in order: the kept first positions the window has left behind, [0, kf), then the window [lo, pos]
	const int kf = min(a.keep_first, lo), total = kf + pos - lo + 1;
	// this CTA's share of the key chunks (the whole range when nsplit == 1)
	const int nchunk = (total + ATT_KC - 1) / ATT_KC, per = (nchunk + a.nsplit - 1) / a.nsplit;
	const int c_begin = (int)blockIdx.z * per * ATT_KC, c_end = min(total - 1, ((int)blockIdx.z + 1) * per * ATT_KC - 1);
	for (int i = tid; i < R * a.kd; i += ATT_THREADS) qs[i] = att_query(a, n, h0 + i / a.kd, i % a.kd);
	if (tid < R) {
		const bool sk = (a.sink || a.add_one) && blockIdx.z == 0; // the sink counts once: in the first share
		mrow[tid] = sk ? (a.add_one ? 0.f : ldf(a.sink + h0 + tid)) : -INFINITY, lrow[tid] = sk ? 1.f : 0.f;
	}
	float acc[ATT_MAXI];
#pragma unroll
	for (int i = 0; i < ATT_MAXI; ++i) acc[i] = 0.f;
	const bool wide = a.vd > 2 * ATT_THREADS;
	__syncthreads();
	for (int c0 = c_begin; c0 <= c_end; c0 += ATT_KC) {
		const int nk = min(ATT_KC, total - c0);
		if (tid < ATT_KC) {
			const int kp = c0 + tid < kf ? c0 + tid : lo + c0 + tid - kf;
			rows[tid] = tid < nk ? cache_row(sb, slot, kp) : 0, dist[tid] = pos - kp;
		}
		__syncthreads();
		// scores: one warp per key, lanes across the key's channels; the lane's slice of the key is read once for all heads
		for (int j = warp; j < ATT_KC; j += nwarp) {
			if (j < nk) {
				const float* kr = a.kc + rows[j] * a.kld + (size_t)kvh * a.kd;
				if (a.kd <= 32 * ATT_KPL) {
					float kv[ATT_KPL];
#pragma unroll
					for (int i = 0; i < ATT_KPL; ++i) kv[i] = i * 32 + lane < a.kd ? kr[i * 32 + lane] : 0.f;
					for (int r0 = 0; r0 < R; r0 += 4) { // four heads' dot products advance together: independent chains and reductions
						float dd[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
						for (int i = 0; i < ATT_KPL; ++i) {
							if (i * 32 < a.kd) {
								const float* qp = qs + r0 * a.kd + min(i * 32 + lane, a.kd - 1);
#pragma unroll
								for (int u = 0; u < 4; ++u)
									if (r0 + u < R) dd[u] = fmaf(qp[u * a.kd], kv[i], dd[u]);
							}
						}
#pragma unroll
						for (int u = 0; u < 4; ++u) dd[u] = warp_sum(dd[u]);
#pragma unroll
						for (int u = 0; u < 4; ++u)
							if (r0 + u < R && lane == u) sc[(r0 + u) * ATT_KC + j] = att_cap(dd[u] * a.scale, a.softcap) - (a.slopes ? a.slopes[h0 + r0 + u] * (float)dist[j] : 0.f);
					}
				} else {
					for (int r = 0; r < R; ++r) {
						float d = 0.f;
						for (int i = lane; i < a.kd; i += 32) d += qs[r * a.kd + i] * kr[i];
						d = warp_sum(d);
						if (lane == 0) sc[r * ATT_KC + j] = att_cap(d * a.scale, a.softcap) - (a.slopes ? a.slopes[h0 + r] * (float)dist[j] : 0.f);
					}
				}
			} else if (lane == 0) {
				for (int r = 0; r < R; ++r) sc[r * ATT_KC + j] = -INFINITY;
			}
		}
		__syncthreads();
		// running maximum, probabilities in place, denominator
		for (int r = warp; r < R; r += nwarp) {
			float mx = -INFINITY;
			for (int j = lane; j < ATT_KC; j += 32) mx = fmaxf(mx, sc[r * ATT_KC + j]);
			mx = warp_max(mx);
			const float mo = mrow[r], mn = fmaxf(mo, mx);
			float ps = 0.f;
			for (int j = lane; j < ATT_KC; j += 32) {
				const float p = expf(sc[r * ATT_KC + j] - mn);
				sc[r * ATT_KC + j] = p, ps += p;
			}
			ps = warp_sum(ps);
			if (lane == 0) {
				const float f = mo == -INFINITY ? 0.f : expf(mo - mn);
				frow[r] = f, lrow[r] = lrow[r] * f + ps, mrow[r] = mn;
			}
		}
		__syncthreads();
		// values: a thread owns value columns tid and tid + 256 for every head of the tile (accumulator c * 16 + r); values wider
		// than 512 run one head per CTA with up to 32 columns per thread (accumulator c)
		if (wide) {
#pragma unroll
			for (int k = 0; k < ATT_MAXI; ++k) {
				const int d = tid + k * ATT_THREADS;
				if (d < a.vd) {
					const float* vcol = a.vc + (size_t)vh * a.vd + d;
					float s = acc[k] * frow[0];
					for (int j = 0; j < nk; ++j) s = fmaf(sc[j], vcol[rows[j] * a.vld], s);
					acc[k] = s;
				}
			}
		} else {
#pragma unroll
			for (int c = 0; c < 2; ++c) {
				const int d = tid + c * ATT_THREADS;
				if (d < a.vd) {
					const float* vcol = a.vc + (size_t)vh * a.vd + d;
#pragma unroll
					for (int r = 0; r < 16; ++r)
						if (r < R) acc[c * 16 + r] *= frow[r];
					for (int j0 = 0; j0 < nk; j0 += 4) {
						float v[4];
#pragma unroll
						for (int u = 0; u < 4; ++u) v[u] = j0 + u < nk ? vcol[rows[j0 + u] * a.vld] : 0.f;
#pragma unroll
						for (int r = 0; r < 16; ++r) {
							if (r < R) {
								const float4 p = *(const float4*)(sc + r * ATT_KC + j0);
								acc[c * 16 + r] = fmaf(p.w, v[3], fmaf(p.z, v[2], fmaf(p.y, v[1], fmaf(p.x, v[0], acc[c * 16 + r]))));
							}
						}
					}
				}
			}
		}
		__syncthreads();
	}
	// accumulator k -> (head of the tile, value column)
	auto head_of = [&](int k) { return wide ? 0 : k % 16; };
	auto col_of = [&](int k) { return tid + (wide ? k : k / 16) * ATT_THREADS; };
	if (a.nsplit > 1 || a.parts) {
		const int pw = a.vd + 2;
#pragma unroll
		for (int k = 0; k < ATT_MAXI; ++k) {
			const int r = head_of(k), d = col_of(k);
			if (r < R && d < a.vd) a.part[(((size_t)n * a.heads + h0 + r) * a.nsplit + blockIdx.z) * pw + d] = acc[k];
		}
		if (tid < R) {
			float* p = a.part + (((size_t)n * a.heads + h0 + tid) * a.nsplit + blockIdx.z) * pw + a.vd;
			p[0] = mrow[tid], p[1] = lrow[tid];
		}
		return;
	}
#pragma unroll
	for (int k = 0; k < ATT_MAXI; ++k) {
		const int r = head_of(k), d = col_of(k);
		if (r < R && d < a.vd) {
			float v = acc[k] / lrow[r];
			if (a.gate) v *= sigmoidf_(a.gate[(size_t)n * a.ldg + (size_t)(h0 + r) * a.ghs + (size_t)d * a.ges]);
			out[((size_t)n * a.heads + h0 + r) * a.vd + d] = to_act<AT>(v);
		}
	}
}
// folds the shares of one (token, head) in share order: one CTA per (token, head, 128 value columns)
#define ATT_MAXSPLIT 128
template <typename AT>
__global__ void __launch_bounds__(128) k_seq_attention_merge(AttArgs a, AT* out) {
	pdl_enter(); // programmatic dependent launch: let the next kernel's launch overlap this one, then wait for the previous one
	__shared__ float wz[ATT_MAXSPLIT], red[2][4];
	const int n = blockIdx.x, h = blockIdx.y, pw = a.vd + 2, z = threadIdx.x, d = blockIdx.z * 128 + threadIdx.x;
	if (a.skip && (a.skip[n] != 0) != (a.merge_skipped != 0)) return;
	const float* p = a.part + ((size_t)n * a.heads + h) * a.nsplit * pw;
	const float m = z < a.nsplit ? p[z * pw + a.vd] : -INFINITY, lz = z < a.nsplit ? p[z * pw + a.vd + 1] : 0.f;
	float mx = warp_max(m);
	if ((z & 31) == 0) red[0][z >> 5] = mx;
	__syncthreads();
	mx = fmaxf(fmaxf(red[0][0], red[0][1]), fmaxf(red[0][2], red[0][3]));
	const float w = m != -INFINITY ? expf(m - mx) : 0.f; // a share without keys counts nothing
	wz[z] = w;
	const float ls = warp_sum(w * lz);
	if ((z & 31) == 0) red[1][z >> 5] = ls;
	__syncthreads();
	if (d >= a.vd) return;
	const float l = (red[1][0] + red[1][1]) + (red[1][2] + red[1][3]);
	float v = 0.f;
#pragma unroll 16
	for (int k = 0; k < a.nsplit; ++k) v = fmaf(p[(size_t)k * pw + d], wz[k], v);
	const float g = (a.gate ? sigmoidf_(a.gate[(size_t)n * a.ldg + (size_t)h * a.ghs + (size_t)d * a.ges]) : 1.f) / l;
	out[((size_t)n * a.heads + h) * a.vd + d] = to_act<AT>(v * g);
}

// The same attention for decoded tokens and short portions on the warp-level tensor cores (bf16 mode): up to 16 query heads that share a
// key/value head are the 16 rows of m16n8k16 products.  Scores and softmax weights keep fp32 accuracy: queries, keys, probabilities and
// values enter as a bf16 value and the bf16 of what that rounding left, hi x hi + hi x lo + lo x hi summed in fp32.  One CTA per (token,
// head tile, share of the keys); keys travel ATM_KC at a time into a double buffer of shared memory by asynchronous copies, once for
// scores and values when the values are the first columns of the key rows (latent attention).
#define ATM_KC 32
#define ATM_TILES 8 // value-column tiles of 8 per warp: values up to 512 wide
__host__ __device__ constexpr int atm_pad(int cols) { return ((cols + 15) & ~15) % 32 == 0 ? ((cols + 15) & ~15) + 8 : ((cols + 15) & ~15) + 24; } // floats per staged row: 8 mod 32, fragment reads meet 32 different banks
__host__ __device__ constexpr int atm_ldq(int kd) { return ((kd + 15) & ~15) + 8; }
__host__ __device__ constexpr size_t atm_smem(int kd, int vd, bool shared_kv) {
	return (size_t)2 * ATM_KC * (atm_pad(kd) + (shared_kv ? 0 : atm_pad(vd))) * 4 + (size_t)2 * 16 * atm_ldq(kd) * 2 + (size_t)(2 * 16 * (ATM_KC + 1) + 3 * 16) * 4;
}
__device__ __forceinline__ void split_pair(float x, float y, uint32_t& hi, uint32_t& lo) {
	const __nv_bfloat162 h = __floats2bfloat162_rn(x, y), l = __floats2bfloat162_rn(x - __bfloat162float(h.x), y - __bfloat162float(h.y));
	hi = *reinterpret_cast<const uint32_t*>(&h), lo = *reinterpret_cast<const uint32_t*>(&l);
}
__device__ __forceinline__ void mma_bf16_16816(float (&c)[4], const uint32_t (&A)[4], const uint32_t (&B)[2]) {
	asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
	             : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
	             : "r"(A[0]), "r"(A[1]), "r"(A[2]), "r"(A[3]), "r"(B[0]), "r"(B[1]));
}
__device__ __forceinline__ void cp_async4(float* dst, const float* src) {
	asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"(smem_u32(dst)), "l"(src) : "memory");
}
__device__ __forceinline__ void cp_async16(float* dst, const float* src) {
	asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(smem_u32(dst)), "l"(src) : "memory");
}
__global__ void __launch_bounds__(256) k_seq_attn_mma(AttArgs a, bf16* out, SeqBatch sb, int shared_kv, int vec) {
	pdl_enter(); // programmatic dependent launch: let the next kernel's launch overlap this one, then wait for the previous one
	extern __shared__ __align__(16) float sm[];
	const int n = blockIdx.x, h0 = blockIdx.y * a.tile, R = a.tile;
	if (a.skip && a.skip[n]) return;
	const int kvh = h0 / a.group, vh = kvh / a.vshare, kd = a.kd, vd = a.vd, kp = (kd + 15) & ~15;
	const int ldk = atm_pad(kd), ldv = shared_kv ? ldk : atm_pad(vd), ldq = atm_ldq(kd);
	const int kbuf = ATM_KC * ldk, vbuf = shared_kv ? 0 : ATM_KC * ldv;
	float* const Ks = sm;                                   // [2][ATM_KC][ldk]
	float* const Vs = shared_kv ? Ks : sm + 2 * kbuf;       // [2][ATM_KC][ldv]
	bf16* const Qh = (bf16*)(sm + 2 * (kbuf + vbuf));       // [16][ldq]
	bf16* const Ql = Qh + 16 * ldq;
	float* const sc = (float*)(Ql + 16 * ldq);              // [2][16][ATM_KC + 1]: the two halves of the scores; [0]: the probabilities
	float *const mrow = sc + 2 * 16 * (ATM_KC + 1), *const lrow = mrow + 16, *const frow = lrow + 16;
	constexpr int LDS_ = ATM_KC + 1;
	const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, g = lane >> 2, t = lane & 3;
	const int slot = sb.tslot[n], pos = sb.tpos[n];
	int lo = a.window > 0 ? max(0, pos - a.window + 1) : 0;
	if (a.chunk > 0) lo = max(lo, pos / a.chunk * a.chunk);
	// visible keys in order: the kept first positions the window has left behind, [0, kf), then the window [lo, pos]; this CTA's share of them
	const int kf = min(a.keep_first, lo), total = kf + pos - lo + 1;
	const int nchunk = (total + ATM_KC - 1) / ATM_KC, per = (nchunk + a.nsplit - 1) / a.nsplit;
	const int c_begin = (int)blockIdx.z * per, c_end = min(nchunk, c_begin + per); // chunks [c_begin, c_end)
	auto key_pos = [&](int j) { return j < kf ? j : lo + j - kf; };
	auto issue = [&](int c) { // one warp per key row
		float *kb = Ks + (c & 1) * kbuf, *vb = Vs + (c & 1) * (shared_kv ? kbuf : vbuf);
		for (int j = warp; j < ATM_KC; j += 8) {
			const int key = c * ATM_KC + j;
			if (key < total) {
				const long row = cache_row(sb, slot, key_pos(key));
				const float *ksrc = a.kc + row * a.kld + (size_t)kvh * kd, *vsrc = a.vc + row * a.vld + (size_t)vh * vd;
				if (vec) {
					for (int i = 4 * lane; i < kd; i += 128) cp_async16(kb + j * ldk + i, ksrc + i);
					if (!shared_kv)
						for (int i = 4 * lane; i < vd; i += 128) cp_async16(vb + j * ldv + i, vsrc + i);
				} else {
					for (int i = lane; i < kd; i += 32) cp_async4(kb + j * ldk + i, ksrc + i);
					if (!shared_kv)
						for (int i = lane; i < vd; i += 32) cp_async4(vb + j * ldv + i, vsrc + i);
				}
				for (int i = kd + lane; i < kp; i += 32) kb[j * ldk + i] = 0.f;
			} else { // past the last key: zeros, so that nothing read here is a NaN
				for (int i = lane; i < kp; i += 32) kb[j * ldk + i] = 0.f;
				if (!shared_kv)
					for (int i = lane; i < vd; i += 32) vb[j * ldv + i] = 0.f;
			}
		}
		asm volatile("cp.async.commit_group;" ::: "memory");
	};
	if (c_begin < c_end) issue(c_begin);
	const int kq = a.qr ? kd - a.rot : kd; // channels read as they are; the rest are turned here
	for (int r = warp; r < 16; r += 8) { // one warp per query row
		bf16 *qh = Qh + r * ldq, *ql = Ql + r * ldq;
		const float* qsrc = a.q + ((size_t)n * a.heads + h0 + r) * kd;
		auto put = [&](int c, float q) {
			const bf16 hi = __float2bfloat16_rn(q);
			qh[c] = hi, ql[c] = __float2bfloat16_rn(q - __bfloat162float(hi));
		};
		if (r < R) {
#pragma unroll 8
			for (int c = lane; c < kq; c += 32) put(c, qsrc[c]);
			for (int i = lane; i < (kd - kq) / 2; i += 32) {
				const float* p = a.qr + (size_t)n * a.ldqr + (size_t)(h0 + r) * a.rot + 2 * i;
				const float2 v = rope_turn(a.cs[(size_t)n * (a.rot / 2) + i], p[0], p[1]);
				put(kq + 2 * i, v.x), put(kq + 2 * i + 1, v.y);
			}
		}
		for (int c = (r < R ? kd : 0) + lane; c < kp; c += 32) put(c, 0.f);
	}
	if (tid < 16) {
		const bool sk = (a.sink || a.add_one) && blockIdx.z == 0 && tid < R; // the sink counts once: in the first share
		mrow[tid] = sk ? (a.add_one ? 0.f : ldf(a.sink + h0 + tid)) : -INFINITY, lrow[tid] = sk ? 1.f : 0.f;
	}
	float acc[ATM_TILES][4];
#pragma unroll
	for (int i = 0; i < ATM_TILES; ++i) acc[i][0] = acc[i][1] = acc[i][2] = acc[i][3] = 0.f;
	for (int c = c_begin; c < c_end; ++c) {
		if (c + 1 < c_end) {
			issue(c + 1);
			asm volatile("cp.async.wait_group 1;" ::: "memory");
		} else asm volatile("cp.async.wait_group 0;" ::: "memory");
		__syncthreads();
		const float *kb = Ks + (c & 1) * kbuf, *vb = Vs + (c & 1) * (shared_kv ? kbuf : vbuf);
		{ // scores: warp = (8 keys, every other 16 channels)
			const int kt = warp & 3, hf = warp >> 2;
			const float* kr = kb + (kt * 8 + g) * ldk + 2 * t;
			const bf16 *q0 = Qh + g * ldq + 2 * t, *q1 = Ql + g * ldq + 2 * t;
			float s0[4] = {0.f, 0.f, 0.f, 0.f}, s1[4] = {0.f, 0.f, 0.f, 0.f}, s2[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll 3
			for (int k0 = hf * 16; k0 < kp; k0 += 32) {
				const float2 x = *(const float2*)(kr + k0), y = *(const float2*)(kr + k0 + 8);
				uint32_t bh[2], bl[2];
				split_pair(x.x, x.y, bh[0], bl[0]), split_pair(y.x, y.y, bh[1], bl[1]);
				const uint32_t ah[4] = {*(const uint32_t*)(q0 + k0), *(const uint32_t*)(q0 + 8 * ldq + k0), *(const uint32_t*)(q0 + k0 + 8), *(const uint32_t*)(q0 + 8 * ldq + k0 + 8)};
				const uint32_t al[4] = {*(const uint32_t*)(q1 + k0), *(const uint32_t*)(q1 + 8 * ldq + k0), *(const uint32_t*)(q1 + k0 + 8), *(const uint32_t*)(q1 + 8 * ldq + k0 + 8)};
				mma_bf16_16816(s0, ah, bh), mma_bf16_16816(s1, ah, bl), mma_bf16_16816(s2, al, bh);
			}
			float* d = sc + hf * 16 * LDS_ + g * LDS_ + kt * 8 + 2 * t;
			d[0] = s0[0] + (s1[0] + s2[0]), d[1] = s0[1] + (s1[1] + s2[1]);
			d[8 * LDS_] = s0[2] + (s1[2] + s2[2]), d[8 * LDS_ + 1] = s0[3] + (s1[3] + s2[3]);
		}
		__syncthreads();
		// softmax: two heads per warp, one key per lane
#pragma unroll
		for (int i = 0; i < 2; ++i) {
			const int r = 2 * warp + i, key = c * ATM_KC + lane;
			float s = -INFINITY;
			if (key < total) {
				s = att_cap((sc[r * LDS_ + lane] + sc[16 * LDS_ + r * LDS_ + lane]) * a.scale, a.softcap);
				if (a.slopes && r < R) s -= a.slopes[h0 + r] * (float)(pos - key_pos(key));
			}
			const float mo = mrow[r], mn = fmaxf(mo, warp_max(s)), p = expf(s - mn);
			sc[r * LDS_ + lane] = p;
			const float ps = warp_sum(p);
			if (lane == 0) {
				const float f = mo == -INFINITY ? 0.f : expf(mo - mn);
				frow[r] = f, lrow[r] = lrow[r] * f + ps, mrow[r] = mn;
			}
		}
		__syncthreads();
		// values: warp = tiles of 8 value columns; inside a 16-key step fragment places (2t, 2t+1, 2t+8, 2t+9) hold keys (t, t+4, t+8, t+12)
		uint32_t ph[2][4], pl[2][4];
#pragma unroll
		for (int s = 0; s < 2; ++s) {
			const float *p0 = sc + g * LDS_ + 16 * s + t, *p1 = p0 + 8 * LDS_;
			split_pair(p0[0], p0[4], ph[s][0], pl[s][0]), split_pair(p1[0], p1[4], ph[s][1], pl[s][1]);
			split_pair(p0[8], p0[12], ph[s][2], pl[s][2]), split_pair(p1[8], p1[12], ph[s][3], pl[s][3]);
		}
		const float f0 = frow[g], f1 = frow[g + 8];
#pragma unroll
		for (int i = 0; i < ATM_TILES; ++i) {
			const int d0 = (warp + 8 * i) * 8;
			if (d0 < vd) {
				acc[i][0] *= f0, acc[i][1] *= f0, acc[i][2] *= f1, acc[i][3] *= f1;
#pragma unroll
				for (int s = 0; s < 2; ++s) {
					const float* vp = vb + (16 * s + t) * ldv + d0 + g;
					uint32_t bh[2], bl[2];
					split_pair(vp[0], vp[4 * ldv], bh[0], bl[0]), split_pair(vp[8 * ldv], vp[12 * ldv], bh[1], bl[1]);
					mma_bf16_16816(acc[i], ph[s], bh), mma_bf16_16816(acc[i], ph[s], bl), mma_bf16_16816(acc[i], pl[s], bh);
				}
			}
		}
		__syncthreads(); // this chunk's buffer may be filled again, its scores overwritten
	}
	if (c_begin >= c_end) __syncthreads(); // a share without keys: mrow and lrow as they were set above
	// Up to eight shares: each CTA leaves its sums where its keys were and finishes 1 / nsplit of the outputs from all of them (a launch of
	// k_seq_attention_merge less: a decode step of six-layer blocks, one sequence at 300 positions, 251 -> 245 us).
	if (a.cluster) {
		const int ns = a.nsplit, z = blockIdx.z;
		float* const own = sm; // [R][vd]
#pragma unroll
		for (int i = 0; i < ATM_TILES; ++i)
#pragma unroll
			for (int e = 0; e < 4; ++e) {
				const int r = g + (e >> 1) * 8, d = (warp + 8 * i) * 8 + 2 * t + (e & 1);
				if (r < R && d < vd) own[r * vd + d] = acc[i][e];
			}
		cluster_sync();
		__shared__ float wz[8][16], inv[16];
		if (tid < 16) {
			float m[8], l = 0.f, mx = -INFINITY;
#pragma unroll
			for (int k = 0; k < 8; ++k) m[k] = k < ns ? cluster_load_f32(cluster_addr(mrow + tid, k)) : -INFINITY, mx = fmaxf(mx, m[k]);
#pragma unroll
			for (int k = 0; k < 8; ++k)
				if (k < ns) {
					const float w = m[k] != -INFINITY ? expf(m[k] - mx) : 0.f; // a share without keys counts nothing
					wz[k][tid] = w, l = fmaf(w, cluster_load_f32(cluster_addr(lrow + tid, k)), l);
				}
			inv[tid] = 1.f / l;
		}
		__syncthreads();
		const int all = R * vd, lo_e = all * z / ns, hi_e = all * (z + 1) / ns;
		for (int e = lo_e + tid; e < hi_e; e += 256) {
			const int r = e / vd, d = e - r * vd;
			const size_t o = (size_t)n * a.heads + h0 + r;
			const float gt = a.gate ? sigmoidf_(a.gate[(size_t)n * a.ldg + (size_t)(h0 + r) * a.ghs + (size_t)d * a.ges]) : 1.f;
			float v = 0.f;
#pragma unroll 8
			for (int k = 0; k < ns; ++k) v = fmaf(cluster_load_f32(cluster_addr(own + e, k)), wz[k][r], v);
			out[o * vd + d] = __float2bfloat16_rn(v * (gt * inv[r]));
		}
		cluster_sync(); // no CTA leaves while another reads its sums
		return;
	}
#pragma unroll
	for (int i = 0; i < ATM_TILES; ++i)
#pragma unroll
		for (int e = 0; e < 4; ++e) {
			const int r = g + (e >> 1) * 8, d = (warp + 8 * i) * 8 + 2 * t + (e & 1);
			if (r >= R || d >= vd) continue;
			const size_t o = (size_t)n * a.heads + h0 + r;
			if (a.nsplit > 1 || a.parts) a.part[(o * a.nsplit + blockIdx.z) * (vd + 2) + d] = acc[i][e];
			else {
				float v = acc[i][e] / lrow[r];
				if (a.gate) v *= sigmoidf_(a.gate[(size_t)n * a.ldg + (size_t)(h0 + r) * a.ghs + (size_t)d * a.ges]);
				out[o * vd + d] = __float2bfloat16_rn(v);
			}
		}
	if ((a.nsplit > 1 || a.parts) && tid < R) {
		float* p = a.part + (((size_t)n * a.heads + h0 + tid) * a.nsplit + blockIdx.z) * (vd + 2) + vd;
		p[0] = mrow[tid], p[1] = lrow[tid];
	}
}

// ---------------------------------------------------------------- prompt attention as products
// For many query tokens of one sequence the scores and the weighted values are matrix products on the tensor cores:
// the keys of the visible range are gathered from the paged cache into a bf16 matrix (values transposed), S = Q K^T per
// head, a row-wise fp32 softmax applies scale, causal / window mask, sink and output gate and writes bf16 probabilities,
// then O = P V.  Single decoded tokens and short portions take k_seq_attn_mma above, the exact mode k_seq_attention.
struct AttGather {
	const float* kc;
	const float* vc;
	int kld, vld, kcol, vcol; // column of this key/value head inside a cache row
	int kd, vd;
	bf16* Kb;   // [C][kd]
	bf16* Vt;   // [vd][Cp]
	int slot, k0, C, Cp;
	int kfb;    // the first kfb gathered keys are positions 0 .. kfb-1 (kept first tokens), the rest k0, k0 + 1, ...
	int split;  // 1: Kb rows are [hi | lo | hi] (3 kd wide: a key as a bf16 value and the bf16 of what the rounding left), Vt rows hold the values twice ([vd][2 Cp])
};
__global__ void k_seq_attn_gather(AttGather a, SeqBatch sb) {
	pdl_enter(); // programmatic dependent launch: let the next kernel's launch overlap this one, then wait for the previous one
	__shared__ float tile[32][33];
	const int j0 = blockIdx.x * 32, tx = threadIdx.x & 31, ty = threadIdx.x >> 5; // 32 x 8 threads
	const int dmax = max(a.kd, a.vd);
	for (int d0 = blockIdx.y * 32; d0 < dmax; d0 += gridDim.y * 32) {
		for (int r = ty; r < 32; r += 8) {
			const int j = j0 + r, d = d0 + tx;
			if (j < a.C) {
				const long row = cache_row(sb, a.slot, j < a.kfb ? j : a.k0 + j - a.kfb);
				if (d < a.kd) {
					const float kv = a.kc[row * a.kld + a.kcol + d];
					const bf16 hi = __float2bfloat16_rn(kv);
					if (a.split) {
						bf16* kr = a.Kb + (size_t)j * 3 * a.kd;
						kr[d] = hi, kr[a.kd + d] = __float2bfloat16_rn(kv - __bfloat162float(hi)), kr[2 * a.kd + d] = hi;
					} else a.Kb[(size_t)j * a.kd + d] = hi;
				}
				tile[r][tx] = d < a.vd ? a.vc[row * a.vld + a.vcol + d] : 0.f;
			} else tile[r][tx] = 0.f;
		}
		__syncthreads();
		for (int r = ty; r < 32; r += 8) {
			const int d = d0 + r, j = j0 + tx;
			if (d < a.vd && j < a.Cp) {
				const bf16 v = __float2bfloat16_rn(tile[tx][r]);
				if (a.split) a.Vt[(size_t)d * 2 * a.Cp + j] = v, a.Vt[(size_t)d * 2 * a.Cp + a.Cp + j] = v;
				else a.Vt[(size_t)d * a.Cp + j] = v;
			}
		}
		__syncthreads();
	}
}
// Which gathered columns a block of query rows sees: row t stands at position qpos0 + t; columns below kfb are the kept first positions, column
// j >= kfb is position k0 + j - kfb.  A row's columns are [0, kept) and [lo(t), hi(t)], both ends growing with t, so what a tile of rows
// sees is known from its first and last row: score tiles outside are not computed, and neither the softmax kernel nor the value product
// touches 64-column blocks that no row of a 128-row tile sees.
struct AttBand {
	int qpos0, k0, kfb, keep_first, window, chunk;
	__device__ __forceinline__ int lo(int t) const {
		const int q = qpos0 + t;
		int p = window > 0 ? max(0, q - window + 1) : 0;
		if (chunk > 0) p = max(p, q / chunk * chunk);
		return max(p - k0, 0) + kfb;
	}
	__device__ __forceinline__ int hi(int t) const { return qpos0 + t - k0 + kfb; }
	__device__ __forceinline__ int kept() const { return max(kfb, keep_first - k0 + kfb); }
	// does any of rows [t0, t1] see any of columns [c0, c1]?
	__device__ __forceinline__ bool meets(int t0, int t1, int c0, int c1) const { return c0 <= hi(t1) && (c1 >= lo(t0) || c0 < kept()); }
};
struct AttSoftmax {
	const float* S; // [heads of the launch][T][Cp]
	bf16* P;        // same shape
	int T, C, Cp;
	AttBand band;
	int banded = 0;      // 1: columns outside the 64-column blocks that a 128-row tile sees are left as they are (the value product skips them)
	const float* slopes = nullptr; // already offset to the first head of the launch, or null: score -= slopes[z] * (row position - column position)
	int add_one = 0;     // 1: one added to the denominator
	float scale;
	const bf16* sink; // already offset to the first head of the launch, or null
	const float* gate; // per head: gate[t * ldg + z], already offset to the first token and head, or null (per-channel gates are applied by the caller)
	int ldg;
	int split = 0;     // 1: P rows are 2 Cp wide: the probabilities as bf16, then the bf16 of what that rounding left
	float softcap = 0.f; // > 0: score = softcap tanh(score / softcap), after the scale
};
// One CTA per (row, head).  A thread takes pairs of neighbouring columns; the first SMX_KEEP pairs of its row stay in registers, so a row of up
// to 512 * SMX_KEEP columns is read once.
#define SMX_KEEP 8
__global__ void __launch_bounds__(256) k_seq_attn_softmax(AttSoftmax a) {
	pdl_enter(); // programmatic dependent launch: let the next kernel's launch overlap this one, then wait for the previous one
	__shared__ float red[2][8];
	const int t = blockIdx.x, z = blockIdx.y, tid = threadIdx.x;
	const float* srow = a.S + ((size_t)z * a.T + t) * a.Cp;
	bf16* prow = a.P + ((size_t)z * a.T + t) * a.Cp * (a.split ? 2 : 1);
	const int qpos = a.band.qpos0 + t, kfb = a.band.kfb;
	const int lo = a.band.lo(t), hi = min(a.C - 1, a.band.hi(t)), kept = a.band.kept();
	// columns written: everything, or the 64-column blocks that some row of this row's 128-row tile sees (a window's kept first positions: from 0 on)
	int w0 = 0, w1 = a.Cp;
	if (a.banded) {
		const int t0 = t & ~127;
		if (kept == 0) w0 = a.band.lo(t0) & ~63;
		w1 = min(a.Cp, (a.band.hi(min(t0 + 127, a.T - 1)) | 63) + 1);
	}
	const float sk = a.add_one ? 0.f : a.sink ? ldf(a.sink + z) : -INFINITY;
	const float slope = a.slopes ? a.slopes[z] : 0.f;
	auto score = [&](int j, float s) { // -inf for a column this row does not see
		if (j > hi || (j < lo && j >= kept)) return -INFINITY;
		return att_cap(s * a.scale, a.softcap) - (a.slopes ? slope * (float)(qpos - (j < kfb ? j : a.band.k0 + j - kfb)) : 0.f);
	};
	auto pair = [&](int j) { // j is even and Cp a multiple of 8: both columns lie inside the row
		if (j > hi || (j + 1 < lo && j >= kept)) return make_float2(-INFINITY, -INFINITY); // nothing was computed there
		const float2 v = *(const float2*)(srow + j);
		return make_float2(score(j, v.x), score(j + 1, v.y));
	};
	float2 keep[SMX_KEEP];
	float mx = sk;
#pragma unroll
	for (int i = 0; i < SMX_KEEP; ++i) {
		if (w0 + 512 * i >= w1) break; // the row ends here (the same for the whole CTA)
		const int j = w0 + 2 * (tid + 256 * i);
		keep[i] = j < w1 ? pair(j) : make_float2(-INFINITY, -INFINITY);
		mx = fmaxf(mx, fmaxf(keep[i].x, keep[i].y));
	}
	for (int j = w0 + 2 * (tid + 256 * SMX_KEEP); j < w1; j += 512) {
		const float2 v = pair(j);
		mx = fmaxf(mx, fmaxf(v.x, v.y));
	}
	mx = warp_max(mx);
	if ((tid & 31) == 0) red[0][tid >> 5] = mx;
	__syncthreads();
#pragma unroll
	for (int w = 0; w < 8; ++w) mx = fmaxf(mx, red[0][w]);
	float sum = 0.f;
#pragma unroll
	for (int i = 0; i < SMX_KEEP; ++i) {
		if (w0 + 512 * i >= w1) break;
		keep[i].x = expf(keep[i].x - mx), keep[i].y = expf(keep[i].y - mx);
		sum += keep[i].x + keep[i].y;
	}
	for (int j = w0 + 2 * (tid + 256 * SMX_KEEP); j < w1; j += 512) {
		const float2 v = pair(j);
		sum += expf(v.x - mx) + expf(v.y - mx);
	}
	sum = warp_sum(sum);
	if ((tid & 31) == 0) red[1][tid >> 5] = sum;
	__syncthreads();
	sum = 0.f;
#pragma unroll
	for (int w = 0; w < 8; ++w) sum += red[1][w];
	if (a.sink || a.add_one) sum += expf(sk - mx);
	const float f = (a.gate ? sigmoidf_(a.gate[(size_t)t * a.ldg + z]) : 1.f) / sum;
	auto put = [&](int j, float x, float y) {
		const __nv_bfloat162 h = __floats2bfloat162_rn(x * f, y * f);
		*(__nv_bfloat162*)(prow + j) = h;
		if (a.split) *(__nv_bfloat162*)(prow + a.Cp + j) = __floats2bfloat162_rn(x * f - __bfloat162float(h.x), y * f - __bfloat162float(h.y));
	};
#pragma unroll
	for (int i = 0; i < SMX_KEEP; ++i) {
		if (w0 + 512 * i >= w1) break;
		const int j = w0 + 2 * (tid + 256 * i);
		if (j < w1) put(j, keep[i].x, keep[i].y);
	}
	for (int j = w0 + 2 * (tid + 256 * SMX_KEEP); j < w1; j += 512) {
		const float2 v = pair(j);
		put(j, expf(v.x - mx), expf(v.y - mx));
	}
}

// ---------------------------------------------------------------- prompt attention in one kernel
// Flash attention for sequences that bring many tokens to a step: attentions over cached keys and values of the same width HD, scores in bf16
// products (not scores_f32, no distance bias, one map), at most with a window, a sink and a gate per channel.  A CTA serves km of
// the query heads that share a key head and tb blocks of 16 tokens, a warp one of each, over one of nsplit shares of the keys
// (flash_shares; partial results then, which k_seq_attention_merge folds in share order); a tile of 64 cached rows (fp32, through the page
// table) is copied to shared memory while the previous one is multiplied, rounded to bf16 once for all its warps, and read as
// mma.m16n8k16 fragments.  Scores, the running maximum, exponentials and the denominator are fp32; queries, keys and values are bf16
// with fp32 accumulation, as in the products that this replaces, and the weights a bf16 value and its remainder (one bf16 there).  Those
// were: gather, score product, softmax and value product per sequence, key head and block of queries, with scores and weights going
// through memory.
// Bound: the MMAs and, with few query heads per key head, the fp32 rows (64 KB a tile from L2).  A 2048-token
// step: 638 us in 16 launches before, 293 here (tensor pipe 13 % active); three sequences of 700 tokens: 700 us in 48 launches, 140 here.
#define AFL_TILE 64
template <int HD>
__host__ __device__ constexpr size_t afl_smem() { // the rows as cached (K, V), then as bf16 (K, V)
	return (size_t)2 * AFL_TILE * HD * (sizeof(float) + sizeof(bf16));
}
__device__ __forceinline__ uint32_t afl_pack(float x, float y) {
	const __nv_bfloat162 h = __floats2bfloat162_rn(x, y);
	return *reinterpret_cast<const uint32_t*>(&h);
}

template <int HD>
__global__ void __launch_bounds__(256, 1) k_seq_attn_flash(const AttArgs a, const bf16* __restrict__ Q, bf16* __restrict__ out, const SeqBatch sb, int km, int tb, int min_count) {
	pdl_enter();
	constexpr int C4 = HD / 4, KS = HD / 16, NT = AFL_TILE / 8;
	extern __shared__ __align__(128) unsigned char afl_sm[];
	float* const raw = reinterpret_cast<float*>(afl_sm);                                   // [K, V][64][HD]
	bf16* const tile = reinterpret_cast<bf16*>(afl_sm + (size_t)2 * AFL_TILE * HD * sizeof(float)); // the same, 16-byte chunks c of row r at c ^ (r & 7)
	const int b = blockIdx.z, cnt = sb.scount[b], c0 = ((int)gridDim.x - 1 - (int)blockIdx.x) * 16 * tb; // first token of the CTA in its sequence (the longest rows first)
	if (cnt < min_count || c0 >= cnt) return;
	const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, g = lane >> 2, t4 = lane & 3;
	const int first = sb.sstart[b], pos0 = sb.spos0[b], slot = sb.sslot[b], per = a.group / km;
	const int hg = blockIdx.y / a.nsplit, share = blockIdx.y % a.nsplit;
	const int kvh = hg / per, head = kvh * a.group + (hg % per) * km + warp % km;
	const int t0 = c0 + (warp / km) * 16; // first token of the warp
	const float* const kbase = a.kc + kvh * HD;
	const float* const vbase = a.vc + kvh * HD;
	const int keep = a.window > 0 ? a.keep_first : 0;
	auto low = [&](int p) { return a.window > 0 ? max(0, p - a.window + 1) : 0; }; // first position that a query at p sees (but for the kept ones)
	const int pa = pos0 + c0, pb = pos0 + min(cnt, c0 + 16 * tb) - 1;       // the CTA's positions
	const int wa = pos0 + t0, wb = pos0 + min(cnt, t0 + 16) - 1;            // the warp's (wb < wa: none)
	// the CTA's tiles: those of the kept positions, then all from the first query's window on; this share of them
	const int from = low(pa) & ~(AFL_TILE - 1), kept = min((keep + AFL_TILE - 1) / AFL_TILE, from / AFL_TILE);
	const int tiles = kept + (pb - from) / AFL_TILE + 1, each = (tiles + a.nsplit - 1) / a.nsplit, end = min(tiles, (share + 1) * each);
	auto key0 = [&](int i) { return i < kept ? i * AFL_TILE : from + (i - kept) * AFL_TILE; };
	auto fetch = [&](int k0) {
		for (int i = tid; i < 2 * AFL_TILE * C4; i += blockDim.x) {
			const int which = i / (AFL_TILE * C4), r = i / C4 % AFL_TILE, c = i % C4, pos = k0 + r;
			if (pos > pb) continue; // the rest of the tile is never visible
			const long row = cache_row(sb, slot, pos);
			cp_async16(raw + ((size_t)which * AFL_TILE + r) * HD + 4 * c, (which ? vbase + row * a.vld : kbase + row * a.kld) + 4 * c);
		}
		asm volatile("cp.async.commit_group;" ::: "memory");
	};
	auto at = [&](int which, int r, int c) { return tile + ((size_t)which * AFL_TILE + r) * HD + ((c ^ (r & 7)) << 3); };
	int ti = share * each;
	if (ti < end) fetch(key0(ti));

	uint32_t q[KS][4];
#pragma unroll
	for (int r = 0; r < 2; ++r) {
		const int t = t0 + g + 8 * r;
		const uint32_t* qp = reinterpret_cast<const uint32_t*>(Q + ((size_t)(first + t) * a.heads + head) * HD) + t4;
#pragma unroll
		for (int k = 0; k < KS; ++k) q[k][r] = t < cnt ? qp[8 * k] : 0u, q[k][2 + r] = t < cnt ? qp[8 * k + 4] : 0u;
	}
	float o[HD / 8][4], m[2], l[2];
#pragma unroll
	for (int n = 0; n < HD / 8; ++n) o[n][0] = o[n][1] = o[n][2] = o[n][3] = 0.f;
	const bool sink = a.sink && share == 0; // counts once
	m[0] = m[1] = sink ? ldf(a.sink + head) : -FLT_MAX;
	if (m[0] == -INFINITY) m[0] = m[1] = -FLT_MAX; // a sink of no weight
	l[0] = l[1] = sink && t4 == 0 ? 1.f : 0.f; // a lane's share of the denominator
	const int wlow = low(wa);
	for (; ti < end; ++ti) {
		const int kt = key0(ti);
		asm volatile("cp.async.wait_group 0;" ::: "memory");
		__syncthreads(); // the tile has arrived, and the bf16 one is no longer being read
		for (int i = tid; i < 2 * AFL_TILE * (HD / 8); i += blockDim.x) {
			const int which = i / (AFL_TILE * (HD / 8)), r = i / (HD / 8) % AFL_TILE, c = i % (HD / 8);
			const float4* s = reinterpret_cast<const float4*>(raw + ((size_t)which * AFL_TILE + r) * HD + 8 * c);
			const bool in = kt + r <= pb; // rows past the last position are zero: a weight of zero must not meet a NaN
			const float4 z = make_float4(0.f, 0.f, 0.f, 0.f), x = in ? s[0] : z, y = in ? s[1] : z;
			*reinterpret_cast<uint4*>(at(which, r, c)) = make_uint4(afl_pack(x.x, x.y), afl_pack(x.z, x.w), afl_pack(y.x, y.y), afl_pack(y.z, y.w));
		}
		__syncthreads();
		if (ti + 1 < end) fetch(key0(ti + 1));
		if (kt > wb || (kt + AFL_TILE <= wlow && kt >= keep)) continue; // (warp-uniform) nothing of this tile is visible to this warp's rows
		float s[NT][4];
#pragma unroll
		for (int n = 0; n < NT; ++n) {
			s[n][0] = s[n][1] = s[n][2] = s[n][3] = 0.f;
#pragma unroll
			for (int k = 0; k < KS; k += 2) {
				uint32_t bb[4];
				ldsm_x4(at(0, n * 8 + (lane & 7), 2 * k + (lane >> 3)), bb);
				const uint32_t b0[2] = {bb[0], bb[1]}, b1[2] = {bb[2], bb[3]};
				mma_bf16_16816(s[n], q[k], b0), mma_bf16_16816(s[n], q[k + 1], b1);
			}
		}
		float mx[2] = {-FLT_MAX, -FLT_MAX};
#pragma unroll
		for (int r = 0; r < 2; ++r) {
			const int p = wa + g + 8 * r, lo = low(p);
#pragma unroll
			for (int n = 0; n < NT; ++n)
#pragma unroll
				for (int e = 0; e < 2; ++e) {
					const int key = kt + n * 8 + 2 * t4 + e;
					float& x = s[n][2 * r + e];
					x = key <= p && (key >= lo || key < keep) ? x * a.scale : -INFINITY;
					mx[r] = fmaxf(mx[r], x);
				}
		}
		float corr[2];
#pragma unroll
		for (int r = 0; r < 2; ++r) {
			mx[r] = fmaxf(mx[r], __shfl_xor_sync(0xffffffffu, mx[r], 1)), mx[r] = fmaxf(mx[r], __shfl_xor_sync(0xffffffffu, mx[r], 2));
			const float mn = fmaxf(m[r], mx[r]);
			corr[r] = expf(m[r] - mn);
			m[r] = mn, l[r] *= corr[r];
		}
#pragma unroll
		for (int n = 0; n < HD / 8; ++n) o[n][0] *= corr[0], o[n][1] *= corr[0], o[n][2] *= corr[1], o[n][3] *= corr[1];
#pragma unroll
		for (int kk = 0; kk < AFL_TILE / 16; ++kk) {
			uint32_t p[4], pl[4];
#pragma unroll
			for (int j = 0; j < 2; ++j)
#pragma unroll
				for (int r = 0; r < 2; ++r) {
					const float x = expf(s[2 * kk + j][2 * r] - m[r]), y = expf(s[2 * kk + j][2 * r + 1] - m[r]);
					l[r] += x + y;
					const __nv_bfloat162 h = __floats2bfloat162_rn(x, y);
					p[2 * j + r] = *reinterpret_cast<const uint32_t*>(&h);
					pl[2 * j + r] = afl_pack(x - __bfloat162float(h.x), y - __bfloat162float(h.y));
				}
#pragma unroll
			for (int n = 0; n < HD / 8; n += 2) {
				uint32_t bb[4];
				ldsm_x4_t(at(1, kk * 16 + (lane & 15), n + (lane >> 4)), bb);
				const uint32_t b0[2] = {bb[0], bb[1]}, b1[2] = {bb[2], bb[3]};
				mma_bf16_16816(o[n], p, b0), mma_bf16_16816(o[n + 1], p, b1);
				mma_bf16_16816(o[n], pl, b0), mma_bf16_16816(o[n + 1], pl, b1);
			}
		}
	}
#pragma unroll
	for (int r = 0; r < 2; ++r) {
		l[r] += __shfl_xor_sync(0xffffffffu, l[r], 1), l[r] += __shfl_xor_sync(0xffffffffu, l[r], 2);
		const int t = t0 + g + 8 * r;
		if (t >= cnt) continue;
		if (a.nsplit > 1) {
			float* p = a.part + (((size_t)(first + t) * a.heads + head) * a.nsplit + share) * (HD + 2);
#pragma unroll
			for (int n = 0; n < HD / 8; ++n) *reinterpret_cast<float2*>(p + 8 * n + 2 * t4) = make_float2(o[n][2 * r], o[n][2 * r + 1]);
			if (t4 == 0) *reinterpret_cast<float2*>(p + HD) = make_float2(l[r] > 0.f ? m[r] : -INFINITY, l[r]); // (no key of the share visible: counts nothing)
			continue;
		}
		const float* gp = a.gate ? a.gate + (size_t)(first + t) * a.ldg + (size_t)head * a.ghs : nullptr;
		const float inv = 1.f / l[r];
		bf16* dst = out + ((size_t)(first + t) * a.heads + head) * HD + 2 * t4;
#pragma unroll
		for (int n = 0; n < HD / 8; ++n) {
			float x = o[n][2 * r] * inv, y = o[n][2 * r + 1] * inv;
			if (gp) x *= sigmoidf_(gp[(size_t)(8 * n + 2 * t4) * a.ges]), y *= sigmoidf_(gp[(size_t)(8 * n + 2 * t4 + 1) * a.ges]);
			*reinterpret_cast<uint32_t*>(dst + 8 * n) = afl_pack(x, y);
		}
	}
}

// ---------------------------------------------------------------- differential attention: two maps of one head
// Head h of key group g has two maps over the same values; the attention kernels run them as query heads (g * 2 + map) * group + j
// of 2 x key heads (j: the head's place in its group).  With their outputs a1, a2: o = a1 - lambda a2, o / sqrt(mean(o^2) + eps) * mul.
struct AttDiff {
	int heads, group, vd; // of the result: out[n][heads * vd]
	float lambda, mul, eps;
	__device__ __forceinline__ int row(int h, int map) const { return (h / group * 2 + map) * group + h % group; } // query head of a map
};
#define ADF_KEEP 8 // value columns per lane kept in registers (heads up to 256 wide; wider ones are formed a second time)
// both maps' outputs as fp32 rows src[n][2 * heads * vd] (the product path): one warp per (token, head).  only: [N] or null, 1 = this token is here
template <typename AT>
__global__ void __launch_bounds__(128) k_seq_attn_diff(AttDiff a, const float* src, AT* out, const int* only, int N) {
	pdl_enter(); // programmatic dependent launch: let the next kernel's launch overlap this one, then wait for the previous one
	const long u = (long)blockIdx.x * 4 + (threadIdx.x >> 5);
	const int lane = threadIdx.x & 31;
	if (u >= (long)N * a.heads) return;
	const int n = (int)(u / a.heads), h = (int)(u % a.heads);
	if (only && !only[n]) return;
	const float* p = src + (size_t)n * 2 * a.heads * a.vd;
	const float *p1 = p + (size_t)a.row(h, 0) * a.vd, *p2 = p + (size_t)a.row(h, 1) * a.vd;
	float keep[ADF_KEEP], ss = 0.f;
#pragma unroll
	for (int i = 0; i < ADF_KEEP; ++i) {
		const int d = i * 32 + lane;
		keep[i] = d < a.vd ? p1[d] - a.lambda * p2[d] : 0.f;
		ss = fmaf(keep[i], keep[i], ss);
	}
	for (int d = ADF_KEEP * 32 + lane; d < a.vd; d += 32) {
		const float v = p1[d] - a.lambda * p2[d];
		ss = fmaf(v, v, ss);
	}
	const float f = a.mul / sqrtf(warp_sum(ss) / (float)a.vd + a.eps);
	AT* o = out + (size_t)u * a.vd;
#pragma unroll
	for (int i = 0; i < ADF_KEEP; ++i)
		if (i * 32 + lane < a.vd) o[i * 32 + lane] = to_act<AT>(keep[i] * f);
	for (int d = ADF_KEEP * 32 + lane; d < a.vd; d += 32) o[d] = to_act<AT>((p1[d] - a.lambda * p2[d]) * f);
}
// the same from the shares that the attention kernels left in t.part (folded in share order, one or more of them): one CTA per (token, head)
template <typename AT>
__global__ void __launch_bounds__(128) k_seq_attn_diff_merge(AttArgs t, AttDiff a, AT* out) {
	pdl_enter(); // programmatic dependent launch: let the next kernel's launch overlap this one, then wait for the previous one
	__shared__ float wz[2][ATT_MAXSPLIT], red[2][2][4], rsum[4];
	const int n = blockIdx.x, h = blockIdx.y, pw = t.vd + 2, z = threadIdx.x, warp = z >> 5;
	if (t.skip && t.skip[n]) return;
	const float *p[2], *b = t.part + (size_t)n * t.heads * t.nsplit * pw;
	float m[2], l[2];
#pragma unroll
	for (int k = 0; k < 2; ++k) {
		p[k] = b + (size_t)a.row(h, k) * t.nsplit * pw;
		m[k] = z < t.nsplit ? p[k][z * pw + t.vd] : -INFINITY, l[k] = z < t.nsplit ? p[k][z * pw + t.vd + 1] : 0.f;
		const float mx = warp_max(m[k]);
		if ((z & 31) == 0) red[0][k][warp] = mx;
	}
	__syncthreads();
#pragma unroll
	for (int k = 0; k < 2; ++k) {
		const float mx = fmaxf(fmaxf(red[0][k][0], red[0][k][1]), fmaxf(red[0][k][2], red[0][k][3]));
		const float w = m[k] != -INFINITY ? expf(m[k] - mx) : 0.f; // a share without keys counts nothing
		wz[k][z] = w;
		const float ls = warp_sum(w * l[k]);
		if ((z & 31) == 0) red[1][k][warp] = ls;
	}
	__syncthreads();
	const float r1 = 1.f / ((red[1][0][0] + red[1][0][1]) + (red[1][0][2] + red[1][0][3]));
	const float r2 = a.lambda / ((red[1][1][0] + red[1][1][1]) + (red[1][1][2] + red[1][1][3]));
	auto value = [&](int d) {
		float v1 = 0.f, v2 = 0.f;
#pragma unroll 8
		for (int k = 0; k < t.nsplit; ++k) v1 = fmaf(p[0][(size_t)k * pw + d], wz[0][k], v1), v2 = fmaf(p[1][(size_t)k * pw + d], wz[1][k], v2);
		return v1 * r1 - v2 * r2;
	};
	float keep[2], ss = 0.f; // value columns z and z + 128 stay in registers
#pragma unroll
	for (int i = 0; i < 2; ++i) {
		keep[i] = i * 128 + z < t.vd ? value(i * 128 + z) : 0.f;
		ss = fmaf(keep[i], keep[i], ss);
	}
	for (int d = 256 + z; d < t.vd; d += 128) {
		const float v = value(d);
		ss = fmaf(v, v, ss);
	}
	const float f = a.mul / sqrtf(cta_sum(ss, rsum) / (float)a.vd + a.eps);
	AT* o = out + ((size_t)n * a.heads + h) * a.vd;
#pragma unroll
	for (int i = 0; i < 2; ++i)
		if (i * 128 + z < t.vd) o[i * 128 + z] = to_act<AT>(keep[i] * f);
	for (int d = 256 + z; d < t.vd; d += 128) o[d] = to_act<AT>(value(d) * f);
}

// ---------------------------------------------------------------- gated delta rule
// One CTA per (sequence, head): the head's state S [dim][vdim] sits in shared memory for all tokens of the step, thread j
// owns value column j.  Per token:  S <- g (.) S (rows);  u = beta (v - S^T k);  S <- S + k u^T;  o = S^T q.
// g = exp(-exp(A_log) softplus(dt + dt_bias)) and beta = sigmoid(.) are formed here in fp32.
struct DeltaArgs {
	const float *q, *k, *v; // [N][kv_heads*dim] x2, [N][heads*vdim]
	const float* proj;      // beta (raw) at column bcol
	int ldp, bcol;
	const float* dt;        // [N][heads*dim] raw
	const bf16 *a_log, *dt_bias;
	float* state;           // [slots][heads][dim][vdim]
	float* o;               // [N][heads*vdim]
	int heads, kv_heads, dim, vdim;
};
__global__ void k_seq_delta_scan(DeltaArgs a, SeqBatch sb) {
	pdl_enter(); // programmatic dependent launch: let the next kernel's launch overlap this one, then wait for the previous one
	extern __shared__ float sm[];
	const int b = blockIdx.x, h = blockIdx.y, D = a.dim, V = a.vdim;
	const int kh = h / (a.heads / a.kv_heads);
	float* S = sm;          // [D][V]
	float* ks = S + D * V;  // [D]
	float* qs = ks + D;
	float* gs = qs + D;
	const int tid = threadIdx.x;
	float* Sg = a.state + ((size_t)sb.sslot[b] * a.heads + h) * D * V;
	for (int i = tid; i < D * V; i += blockDim.x) S[i] = Sg[i];
	const float A = expf(ldf(a.a_log + h));
	const int start = sb.sstart[b], cnt = sb.scount[b];
	for (int t = 0; t < cnt; ++t) {
		const int n = start + t;
		__syncthreads();
		for (int i = tid; i < D; i += blockDim.x) {
			ks[i] = a.k[((size_t)n * a.kv_heads + kh) * D + i];
			qs[i] = a.q[((size_t)n * a.kv_heads + kh) * D + i];
			gs[i] = expf(-A * softplusf_(a.dt[((size_t)n * a.heads + h) * D + i] + ldf(a.dt_bias + h * D + i)));
		}
		__syncthreads();
		if (tid < V) {
			float dot = 0.f;
			for (int i = 0; i < D; ++i) {
				const float s = gs[i] * S[i * V + tid];
				S[i * V + tid] = s;
				dot += s * ks[i];
			}
			const float beta = sigmoidf_(a.proj[(size_t)n * a.ldp + a.bcol + h]);
			const float u = beta * (a.v[((size_t)n * a.heads + h) * V + tid] - dot);
			float o = 0.f;
			for (int i = 0; i < D; ++i) {
				const float s = S[i * V + tid] + ks[i] * u;
				S[i * V + tid] = s;
				o += s * qs[i];
			}
			a.o[((size_t)n * a.heads + h) * V + tid] = o;
		}
	}
	__syncthreads();
	for (int i = tid; i < D * V; i += blockDim.x) Sg[i] = S[i];
}
// The same recurrence with the state in registers.  Value columns are independent: a CTA takes DELTA_VC of them, eight lanes share a
// pair of columns and each holds D/8 rows of both.  Tokens are staged DELTA_TB at a time: while one block of tokens is applied (no
// barrier between its tokens, only shuffles inside a pair's eight lanes), the next block's k, q, decay, v and beta travel from global
// memory into the other half of a double buffer; k, q and the decay are read back as float4 (eighths padded so that the eight lanes
// hit different banks).  The lanes' shares of a block's read-outs are folded together at its end, so that lane i ends with the i-th of
// the pair's 2 DELTA_TB values.
// Bound: shared-memory reads, D/4 float4 of k and q and D/8 of the decay per lane group and token, and the chain of a token (dot,
// shuffles, update).  With all columns of a head in one CTA and a column per four lanes, 48 CTAs took 845 us
// for 3 x 700 tokens of 16 heads of 128; 192 CTAs of a quarter of the columns and half the reads per column take 522.
#define DELTA_TB 4
#define DELTA_VC 32
__host__ __device__ constexpr int delta_qp(int D) { return D / 8 == 4 ? 4 : D / 8 + 4; }
__host__ __device__ constexpr int delta_tok(int D) { return 3 * 8 * delta_qp(D) + DELTA_VC + 4; } // k, q, g (padded eighths), v, beta
template <int D>
__global__ void __launch_bounds__(128) k_seq_delta_scan_reg(DeltaArgs a, SeqBatch sb) {
	pdl_enter(); // programmatic dependent launch: let the next kernel's launch overlap this one, then wait for the previous one
	constexpr int Q = D / 8, QP = delta_qp(D), TOK = delta_tok(D), VAT = 3 * 8 * QP, BAT = VAT + DELTA_VC;
	constexpr int ITEMS = (3 * D + DELTA_VC) / 4 + 1, ROUNDS = (DELTA_TB * ITEMS + 127) / 128;
	__shared__ __align__(16) float sm[2 * DELTA_TB * TOK];
	const int b = blockIdx.x, h = blockIdx.y, V = a.vdim, v0 = blockIdx.z * DELTA_VC;
	const int kh = h / (a.heads / a.kv_heads);
	const int tid = threadIdx.x, part = tid & 7, cl = (tid >> 3) * 2;
	const bool live = v0 + cl < V; // (V is a multiple of 4: both columns or none) lanes past the last column run along on a copy of it
	const int col = live ? v0 + cl : V - 2;
	float S[Q][2];
	float* Sg = a.state + ((size_t)sb.sslot[b] * a.heads + h) * D * V + (size_t)part * Q * V + col;
#pragma unroll
	for (int i = 0; i < Q; ++i) {
		const float2 t = *(const float2*)(Sg + (size_t)i * V);
		S[i][0] = t.x, S[i][1] = t.y;
	}
	const float A = expf(ldf(a.a_log + h));
	const int start = sb.sstart[b], cnt = sb.scount[b];
	// Staging.  A token's inputs are 3 D / 4 + DELTA_VC / 4 float4 items (k, q, raw decay input, v) and one scalar (beta's input); item e
	// of a block belongs to token e / ITEMS.  A thread serves the same items of every block, so where they come from and go to is worked
	// out once; per block it issues its 16-byte loads before the running block's arithmetic and finishes them (decay, beta) after it.
	const float* src[ROUNDS];
	float4 bias[ROUNDS];                                // decay items: their dt_bias entries
	int stride[ROUNDS], slot[ROUNDS], kind[ROUNDS];     // kind: 0 plain float4, 1 decay input, 2 beta input (scalar), -1 none
#pragma unroll
	for (int r = 0; r < ROUNDS; ++r) {
		const int e = tid + r * 128, tt = e / ITEMS, i0 = 4 * (e % ITEMS);
		kind[r] = -1, src[r] = a.k, stride[r] = 0, slot[r] = 0, bias[r] = make_float4(0.f, 0.f, 0.f, 0.f);
		if (tt >= DELTA_TB) continue;
		if (i0 < 3 * D) {
			const int seg = i0 / D, w = i0 % D;
			kind[r] = seg == 2 ? 1 : 0;
			stride[r] = seg == 2 ? a.heads * D : a.kv_heads * D;
			src[r] = (seg == 0 ? a.k + (size_t)kh * D : seg == 1 ? a.q + (size_t)kh * D : a.dt + (size_t)h * D) + w + (size_t)(start + tt) * stride[r];
			slot[r] = tt * TOK + seg * 8 * QP + (w / Q) * QP + w % Q;
			if (seg == 2) {
				const bf16* bp = a.dt_bias + h * D + w;
				bias[r] = make_float4(ldf(bp), ldf(bp + 1), ldf(bp + 2), ldf(bp + 3));
			}
		} else if (i0 < 3 * D + DELTA_VC) {
			const int i = i0 - 3 * D;
			if (v0 + i >= V) continue;
			kind[r] = 0, stride[r] = a.heads * V;
			src[r] = a.v + (size_t)h * V + v0 + i + (size_t)(start + tt) * stride[r];
			slot[r] = tt * TOK + VAT + i;
		} else {
			kind[r] = 2, stride[r] = a.ldp;
			src[r] = a.proj + a.bcol + h + (size_t)(start + tt) * stride[r];
			slot[r] = tt * TOK + BAT;
		}
	}
	auto fetch_block = [&](int blk, float4 (&pre)[ROUNDS]) {
		const int nt = min(DELTA_TB, cnt - blk * DELTA_TB);
#pragma unroll
		for (int r = 0; r < ROUNDS; ++r) {
			pre[r] = make_float4(0.f, 0.f, 0.f, 0.f);
			if (kind[r] >= 0 && (tid + r * 128) / ITEMS < nt) {
				const float* p = src[r] + (size_t)blk * DELTA_TB * stride[r];
				if (kind[r] == 2) pre[r].x = __ldg(p);
				else pre[r] = __ldg((const float4*)p);
			}
		}
	};
	auto put_block = [&](float* st, int blk, const float4 (&pre)[ROUNDS]) {
		const int nt = min(DELTA_TB, cnt - blk * DELTA_TB);
#pragma unroll
		for (int r = 0; r < ROUNDS; ++r) {
			if (kind[r] >= 0 && (tid + r * 128) / ITEMS < nt) {
				float4 v = pre[r];
				if (kind[r] == 1) {
					v.x = expf(-A * softplusf_(v.x + bias[r].x)), v.y = expf(-A * softplusf_(v.y + bias[r].y));
					v.z = expf(-A * softplusf_(v.z + bias[r].z)), v.w = expf(-A * softplusf_(v.w + bias[r].w));
				}
				if (kind[r] == 2) st[slot[r]] = sigmoidf_(v.x);
				else *(float4*)(st + slot[r]) = v;
			}
		}
	};
	const int nblk = (cnt + DELTA_TB - 1) / DELTA_TB, vcol = live ? cl : 0; // (a staged column; what the others compute goes nowhere)
	float4 pre[ROUNDS];
	fetch_block(0, pre);
	put_block(sm, 0, pre);
	__syncthreads();
	for (int blk = 0; blk < nblk; ++blk) {
		const float* __restrict__ cur = sm + (blk & 1) * DELTA_TB * TOK;
		if (blk + 1 < nblk) fetch_block(blk + 1, pre);
		const int nt = min(DELTA_TB, cnt - blk * DELTA_TB);
		float o[2 * DELTA_TB];
		auto apply = [&](int tt, float& oa, float& ob) { // one token: decay, correction, this lane's share of the read-out
			const float* tk = cur + tt * TOK;
			const float4 *ks = (const float4*)(tk + part * QP), *qs = (const float4*)(tk + 8 * QP + part * QP), *gs = (const float4*)(tk + 16 * QP + part * QP);
			const float2 v = *(const float2*)(tk + VAT + vcol);
			float dot[2][2] = {};
#pragma unroll
			for (int i = 0; i < Q / 4; ++i) {
				const float4 g4 = gs[i], k4 = ks[i];
				const float g[4] = {g4.x, g4.y, g4.z, g4.w}, k[4] = {k4.x, k4.y, k4.z, k4.w};
#pragma unroll
				for (int e = 0; e < 4; ++e)
#pragma unroll
					for (int c = 0; c < 2; ++c) S[4 * i + e][c] *= g[e], dot[c][e & 1] = fmaf(S[4 * i + e][c], k[e], dot[c][e & 1]);
			}
			float u[2] = {dot[0][0] + dot[0][1], dot[1][0] + dot[1][1]};
#pragma unroll
			for (int w = 1; w < 8; w <<= 1) u[0] += __shfl_xor_sync(0xffffffffu, u[0], w), u[1] += __shfl_xor_sync(0xffffffffu, u[1], w);
			u[0] = tk[BAT] * (v.x - u[0]), u[1] = tk[BAT] * (v.y - u[1]);
			float r[2][2] = {};
#pragma unroll
			for (int i = 0; i < Q / 4; ++i) {
				const float4 k4 = ks[i], q4 = qs[i];
				const float k[4] = {k4.x, k4.y, k4.z, k4.w}, q[4] = {q4.x, q4.y, q4.z, q4.w};
#pragma unroll
				for (int e = 0; e < 4; ++e)
#pragma unroll
					for (int c = 0; c < 2; ++c) S[4 * i + e][c] = fmaf(k[e], u[c], S[4 * i + e][c]), r[c][e & 1] = fmaf(S[4 * i + e][c], q[e], r[c][e & 1]);
			}
			oa = r[0][0] + r[0][1], ob = r[1][0] + r[1][1];
		};
		if (nt == DELTA_TB) { // no branch between the tokens: loads of later ones move up past the arithmetic of earlier ones
#pragma unroll
			for (int tt = 0; tt < DELTA_TB; ++tt) apply(tt, o[2 * tt], o[2 * tt + 1]);
		} else {
#pragma unroll
			for (int tt = 0; tt < DELTA_TB; ++tt) {
				o[2 * tt] = o[2 * tt + 1] = 0.f;
				if (tt < nt) apply(tt, o[2 * tt], o[2 * tt + 1]);
			}
		}
#pragma unroll
		for (int w = 4; w > 0; w >>= 1) { // lane bit w keeps the half of the values that has it
			const bool up = part & w;
#pragma unroll
			for (int i = 0; i < w; ++i) {
				const float other = __shfl_xor_sync(0xffffffffu, up ? o[i] : o[i + w], w);
				o[i] = (up ? o[i + w] : o[i]) + other;
			}
		}
		if (live && (part >> 1) < nt) a.o[((size_t)(start + blk * DELTA_TB + (part >> 1)) * a.heads + h) * V + col + (part & 1)] = o[0];
		if (blk + 1 < nblk) put_block(sm + ((blk + 1) & 1) * DELTA_TB * TOK, blk + 1, pre);
		__syncthreads();
	}
	if (live) {
#pragma unroll
		for (int i = 0; i < Q; ++i) *(float2*)(Sg + (size_t)i * V) = make_float2(S[i][0], S[i][1]);
	}
}
// The same recurrence, blocks of DELTA_BK tokens at a time.  Inside a block, with S the state before it, G_t the product of the decays up to token t and
// D(t, s) that of the decays after s up to t (per key channel, nothing is divided):
//   u_t = beta_t (v_t - (k_t G_t) S - sum_{s<t} A_ts u_s),   A_ts = k_t . D(t, s) k_s
//   o_t = (q_t G_t) S + sum_{s<=t} B_ts u_s,                 B_ts = q_t . D(t, s) k_s
//   S'  = G_T S + sum_s (D(T, s) k_s) u_s
// so the corrections of a block are one triangular system, U = X (V - (K G) S) with X = (1 + diag(beta) A)^-1 diag(beta), and the read-outs are (Q G) S + (B X) (V - (K G) S).
// X and B X depend on no value: k_seq_delta_system forms them for all blocks side by side (and turns the raw decay inputs into decays, in place), and
// k_seq_delta_blocks walks the state from block to block with products whose terms do not wait for one another.  The scan's chain of a token (dot, shuffles,
// update: 0.6 us, 1.7 where the CTAs take three waves) becomes a block's, 4.5 us, or 10 for three CTAs to an SM: 3 x 700 tokens of 16 heads of 128 x 128 504 -> 313 us, one
// sequence of 2048 1263 -> 598, sixteen of 128 340 -> 211 (both kernels, timed apart).
#define DELTA_BK 16
struct DeltaBlocks {
	float* sys; // [block][heads][2][DELTA_BK][DELTA_BK]: X, B X; block j of sequence b is number sstart[b] / DELTA_BK + b + j (one more than fit a portion at most)
	float* dt;  // DeltaArgs::dt, written
	int count;  // blocks of the longest portion
};
__global__ void __launch_bounds__(512) k_seq_delta_system(DeltaArgs a, DeltaBlocks c, SeqBatch sb) {
	pdl_enter(); // programmatic dependent launch: let the next kernel's launch overlap this one, then wait for the previous one
	constexpr int D = 128, T = DELTA_BK; // a warp per token, four channels per lane
	__shared__ __align__(16) float ks[T][D], qs[T][D], gs[T][D];
	__shared__ float A[T][T + 1], Bm[T][T + 1], X[T][T + 1], beta[T];
	const int b = blockIdx.x / c.count, blk = blockIdx.x % c.count, h = blockIdx.y, kh = h / (a.heads / a.kv_heads);
	const int t0 = blk * T, nt = min(T, sb.scount[b] - t0);
	if (nt <= 0) return;
	const int tid = threadIdx.x, w = tid >> 5, lane = tid & 31, i = 4 * lane;
	const size_t n = (size_t)sb.sstart[b] + t0 + w;
	float4 k = make_float4(0.f, 0.f, 0.f, 0.f), q = k, g = make_float4(1.f, 1.f, 1.f, 1.f); // tokens past the portion change nothing
	if (w < nt) {
		k = __ldg((const float4*)(a.k + (n * a.kv_heads + kh) * D + i)), q = __ldg((const float4*)(a.q + (n * a.kv_heads + kh) * D + i));
		float4* const dt = (float4*)(c.dt + (n * a.heads + h) * D + i);
		const float4 z = *dt;
		const bf16* bp = a.dt_bias + h * D + i;
		const float e = expf(ldf(a.a_log + h));
		g = make_float4(expf(-e * softplusf_(z.x + ldf(bp))), expf(-e * softplusf_(z.y + ldf(bp + 1))), expf(-e * softplusf_(z.z + ldf(bp + 2))), expf(-e * softplusf_(z.w + ldf(bp + 3))));
		*dt = g;
	}
	*(float4*)(ks[w] + i) = k, *(float4*)(qs[w] + i) = q, *(float4*)(gs[w] + i) = g;
	if (lane == 0) beta[w] = w < nt ? sigmoidf_(a.proj[n * a.ldp + a.bcol + h]) : 0.f;
	__syncthreads();
	// warp w: column s = w of A and B; its key decays on its way through the later tokens
	float v[2 * T];
#pragma unroll
	for (int t = 0; t < T; ++t) {
		v[t] = v[T + t] = 0.f;
		if (t < w) continue;
		const float4 kt = *(const float4*)(ks[t] + i), qt = *(const float4*)(qs[t] + i);
		if (t > w) {
			const float4 gt = *(const float4*)(gs[t] + i);
			k.x *= gt.x, k.y *= gt.y, k.z *= gt.z, k.w *= gt.w;
			v[t] = fmaf(kt.x, k.x, kt.y * k.y) + fmaf(kt.z, k.z, kt.w * k.w);
		}
		v[T + t] = fmaf(qt.x, k.x, qt.y * k.y) + fmaf(qt.z, k.z, qt.w * k.w);
	}
#pragma unroll
	for (int o = 16; o > 0; o >>= 1) { // lane l ends with the sum of value l
		const bool up = lane & o;
#pragma unroll
		for (int j = 0; j < o; ++j) {
			const float other = __shfl_xor_sync(0xffffffffu, up ? v[j] : v[j + o], o);
			v[j] = (up ? v[j + o] : v[j]) + other;
		}
	}
	(lane < T ? A[lane] : Bm[lane - T])[w] = v[0];
	__syncthreads();
	if (tid < T) { // column `tid` of X by forward substitution
		float x[T];
#pragma unroll
		for (int t = 0; t < T; ++t) {
			float r = t == tid ? 1.f : 0.f;
#pragma unroll
			for (int s = 0; s < t; ++s) r = fmaf(-A[t][s], x[s], r);
			x[t] = beta[t] * r;
			X[t][tid] = x[t];
		}
	}
	__syncthreads();
	if (tid < T * T) {
		const int t = tid / T, j = tid % T;
		float r = 0.f;
		for (int s = j; s <= t; ++s) r = fmaf(Bm[t][s], X[s][j], r);
		float* out = c.sys + ((size_t)(sb.sstart[b] / T + b + blk) * a.heads + h) * 2 * T * T + tid;
		out[0] = X[t][j], out[T * T] = r;
	}
}
// One CTA of four warps per (sequence, head, DELTA_VC value columns).  16 lanes share four columns and hold eight key channels of each.
__host__ __device__ constexpr int delta_block_floats() { return 3 * DELTA_BK * 128 + DELTA_BK * DELTA_VC + 2 * DELTA_BK * DELTA_BK; } // k, q, decay, v, X, B X
__host__ __device__ constexpr size_t delta_block_smem() { return (size_t)(2 * delta_block_floats() + 3 * DELTA_BK * DELTA_VC + 128) * sizeof(float); }
__global__ void __launch_bounds__(128) k_seq_delta_blocks(DeltaArgs a, DeltaBlocks c, SeqBatch sb) {
	pdl_enter(); // programmatic dependent launch: let the next kernel's launch overlap this one, then wait for the previous one
	constexpr int D = 128, T = DELTA_BK, VC = DELTA_VC, BUF = delta_block_floats();
	extern __shared__ __align__(16) float sm[];
	float* const rest = sm + 2 * BUF; // V - (K G) S, then
	float* const read = rest + T * VC; // (Q G) S and
	float* const corr = read + T * VC; // U, [token][column] each
	float* const last = corr + T * VC; // [D] G_T
	const int b = blockIdx.x, h = blockIdx.y, V = a.vdim, v0 = blockIdx.z * VC, kh = h / (a.heads / a.kv_heads);
	const int tid = threadIdx.x, part = tid & 15, cl = (tid >> 4) * 4;
	const int start = sb.sstart[b], cnt = sb.scount[b], nblk = (cnt + T - 1) / T;
	const bool live = v0 + cl < V; // (V is a multiple of 4) lanes past the last column run along on the last ones
	float* const Sg = a.state + ((size_t)sb.sslot[b] * a.heads + h) * D * V + (live ? v0 + cl : V - 4);
	auto channel = [&](int e) { return (e >> 2) * (D / 2) + 4 * part + (e & 3); }; // this lane's channel e of 8
	float2 S[4][4]; // [column][pair of channels]
#pragma unroll
	for (int p = 0; p < 4; ++p) {
		const float4 x = *(const float4*)(Sg + (size_t)channel(2 * p) * V), y = *(const float4*)(Sg + (size_t)channel(2 * p + 1) * V);
		S[0][p] = make_float2(x.x, y.x), S[1][p] = make_float2(x.y, y.y), S[2][p] = make_float2(x.z, y.z), S[3][p] = make_float2(x.w, y.w);
	}
	auto issue = [&](int blk) { // a block's inputs in 16-byte pieces; tokens past the portion: zero keys, queries and values, decays of one
		float* const to = sm + (blk & 1) * BUF;
		const int nt = min(T, cnt - blk * T);
		const size_t n0 = (size_t)start + blk * T;
		for (int e = tid; e < 3 * T * D / 4; e += 128) {
			const int which = e / (T * D / 4), t = e / (D / 4) % T, i = 4 * (e % (D / 4));
			float* const d = to + 4 * e;
			if (t < nt) cp_async16(d, which == 2 ? c.dt + ((n0 + t) * a.heads + h) * D + i : (which == 0 ? a.k : a.q) + ((n0 + t) * a.kv_heads + kh) * D + i);
			else *(float4*)d = which == 2 ? make_float4(1.f, 1.f, 1.f, 1.f) : make_float4(0.f, 0.f, 0.f, 0.f);
		}
		float* const vt = to + 3 * T * D;
		{
			const int t = tid / (VC / 4), i = 4 * (tid % (VC / 4)); // T * VC / 4 = 128 pieces
			if (t < nt && v0 + i < V) cp_async16(vt + 4 * tid, a.v + ((n0 + t) * a.heads + h) * V + v0 + i);
			else *(float4*)(vt + 4 * tid) = make_float4(0.f, 0.f, 0.f, 0.f);
		}
		cp_async16(vt + T * VC + 4 * tid, c.sys + ((size_t)(start / T + b + blk) * a.heads + h) * 2 * T * T + 4 * tid); // 2 T T / 4 = 128 pieces
		asm volatile("cp.async.commit_group;" ::: "memory");
	};
	static_assert(T * VC / 4 == 128 && 2 * T * T / 4 == 128 && D == 128, "one piece of v and of the system, and one channel, per thread");
	issue(0);
	for (int blk = 0; blk < nblk; ++blk) {
		float* const ks = sm + (blk & 1) * BUF;
		float *const qs = ks + T * D, *const gs = qs + T * D, *const vs = gs + T * D;
		const float *const X = vs + T * VC, *const BX = X + T * T;
		if (blk + 1 < nblk) {
			issue(blk + 1); // into the half that the block before has been done with since its last barrier
			asm volatile("cp.async.wait_group 1;" ::: "memory");
		} else asm volatile("cp.async.wait_group 0;" ::: "memory");
		__syncthreads();
		{ // in place, a channel per thread: decay -> k G, q -> q G, k -> D(T, s) k
			float g[T], G = 1.f;
#pragma unroll
			for (int t = 0; t < T; ++t) g[t] = gs[t * D + tid];
#pragma unroll
			for (int t = 0; t < T; ++t) G *= g[t], gs[t * D + tid] = ks[t * D + tid] * G, qs[t * D + tid] *= G;
			last[tid] = G, G = 1.f;
#pragma unroll
			for (int t = T - 1; t >= 0; --t) ks[t * D + tid] *= G, G *= g[t];
		}
		__syncthreads();
#pragma unroll 1
		for (int t0 = 0; t0 < T; t0 += 4) { // (K G) S and (Q G) S, four tokens' shares at a time
			float r[32]; // [token][K, Q][column]
#pragma unroll
			for (int x = 0; x < 8; ++x) {
				const float* at = (x & 1 ? qs : gs) + (t0 + x / 2) * D + 4 * part;
				const float4 lo = *(const float4*)at, hi = *(const float4*)(at + D / 2);
				const float2 y[4] = {make_float2(lo.x, lo.y), make_float2(lo.z, lo.w), make_float2(hi.x, hi.y), make_float2(hi.z, hi.w)};
#pragma unroll
				for (int j = 0; j < 4; ++j) {
					float2 z = __fmul2_rn(y[0], S[j][0]);
#pragma unroll
					for (int p = 1; p < 4; ++p) z = __ffma2_rn(y[p], S[j][p], z);
					r[4 * x + j] = z.x + z.y;
				}
			}
#pragma unroll
			for (int o = 8, left = 16; o > 0; o >>= 1, left >>= 1) { // over the 16 lanes, each keeping half of the values: lane `part` ends with two
				const bool up = part & o;
#pragma unroll
				for (int i = 0; i < left; ++i) {
					const float other = __shfl_xor_sync(0xffffffffu, up ? r[i] : r[i + left], o);
					r[i] = (up ? r[i + left] : r[i]) + other;
				}
			}
			const int at = (t0 + (part >> 2)) * VC + cl + 2 * (part & 1);
			if (part & 2) *(float2*)(read + at) = make_float2(r[0], r[1]);
			else {
				const float2 v = *(const float2*)(vs + at);
				*(float2*)(rest + at) = make_float2(v.x - r[0], v.y - r[1]);
			}
		}
		__syncthreads();
		{ // four tokens of one column per thread: U and the read-outs
			const int col = tid & (VC - 1), r0 = 4 * (tid / VC);
			float u[4] = {}, o[4];
#pragma unroll
			for (int j = 0; j < 4; ++j) o[j] = read[(r0 + j) * VC + col];
			// both matrices are lower triangular; on the diagonal their zeros are left out: times a later token's NaN or infinity they would not be zero
			auto four = [&](int s0, auto diagonal) {
				float x[4];
#pragma unroll
				for (int i = 0; i < 4; ++i) x[i] = rest[(s0 + i) * VC + col];
#pragma unroll
				for (int j = 0; j < 4; ++j) {
					const float4 p4 = *(const float4*)(X + (r0 + j) * T + s0), q4 = *(const float4*)(BX + (r0 + j) * T + s0);
					const float p[4] = {p4.x, p4.y, p4.z, p4.w}, q[4] = {q4.x, q4.y, q4.z, q4.w};
#pragma unroll
					for (int i = 0; i < 4; ++i)
						if (!decltype(diagonal)::value || i <= j) u[j] = fmaf(p[i], x[i], u[j]), o[j] = fmaf(q[i], x[i], o[j]);
				}
			};
#pragma unroll 1
			for (int s0 = 0; s0 < r0; s0 += 4) four(s0, std::false_type{});
			four(r0, std::true_type{});
#pragma unroll
			for (int j = 0; j < 4; ++j) {
				corr[(r0 + j) * VC + col] = u[j];
				const int t = blk * T + r0 + j;
				if (t < cnt && v0 + col < V) a.o[((size_t)(start + t) * a.heads + h) * V + v0 + col] = o[j];
			}
		}
		__syncthreads();
		{
			const float4 lo = *(const float4*)(last + 4 * part), hi = *(const float4*)(last + D / 2 + 4 * part);
			const float2 G[4] = {make_float2(lo.x, lo.y), make_float2(lo.z, lo.w), make_float2(hi.x, hi.y), make_float2(hi.z, hi.w)};
#pragma unroll
			for (int j = 0; j < 4; ++j)
#pragma unroll
				for (int p = 0; p < 4; ++p) S[j][p] = __fmul2_rn(S[j][p], G[p]);
		}
#pragma unroll 4
		for (int t = 0; t < T; ++t) {
			const float4 lo = *(const float4*)(ks + t * D + 4 * part), hi = *(const float4*)(ks + t * D + D / 2 + 4 * part), u4 = *(const float4*)(corr + t * VC + cl);
			const float2 y[4] = {make_float2(lo.x, lo.y), make_float2(lo.z, lo.w), make_float2(hi.x, hi.y), make_float2(hi.z, hi.w)};
			const float u[4] = {u4.x, u4.y, u4.z, u4.w};
#pragma unroll
			for (int j = 0; j < 4; ++j)
#pragma unroll
				for (int p = 0; p < 4; ++p) S[j][p] = __ffma2_rn(y[p], make_float2(u[j], u[j]), S[j][p]);
		}
		__syncthreads(); // the block's buffer, its corrections and G_T have been read
	}
	if (live) {
#pragma unroll
		for (int p = 0; p < 4; ++p) {
			*(float4*)(Sg + (size_t)channel(2 * p) * V) = make_float4(S[0][p].x, S[1][p].x, S[2][p].x, S[3][p].x);
			*(float4*)(Sg + (size_t)channel(2 * p + 1) * V) = make_float4(S[0][p].y, S[1][p].y, S[2][p].y, S[3][p].y);
		}
	}
}
// read-out: o / rms(o) (per head) * w * sigmoid(gate); one warp per (token, head)
// (the gate goes through a sigmoid, or through SiLU when silu_gate is set; it is read at gate[token * ldg + head * vdim + i])
template <typename AT>
__global__ void k_seq_delta_out(AT* out, const float* o, const float* gate, int ldg, const bf16* w, int N, int heads, int vdim, float eps, int silu_gate) {
	pdl_enter(); // programmatic dependent launch: let the next kernel's launch overlap this one, then wait for the previous one
	const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
	const size_t u = (size_t)blockIdx.x * (blockDim.x >> 5) + warp;
	if (u >= (size_t)N * heads) return;
	const float* src = o + u * vdim;
	float ss = 0.f;
	for (int i = lane; i < vdim; i += 32) ss += src[i] * src[i];
	ss = warp_sum(ss);
	const float r = 1.f / sqrtf(ss / (float)vdim + eps);
	const float* gp = gate + (u / heads) * (size_t)ldg + (u % heads) * (size_t)vdim;
	for (int i = lane; i < vdim; i += 32) {
		const float g = gp[i], sg = sigmoidf_(g);
		out[u * vdim + i] = to_act<AT>(src[i] * r * ldf(w + i) * (silu_gate ? g * sg : sg));
	}
}

// ---------------------------------------------------------------- gated linear attention
// Per (sequence, head): S [dim][vdim] fp32;  per token  S <- diag(a) S + k v^T,  o = S^T q * qscale  with one decay a per key
// channel (formed in fp32 by the decay projection's epilogue, EPI_DECAY).  q, k, v are columns of the stacked projection (row
// stride ldp).
struct GlaArgs {
	const float* proj;
	int ldp, qcol, kcol, vcol;
	const float* decay;  // [N][heads*dim]
	float qscale;
	float* state;        // [slots][heads][vdim][ldstate]: a value column's key channels side by side (channels past dim stay zero)
	int ldstate;
	float* o;            // [N][heads*vdim]
	int heads, dim, vdim;
	int vec;             // rows, columns and bases are 16-byte aligned: tokens are staged with 16-byte copies instead of 4-byte ones
};
// One CTA of 128 threads per (sequence, head, 128 / P value columns).  The state sits in registers: P lanes share a value column,
// each holding R of its key channels (P = 4, 8 or 16: the host takes more lanes per column when sequences x heads alone would
// leave SMs idle, since per token a warp issues ~3 R arithmetic instructions and that, not memory, bounds a long prompt).
// Tokens are staged GLA_TB at a time into a double buffer with asynchronous copies (k, q and the decay in P segments padded by 4
// floats, so that the lanes of a column read different banks as float4; the CTA's values of v), so a block's tokens are applied
// without a barrier between them -- log2(P) shuffles fold a column's read-out -- while the next block travels.  Read-outs
// leave through shared memory, one coalesced store per block.
#define GLA_TB 16
template <int R, int P>
__global__ void __launch_bounds__(128) k_seq_gla_scan(GlaArgs a, SeqBatch sb) {
	pdl_enter(); // programmatic dependent launch: let the next kernel's launch overlap this one, then wait for the previous one
	constexpr int QP = R + 4, VC = 128 / P, TOK = 3 * P * QP + VC;
	extern __shared__ __align__(16) float sm[];
	float* const buf0 = sm;
	float* const obuf = sm + 2 * GLA_TB * TOK; // [2][GLA_TB][VC]
	const int b = blockIdx.x, h = blockIdx.y, D = a.dim, V = a.vdim, v0 = blockIdx.z * VC;
	const int tid = threadIdx.x, part = tid % P, cl = tid / P;
	const bool live = v0 + cl < V;
	const int start = sb.sstart[b], cnt = sb.scount[b], nblk = (cnt + GLA_TB - 1) / GLA_TB;
	// the padding (channels past dim, columns past vdim) is never copied over: zero what this step will use, once
	for (int i = tid; i < min(cnt, 2 * GLA_TB) * TOK; i += 128) sm[i] = 0.f;
	float S[R];
	float* Sg = a.state + (((size_t)sb.sslot[b] * a.heads + h) * V + min(v0 + cl, V - 1)) * a.ldstate + part * R;
#pragma unroll
	for (int i = 0; i < R; i += 4) {
		const float4 t = *(const float4*)(Sg + i);
		S[i] = t.x, S[i + 1] = t.y, S[i + 2] = t.z, S[i + 3] = t.w;
	}
	// 16-byte staging: a thread copies the same (at most two) chunks of every token, so where they come from and go to is worked out once
	const float* vsrc[2] = {nullptr, nullptr};
	long vstride[2] = {0, 0};
	int vdst[2] = {0, 0};
	if (a.vec) {
		const int dc = D / 4;
#pragma unroll
		for (int r = 0; r < 2; ++r) {
			const int c = tid + r * 128;
			if (c < 3 * dc) {
				const int sgm = c / dc, i = 4 * (c % dc);
				vsrc[r] = sgm == 2 ? a.decay + ((size_t)start * a.heads + h) * D + i : a.proj + (size_t)start * a.ldp + (sgm == 0 ? a.kcol : a.qcol) + h * D + i;
				vstride[r] = sgm == 2 ? (long)a.heads * D : a.ldp;
				vdst[r] = sgm * P * QP + (i / R) * QP + i % R;
			} else if (c < 3 * dc + VC / 4 && v0 + 4 * (c - 3 * dc) < V) {
				const int i = 4 * (c - 3 * dc);
				vsrc[r] = a.proj + (size_t)start * a.ldp + a.vcol + h * V + v0 + i, vstride[r] = a.ldp, vdst[r] = 3 * P * QP + i;
			}
		}
	}
	__syncthreads();
	auto issue = [&](int blk) {
		float* dst = buf0 + (blk & 1) * GLA_TB * TOK;
		const int t0 = blk * GLA_TB, nt = min(GLA_TB, cnt - t0);
		if (a.vec) {
#pragma unroll
			for (int r = 0; r < 2; ++r)
				if (vsrc[r])
					for (int tt = 0; tt < nt; ++tt) cp_async16(dst + tt * TOK + vdst[r], vsrc[r] + (t0 + tt) * vstride[r]);
		} else {
			const int per = 3 * D + VC;
			for (int e = tid; e < nt * per; e += 128) {
				const int tt = e / per, c = e % per;
				const float* row = a.proj + (size_t)(start + t0 + tt) * a.ldp;
				if (c < 3 * D) {
					const int sgm = c / D, i = c % D;
					const float* src = sgm == 0 ? row + a.kcol + h * D + i : sgm == 1 ? row + a.qcol + h * D + i : a.decay + ((size_t)(start + t0 + tt) * a.heads + h) * D + i;
					cp_async4(dst + tt * TOK + sgm * P * QP + (i / R) * QP + i % R, src);
				} else {
					const int i = c - 3 * D;
					if (v0 + i < V) cp_async4(dst + tt * TOK + 3 * P * QP + i, row + a.vcol + h * V + v0 + i);
				}
			}
		}
		asm volatile("cp.async.commit_group;" ::: "memory");
	};
	auto write_out = [&](int blk) { // the read-outs of a finished block: consecutive threads, consecutive columns
		const int nt = min(GLA_TB, cnt - blk * GLA_TB);
		const float* ob = obuf + (blk & 1) * GLA_TB * VC;
		for (int e = tid; e < nt * VC; e += 128) {
			const int tt = e / VC, c = e % VC;
			if (v0 + c < V) a.o[((size_t)(start + blk * GLA_TB + tt) * a.heads + h) * V + v0 + c] = ob[e];
		}
	};
	issue(0);
	for (int blk = 0; blk < nblk; ++blk) {
		if (blk + 1 < nblk) {
			issue(blk + 1);
			asm volatile("cp.async.wait_group 1;" ::: "memory");
		} else {
			asm volatile("cp.async.wait_group 0;" ::: "memory");
		}
		__syncthreads();
		if (blk > 0) write_out(blk - 1);
		const float* __restrict__ cur = buf0 + (blk & 1) * GLA_TB * TOK;
		float* __restrict__ ob = obuf + (blk & 1) * GLA_TB * VC;
		const int nt = min(GLA_TB, cnt - blk * GLA_TB);
		// the block's tokens, unrolled: each lane's share of a read-out stays in a register until the block is done, then the shares are
		// folded for all tokens at once -- independent shuffles that overlap, instead of one dependent chain per token
		float oacc[GLA_TB];
		auto apply = [&](int tt) { // one token: decay, write, this lane's share of the read-out
			const float* tk = cur + tt * TOK;
			const float4 *kp = (const float4*)(tk + part * QP), *qp = (const float4*)(tk + P * QP + part * QP), *gp = (const float4*)(tk + 2 * P * QP + part * QP);
			const float v = tk[3 * P * QP + cl];
			float o0 = 0.f, o1 = 0.f;
#pragma unroll
			for (int i = 0; i < R / 4; ++i) {
				const float4 g4 = gp[i], k4 = kp[i], q4 = qp[i];
				S[4 * i] = fmaf(g4.x, S[4 * i], k4.x * v), S[4 * i + 1] = fmaf(g4.y, S[4 * i + 1], k4.y * v);
				S[4 * i + 2] = fmaf(g4.z, S[4 * i + 2], k4.z * v), S[4 * i + 3] = fmaf(g4.w, S[4 * i + 3], k4.w * v);
				o0 = fmaf(S[4 * i], q4.x, o0), o1 = fmaf(S[4 * i + 1], q4.y, o1), o0 = fmaf(S[4 * i + 2], q4.z, o0), o1 = fmaf(S[4 * i + 3], q4.w, o1);
			}
			return o0 + o1;
		};
		if (nt == GLA_TB) { // a full block has no branch between its tokens: the loads of later tokens move up past the arithmetic of earlier ones
#pragma unroll
			for (int tt = 0; tt < GLA_TB; ++tt) oacc[tt] = apply(tt);
		} else {
#pragma unroll
			for (int tt = 0; tt < GLA_TB; ++tt) oacc[tt] = tt < nt ? apply(tt) : 0.f;
		}
#pragma unroll
		for (int w = 1; w < P; w <<= 1)
#pragma unroll
			for (int tt = 0; tt < GLA_TB; ++tt) oacc[tt] += __shfl_xor_sync(0xffffffffu, oacc[tt], w);
#pragma unroll
		for (int tt = 0; tt < GLA_TB; ++tt)
			if (tt % P == part) ob[tt * VC + cl] = oacc[tt] * a.qscale; // every lane of a column holds the sums: the lanes share the stores out
		__syncthreads(); // this block's buffer may be refilled and its read-outs are complete
	}
	write_out(nblk - 1);
	if (live) {
#pragma unroll
		for (int i = 0; i < R; i += 4) *(float4*)(Sg + i) = make_float4(S[i], S[i + 1], S[i + 2], S[i + 3]);
	}
}

// One token per sequence (decode): the recurrence is a stream over the states.  A warp takes COLS value columns, a lane 4 NV of their key channels, so a column
// travels as whole 512-byte lines and all of a warp's columns are on their way at once; the read-outs of its columns are transposed and
// folded together.  (The scan's lane holds R channels of one column: 16 bytes of 32 lines per request, 19 us a layer of 16 sequences x 16 heads of
// 128 x 128, whose 33.5 MB take 5.1 at the memory's rate.)
template <int NV>
__global__ void __launch_bounds__(128) k_seq_gla_step(GlaArgs a, SeqBatch sb) {
	pdl_enter(); // programmatic dependent launch: let the next kernel's launch overlap this one, then wait for the previous one
	constexpr int COLS = 16 / NV;
	const int b = blockIdx.x, h = blockIdx.y, lane = threadIdx.x & 31, v0 = (blockIdx.z * 4 + (threadIdx.x >> 5)) * COLS, n = sb.sstart[b];
	if (v0 >= a.vdim) return;
	float* const Sg = a.state + (((size_t)sb.sslot[b] * a.heads + h) * a.vdim + v0) * a.ldstate;
	const float* const row = a.proj + (size_t)n * a.ldp;
	const float4 none = make_float4(0.f, 0.f, 0.f, 0.f);
	float4 S[COLS][NV], k4[NV], q4[NV], g4[NV];
#pragma unroll
	for (int i = 0; i < COLS; ++i)
#pragma unroll
		for (int j = 0; j < NV; ++j) S[i][j] = v0 + i < a.vdim && 4 * lane + 128 * j < a.dim ? *(const float4*)(Sg + (size_t)i * a.ldstate + 4 * lane + 128 * j) : none;
#pragma unroll
	for (int j = 0; j < NV; ++j) {
		const int c = 4 * lane + 128 * j;
		const bool in = c < a.dim;
		k4[j] = in ? *(const float4*)(row + a.kcol + h * a.dim + c) : none, q4[j] = in ? *(const float4*)(row + a.qcol + h * a.dim + c) : none;
		g4[j] = in ? *(const float4*)(a.decay + ((size_t)n * a.heads + h) * a.dim + c) : none;
	}
	const float mine = lane < COLS && v0 + lane < a.vdim ? row[a.vcol + h * a.vdim + v0 + lane] : 0.f;
	float o[COLS];
#pragma unroll
	for (int i = 0; i < COLS; ++i) {
		const float v = __shfl_sync(0xffffffffu, mine, i);
		float o0 = 0.f, o1 = 0.f;
#pragma unroll
		for (int j = 0; j < NV; ++j) {
			float4& t = S[i][j];
			t.x = fmaf(g4[j].x, t.x, k4[j].x * v), t.y = fmaf(g4[j].y, t.y, k4[j].y * v), t.z = fmaf(g4[j].z, t.z, k4[j].z * v), t.w = fmaf(g4[j].w, t.w, k4[j].w * v);
			o0 = fmaf(t.x, q4[j].x, o0), o1 = fmaf(t.y, q4[j].y, o1), o0 = fmaf(t.z, q4[j].z, o0), o1 = fmaf(t.w, q4[j].w, o1);
			if (v0 + i < a.vdim && 4 * lane + 128 * j < a.dim) *(float4*)(Sg + (size_t)i * a.ldstate + 4 * lane + 128 * j) = t;
		}
		o[i] = o0 + o1;
	}
	int col = 0; // of this lane in the end
#pragma unroll
	for (int half = COLS / 2, m = 16; half >= 1; half >>= 1, m >>= 1) {
		const bool up = lane & m;
#pragma unroll
		for (int i = 0; i < half; ++i) {
			const float send = up ? o[i] : o[i + half];
			o[i] = (up ? o[i + half] : o[i]) + __shfl_xor_sync(0xffffffffu, send, m);
		}
		col += up ? half : 0;
	}
#pragma unroll
	for (int m = 16 / COLS; m >= 1; m >>= 1) o[0] += __shfl_xor_sync(0xffffffffu, o[0], m);
	if (!(lane & (32 / COLS - 1)) && v0 + col < a.vdim) a.o[((size_t)n * a.heads + h) * a.vdim + v0 + col] = o[0] * a.qscale;
}

// The same recurrence for long portions, cut into chunks of tokens that run side by side: (1) k_seq_gla_local forms what a chunk adds to a zero
// state and the product of its decays, (2) k_seq_gla_starts walks a state element through the chunks, leaving every chunk's first state in place
// of what it adds, and updates the slot's state, (3) k_seq_gla_apply runs each chunk's tokens from there for the read-outs.
// k_seq_gla_scan is a chain over all tokens on as many SMs as sequences x heads x columns give (2048 tokens of 16 heads of 128 x 128: 469 us,
// 230 ns a token whatever the arithmetic); here (1) and (3) fill the SMs: 148 us, each launch alone with cold caches 47 + 18 + 94.
struct GlaChunks {
	float* add;  // [B][count][heads][vdim][dim]: what a chunk adds, then the state it starts from
	float* keep; // [B][count][heads][dim]: product of the chunk's decays
	int len, count;
};
// (1): S[v][d] = sum over tokens of v (x) k scaled by the decays that follow, a block of GLC_TB tokens at a time: inside a block the keys carry the
// product of the later tokens' decays (nothing is divided), so that an element costs one FMA per token and one multiplication per block.
// One CTA per (chunk, head, 128 value columns), 2 D threads of 8 x 8 elements each, multiplied in pairs (an FMA pipe is as fast on single ones, but pairs
// leave every second issue slot to the loads).  Blocks travel two ahead by asynchronous copies, and a block's keys are scaled while the one before is
// multiplied.
#define GLC_TB 8
#define GLC_STAGES 4
__host__ __device__ constexpr int glc_tok(int D) { return 2 * D + 128; } // k, decay, v
__host__ __device__ constexpr size_t glc_smem(int D) { return ((size_t)GLC_STAGES * GLC_TB * glc_tok(D) + 2 * (GLC_TB + 1) * D) * sizeof(float); }
template <int D>
__global__ void __launch_bounds__(2 * D, 256 / D) k_seq_gla_local(GlaArgs a, GlaChunks c, SeqBatch sb) {
	pdl_enter(); // programmatic dependent launch: let the next kernel's launch overlap this one, then wait for the previous one
	constexpr int TX = D / 8, TOK = glc_tok(D), ITEMS = TOK / 4, ROUNDS = (ITEMS + 2 * D - 1) / (2 * D);
	extern __shared__ __align__(16) float sm[];
	float* const scaled = sm + GLC_STAGES * GLC_TB * TOK; // [2][GLC_TB scaled keys, then the block's decays][D]
	const int b = blockIdx.x / c.count, ch = blockIdx.x % c.count, h = blockIdx.y, v0 = blockIdx.z * 128, V = a.vdim;
	const int t0 = ch * c.len, nt = min(c.len, sb.scount[b] - t0);
	if (nt <= 0) return;
	const int tid = threadIdx.x, tx = tid % TX, ty = tid / TX, nblk = (nt + GLC_TB - 1) / GLC_TB;
	const size_t first = (size_t)sb.sstart[b] + t0;
	// a thread copies the same 16-byte items of every token; columns past the last one are zero
	const float* src[ROUNDS];
	long stride[ROUNDS];
#pragma unroll
	for (int r = 0; r < ROUNDS; ++r) {
		const int i = 4 * (tid + r * 2 * D);
		src[r] = nullptr, stride[r] = a.ldp;
		if (i < D) src[r] = a.proj + first * a.ldp + a.kcol + h * D + i;
		else if (i < 2 * D) src[r] = a.decay + (first * a.heads + h) * D + i - D, stride[r] = (long)a.heads * D;
		else if (i < TOK && v0 + i - 2 * D < V) src[r] = a.proj + first * a.ldp + a.vcol + h * V + v0 + i - 2 * D;
		else if (i < TOK)
			for (int t = 0; t < GLC_STAGES * GLC_TB; ++t) *(float4*)(sm + t * TOK + i) = make_float4(0.f, 0.f, 0.f, 0.f);
	}
	auto issue = [&](int blk) {
		const int n = min(GLC_TB, nt - blk * GLC_TB);
		float* dst = sm + blk % GLC_STAGES * GLC_TB * TOK;
#pragma unroll
		for (int r = 0; r < ROUNDS; ++r)
			if (src[r])
				for (int t = 0; t < n; ++t) cp_async16(dst + t * TOK + 4 * (tid + r * 2 * D), src[r] + (blk * GLC_TB + t) * stride[r]);
		asm volatile("cp.async.commit_group;" ::: "memory"); // (an empty group past the last block)
	};
	float all = 1.f; // threads that scale keys: the decays of the chunk so far
	auto scale = [&](int blk) {
		const int n = min(GLC_TB, nt - blk * GLC_TB);
		const float* raw = sm + blk % GLC_STAGES * GLC_TB * TOK + tid;
		float* to = scaled + (blk & 1) * (GLC_TB + 1) * D + tid;
		float w = 1.f;
#pragma unroll
		for (int t = GLC_TB - 1; t >= 0; --t) {
			to[t * D] = t < n ? raw[t * TOK] * w : 0.f;
			if (t < n) w *= raw[t * TOK + D];
		}
		to[GLC_TB * D] = w, all *= w;
	};
	float2 S[8][4] = {}; // [value column][pair of key channels], both as two groups of four: 4 ty + {0, 64}, 4 tx + {0, D / 2}
	issue(0), issue(1), issue(2);
	asm volatile("cp.async.wait_group 2;" ::: "memory");
	__syncthreads();
	if (tid < D) scale(0);
	for (int blk = 0; blk < nblk; ++blk) {
		asm volatile("cp.async.wait_group 1;" ::: "memory");
		__syncthreads(); // block blk + 1 is there, block blk scaled, block blk - 1 done with
		issue(blk + 3);
		if (tid < D && blk + 1 < nblk) scale(blk + 1);
		const float* kk = scaled + (blk & 1) * (GLC_TB + 1) * D + 4 * tx;
		const float* vv = sm + blk % GLC_STAGES * GLC_TB * TOK + 2 * D + 4 * ty;
		float2 k[4];
		auto row = [&](int t) {
			const float4 x = *(const float4*)(kk + t * D), y = *(const float4*)(kk + t * D + D / 2);
			k[0] = make_float2(x.x, x.y), k[1] = make_float2(x.z, x.w), k[2] = make_float2(y.x, y.y), k[3] = make_float2(y.z, y.w);
		};
		row(GLC_TB);
#pragma unroll
		for (int j = 0; j < 8; ++j)
#pragma unroll
			for (int i = 0; i < 4; ++i) S[j][i] = __fmul2_rn(S[j][i], k[i]);
		const int n = min(GLC_TB, nt - blk * GLC_TB);
#pragma unroll 4
		for (int t = 0; t < n; ++t) {
			row(t);
			const float4 x = *(const float4*)(vv + t * TOK), y = *(const float4*)(vv + t * TOK + 64);
			const float v[8] = {x.x, x.y, x.z, x.w, y.x, y.y, y.z, y.w};
#pragma unroll
			for (int j = 0; j < 8; ++j)
#pragma unroll
				for (int i = 0; i < 4; ++i) S[j][i] = __ffma2_rn(make_float2(v[j], v[j]), k[i], S[j][i]);
		}
	}
	const size_t unit = ((size_t)b * c.count + ch) * a.heads + h;
#pragma unroll
	for (int j = 0; j < 8; ++j) {
		const int v = v0 + (j >> 2) * 64 + 4 * ty + (j & 3);
		if (v >= V) continue;
		float* o = c.add + (unit * V + v) * D;
		*(float4*)(o + 4 * tx) = make_float4(S[j][0].x, S[j][0].y, S[j][1].x, S[j][1].y);
		*(float4*)(o + D / 2 + 4 * tx) = make_float4(S[j][2].x, S[j][2].y, S[j][3].x, S[j][3].y);
	}
	if (tid < D && blockIdx.z == 0) c.keep[unit * D + tid] = all;
}
// (2): four key channels of one value column per thread
template <int D>
__global__ void __launch_bounds__(128) k_seq_gla_starts(GlaArgs a, GlaChunks c, SeqBatch sb) {
	pdl_enter(); // programmatic dependent launch: let the next kernel's launch overlap this one, then wait for the previous one
	const int b = blockIdx.y, e = blockIdx.x * 128 + threadIdx.x, d = e % (D / 4) * 4, hv = e / (D / 4);
	if (hv >= a.heads * a.vdim) return;
	const int h = hv / a.vdim, nc = (sb.scount[b] + c.len - 1) / c.len;
	float4* const st = (float4*)(a.state + ((size_t)sb.sslot[b] * a.heads * a.vdim + hv) * a.ldstate + d);
	float4* ap = (float4*)(c.add + ((size_t)b * c.count * a.heads * a.vdim + hv) * D + d);
	const float4* kp = (const float4*)(c.keep + ((size_t)b * c.count * a.heads + h) * D + d);
	const size_t as = (size_t)a.heads * a.vdim * D / 4, ks = (size_t)a.heads * D / 4;
	float4 s = *st;
	for (int i0 = 0; i0 < nc; i0 += 4, ap += 4 * as, kp += 4 * ks) {
		float4 x[4], k[4];
#pragma unroll
		for (int i = 0; i < 4; ++i)
			if (i0 + i < nc) x[i] = ap[i * as], k[i] = kp[i * ks];
#pragma unroll
		for (int i = 0; i < 4; ++i)
			if (i0 + i < nc) {
				ap[i * as] = s;
				s = make_float4(fmaf(k[i].x, s.x, x[i].x), fmaf(k[i].y, s.y, x[i].y), fmaf(k[i].z, s.z, x[i].z), fmaf(k[i].w, s.w, x[i].w));
			}
	}
	*st = s;
}
// (3): one CTA of four warps per (chunk, head, gla_cols(D) value columns); D / 8 lanes share four columns and hold eight key channels of each, so that
// the seven 16-byte shared-memory reads of a token serve 96 multiplications and multiply-adds per lane (k_seq_gla_scan: six for 24).  Bound by those: the
// FMA pipe is at two thirds, and pairs of them (half as many instructions, the same pipe time) are as fast as single ones, 94 and 96 us.
#define GLA_TC 8
__host__ __device__ constexpr int gla_cols(int D) { return 128 / (D / 8) * 4; }
template <int D>
__global__ void __launch_bounds__(128, 4) k_seq_gla_apply(GlaArgs a, GlaChunks c, SeqBatch sb) {
	pdl_enter(); // programmatic dependent launch: let the next kernel's launch overlap this one, then wait for the previous one
	constexpr int P = D / 8, VC = gla_cols(D), TOK = 3 * D + VC, ITEMS = TOK / 4;
	__shared__ __align__(16) float sm[2][GLA_TC * TOK]; // per token k, q, decay, v
	const int b = blockIdx.x / c.count, ch = blockIdx.x % c.count, h = blockIdx.y, V = a.vdim, v0 = blockIdx.z * VC;
	const int t0 = ch * c.len, nt = min(c.len, sb.scount[b] - t0);
	if (nt <= 0) return;
	const int tid = threadIdx.x, part = tid % P, cl = tid / P * 4;
	const bool live = v0 + cl < V; // (V is a multiple of 4) lanes past the last column run along on the last group's state
	const size_t first = (size_t)sb.sstart[b] + t0;
	float2 S[4][4]; // [value column][pairs of the key channels 4 part + {0..3}, D / 2 + 4 part + {0..3}]
	const float* Sg = c.add + ((((size_t)b * c.count + ch) * a.heads + h) * V + (live ? v0 + cl : V - 4)) * D + 4 * part;
#pragma unroll
	for (int j = 0; j < 4; ++j) {
		const float4 x = *(const float4*)(Sg + j * D), y = *(const float4*)(Sg + j * D + D / 2);
		S[j][0] = make_float2(x.x, x.y), S[j][1] = make_float2(x.z, x.w), S[j][2] = make_float2(y.x, y.y), S[j][3] = make_float2(y.z, y.w);
	}
	// a thread copies the same (at most two) 16-byte items of every token
	const float* src[2] = {nullptr, nullptr};
	long stride[2] = {0, 0};
#pragma unroll
	for (int r = 0; r < 2; ++r) {
		const int i = 4 * (tid + r * 128);
		if (tid + r * 128 >= ITEMS) continue;
		if (i < 2 * D) src[r] = a.proj + first * a.ldp + (i < D ? a.kcol + i : a.qcol + i - D) + h * D, stride[r] = a.ldp;
		else if (i < 3 * D) src[r] = a.decay + (first * a.heads + h) * D + i - 2 * D, stride[r] = (long)a.heads * D;
		else if (v0 + i - 3 * D < V) src[r] = a.proj + first * a.ldp + a.vcol + h * V + v0 + i - 3 * D, stride[r] = a.ldp;
	}
	auto issue = [&](int blk) {
		const int n = min(GLA_TC, nt - blk * GLA_TC);
#pragma unroll
		for (int r = 0; r < 2; ++r)
			if (src[r])
				for (int t = 0; t < n; ++t) cp_async16(sm[blk & 1] + t * TOK + 4 * (tid + r * 128), src[r] + (blk * GLA_TC + t) * stride[r]);
		asm volatile("cp.async.commit_group;" ::: "memory");
	};
	const int nblk = (nt + GLA_TC - 1) / GLA_TC;
	issue(0);
	for (int blk = 0; blk < nblk; ++blk) {
		if (blk + 1 < nblk) {
			issue(blk + 1);
			asm volatile("cp.async.wait_group 1;" ::: "memory");
		} else asm volatile("cp.async.wait_group 0;" ::: "memory");
		__syncthreads();
		const float* __restrict__ cur = sm[blk & 1];
		const int n = min(GLA_TC, nt - blk * GLA_TC);
		float o[4 * GLA_TC]; // this lane's shares of the read-outs [token][column]
		auto apply = [&](int t) {
			const float* tk = cur + t * TOK;
			const float4 va = *(const float4*)(tk + 3 * D + cl);
			const float v[4] = {va.x, va.y, va.z, va.w};
			float2 r[4] = {};
#pragma unroll
			for (int half = 0; half < 2; ++half) {
				const float* at = tk + half * (D / 2) + 4 * part;
				const float4 k4 = *(const float4*)at, q4 = *(const float4*)(at + D), g4 = *(const float4*)(at + 2 * D);
				const float2 k[2] = {make_float2(k4.x, k4.y), make_float2(k4.z, k4.w)}, q[2] = {make_float2(q4.x, q4.y), make_float2(q4.z, q4.w)}, g[2] = {make_float2(g4.x, g4.y), make_float2(g4.z, g4.w)};
#pragma unroll
				for (int j = 0; j < 4; ++j)
#pragma unroll
					for (int i = 0; i < 2; ++i) {
						float2& s = S[j][2 * half + i];
						s = __ffma2_rn(g[i], s, __fmul2_rn(k[i], make_float2(v[j], v[j]))), r[j] = __ffma2_rn(s, q[i], r[j]);
					}
			}
#pragma unroll
			for (int j = 0; j < 4; ++j) o[4 * t + j] = r[j].x + r[j].y;
		};
		if (n == GLA_TC) {
#pragma unroll
			for (int t = 0; t < GLA_TC; ++t) apply(t);
		} else {
#pragma unroll
			for (int t = 0; t < GLA_TC; ++t) {
				if (t < n) apply(t);
				else o[4 * t] = o[4 * t + 1] = o[4 * t + 2] = o[4 * t + 3] = 0.f;
			}
		}
		// folded over the column's lanes, each keeping half of the values at every step: lane `part` ends with values E part .. E part + E - 1
		constexpr int E = 4 * GLA_TC / P;
#pragma unroll
		for (int w = P / 2, left = 2 * GLA_TC; w > 0; w >>= 1, left >>= 1) {
			const bool up = part & w;
#pragma unroll
			for (int i = 0; i < left; ++i) {
				const float other = __shfl_xor_sync(0xffffffffu, up ? o[i] : o[i + left], w);
				o[i] = (up ? o[i + left] : o[i]) + other;
			}
		}
		const int t = part * E / 4;
		if (live && t < n) {
			float* dst = a.o + ((first + blk * GLA_TC + t) * a.heads + h) * V + v0 + cl + part * E % 4;
			if constexpr (E == 2) *(float2*)dst = make_float2(o[0] * a.qscale, o[1] * a.qscale);
			else *(float4*)dst = make_float4(o[0] * a.qscale, o[1] * a.qscale, o[2] * a.qscale, o[3] * a.qscale);
		}
		__syncthreads(); // this half of the buffer may be filled again
	}
}

// ---------------------------------------------------------------- query / key preparation of grouped-query attention
// One CTA per token (or, with norms per head, several: gridDim.y slices of the heads), on the stacked (biased) projection [q | k | v | ...]: an RMS norm over the WHOLE query projection and one over
// the whole key projection (all heads at once, weights qw / kw; null: no norm), then the first rot_dims channels of every head turn
// by the token's position (channel i with channel i + rot_dims/2, angle = position * freq[i], cos and sin times `mag`); queries go
// to an activation-independent fp32 matrix, keys and values to their cache rows.  Angles are formed in double: a position in the
// thousands times a frequency near one leaves fp32 with too few fraction bits.
struct QkArgs {
	const float* proj;
	int ldp;
	int heads, kv_heads, dim, vdim;
	const bf16 *qw, *kw;
	float eps;
	int rot_dims;
	const double* freq; // [rot_dims / 2]
	float mag;
	float* q;           // [N][heads*dim]
	float* kc;          // cache rows [kv_heads*dim]
	float* vc;          // cache rows [kv_heads*vdim]
	int v_norm = 0;     // 1: every value head is divided by its root mean square over vdim (eps inside the root, no weight)
	int per_head = 0;   // 1: the RMS norms run over each head's `dim` channels, qw / kw are [dim] and serve every head
	int vheads;         // value heads (kv_heads, or fewer when neighbouring key heads share one)
	int v_from_k = 0;   // 1: the values are the keys as projected, before norm and rotation (the projection has no value columns)
	int pairs2 = 0;     // 1: rotation turns channels 2i and 2i + 1 together, 0: i and i + rot_dims/2
	bf16* qb = nullptr; // given: the queries leave in the activation type for the product path instead, as they are (qsplit 0) or as
	int qsplit = 0;     //        [hi | hi | lo] rows of `dim` columns each per head (see k_seq_split_q)
};
// TH threads: 1024 where few tokens have a CTA each (16 tokens, 16 + 4 heads of 128 normed as a whole: 15.5 us with 256, most of it ten steps of two loads one after the other)
template <int TH>
__global__ void __launch_bounds__(TH) k_seq_qk_rope(QkArgs a, SeqBatch sb) {
	pdl_enter(); // programmatic dependent launch: let the next kernel's launch overlap this one, then wait for the previous one
	extern __shared__ float cs[]; // [rot_dims/2] cos, [rot_dims/2] sin, then (per_head) [heads + kv_heads] reciprocal root mean squares
	__shared__ float red[2][TH / 32];
	const int n = blockIdx.x, tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
	const int Q = a.heads * a.dim, K = a.kv_heads * a.dim, Vn = a.vheads * a.vdim, half = a.rot_dims / 2;
	const float* pr = a.proj + (size_t)n * a.ldp;
	const int units = a.heads + a.kv_heads, per = (units + (int)gridDim.y - 1) / (int)gridDim.y; // this CTA's head vectors: query heads, then key heads
	const int u0 = min(units, (int)blockIdx.y * per), u1 = min(units, u0 + per);
	const int pos = sb.tpos[n];
	const long row = cache_row(sb, sb.tslot[n], pos);
	for (int i = tid; i < half; i += blockDim.x) {
		double s, c;
		sincos((double)pos * a.freq[i], &s, &c);
		cs[i] = (float)c * a.mag, cs[half + i] = (float)s * a.mag;
	}
	float sq = 0.f, sk = 0.f;
	float* rh = cs + 2 * max(half, 1);
	if (a.qw && a.per_head) { // one warp per head vector, query heads first: the key heads follow them in the projection
		for (int u = u0 + warp; u < u1; u += (int)(blockDim.x >> 5)) {
			const float* src = pr + (size_t)u * a.dim;
			float ss = 0.f;
			for (int i = lane; i < a.dim; i += 32) ss = fmaf(src[i], src[i], ss);
			ss = warp_sum(ss);
			if (lane == 0) rh[u - u0] = 1.f / sqrtf(ss / (float)a.dim + a.eps);
		}
	} else if (a.qw) {
		for (int i = tid; i < Q; i += blockDim.x) sq = fmaf(pr[i], pr[i], sq);
		for (int i = tid; i < K; i += blockDim.x) sk = fmaf(pr[Q + i], pr[Q + i], sk);
		sq = warp_sum(sq), sk = warp_sum(sk);
		if (lane == 0) red[0][warp] = sq, red[1][warp] = sk;
	}
	__syncthreads();
	float rq = 1.f, rk = 1.f;
	if (a.qw && !a.per_head) {
		sq = sk = 0.f;
		for (int w = 0; w < (int)(blockDim.x >> 5); ++w) sq += red[0][w], sk += red[1][w];
		rq = 1.f / sqrtf(sq / (float)Q + a.eps), rk = 1.f / sqrtf(sk / (float)K + a.eps);
	}
	float* kd = a.kc + row * K;
	for (int e = u0 * a.dim + tid; e < u1 * a.dim; e += blockDim.x) {
		const bool isq = e < Q;
		const int c = isq ? e : e - Q, d = c % a.dim;
		const bf16* w = isq ? a.qw : a.kw;
		const float r = a.per_head && w ? rh[e / a.dim - u0] : isq ? rq : rk; // e / dim: query heads, then key heads
		const float* src = pr + (isq ? 0 : Q);
		const int wo = a.per_head ? c - d : 0; // a weight shared by the heads is indexed by the channel inside the head
		float v = src[c] * r * (w ? ldf(w + c - wo) : 1.f);
		if (d < a.rot_dims) {
			const bool first = a.pairs2 ? !(d & 1) : d < half; // the pair's first channel?
			const int i = a.pairs2 ? d >> 1 : first ? d : d - half, o = a.pairs2 ? (first ? c + 1 : c - 1) : first ? c + half : c - half;
			const float other = src[o] * r * (w ? ldf(w + o - wo) : 1.f);
			v = first ? v * cs[i] - other * cs[half + i] : v * cs[i] + other * cs[half + i];
		}
		if (isq && a.qb) {
			const bf16 hi = __float2bfloat16_rn(v);
			if (a.qsplit) {
				bf16* qd = a.qb + (size_t)n * 3 * Q + 3 * (c - d) + d;
				qd[0] = hi, qd[a.dim] = hi, qd[2 * a.dim] = __float2bfloat16_rn(v - __bfloat162float(hi));
			} else a.qb[(size_t)n * Q + c] = hi;
		} else if (isq) a.q[(size_t)n * Q + c] = v;
		else kd[c] = v;
	}
	float* vd = a.vc + row * Vn;
	const float* const vp = pr + Q + (a.v_from_k ? 0 : K);
	if (a.v_norm) { // one warp per value head
		for (int g = blockIdx.y * (int)(blockDim.x >> 5) + warp; g < a.vheads; g += (int)(gridDim.y * (blockDim.x >> 5))) {
			const float* src = vp + g * a.vdim;
			float ss = 0.f;
			for (int i = lane; i < a.vdim; i += 32) ss = fmaf(src[i], src[i], ss);
			ss = warp_sum(ss);
			const float rv = 1.f / sqrtf(ss / (float)a.vdim + a.eps);
			for (int i = lane; i < a.vdim; i += 32) vd[g * a.vdim + i] = src[i] * rv;
		}
		return;
	}
	for (int i = blockIdx.y * blockDim.x + tid; i < Vn; i += gridDim.y * blockDim.x) vd[i] = vp[i];
}

// ---------------------------------------------------------------- routed experts
// Router: per token the `top` highest-scoring experts (lowest index wins a tie) and a softmax restricted to their scores.  One warp per token.
// mode 1: scores are a softmax over ALL `experts` router outputs; the choice is made on score + correction (bf16 [experts] or null), the
// weights are the chosen scores times `scale`, not renormalised.  mode 2: scores are sigmoid(output), choice and weight alike.
__device__ __forceinline__ void moe_route_token(int n, int lane, const float* logits, int ld, int experts, int top, int* sel, float* wt, int mode, const bf16* correction, float scale) {
	const float* z = logits + (size_t)n * ld;
	if (mode == 1) {
		float mx = -INFINITY;
		for (int e = lane; e < experts; e += 32) mx = fmaxf(mx, z[e]);
		mx = warp_max(mx);
		float den = 0.f;
		for (int e = lane; e < experts; e += 32) den += expf(z[e] - mx);
		den = warp_sum(den);
		for (int k = 0; k < top; ++k) {
			float bv = -INFINITY, bs = 0.f;
			int bi = 0x7fffffff;
			for (int e = lane; e < experts; e += 32) {
				bool taken = false;
				for (int j = 0; j < k; ++j) taken |= sel[(size_t)n * top + j] == e;
				const float sc = expf(z[e] - mx) / den, c = sc + (correction ? ldf(correction + e) : 0.f);
				if (!taken && c > bv) bv = c, bi = e, bs = sc;
			}
			for (int o = 16; o > 0; o >>= 1) {
				const float ov = __shfl_xor_sync(0xffffffffu, bv, o), os = __shfl_xor_sync(0xffffffffu, bs, o);
				const int oi = __shfl_xor_sync(0xffffffffu, bi, o);
				if (ov > bv || (ov == bv && oi < bi)) bv = ov, bi = oi, bs = os;
			}
			if (lane == 0) sel[(size_t)n * top + k] = bi, wt[(size_t)n * top + k] = bs * scale;
			__syncwarp();
		}
		return;
	}
	if (mode == 2) { // scores sigmoid(z); the `top` largest, each weighted by its own score
		for (int k = 0; k < top; ++k) {
			float bv = -INFINITY;
			int bi = 0x7fffffff;
			for (int e = lane; e < experts; e += 32) {
				bool taken = false;
				for (int j = 0; j < k; ++j) taken |= sel[(size_t)n * top + j] == e;
				const float sc = sigmoidf_(z[e]);
				if (!taken && sc > bv) bv = sc, bi = e;
			}
			for (int o = 16; o > 0; o >>= 1) {
				const float ov = __shfl_xor_sync(0xffffffffu, bv, o);
				const int oi = __shfl_xor_sync(0xffffffffu, bi, o);
				if (ov > bv || (ov == bv && oi < bi)) bv = ov, bi = oi;
			}
			if (lane == 0) sel[(size_t)n * top + k] = bi, wt[(size_t)n * top + k] = bv * scale;
			__syncwarp();
		}
		return;
	}
	float first = 0.f, sum = 0.f;
	for (int k = 0; k < top; ++k) {
		float bv = -INFINITY;
		int bi = 0x7fffffff;
		for (int e = lane; e < experts; e += 32) {
			bool taken = false;
			for (int j = 0; j < k; ++j) taken |= sel[(size_t)n * top + j] == e; // written by lane 0 below, visible after the warp barrier
			if (!taken && z[e] > bv) bv = z[e], bi = e;
		}
		for (int o = 16; o > 0; o >>= 1) {
			const float ov = __shfl_xor_sync(0xffffffffu, bv, o);
			const int oi = __shfl_xor_sync(0xffffffffu, bi, o);
			if (ov > bv || (ov == bv && oi < bi)) bv = ov, bi = oi;
		}
		if (k == 0) first = bv;
		const float p = expf(bv - first); // the first chosen logit is the largest: the softmax's maximum
		sum += p;
		if (lane == 0) sel[(size_t)n * top + k] = bi, wt[(size_t)n * top + k] = p;
		__syncwarp();
	}
	for (int k = lane; k < top; k += 32) wt[(size_t)n * top + k] /= sum;
}
__global__ void k_seq_moe_route(const float* logits, int ld, int experts, int top, int N, int* sel, float* wt, int mode, const bf16* correction, float scale) {
	pdl_enter(); // programmatic dependent launch: let the next kernel's launch overlap this one, then wait for the previous one
	const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
	const int n = blockIdx.x * (blockDim.x >> 5) + warp;
	if (n >= N) return;
	moe_route_token(n, lane, logits, ld, experts, top, sel, wt, mode, correction, scale);
}
// Few tokens (a decode step): routing and grouping in ONE CTA.  The warps route the tokens, then thread e places expert e's pairs in
// token order behind those of the lower experts (same result as k_seq_moe_route followed by k_seq_moe_group).
#define MOE_SMALL_TOKENS 64
__global__ void __launch_bounds__(256) k_seq_moe_route_group(const float* logits, int ld, int experts, int top, int N, int* sel, float* wt, int mode, const bf16* correction, float scale,
                                                             int* seg, int* perm, int* inv) {
	pdl_enter(); // programmatic dependent launch: let the next kernel's launch overlap this one, then wait for the previous one
	const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
	for (int n = warp; n < N; n += 8) moe_route_token(n, lane, logits, ld, experts, top, sel, wt, mode, correction, scale);
	__syncthreads();
	const int pairs = N * top;
	for (int e = threadIdx.x; e < experts; e += 256) {
		int below = 0;
		for (int i = 0; i < pairs; ++i) below += sel[i] < e;
		seg[e] = below;
		if (e == experts - 1) seg[experts] = pairs;
		for (int i = 0; i < pairs; ++i)
			if (sel[i] == e) perm[below] = i, inv[i] = below, ++below;
	}
}
// Groups the (token, choice) pairs by expert, pairs of one expert in token order: one CTA per expert counts the pairs of lower
// experts (its group's first row) and places its own.  seg[e] .. seg[e+1] are expert e's rows, perm[row] = pair, inv[pair] = row.
__global__ void __launch_bounds__(256) k_seq_moe_group(const int* sel, int pairs, int experts, int* seg, int* perm, int* inv) {
	pdl_enter(); // programmatic dependent launch: let the next kernel's launch overlap this one, then wait for the previous one
	__shared__ int wsum[8], base_s, run_s;
	const int e = blockIdx.x, tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
	int below = 0;
	for (int i = tid; i < pairs; i += 256) below += sel[i] < e;
	for (int o = 16; o > 0; o >>= 1) below += __shfl_xor_sync(0xffffffffu, below, o);
	if (lane == 0) wsum[warp] = below;
	__syncthreads();
	if (tid == 0) {
		int s = 0;
		for (int w = 0; w < 8; ++w) s += wsum[w];
		base_s = s, run_s = 0;
		seg[e] = s;
		if (e == experts - 1) seg[experts] = pairs;
	}
	__syncthreads();
	const int base = base_s;
	for (int i0 = 0; i0 < pairs; i0 += 256) {
		const int i = i0 + tid;
		const bool mine = i < pairs && sel[i] == e;
		const unsigned bal = __ballot_sync(0xffffffffu, mine);
		__syncthreads(); // the previous pass's readers of wsum / run_s are done
		if (lane == 0) wsum[warp] = __popc(bal);
		__syncthreads();
		int before = run_s;
		for (int w = 0; w < warp; ++w) before += wsum[w];
		if (mine) {
			const int r = base + before + __popc(bal & ((1u << lane) - 1));
			perm[r] = i, inv[i] = r;
		}
		__syncthreads();
		if (tid == 0) {
			int s = run_s;
			for (int w = 0; w < 8; ++w) s += wsum[w];
			run_s = s;
		}
	}
}
// rows of the grouped activation matrix: Xp[row] = h[perm[row] / top]  (T: an element, or 16 bytes of a row; width counts in T)
template <typename T>
__global__ void k_seq_moe_gather(T* xp, const T* h, const int* perm, int top, int pairs, int width) {
	pdl_enter(); // programmatic dependent launch: let the next kernel's launch overlap this one, then wait for the previous one
	const size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
	if (i >= (size_t)pairs * width) return;
	const size_t r = i / width, c = i % width;
	xp[i] = h[(size_t)(perm[r] / top) * width + c];
}
// x[n] += (res ? res[n] : 0) + sum_k wt[n][k] * y[inv[n * top + k]]   (choices in order of rank; `store`: x[n] = the sum alone)
// A choice sel >= real is an identity expert: its output is the token's own input row h[n].
template <typename AT>
__global__ void k_seq_moe_combine(float* x, const float* res, const float* y, const int* inv, const float* wt, int top, int N, int width, const int* sel, int real, const AT* h,
                                  int store) {
	pdl_enter(); // programmatic dependent launch: let the next kernel's launch overlap this one, then wait for the previous one
	const size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
	if (i >= (size_t)N * width) return;
	const size_t n = i / width, c = i % width;
	float s = 0.f;
	for (int k = 0; k < top; ++k) {
		const float v = sel[n * top + k] >= real ? ldf(h + i) : y[(size_t)inv[n * top + k] * width + c];
		s = fmaf(wt[n * top + k], v, s);
	}
	if (store) x[i] = s;
	else x[i] += res ? res[i] + s : s;
}

// ---------------------------------------------------------------- hyper-connections: several copies of the residual stream
// x is [N][streams][width].  Read: u = sum_s in[s] x_s (in == null: every stream counts once), then the RMS norm of u with a weight
// per column (w_len = width) or one number for all (w_len = 1); one CTA per row, rows[] picks tokens (the rows whose logits are wanted).
template <typename AT>
__global__ void __launch_bounds__(256) k_seq_hc_read(AT* out, const float* x, const int* rows, const bf16* in, const bf16* w, int w_len, float offset, float eps, int R, int width,
                                                     int streams) {
	pdl_enter(); // programmatic dependent launch: let the next kernel's launch overlap this one, then wait for the previous one
	__shared__ float red[8];
	const int tid = threadIdx.x, nt = blockDim.x, r = blockIdx.x;
	const float* src = x + (size_t)(rows ? rows[r] : r) * streams * width;
	auto mixed = [&](int c) {
		float u = 0.f;
		for (int s = 0; s < streams; ++s) u = fmaf(in ? ldf(in + s) : 1.f, src[(size_t)s * width + c], u);
		return u;
	};
	float keep[RMS_KEEP];
	float ss = 0.f;
#pragma unroll
	for (int i = 0; i < RMS_KEEP; ++i) {
		const int c = i * nt + tid;
		keep[i] = c < width ? mixed(c) : 0.f;
		ss = fmaf(keep[i], keep[i], ss);
	}
	for (int c = RMS_KEEP * nt + tid; c < width; c += nt) {
		const float u = mixed(c);
		ss = fmaf(u, u, ss);
	}
	ss = warp_sum(ss);
	if ((tid & 31) == 0) red[tid >> 5] = ss;
	__syncthreads();
	ss = 0.f;
	for (int i = 0; i < (nt >> 5); ++i) ss += red[i];
	const float rinv = 1.f / sqrtf(ss / (float)width + eps);
	AT* d = out + (size_t)r * width;
#pragma unroll
	for (int i = 0; i < RMS_KEEP; ++i) {
		const int c = i * nt + tid;
		if (c < width) d[c] = to_act<AT>(keep[i] * rinv * (ldf(w + (w_len == 1 ? 0 : c)) + offset));
	}
	for (int c = RMS_KEEP * nt + tid; c < width; c += nt) d[c] = to_act<AT>(mixed(c) * rinv * (ldf(w + (w_len == 1 ? 0 : c)) + offset));
}
// Write: x_t <- sum_s mix[s][t] x_s + out[t] y for every stream t at once, from the old streams.  y = base (the sublayer's last product,
// or null) + the routed experts' weighted sum when `moe.y` is set (choices in order of rank; identity experts return the input row h).
#define HC_MAX 16
struct HcMoe {
	const float* y;  // [pairs][width] grouped expert outputs, or null: no routed part
	const int* inv;
	const int* sel;
	const float* wt;
	int top, real;
};
// One CTA per token.  When `rd.out` is set the same pass also forms the NEXT sublayer's input from the streams it has just written
// (u = sum_t in[t] x_t, RMS norm, weight), so the streams are not read again: hc_write followed by hc_read in one kernel.  The row of h
// that identity experts read may be the very row rd.out overwrites: all reads of it come before the barrier, all writes after.
struct HcRead {
	void* out;       // [N][width] of the activation type, or null: write only
	const bf16* in;  // [streams]
	const bf16* w;
	int w_len;
	float offset, eps;
};
// (a thread's columns alternate loads and stores of the same matrix, which do not overlap in time, so a thread should have one
// group of columns, or few)
#define HC_KEEP 4
template <int V>
struct HcVec { float v[V]; };
template <int V>
__device__ __forceinline__ HcVec<V> hc_load(const float* p) {
	HcVec<V> r;
	if constexpr (V == 4) {
		const float4 t = *(const float4*)p;
		r.v[0] = t.x, r.v[1] = t.y, r.v[2] = t.z, r.v[3] = t.w;
	} else r.v[0] = *p;
	return r;
}
template <int V>
__device__ __forceinline__ void hc_store(float* p, const HcVec<V>& r) {
	if constexpr (V == 4) *(float4*)p = make_float4(r.v[0], r.v[1], r.v[2], r.v[3]);
	else *p = r.v[0];
}
// V = 4: width is a multiple of 4 and a thread owns four neighbouring columns (16-byte loads and stores); V = 1: any width.
// SM: the most streams this instance holds in registers (4 or HC_MAX)
template <typename AT, int V, int SM>
__global__ void __launch_bounds__(V == 4 ? 512 : 1024) k_seq_hc_write(float* x, const float* base, const bf16* mix, const bf16* outw, int N, int width, int streams, HcMoe moe, const AT* h, HcRead rd) {
	pdl_enter(); // programmatic dependent launch: let the next kernel's launch overlap this one, then wait for the previous one
	__shared__ float red[32];
	const int tid = threadIdx.x, nt = blockDim.x;
	const size_t n = blockIdx.x;
	// the few coefficients (mix, out, the next read's in) are read where they are used: every lane the same address, served by L1; no
	// staging and no barrier before the first loads of the streams go out
	auto c_mix = [&](int s, int t) { return ldf(mix + s * streams + t); };
	auto c_out = [&](int t) { return ldf(outw + t); };
	auto c_in = [&](int t) { return rd.out ? ldf(rd.in + t) : 0.f; };
	float* xr = x + n * streams * width;
	auto column = [&](int c) { // writes the new streams of columns c .. c + V - 1, returns the next read's weighted sum of them
		const size_t i = n * width + c;
		HcVec<V> y;
#pragma unroll
		for (int e = 0; e < V; ++e) y.v[e] = 0.f;
		if (base) y = hc_load<V>(base + i);
		if (moe.y) {
			HcVec<V> sacc;
#pragma unroll
			for (int e = 0; e < V; ++e) sacc.v[e] = 0.f;
			for (int k = 0; k < moe.top; ++k) {
				HcVec<V> v;
				if (moe.sel[n * moe.top + k] >= moe.real) {
#pragma unroll
					for (int e = 0; e < V; ++e) v.v[e] = ldf(h + i + e);
				} else v = hc_load<V>(moe.y + (size_t)moe.inv[n * moe.top + k] * width + c);
				const float wk = moe.wt[n * moe.top + k];
#pragma unroll
				for (int e = 0; e < V; ++e) sacc.v[e] = fmaf(wk, v.v[e], sacc.v[e]);
			}
#pragma unroll
			for (int e = 0; e < V; ++e) y.v[e] += sacc.v[e];
		}
		HcVec<V> old[SM];
#pragma unroll
		for (int s = 0; s < SM; ++s)
			if (s < streams) old[s] = hc_load<V>(xr + (size_t)s * width + c);
		HcVec<V> u;
#pragma unroll
		for (int e = 0; e < V; ++e) u.v[e] = 0.f;
		for (int t = 0; t < streams; ++t) {
			HcVec<V> v;
#pragma unroll
			for (int e = 0; e < V; ++e) v.v[e] = 0.f;
#pragma unroll
			for (int s = 0; s < SM; ++s)
				if (s < streams) {
					const float mx = c_mix(s, t);
#pragma unroll
					for (int e = 0; e < V; ++e) v.v[e] = fmaf(mx, old[s].v[e], v.v[e]);
				}
			const float co = c_out(t), ci = c_in(t);
#pragma unroll
			for (int e = 0; e < V; ++e) v.v[e] = fmaf(co, y.v[e], v.v[e]), u.v[e] = fmaf(ci, v.v[e], u.v[e]);
			hc_store<V>(xr + (size_t)t * width + c, v);
		}
		return u;
	};
	HcVec<V> keep[HC_KEEP];
	float ss = 0.f;
#pragma unroll
	for (int i = 0; i < HC_KEEP; ++i) {
		const int c = (i * nt + tid) * V;
		if (c < width) keep[i] = column(c);
		else {
#pragma unroll
			for (int e = 0; e < V; ++e) keep[i].v[e] = 0.f;
		}
#pragma unroll
		for (int e = 0; e < V; ++e) ss = fmaf(keep[i].v[e], keep[i].v[e], ss);
	}
	for (int c = (HC_KEEP * nt + tid) * V; c < width; c += nt * V) {
		const HcVec<V> u = column(c);
#pragma unroll
		for (int e = 0; e < V; ++e) ss = fmaf(u.v[e], u.v[e], ss);
	}
	if (!rd.out) return;
	ss = warp_sum(ss);
	if ((tid & 31) == 0) red[tid >> 5] = ss;
	__syncthreads();
	ss = 0.f;
	for (int i = 0; i < (nt >> 5); ++i) ss += red[i];
	const float rinv = 1.f / sqrtf(ss / (float)width + rd.eps);
	AT* d = (AT*)rd.out + n * width;
#pragma unroll
	for (int i = 0; i < HC_KEEP; ++i) {
		const int c = (i * nt + tid) * V;
		if (c < width) {
#pragma unroll
			for (int e = 0; e < V; ++e) d[c + e] = to_act<AT>(keep[i].v[e] * rinv * (ldf(rd.w + (rd.w_len == 1 ? 0 : c + e)) + rd.offset));
		}
	}
	for (int c = (HC_KEEP * nt + tid) * V; c < width; c += nt * V) { // wider rows: the sum is formed again from the streams just written (by this thread)
#pragma unroll
		for (int e = 0; e < V; ++e) {
			float u = 0.f;
			for (int t = 0; t < streams; ++t) u = fmaf(c_in(t), xr[(size_t)t * width + c + e], u);
			d[c + e] = to_act<AT>(u * rinv * (ldf(rd.w + (rd.w_len == 1 ? 0 : c + e)) + rd.offset));
		}
	}
}
// Post-norm blocks: x[n] += y / sqrt(mean(y^2) + eps) * (w + offset) (LN: y's mean is taken off it first), where y = base (a sublayer's last product, or null) + the routed
// experts' sum when `moe.y` is set (choices in order of rank, each times its weight, or times one when moe.wt is null: the weight went
// in at the expert's input).  The same pass writes the new row of x in the activation type: the input of the sublayer that follows.
// One CTA per token.  V = 4: width is a multiple of 4 and a thread owns groups of four neighbouring columns (16-byte loads and stores);
// V = 1: any width.  A thread keeps PN_KEEP groups of y in registers (wider rows form y a second time).
#define PN_KEEP 4
template <typename AT, int V>
__device__ __forceinline__ void pn_store_act(AT* p, const HcVec<V>& r) {
	if constexpr (V == 4 && sizeof(AT) == 2) {
		__nv_bfloat162 lo = __floats2bfloat162_rn(r.v[0], r.v[1]), hi = __floats2bfloat162_rn(r.v[2], r.v[3]);
		uint2 u;
		u.x = *reinterpret_cast<unsigned*>(&lo), u.y = *reinterpret_cast<unsigned*>(&hi);
		*reinterpret_cast<uint2*>(p) = u;
	} else {
#pragma unroll
		for (int e = 0; e < V; ++e) p[e] = to_act<AT>(r.v[e]);
	}
}
template <typename AT, int V, bool LN = false>
__global__ void __launch_bounds__(256) k_seq_post_norm(float* x, AT* act, const float* base, HcMoe moe, const bf16* w, float offset, float eps, int N, int width) {
	pdl_enter(); // programmatic dependent launch: let the next kernel's launch overlap this one, then wait for the previous one
	__shared__ float red[8], redm[8];
	const int tid = threadIdx.x, nt = blockDim.x;
	const size_t n = blockIdx.x;
	auto yval = [&](int c) {
		HcVec<V> y;
#pragma unroll
		for (int e = 0; e < V; ++e) y.v[e] = 0.f;
		if (base) y = hc_load<V>(base + n * width + c);
		if (moe.y)
			for (int k = 0; k < moe.top; ++k) {
				const HcVec<V> v = hc_load<V>(moe.y + (size_t)moe.inv[n * moe.top + k] * width + c);
				const float wk = moe.wt ? moe.wt[n * moe.top + k] : 1.f;
#pragma unroll
				for (int e = 0; e < V; ++e) y.v[e] = moe.wt ? fmaf(wk, v.v[e], y.v[e]) : y.v[e] + v.v[e];
			}
		return y;
	};
	HcVec<V> keep[PN_KEEP];
	float ss = 0.f, sum = 0.f, mean = 0.f;
#pragma unroll
	for (int i = 0; i < PN_KEEP; ++i) {
		const int c = (i * nt + tid) * V;
		if (c < width) keep[i] = yval(c);
		else {
#pragma unroll
			for (int e = 0; e < V; ++e) keep[i].v[e] = 0.f;
		}
#pragma unroll
		for (int e = 0; e < V; ++e) {
			if constexpr (LN) sum += keep[i].v[e];
			else ss = fmaf(keep[i].v[e], keep[i].v[e], ss);
		}
	}
	if constexpr (LN) {
		for (int c = (PN_KEEP * nt + tid) * V; c < width; c += nt * V) {
			const HcVec<V> y = yval(c);
#pragma unroll
			for (int e = 0; e < V; ++e) sum += y.v[e];
		}
		mean = cta_sum(sum, redm) / (float)width;
#pragma unroll
		for (int i = 0; i < PN_KEEP; ++i)
			if ((i * nt + tid) * V < width) {
#pragma unroll
				for (int e = 0; e < V; ++e) keep[i].v[e] -= mean, ss = fmaf(keep[i].v[e], keep[i].v[e], ss);
			}
	}
	auto wide = [&](int c) { // columns beyond the registers: formed again
		HcVec<V> y = yval(c);
		if constexpr (LN) {
#pragma unroll
			for (int e = 0; e < V; ++e) y.v[e] -= mean;
		}
		return y;
	};
	for (int c = (PN_KEEP * nt + tid) * V; c < width; c += nt * V) {
		const HcVec<V> y = wide(c);
#pragma unroll
		for (int e = 0; e < V; ++e) ss = fmaf(y.v[e], y.v[e], ss);
	}
	ss = warp_sum(ss);
	if ((tid & 31) == 0) red[tid >> 5] = ss;
	__syncthreads();
	ss = 0.f;
	for (int i = 0; i < (nt >> 5); ++i) ss += red[i]; // every thread adds the warps' sums in the same order
	const float rinv = 1.f / sqrtf(ss / (float)width + eps);
	float* xr = x + n * width;
	AT* ar = act + n * width;
	auto put = [&](int c, const HcVec<V>& y) {
		HcVec<V> v = hc_load<V>(xr + c);
#pragma unroll
		for (int e = 0; e < V; ++e) v.v[e] += y.v[e] * rinv * (ldf(w + c + e) + offset);
		hc_store<V>(xr + c, v);
		pn_store_act<AT, V>(ar + c, v);
	};
#pragma unroll
	for (int i = 0; i < PN_KEEP; ++i) {
		const int c = (i * nt + tid) * V;
		if (c < width) put(c, keep[i]);
	}
	for (int c = (PN_KEEP * nt + tid) * V; c < width; c += nt * V) put(c, wide(c));
}
// Sandwich blocks: what follows a sublayer's last product, in one pass over the row.
//   y = (base + the routed experts' sum) * sigmoid(gate),  v = x[n] + y / sqrt(mean(y^2) + eps) * (w + offset);
//   with a depth average (dwa): X_k = v is kept in hist[k] and v becomes dwa[k] v + sum_(j < k) dwa[j] hist[j];
//   x[n] = v;  act[n] = v / sqrt(mean(v^2) + eps) * (w_next + offset), the normed input of the sublayer that follows (w_next null: none).
// One CTA per token; V and PN_KEEP as in k_seq_post_norm.
struct Sandwich {
	const float* base; // a sublayer's last product, or null
	HcMoe moe;
	const float* gate; // gate[n * ldg + c], raw; null: none
	long ldg;
	const bf16* w;
	float* hist;       // [k + 1 ..][N][width]
	const bf16* dwa;   // [k + 1], or null
	int k;
	const bf16* w_next;
	float offset, eps;
};
template <typename AT, int V>
__global__ void __launch_bounds__(256) k_seq_sandwich(float* x, AT* act, Sandwich a, int N, int width) {
	pdl_enter(); // programmatic dependent launch: let the next kernel's launch overlap this one, then wait for the previous one
	__shared__ float red[2][8];
	const int tid = threadIdx.x, nt = blockDim.x;
	const size_t n = blockIdx.x;
	auto yval = [&](int c) {
		HcVec<V> y;
#pragma unroll
		for (int e = 0; e < V; ++e) y.v[e] = 0.f;
		if (a.base) y = hc_load<V>(a.base + n * width + c);
		if (a.moe.y)
			for (int k = 0; k < a.moe.top; ++k) {
				const HcVec<V> v = hc_load<V>(a.moe.y + (size_t)a.moe.inv[n * a.moe.top + k] * width + c);
				const float wk = a.moe.wt ? a.moe.wt[n * a.moe.top + k] : 1.f;
#pragma unroll
				for (int e = 0; e < V; ++e) y.v[e] = a.moe.wt ? fmaf(wk, v.v[e], y.v[e]) : y.v[e] + v.v[e];
			}
		if (a.gate) {
			const HcVec<V> g = hc_load<V>(a.gate + n * a.ldg + c);
#pragma unroll
			for (int e = 0; e < V; ++e) y.v[e] *= sigmoidf_(g.v[e]);
		}
		return y;
	};
	auto row_sum = [&](float ss, float* r) { // every thread adds the warps' sums in the same order
		ss = warp_sum(ss);
		if ((tid & 31) == 0) r[tid >> 5] = ss;
		__syncthreads();
		ss = 0.f;
		for (int i = 0; i < (nt >> 5); ++i) ss += r[i];
		return ss;
	};
	HcVec<V> keep[PN_KEEP];
	float ss = 0.f;
#pragma unroll
	for (int i = 0; i < PN_KEEP; ++i) {
		const int c = (i * nt + tid) * V;
		if (c < width) keep[i] = yval(c);
		else {
#pragma unroll
			for (int e = 0; e < V; ++e) keep[i].v[e] = 0.f;
		}
#pragma unroll
		for (int e = 0; e < V; ++e) ss = fmaf(keep[i].v[e], keep[i].v[e], ss);
	}
	for (int c = (PN_KEEP * nt + tid) * V; c < width; c += nt * V) {
		const HcVec<V> y = yval(c);
#pragma unroll
		for (int e = 0; e < V; ++e) ss = fmaf(y.v[e], y.v[e], ss);
	}
	const float rinv = 1.f / sqrtf(row_sum(ss, red[0]) / (float)width + a.eps);
	float* xr = x + n * width;
	auto put = [&](int c, const HcVec<V>& y) { // the new row's columns c .. c + V - 1
		HcVec<V> v = hc_load<V>(xr + c);
#pragma unroll
		for (int e = 0; e < V; ++e) v.v[e] += y.v[e] * rinv * (ldf(a.w + c + e) + a.offset);
		if (a.dwa) {
			const size_t o = n * width + c, layer = (size_t)N * width;
			hc_store<V>(a.hist + a.k * layer + o, v);
			HcVec<V> m;
#pragma unroll
			for (int e = 0; e < V; ++e) m.v[e] = 0.f;
#pragma unroll 4
			for (int j = 0; j < a.k; ++j) {
				const HcVec<V> h = hc_load<V>(a.hist + j * layer + o);
				const float wj = ldf(a.dwa + j);
#pragma unroll
				for (int e = 0; e < V; ++e) m.v[e] = fmaf(wj, h.v[e], m.v[e]);
			}
			const float wk = ldf(a.dwa + a.k);
#pragma unroll
			for (int e = 0; e < V; ++e) v.v[e] = fmaf(wk, v.v[e], m.v[e]);
		}
		hc_store<V>(xr + c, v);
		return v;
	};
	ss = 0.f;
#pragma unroll
	for (int i = 0; i < PN_KEEP; ++i) {
		const int c = (i * nt + tid) * V;
		if (c < width) keep[i] = put(c, keep[i]);
#pragma unroll
		for (int e = 0; e < V; ++e) ss = fmaf(keep[i].v[e], keep[i].v[e], ss); // columns past the row are still zero
	}
	for (int c = (PN_KEEP * nt + tid) * V; c < width; c += nt * V) {
		const HcVec<V> v = put(c, yval(c));
#pragma unroll
		for (int e = 0; e < V; ++e) ss = fmaf(v.v[e], v.v[e], ss);
	}
	if (!a.w_next) return;
	const float rnext = 1.f / sqrtf(row_sum(ss, red[1]) / (float)width + a.eps);
	AT* ar = act + n * width;
	auto normed = [&](int c, HcVec<V> v) {
#pragma unroll
		for (int e = 0; e < V; ++e) v.v[e] *= rnext * (ldf(a.w_next + c + e) + a.offset);
		pn_store_act<AT, V>(ar + c, v);
	};
#pragma unroll
	for (int i = 0; i < PN_KEEP; ++i) {
		const int c = (i * nt + tid) * V;
		if (c < width) normed(c, keep[i]);
	}
	for (int c = (PN_KEEP * nt + tid) * V; c < width; c += nt * V) normed(c, hc_load<V>(xr + c)); // written by this very thread
}
// out[n] = sum of the streams of token n
__global__ void k_seq_stream_sum(float* out, const float* x, int N, int width, int streams) {
	pdl_enter(); // programmatic dependent launch: let the next kernel's launch overlap this one, then wait for the previous one
	const size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
	if (i >= (size_t)N * width) return;
	const size_t n = i / width, c = i % width;
	float v = 0.f;
	for (int s = 0; s < streams; ++s) v += x[(n * streams + s) * width + c];
	out[i] = v;
}

// ---------------------------------------------------------------- linear recurrences served by the gated-linear-attention scan
// mLSTM, HGRN2 and Mamba-2 are all S <- diag(a) S + k v^T, o = S^T q per head; what differs is how a, k, v, q come out of the
// projection and what happens to o.  A preparation kernel writes them as the scan's input (`lin`: rows [q | k | v] per token, and
// the decay matrix), the scan itself is k_seq_gla_scan, k_seq_lin_out finishes.

// mLSTM gates.  Per (sequence, head), over the step's tokens in order, with the running maximum m carried in the slot state:
//   li = cap tanh((i_raw) / cap), lf = logsigmoid(cap tanh(f_raw / cap)), m_t = max(lf + m_(t-1), li),
//   keep_t = exp(lf + m_(t-1) - m_t), take_t = exp(li - m_t).
// One warp per (sequence, head), 32 tokens per round: with F the running sum of lf inside the round, m_t = F_t + max(m_in, max_(s<=t)(li_s - F_s)).
struct MlstmGates {
	const float* proj; // biased projection; raw gates at columns icol + h, fcol + h
	int ldp, icol, fcol, heads;
	float cap;
	float* m_state;    // [slots][heads]
	float* keep;       // [N][heads]
	float* take;       // [N][heads]
	float* m_out;      // [N][heads]
};
__global__ void k_seq_mlstm_gates(MlstmGates a, SeqBatch sb) {
	pdl_enter(); // programmatic dependent launch: let the next kernel's launch overlap this one, then wait for the previous one
	const int b = blockIdx.x, h = blockIdx.y, lane = threadIdx.x;
	const int start = sb.sstart[b], cnt = sb.scount[b];
	float* mp = a.m_state + (size_t)sb.sslot[b] * a.heads + h;
	float m_in = *mp;
	for (int t0 = 0; t0 < cnt; t0 += 32) {
		const int t = t0 + lane;
		const bool live = t < cnt;
		float li = -INFINITY, lf = 0.f;
		if (live) {
			const float* pr = a.proj + (size_t)(start + t) * a.ldp;
			li = a.cap * tanhf(pr[a.icol + h] / a.cap);
			const float fr = a.cap * tanhf(pr[a.fcol + h] / a.cap);
			lf = -softplusf_(-fr);
		}
		// the two scans run in double: a round's sum of log forget gates can reach hundreds, where a float keeps four decimals only
		double F = lf;
		for (int o = 1; o < 32; o <<= 1) {
			const double up = __shfl_up_sync(0xffffffffu, F, o);
			if (lane >= o) F += up;
		}
		double A = live ? (double)li - F : -INFINITY;
		for (int o = 1; o < 32; o <<= 1) {
			const double up = __shfl_up_sync(0xffffffffu, A, o);
			if (lane >= o) A = fmax(A, up);
		}
		const double m = F + fmax((double)m_in, A);
		double m_prev = __shfl_up_sync(0xffffffffu, m, 1);
		if (lane == 0) m_prev = m_in;
		if (live) {
			const size_t o = (size_t)(start + t) * a.heads + h;
			a.keep[o] = expf((float)((double)lf + m_prev - m)), a.take[o] = expf((float)((double)li - m)), a.m_out[o] = (float)m;
		}
		m_in = (float)__shfl_sync(0xffffffffu, m, min(31, cnt - t0 - 1));
	}
	if (lane == 0) *mp = m_in;
}

// Scan input of one token and head.  lin row: [q: heads*dim | k: heads*dim | v: heads*vs], decay row: [heads*dim].
//   LIN_MLSTM : q, k as projected; v' = take * [v, 1, 0..] (vs = vdim rounded up past one extra column: the normaliser n rides as a value
//               column of ones); decay = keep for every channel.
//   LIN_HGRN2 : q = silu(q_raw); f = l + (1 - l) sigmoid(f_raw); k = 1 - f; decay = f; v as projected.
//   LIN_MAMBA2: q = C and k = B of the head's group (after the convolution); dt = softplus(dt_raw + dt_bias); v' = dt x; decay = exp(-exp(A_log) dt).
enum { LIN_MLSTM = 0, LIN_HGRN2 = 1, LIN_MAMBA2 = 2 };
struct LinPack {
	int mode;
	const float* proj;
	int ldp, qcol, kcol, vcol; // HGRN2: kcol = the raw forget gate's column
	const float *keep, *take;  // LIN_MLSTM
	const bf16* lower;         // LIN_HGRN2
	const float *xs, *bs, *cs; // LIN_MAMBA2: convolved x [N][heads*vdim], B and C [N][groups*dim]
	int dtcol, groups;
	const bf16 *dt_bias, *a_log;
	float* lin;
	float* decay;
	int heads, dim, vdim, vs;
};
__global__ void k_seq_lin_pack(LinPack a, int N) {
	pdl_enter(); // programmatic dependent launch: let the next kernel's launch overlap this one, then wait for the previous one
	const int n = blockIdx.x, h = blockIdx.y, tid = threadIdx.x, H = a.heads, D = a.dim, V = a.vdim;
	const int ldl = 2 * H * D + H * a.vs;
	const float* pr = a.proj + (size_t)n * a.ldp;
	float* lq = a.lin + (size_t)n * ldl + h * D;
	float* lk = lq + H * D;
	float* lv = a.lin + (size_t)n * ldl + 2 * H * D + h * a.vs;
	float* dc = a.decay + ((size_t)n * H + h) * D;
	if (a.mode == LIN_MLSTM) {
		const float keep = a.keep[(size_t)n * H + h], take = a.take[(size_t)n * H + h];
		for (int i = tid; i < D; i += blockDim.x) lq[i] = pr[a.qcol + h * D + i], lk[i] = pr[a.kcol + h * D + i], dc[i] = keep;
		for (int i = tid; i < a.vs; i += blockDim.x) lv[i] = i < V ? take * pr[a.vcol + h * V + i] : i == V ? take : 0.f;
	} else if (a.mode == LIN_HGRN2) {
		for (int i = tid; i < D; i += blockDim.x) {
			const float q = pr[a.qcol + h * D + i], l = ldf(a.lower + h * D + i);
			const float f = l + (1.f - l) * sigmoidf_(pr[a.kcol + h * D + i]);
			lq[i] = q * sigmoidf_(q), lk[i] = 1.f - f, dc[i] = f;
		}
		for (int i = tid; i < a.vs; i += blockDim.x) lv[i] = i < V ? pr[a.vcol + h * V + i] : 0.f;
	} else {
		const int g = h / (H / a.groups);
		const float dt = softplusf_(pr[a.dtcol + h] + ldf(a.dt_bias + h));
		const float dec = expf(-expf(ldf(a.a_log + h)) * dt);
		for (int i = tid; i < D; i += blockDim.x) {
			lq[i] = a.cs[((size_t)n * a.groups + g) * D + i], lk[i] = a.bs[((size_t)n * a.groups + g) * D + i], dc[i] = dec;
		}
		for (int i = tid; i < a.vs; i += blockDim.x) lv[i] = i < V ? dt * a.xs[((size_t)n * H + h) * V + i] : 0.f;
	}
}

// Read-out of a linear recurrence.  The token's heads*vdim outputs (o[n*ldo + h*ohs + d]) are taken in units of `unit` columns (vdim: per
// head; heads*vdim / groups: equal parts); one warp per (token, unit):
//   mLSTM (m_t given): o /= max(|o[.., vdim]|, exp(-m_t)) + 1e-6 first (column vdim of the head holds n . q);
//   skip given: o += skip_w[h] * skip[n][h*vdim + d];   gate_mode 3: o *= silu(gate) BEFORE the norm;
//   then RMS over the unit (eps inside the root), times w[col % w_mod] (null: no weight), times sigmoid(gate) (gate_mode 1), times mul.
struct LinOut {
	const float* o;
	int ldo, ohs, heads, vdim, unit;
	const bf16* w;
	int w_mod;
	const float* gate;
	int ldg, gate_mode;
	const float* m_t;     // [N][heads] or null
	const float* skip;    // [N][heads*vdim] or null
	const bf16* skip_w;   // [heads]
	float eps, mul;
};
template <typename AT>
__global__ void k_seq_lin_out(AT* out, LinOut a, int N) {
	pdl_enter(); // programmatic dependent launch: let the next kernel's launch overlap this one, then wait for the previous one
	const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
	const int inner = a.heads * a.vdim, units = inner / a.unit;
	const size_t u = (size_t)blockIdx.x * (blockDim.x >> 5) + warp;
	if (u >= (size_t)N * units) return;
	const size_t n = u / units;
	const int c0 = (int)(u % units) * a.unit;
	// a unit that is one head (mLSTM, HGRN2): the head, its row of o and the mLSTM's denominator are the same for the whole warp
	const bool one_head = a.unit == a.vdim;
	const int h0 = c0 / a.vdim;
	auto denominator = [&](int h) { return fmaxf(fabsf(a.o[n * a.ldo + (size_t)h * a.ohs + a.vdim]), expf(-a.m_t[n * a.heads + h])) + 1e-6f; };
	const float den0 = a.m_t && one_head ? denominator(h0) : 1.f;
	auto value = [&](int c) {
		const int h = one_head ? h0 : c / a.vdim, d = one_head ? c - c0 : c % a.vdim;
		const float* oh = a.o + n * a.ldo + (size_t)h * a.ohs;
		float v = oh[d];
		if (a.m_t) v /= one_head ? den0 : denominator(h);
		if (a.skip) v = fmaf(ldf(a.skip_w + h), a.skip[n * inner + c], v);
		if (a.gate_mode == 3) {
			const float g = a.gate[n * a.ldg + c];
			v *= g * sigmoidf_(g);
		}
		return v;
	};
	// two passes over the unit, both straight from memory: holding the values in registers between them was measured slower (the
	// unrolled rounds cost more than the second read, which comes from L1 / L2)
	float ss = 0.f;
	for (int i = lane; i < a.unit; i += 32) {
		const float v = value(c0 + i);
		ss = fmaf(v, v, ss);
	}
	ss = warp_sum(ss);
	const float r = 1.f / sqrtf(ss / (float)a.unit + a.eps) * a.mul;
	for (int i = lane; i < a.unit; i += 32) {
		const int c = c0 + i;
		float v = value(c) * r;
		if (a.w) v *= ldf(a.w + c % a.w_mod);
		if (a.gate_mode == 1) v *= sigmoidf_(a.gate[n * a.ldg + c]);
		out[n * inner + c] = to_act<AT>(v);
	}
}

// ---------------------------------------------------------------- gated recurrence whose gates read only the current token (minGRU)
// Per channel  S <- (1 - z) S + z c,  z = sigmoid(raw z),  c = u + 1/2 (u >= 0) or sigmoid(u) (u < 0);  output S silu(g).  Raw z, u and g are
// columns 0, width and 2 width of the projection.  The map of a stretch of tokens on the state is S -> A S + B, so a prompt is cut into
// chunks of `chunk` tokens: k_seq_mingru_chunk forms every chunk's (A, B) but the last's, k_seq_mingru_apply folds those before its chunk
// into the state its chunk starts from and runs the tokens.  A sequence of at most `chunk` new tokens (a decoded one) needs the second kernel only.
struct MinGruArgs {
	const float* proj;
	int ldp, width;
	float* state;  // [slots][width]
	float2* carry; // [B][slots of carry][width]: entry 0 = (0, state before the step), entry k + 1 = (A, B) of chunk k
	int chunk, carries;
};
__device__ __forceinline__ void mingru_step(float zr, float u, float& keep, float& take) { // S <- keep S + take
	const float z = sigmoidf_(zr);
	keep = 1.f - z, take = z * (u >= 0.f ? u + 0.5f : sigmoidf_(u));
}
#define MINGRU_U 8 // tokens whose inputs are requested together
__global__ void __launch_bounds__(64) k_seq_mingru_chunk(MinGruArgs a, SeqBatch sb) {
	pdl_enter(); // programmatic dependent launch: let the next kernel's launch overlap this one, then wait for the previous one
	const int ch = blockIdx.x * 64 + threadIdx.x, k = blockIdx.y, b = blockIdx.z, cnt = sb.scount[b];
	if (ch >= a.width || (long)(k + 1) * a.chunk >= cnt) return; // the last chunk's map is not needed
	float2* cr = a.carry + (size_t)b * a.carries * a.width + ch;
	if (k == 0) cr[0] = make_float2(0.f, a.state[(size_t)sb.sslot[b] * a.width + ch]);
	const float* p = a.proj + (size_t)(sb.sstart[b] + k * a.chunk) * a.ldp + ch; // walks down the tokens
	float A = 1.f, B = 0.f;
	for (int t0 = 0; t0 < a.chunk; t0 += MINGRU_U) {
		float zr[MINGRU_U], u[MINGRU_U];
#pragma unroll
		for (int i = 0; i < MINGRU_U; ++i, p += a.ldp)
			if (t0 + i < a.chunk) zr[i] = p[0], u[i] = p[a.width];
#pragma unroll
		for (int i = 0; i < MINGRU_U; ++i)
			if (t0 + i < a.chunk) {
				float keep, take;
				mingru_step(zr[i], u[i], keep, take);
				A *= keep, B = fmaf(keep, B, take);
			}
	}
	cr[(size_t)(k + 1) * a.width] = make_float2(A, B);
}
template <typename AT>
__global__ void __launch_bounds__(64) k_seq_mingru_apply(MinGruArgs a, AT* out, SeqBatch sb) {
	pdl_enter(); // programmatic dependent launch: let the next kernel's launch overlap this one, then wait for the previous one
	const int ch = blockIdx.x * 64 + threadIdx.x, k = blockIdx.y, b = blockIdx.z, cnt = sb.scount[b];
	if (ch >= a.width || (long)k * a.chunk >= cnt) return;
	float* st = a.state + (size_t)sb.sslot[b] * a.width + ch;
	float S;
	if (cnt <= a.chunk) S = *st;
	else { // the state itself is written below by the last chunk while others still start: all of them read entry 0 instead
		S = 0.f;
		const float2* cr = a.carry + (size_t)b * a.carries * a.width + ch;
#pragma unroll 8
		for (int j = 0; j <= k; ++j) {
			const float2 m = cr[(size_t)j * a.width];
			S = fmaf(m.x, S, m.y);
		}
	}
	const int first = sb.sstart[b] + k * a.chunk, nt = min(a.chunk, cnt - k * a.chunk);
	const float* p = a.proj + (size_t)first * a.ldp + ch;
	AT* o = out + (size_t)first * a.width + ch;
	for (int t0 = 0; t0 < nt; t0 += MINGRU_U) {
		float zr[MINGRU_U], u[MINGRU_U], g[MINGRU_U];
#pragma unroll
		for (int i = 0; i < MINGRU_U; ++i, p += a.ldp)
			if (t0 + i < nt) zr[i] = p[0], u[i] = p[a.width], g[i] = p[2 * a.width];
#pragma unroll
		for (int i = 0; i < MINGRU_U; ++i, o += a.width)
			if (t0 + i < nt) {
				float keep, take;
				mingru_step(zr[i], u[i], keep, take);
				S = fmaf(keep, S, take);
				*o = to_act<AT>(S * g[i] * sigmoidf_(g[i]));
			}
	}
	if (k * a.chunk + nt == cnt) *st = S;
}

// ---------------------------------------------------------------- products  Y[n][m] = sum_k X[n][k] W[m][k]
// blockIdx.z = batch (per-head products): X, W, Y advance by xbs, wbs, ybs elements.
enum { EPI_F32 = 0, EPI_ACT = 1, EPI_DYT_RES = 2, EPI_RES = 3, EPI_ACT_RELU2 = 4, EPI_DECAY = 5, EPI_SPLIT3 = 6, EPI_GLU = 7 };
struct GemmArgs {
	const void* X;
	long ldx, xbs;
	const bf16* W;
	long ldw, wbs;
	void* Y;
	long ldy, ybs;
	int N, M, K;
	int epi;                 // EPI_F32: Y fp32; EPI_ACT: Y of the activation type; EPI_DYT_RES: Y fp32 residual += tanh(alpha acc) w + b, and
	                         // with xw the new value's own Dynamic Tanh norm (xa, xw, xb), the next sublayer's input, to Y2 (activation type);
	                         // EPI_RES: Y fp32 residual += (res ? res : 0) + acc; EPI_ACT_RELU2: Y of the activation type = relu(acc)^2;
	                         // EPI_DECAY: Y fp32 = sigmoid(acc)^epi_f = exp(-softplus(-acc) * epi_f);
	                         // EPI_SPLIT3: Y of the activation type, three columns `split3` apart: hi, hi, lo (value and remainder of its rounding);
	                         // EPI_GLU: rows of W alternate gate and up, Y[n][m / 2] of the activation type = glu_unit(gate, up)
	float epi_f;
	const bf16 *nw, *nb, *na;
	const bf16 *xw, *xb, *xa;
	int w_immutable;         // W is a model weight: it may be read before the previous kernel has finished (products of gathered keys set 0)
	const bf16* bias;        // [batch][M] or null: added to the accumulator first
	const float* res;        // EPI_RES: a second addend laid out like Y, or null
	const float* gate;       // EPI_ACT: the output is multiplied by sigmoid(gate[z * gbs + n * ldgate + m]); null: none
	long ldgate, gbs;
	const int* seg;          // grouped products: batch z owns rows [seg[z], seg[z+1]) of X and Y (xbs = ybs = 0), N bounds one group; null: none
	int x_rows;              // grouped products: rows of X and Y over all groups
	int split;               // > 0: output columns m >= split leave in the activation type to Y2[n][m - split] (row stride ldy2), whatever epi says:
	int split_act = 0;       //      as relu(acc)^2 (0) or as they are (1)
	void* Y2;
	long ldy2;
	float out_scale = 0.f;   // != 0: the accumulator (after the bias) is multiplied by it
	float out_cap = 0.f;     // > 0: then out_cap tanh(. / out_cap)
	const float* rs = nullptr; // a factor per row on the accumulator (after the bias): rs[(rs_idx ? rs_idx[row] : row) * rs_ld], through a sigmoid when rs_act is 1
	const int* rs_idx = nullptr;
	long rs_ld = 1;
	int rs_act = 0;
	int split3 = 0;
	int glu_mode = 0;        // EPI_GLU: as k_seq_ff_act
	float glu_limit = 0.f;
	const int* x_idx = nullptr; // k_seq_gemm_skinny only: row r of X is X[x_idx[r] / x_div] (r counts from the group's first row on)
	int x_div = 1;
	int band_mode = 0;       // k_seq_gemm_tc only.  1: tiles of Y (rows n, columns m) that `band` does not meet are left out; 2: so are 64-deep steps of the
	AttBand band;            // sum over k (columns of the band; with band_cp > 0 the columns are held twice, band_cp apart) that a tile's rows do not meet
	int band_cp = 0;
};
// rows of batch z: first row and count
struct GemmRows {
	int base, count;
};
__device__ __forceinline__ GemmRows gemm_rows(const GemmArgs& a, int z) {
	if (!a.seg) return GemmRows{0, a.N};
	const int b = a.seg[z];
	return GemmRows{b, a.seg[z + 1] - b};
}
template <typename AT>
__device__ __forceinline__ void gemm_store(const GemmArgs& a, int z, const GemmRows& gr, int n, int m, float acc) {
	if (n >= gr.count || m >= a.M) return;
	const size_t o = (size_t)z * a.ybs + (size_t)(gr.base + n) * a.ldy + m;
	if (a.bias) acc += ldf(a.bias + (size_t)z * a.M + m);
	if (a.out_scale != 0.f) acc *= a.out_scale;
	if (a.out_cap > 0.f) acc = a.out_cap * tanhf(acc / a.out_cap);
	if (a.rs) {
		const float f = a.rs[(size_t)(a.rs_idx ? a.rs_idx[gr.base + n] : gr.base + n) * a.rs_ld];
		acc *= a.rs_act ? sigmoidf_(f) : f;
	}
	if (a.split > 0 && m >= a.split) {
		const float r = fmaxf(acc, 0.f);
		((AT*)a.Y2)[(size_t)(gr.base + n) * a.ldy2 + (m - a.split)] = to_act<AT>(a.split_act ? acc : r * r);
		return;
	}
	if (a.epi == EPI_F32) ((float*)a.Y)[o] = acc;
	else if (a.epi == EPI_SPLIT3) {
		AT* y = (AT*)a.Y + o;
		y[0] = to_act<AT>(acc), y[a.split3] = y[0], y[2 * a.split3] = to_act<AT>(acc - ldf(y));
	} else if (a.epi == EPI_ACT) {
		if (a.gate) acc *= sigmoidf_(a.gate[(size_t)z * a.gbs + (size_t)(gr.base + n) * a.ldgate + m]);
		((AT*)a.Y)[o] = to_act<AT>(acc);
	} else if (a.epi == EPI_RES) ((float*)a.Y)[o] += a.res ? a.res[o] + acc : acc;
	else if (a.epi == EPI_DECAY) ((float*)a.Y)[o] = expf(-softplusf_(-acc) * a.epi_f);
	else if (a.epi == EPI_ACT_RELU2) {
		const float r = fmaxf(acc, 0.f);
		((AT*)a.Y)[o] = to_act<AT>(r * r);
	} else {
		const float y = ((float*)a.Y)[o] + (tanhf(ldf(a.na) * acc) * ldf(a.nw + m) + ldf(a.nb + m));
		((float*)a.Y)[o] = y;
		if (a.xw) ((AT*)a.Y2)[(size_t)(gr.base + n) * a.ldy2 + m] = to_act<AT>(tanhf(ldf(a.xa) * y) * ldf(a.xw + m) + ldf(a.xb + m));
	}
}

// EPI_GLU: the pair of columns m (even: gate) and m + 1 (up)
template <typename AT>
__device__ __forceinline__ void gemm_store_glu(const GemmArgs& a, int z, const GemmRows& gr, int n, int m, float gate, float up) {
	if (n >= gr.count || m >= a.M) return;
	((AT*)a.Y)[(size_t)z * a.ybs + (size_t)(gr.base + n) * a.ldy + (m >> 1)] = to_act<AT>(glu_unit(gate, up, a.glu_limit, a.glu_mode));
}
// columns m (even) and m + 1 of row n
template <typename AT>
__device__ __forceinline__ void gemm_store2(const GemmArgs& a, int z, const GemmRows& gr, int n, int m, float x, float y) {
	if (a.epi == EPI_GLU) gemm_store_glu<AT>(a, z, gr, n, m, x, y);
	else gemm_store<AT>(a, z, gr, n, m, x), gemm_store<AT>(a, z, gr, n, m + 1, y);
}

// exact mode: fp32 FMA, 64 x 64 tile, 16-deep steps, 256 threads with 4 x 4 outputs each
__global__ void __launch_bounds__(256) k_seq_gemm_f32(GemmArgs a) {
	pdl_enter(); // programmatic dependent launch: let the next kernel's launch overlap this one, then wait for the previous one
	__shared__ float Xs[16][64 + 4], Ws[16][64 + 4];
	const int z = blockIdx.z, n0 = blockIdx.y * 64, m0 = blockIdx.x * 64, tid = threadIdx.x;
	const GemmRows gr = gemm_rows(a, z);
	if (n0 >= gr.count) return;
	const float* X = (const float*)a.X + (size_t)z * a.xbs + (size_t)gr.base * a.ldx;
	const bf16* W = a.W + (size_t)z * a.wbs;
	const int tn = (tid / 16) * 4, tm = (tid % 16) * 4;
	float acc[4][4] = {};
	for (int k0 = 0; k0 < a.K; k0 += 16) {
		for (int i = tid; i < 64 * 16; i += 256) {
			const int r = i / 16, k = i % 16;
			Xs[k][r] = (n0 + r < gr.count && k0 + k < a.K) ? X[(size_t)(n0 + r) * a.ldx + k0 + k] : 0.f;
			Ws[k][r] = (m0 + r < a.M && k0 + k < a.K) ? ldf(W + (size_t)(m0 + r) * a.ldw + k0 + k) : 0.f;
		}
		__syncthreads();
#pragma unroll
		for (int k = 0; k < 16; ++k) {
			float xv[4], wv[4];
#pragma unroll
			for (int i = 0; i < 4; ++i) xv[i] = Xs[k][tn + i], wv[i] = Ws[k][tm + i];
#pragma unroll
			for (int i = 0; i < 4; ++i)
#pragma unroll
				for (int j = 0; j < 4; ++j) acc[i][j] = fmaf(xv[i], wv[j], acc[i][j]);
		}
		__syncthreads();
	}
#pragma unroll
	for (int i = 0; i < 4; ++i)
#pragma unroll
		for (int j = 0; j < 4; j += 2) gemm_store2<float>(a, z, gr, n0 + tn + i, m0 + tm + j, acc[i][j], acc[i][j + 1]);
}

// bf16 x bf16 -> fp32 on the tensor cores for ANY shape (edges are zero-filled in shared memory): 64 tokens x 64 rows per
// CTA, 32-deep steps, four warps of 32 x 32.  The tcgen05 kernel below takes the shapes that fill its tiles.
#define GB_LD 40 // bf16 per shared-memory row: 32 + 8 keeps the fragment reads conflict-free
__device__ __forceinline__ void gemm_fill_tile(bf16 (*dst)[GB_LD], const bf16* src, long ld, int r0, int rows, int k0, int K, int tid) {
	// 64 rows x 32 columns as 256 groups of 8: two per thread
	for (int i = tid; i < 256; i += 128) {
		const int r = i >> 2, c = (i & 3) * 8;
		const bf16* p = src + (size_t)(r0 + r) * ld + k0 + c;
		uint4 v = make_uint4(0, 0, 0, 0);
		if (r0 + r < rows) {
			if (k0 + c + 8 <= K && (((uintptr_t)p) & 15) == 0) v = *(const uint4*)p;
			else {
				bf16 t[8];
#pragma unroll
				for (int e = 0; e < 8; ++e) t[e] = k0 + c + e < K ? p[e] : __float2bfloat16_rn(0.f);
				v = *(const uint4*)t;
			}
		}
		*(uint4*)&dst[r][c] = v;
	}
}
__global__ void __launch_bounds__(128) k_seq_gemm_bf16(GemmArgs a) {
	pdl_enter(); // programmatic dependent launch: let the next kernel's launch overlap this one, then wait for the previous one
	__shared__ __align__(16) bf16 Xs[64][GB_LD], Ws[64][GB_LD];
	const int z = blockIdx.z, n0 = blockIdx.y * 64, m0 = blockIdx.x * 64, tid = threadIdx.x;
	const GemmRows gr = gemm_rows(a, z);
	if (n0 >= gr.count) return;
	const bf16* X = (const bf16*)a.X + (size_t)z * a.xbs + (size_t)gr.base * a.ldx;
	const bf16* W = a.W + (size_t)z * a.wbs;
	const int warp = tid >> 5, lane = tid & 31, g = lane >> 2, t = lane & 3;
	const int wn = (warp >> 1) * 32, wm = (warp & 1) * 32;
	float acc[2][4][4] = {};
	for (int k0 = 0; k0 < a.K; k0 += 32) {
		gemm_fill_tile(Xs, X, a.ldx, n0, gr.count, k0, a.K, tid);
		gemm_fill_tile(Ws, W, a.ldw, m0, a.M, k0, a.K, tid);
		__syncthreads();
#pragma unroll
		for (int kk = 0; kk < 32; kk += 16) {
			uint32_t A[2][4], B[4][2];
#pragma unroll
			for (int i = 0; i < 2; ++i) {
				const int r = wn + i * 16 + g;
				A[i][0] = *(const uint32_t*)&Xs[r][kk + 2 * t], A[i][1] = *(const uint32_t*)&Xs[r + 8][kk + 2 * t];
				A[i][2] = *(const uint32_t*)&Xs[r][kk + 2 * t + 8], A[i][3] = *(const uint32_t*)&Xs[r + 8][kk + 2 * t + 8];
			}
#pragma unroll
			for (int j = 0; j < 4; ++j) {
				const int r = wm + j * 8 + g;
				B[j][0] = *(const uint32_t*)&Ws[r][kk + 2 * t], B[j][1] = *(const uint32_t*)&Ws[r][kk + 2 * t + 8];
			}
#pragma unroll
			for (int i = 0; i < 2; ++i)
#pragma unroll
				for (int j = 0; j < 4; ++j) mma_bf16_16816(acc[i][j], A[i], B[j]);
		}
		__syncthreads();
	}
#pragma unroll
	for (int i = 0; i < 2; ++i)
#pragma unroll
		for (int j = 0; j < 4; ++j) {
			const int n = n0 + wn + i * 16 + g, m = m0 + wm + j * 8 + 2 * t;
			gemm_store2<bf16>(a, z, gr, n, m, acc[i][j][0], acc[i][j][1]), gemm_store2<bf16>(a, z, gr, n + 8, m, acc[i][j][2], acc[i][j][3]);
		}
}

// Few tokens (decode): every weight is used once, so the kernel is a stream over W.  A CTA owns 16 weight rows, its warps (8, or 16 when the matrix has few rows)
// take interleaved 32-wide slices of K; a lane loads 16 bytes of row g and of row g + 8 per slice straight into the A
// fragments of two m16n8k16 MMAs (the k order inside a slice is permuted the same way for A and B, which a sum over k does
// not see); tokens are the MMA's N.  The warps' partial tiles are added in warp order through shared memory.
template <int NT, int NW>
__global__ void __launch_bounds__(NW * 32) k_seq_gemm_skinny(GemmArgs a) {
	__shared__ float red[NW][16][NT * 8 + 1];
	const int z = blockIdx.z, m0 = blockIdx.x * 16, tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, g = lane >> 2, t = lane & 3;
	bool waited = false;
	pdl_launch_next();
	GemmRows gr{0, a.N};
	if (a.seg) { // the groups come from the previous kernel: a group without rows leaves before it touches its weights
		pdl_wait_prev(), waited = true;
		gr = gemm_rows(a, z);
		if (gr.count == 0) return;
	}
	const bf16* X = (const bf16*)a.X + (size_t)z * a.xbs + (a.x_idx ? 0 : (size_t)gr.base * a.ldx);
	const bf16* W = a.W + (size_t)z * a.wbs;
	const bf16* w0 = W + (size_t)min(m0 + g, a.M - 1) * a.ldw;
	const bf16* w1 = W + (size_t)min(m0 + g + 8, a.M - 1) * a.ldw;
	float acc[NT][4] = {};
	const int nslice = (a.K + 31) / 32;
	constexpr int U = 4; // slices requested before the first is used: 8 x 16 bytes in flight per lane
	if (!a.w_immutable && !waited) pdl_wait_prev(), waited = true;
	long xrow[NT]; // this lane's rows of X (a routed token's own row where the rows are not grouped)
#pragma unroll
	for (int j = 0; j < NT; ++j) {
		const int n = j * 8 + g;
		xrow[j] = a.x_idx ? (n < gr.count ? (long)(a.x_idx[gr.base + n] / a.x_div) * a.ldx : 0) : (long)n * a.ldx; // x_idx comes with groups: the previous kernel has been waited for
	}
	for (int s0 = warp; s0 < nslice; s0 += NW * U) {
		uint4 A0[U], A1[U];
#pragma unroll
		for (int u = 0; u < U; ++u) {
			const int k = (s0 + NW * u) * 32 + 8 * t;
			A0[u] = A1[u] = make_uint4(0, 0, 0, 0);
			if (k < a.K) A0[u] = __ldcs((const uint4*)(w0 + k)), A1[u] = __ldcs((const uint4*)(w1 + k));
		}
		if (!waited) pdl_wait_prev(), waited = true; // the first weights (immutable) are already on their way; the activations need the previous kernel
#pragma unroll
		for (int u = 0; u < U; ++u) {
			const int k = (s0 + NW * u) * 32 + 8 * t;
			const uint32_t F0[4] = {A0[u].x, A1[u].x, A0[u].y, A1[u].y}, F1[4] = {A0[u].z, A1[u].z, A0[u].w, A1[u].w};
#pragma unroll
			for (int j = 0; j < NT; ++j) {
				uint4 B = make_uint4(0, 0, 0, 0);
				const int n = j * 8 + g;
				if (n < gr.count && k < a.K) B = *(const uint4*)(X + xrow[j] + k);
				const uint32_t B0[2] = {B.x, B.y}, B1[2] = {B.z, B.w};
				mma_bf16_16816(acc[j], F0, B0);
				mma_bf16_16816(acc[j], F1, B1);
			}
		}
	}
	if (!waited) pdl_wait_prev(); // a warp without a slice still must not write before the previous kernel is done
#pragma unroll
	for (int j = 0; j < NT; ++j) {
		red[warp][g][j * 8 + 2 * t] = acc[j][0], red[warp][g][j * 8 + 2 * t + 1] = acc[j][1];
		red[warp][g + 8][j * 8 + 2 * t] = acc[j][2], red[warp][g + 8][j * 8 + 2 * t + 1] = acc[j][3];
	}
	__syncthreads();
	for (int i = tid; i < 16 * NT * 8; i += NW * 32) {
		const int n = i / 16, r = i % 16; // consecutive threads: consecutive weight rows of one token
		float v = 0.f;
#pragma unroll
		for (int w = 0; w < NW; ++w) v += red[w][r][n];
		if (a.epi == EPI_GLU) { // whole warps get here: 16 * NT * 8 is a multiple of 32
			const float up = __shfl_down_sync(0xffffffffu, v, 1);
			if (!(r & 1)) gemm_store_glu<bf16>(a, z, gr, n, m0 + r, v, up);
		} else gemm_store<bf16>(a, z, gr, n, m0 + r, v);
	}
}

// ---------------------------------------------------------------- sampling helper
// One CTA per row, 16-byte loads (rows of whole float4s), four of them out at a time per thread: 16 rows of 32000 logits 33 us with 256 threads and one float after the
// other, now 6.3.
__global__ void __launch_bounds__(1024) k_seq_argmax(const float* logits, int vocab, int* out) {
	pdl_enter(); // programmatic dependent launch: let the next kernel's launch overlap this one, then wait for the previous one
	__shared__ float bv[32];
	__shared__ int bi[32];
	const float* row = logits + (size_t)blockIdx.x * vocab;
	float v = -INFINITY;
	int ix = 0x7fffffff;
	auto see = [&](float z, int i) { // ascending i per thread: the first maximum stays
		if (z > v) v = z, ix = i;
	};
	int i = threadIdx.x;
	if (vocab % 4 == 0) {
		const float4* row4 = reinterpret_cast<const float4*>(row);
		const int n4 = vocab / 4, nt = blockDim.x;
		auto four = [&](float4 q, int k) { see(q.x, 4 * k), see(q.y, 4 * k + 1), see(q.z, 4 * k + 2), see(q.w, 4 * k + 3); };
		for (; i + 3 * nt < n4; i += 4 * nt) {
			const float4 a = row4[i], b = row4[i + nt], c = row4[i + 2 * nt], d = row4[i + 3 * nt];
			four(a, i), four(b, i + nt), four(c, i + 2 * nt), four(d, i + 3 * nt);
		}
		for (; i < n4; i += nt) four(row4[i], i);
	} else
#pragma unroll 4
		for (; i < vocab; i += blockDim.x) see(row[i], i);
	for (int o = 16; o > 0; o >>= 1) {
		const float ov = __shfl_xor_sync(0xffffffffu, v, o);
		const int oi = __shfl_xor_sync(0xffffffffu, ix, o);
		if (ov > v || (ov == v && oi < ix)) v = ov, ix = oi;
	}
	if ((threadIdx.x & 31) == 0) bv[threadIdx.x >> 5] = v, bi[threadIdx.x >> 5] = ix;
	__syncthreads();
	if (threadIdx.x == 0) {
		for (int w = 1; w < (int)(blockDim.x >> 5); ++w)
			if (bv[w] > v || (bv[w] == v && bi[w] < ix)) v = bv[w], ix = bi[w];
		out[blockIdx.x] = ix;
	}
}
