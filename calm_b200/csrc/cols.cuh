// cols.cuh -- the matvec stages of a token (q/k/v, wo, FFN up, FFN down) on the tensor cores, with the weights requested ahead of the previous
// kernel's end.  fp8 and fp16 models (gf4: unpacking the words into f16 pairs took 23 us for FFN up, k_ffn_up_ring 22).
//
// Why: a token is a chain of short launches, and between the last byte of one and the first use of the next the memory stands still: the
// predecessor's last rows, its flush, the activation vector on its way, a DRAM round trip.  Here a CTA (one per SM) owns a contiguous
// range of rows, and two warps of it do nothing but copy their pieces into a ring of stages with cp.async.bulk.  They depend on nothing that the
// previous kernel writes, so they start the moment the CTA is resident; ring, registers and threads are at most half of an SM's, so that the
// CTA IS resident while the previous kernel still runs (programmatic dependent launch), and the ring is full when the dependency wait returns.
//
// Arithmetic: mma.m16n8k16, f16 x f16 -> f32, 8 rows of weights at a time.  Weights are exact in f16 (e5m2: a byte permute), the
// activations are three f16 pieces of a value scaled by the power of two that brings a warp's largest one (of a row; of a piece of it in wo and w2) to 2^14: all 24 bits down to 2^-34 of
// it, steps of 2^-58 of it below (with the pieces at one scale and 2^7 the 24 bits ended at 2^-9, and rows whose weights met only entries of 2^-20 of the largest were 3e-5 off, of 2^-26
// 4e-3; 1e-7 now).  A row of weights goes through a product
// twice at once: rows g of A are 64 bytes (a step) of row g, rows g + 8 the next step of the same row, columns 0 - 2 of B the pieces of the first step's activations
// and columns 3 - 5 of the second's; the sums wanted are those of rows 0 - 7 in columns 0 - 2 and of rows 8 - 15 in columns 3 - 5.  So no product is
// spent on padding rows and a warp's activations take half the registers.  A warp of 8 owns two or four steps of every 2 KB of a row; lane (g, t) reads 16
// contiguous bytes for a step and takes their k in the order they lie in -- B has the same order.  An SM starts one such product every two cycles (measured,
// 16 warps).  Dot products of packed FP32 FMA in this frame took 4.3 instructions a weight at 60 % of the issue slots (conversions, a transposing
// reduction per row: FFN up 25.6 us against 24).
// The tensor core truncates where it aligns and adds, so the first piece has 8 bits and two products (fp16) or those of a stage, eight at most (fp8), add up in it before an FP32 addition.
// Distance from 64 bits, as a share of that of the FP32 dot products of ring.cuh (1.3 to 1.7e-7 for a row of w2, 2 to 3e-7 for FFN up): fp8 rows of 4096, 14336 and 28672 weights, normal
// and gated activations, 0.48 to 0.71, FFN up 0.55 and 0.68 (2048); fp16 0.84 to 0.98, FFN up 0.63 and 0.86 (1024).  Whole rows of fp8 in the tensor core were 1.5 (4096) to 11 times (28672) as far off as the ring's.
// The 8 warps' sums of a tile of 8 rows go through shared memory to one more warp, which adds them in order (deterministic) and applies the
// stage's epilogue while the others are at the next tile (left to the last of the 8, this held up the slowest one: FFN up 29 us instead of 24).
//
// Two warps copy, in turn: a warp issues a bulk copy every 95 cycles, which is what 2 KB take at the memory's rate.
//
// Two orders of the pieces of a CTA's rows: tile by tile with the whole vector's pieces in registers (q/k/v, FFN up), or one piece of all
// rows after the other with one accumulator per tile and the vector's pieces made as they are needed (wo, w2: few rows, long ones).
//
// Measured, a whole token: Qwen2-0.5B fp16 at 131 positions 906 -> 639 us, Llama-3-8B fp8 at 4095 2215 -> 2149; tokens of six layers between those
// widths 1.00 to 1.26 times as fast (k_qkv, k_matres, ring.cuh before), four layers of 5120 to 8192 wide models 1.02 to 1.32 times.  By stage, Llama-3-8B fp8: q/k/v 8.5 -> 6.9 us, wo 7.4 -> 6.9,
// FFN up 19.9, w2 13.9 -> 14.1; 0.5B: 4.2 -> 1.8, 3.5 -> 1.5, 6.7 -> 4.2, 7.8 -> 3.6.  Rows of 4096 fp16 weights are where the ring is as good: w2 18.0 us there, 20.2 here.
// What bounds it now: about 2 us from the last store of a stage to the first product of the next (the grid's end is seen after 1.1 us, the vector's way to the registers and its pieces take
// the rest), then the memory's rate.
#pragma once

#include "stages.cuh"
#include "tc05.cuh"

#define COLS_WARPS 8                         // multiplying warps; then two that copy and the epilogue's
#define COLS_THREADS (32 * (COLS_WARPS + 3))
#define COLS_CHUNK 2048                      // bytes of a row in a stage, at most: 8 warps x 4 steps of 64
#define COLS_PITCH (COLS_CHUNK + 64)         // of the rows of a stage: 8 lanes read 64 bytes of two rows at a time, without bank conflicts
#define COLS_STAGE (8 * COLS_PITCH)
#define COLS_STAGES 6
#define COLS_PARTS 8                         // tiles whose sums may wait for the epilogue
#define COLS_PAIRS 64                        // row pairs of a CTA whose angles and biases are loaded ahead
#define COLS_TILES 8                         // tiles of a CTA in the second order, at most
// dynamic shared memory: ring, the warps' sums, their scratch for splitting activations (3 pieces of 128)
#define COLS_SMEM (COLS_STAGES * COLS_STAGE + COLS_PARTS * COLS_WARPS * 8 * 4 + COLS_WARPS * 768)

template <int DBITS>
struct ColsStep { // 64 bytes of a row
	static constexpr int K = 64 * 8 / DBITS; // weights
	static constexpr int B = K / 8;          // registers of a lane's activations of two steps
	static constexpr int F = 4 * K / 32;     // a lane's activations of its steps, as they are loaded
};

// The chain keeps one CTA of each of two kernels on an SM only if it starts so: where a kernel follows one that leaves no room for it (attention), the SMs that are
// free first would take two of its CTAs, the last ones none, and every kernel behind it would inherit that (FFN up of Llama-3-8B fp8: 27 us, 20 evenly).
// wo asks for this much shared memory: two of its CTAs do not fit an SM, one beside one of FFN up's does.
#define COLS_ALONE 115200

// An activation is three f16 pieces: its first 8 bits, what they leave times COLS_MID, what that leaves times COLS_LO (a piece has columns, and so sums, of its own)
#define COLS_MID 256.f
#define COLS_LO 524288.f

struct ColsRun {
	int steps, chunk_steps; // 64-byte steps of a row, and of its pieces in a stage (the last may have fewer)
	int own;                // of a piece's steps, those of a warp: 2 or 4
	int* err;               // mapped host word: a wait that gave up
	unsigned tries;         // of a wait before it gives up (the multiplying warps of k_matres_cols: none if this is 0, else MBAR_SPINS; a limit in a register cost 0.3 us a launch there)
};

struct ColsShared {
	uint64_t full[COLS_STAGES], empty[COLS_STAGES], part_full[COLS_PARTS], part_empty[COLS_PARTS];
	float ss[COLS_WARPS]; // sums of squares
	float rows[8 * COLS_TILES]; // wo, w2: what the rows' sums are added to; tensor parallelism: this rank's partials, summed over the ranks at the end
	float4 pair[COLS_PAIRS];    // q/k/v: angle (cos, sin) and bias of the CTA's first row pairs, loaded ahead of their use
	int gave_up;
};

__device__ __forceinline__ void cols_init(ColsShared* sh) {
	if (threadIdx.x < COLS_STAGES) mbar_init(&sh->full[threadIdx.x], 1), mbar_init(&sh->empty[threadIdx.x], COLS_WARPS);
	if (threadIdx.x < COLS_PARTS) {
		mbar_init(&sh->part_full[threadIdx.x], COLS_WARPS), mbar_init(&sh->part_empty[threadIdx.x], 1);
		mbar_init_fence();
	}
	if (threadIdx.x == 0) sh->gave_up = 0;
	__syncthreads();
}

// a CTA's share of n units
__device__ __forceinline__ int cols_share(int n, int b) {
	return (int)(((long long)b * n) / gridDim.x);
}

// The dependency wait of a CTA: one warp waits for the grid, the others at a barrier.
__device__ __forceinline__ void cols_wait_prev(bool polls) {
	if (polls) pdl_wait_prev();
	asm volatile("bar.sync 1, %0;" ::"n"(COLS_THREADS) : "memory");
}

// Every wait is bounded: a role whose wait gives up leaves its loop with a code, and the others' waits then run out too.  Nearly all waits end with their first try; what follows
// is kept out of the way, since a kernel's code is read anew in every launch and most launches are short (q/k/v and FFN up of Llama-3-8B fp8 6.9 and 19.8 us; with the loop in place 7.3 and 21.7).
static __device__ __noinline__ bool cols_wait_on(ColsShared* sh, uint64_t* bar, uint32_t parity, unsigned tries, int code) {
	if (mbar_wait_warp(bar, parity, tries)) return true;
	if ((threadIdx.x & 31) == 0) sh->gave_up = code;
	return false;
}
__device__ __forceinline__ bool cols_wait(ColsShared* sh, uint64_t* bar, uint32_t parity, const ColsRun& r, int code) {
	return __all_sync(0xffffffffu, mbar_try_wait(bar, parity) && r.tries) || cols_wait_on(sh, bar, parity, r.tries, code);
}

// A copying warp (of two: they take the stages in turn).  order(i, tile, chunk): what stage i holds; row(tile, slot): where the weights of the tile's row `slot` begin, NULL: no such row.
// Whichever role gives up, nothing is in flight into this CTA's shared memory when it exits: these warps wait for their last copies themselves, at a time when others need those too.
template <typename OrderFn, typename RowFn>
__device__ __forceinline__ void cols_produce(ColsShared* sh, const ColsRun& r, unsigned char* ring, int nst, OrderFn order, RowFn row) {
	const int lane = threadIdx.x & 31, which = (threadIdx.x >> 5) - COLS_WARPS;
	const uint64_t policy = l2_policy_evict_first();
	bool waited = false;
	int i = which;
	for (; i < nst; i += 2) {
		const int slot = i % COLS_STAGES;
		if (i >= COLS_STAGES) {
			if (!waited) cols_wait_prev(which == 0), waited = true; // no stage is free before the others have activations
			if (!cols_wait(sh, &sh->empty[slot], ((i / COLS_STAGES) & 1) ^ 1, r, 9401)) break;
		}
		int tile, chunk;
		order(i, tile, chunk);
		const uint32_t bytes = min(r.chunk_steps, r.steps - chunk * r.chunk_steps) * 64;
		const unsigned char* src = lane < 8 ? row(tile, lane) : nullptr;
		const unsigned n = __popc(__ballot_sync(0xffffffffu, src != nullptr));
		if (lane == 0) mbar_expect_tx(&sh->full[slot], n * bytes);
		__syncwarp();
		if (src) tma_load_1d_hint(ring + slot * COLS_STAGE + lane * COLS_PITCH, src + (size_t)chunk * r.chunk_steps * 64, bytes, &sh->full[slot], policy);
	}
	if (!waited) cols_wait_prev(which == 0);
	for (int k = i - 2; k >= max(0, i - COLS_STAGES); k -= 2) mbar_wait_warp(&sh->full[k % COLS_STAGES], (k / COLS_STAGES) & 1); // the last stage of each of its slots
}

__device__ __forceinline__ void mma16816(float (&d)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0, uint32_t b1) {
	asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
	             : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
	             : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}

// biased exponent of the largest magnitude, and the power of two that brings it to [2^14, 2^15)
__device__ __forceinline__ int cols_exponent(float m) { return max((int)(__float_as_uint(m) >> 23), 37); } // (below 2^-90 the third piece's steps are FP32's; an infinity stays one)
__device__ __forceinline__ float cols_scale(int e) { return __uint_as_float((uint32_t)(268 - e) << 23); }
__device__ __forceinline__ float cols_unscale(int e) { return __uint_as_float((uint32_t)(e - 14) << 23); }
// a warp's activations at the scale that their largest magnitude asks for; returns what undoes it
template <int N>
__device__ __forceinline__ float cols_to_scale(float (&f)[N]) {
	float most = 0.f;
#pragma unroll
	for (int k = 0; k < N; ++k) most = fmaxf(most, fabsf(f[k]));
	const int e = cols_exponent(warp_max(most));
	const float scale = cols_scale(e);
#pragma unroll
	for (int k = 0; k < N; ++k) f[k] *= scale;
	return cols_unscale(e);
}

struct ColsLane {
	int lane, warp, g, t;
	__device__ __forceinline__ ColsLane() : lane(threadIdx.x & 31), warp(threadIdx.x >> 5), g(lane >> 2), t(lane & 3) {}
	// steps of this warp in chunk c of a row
	__device__ __forceinline__ int own(const ColsRun& r, int c) const {
		const int steps = min(r.chunk_steps, r.steps - c * r.chunk_steps);
		return max(0, min(r.own, steps - r.own * warp));
	}
	__device__ __forceinline__ float2 worth(float unscale) const { // of a sum in either of its two columns (pieces 0 1 | 2 0 | 1 2)
		constexpr float mid = 1.f / COLS_MID, lo = 1.f / COLS_LO;
		return make_float2(unscale * (t == 0 ? 1.f : t == 1 ? lo : mid), unscale * (t == 0 ? mid : t == 1 ? 1.f : lo));
	}
	// this warp's first activation in chunk c
	template <int DBITS>
	__device__ __forceinline__ size_t at(const ColsRun& r, int c) const { return (size_t)(c * r.chunk_steps + r.own * warp) * ColsStep<DBITS>::K; }
};

// The pieces of 64 activations (f0, f1: elements 2 lane and 2 lane + 1, scaled) into 384 bytes of the warp's own.
__device__ __forceinline__ void cols_split(uint32_t* buf, int lane, float f0, float f1) {
	// The first piece is 8 bits, not 11: a product of 16 terms aligns them to the largest and drops what falls off its end, which is less the shorter they are
	// (8 + 11 + 11 bits still hold all 24).
	const __half2 hi = __floats2half2_rn(__uint_as_float(__float_as_uint(f0) & 0xffff0000u), __uint_as_float(__float_as_uint(f1) & 0xffff0000u));
	float r0 = f0 - __low2float(hi), r1 = f1 - __high2float(hi);
	r0 = fabsf(f0) <= FLT_MAX ? r0 : 0.f, r1 = fabsf(f1) <= FLT_MAX ? r1 : 0.f; // an infinity has no remainder
	r0 *= COLS_MID, r1 *= COLS_MID;
	const __half2 mid = __floats2half2_rn(r0, r1);
	constexpr float next = COLS_LO / COLS_MID;
	const __half2 lo = __floats2half2_rn((r0 - __low2float(mid)) * next, (r1 - __high2float(mid)) * next);
	buf[lane] = *reinterpret_cast<const uint32_t*>(&hi), buf[32 + lane] = *reinterpret_cast<const uint32_t*>(&mid), buf[64 + lane] = *reinterpret_cast<const uint32_t*>(&lo);
}
// A warp's activations of one chunk as B fragments: f[2 k], f[2 k + 1] are elements 64 k + 2 lane, + 1, scaled.
template <int DBITS>
struct ColsFragments {
	static constexpr int B = ColsStep<DBITS>::B, F = ColsStep<DBITS>::F;
	uint32_t b[2][B];

	__device__ __forceinline__ void make(uint32_t* buf, const ColsLane& l, const float* f) {
		const int which = l.g >= 3, piece = l.g - 3 * which; // lanes of g = 6, 7 hold nothing
		auto take = [&](uint32_t* d, const uint32_t* from, int at, bool on) { // eight halves
			if (on && l.g < 6) {
				const uint4 v = *reinterpret_cast<const uint4*>(from + piece * 32 + at * 4);
				d[0] = v.x, d[1] = v.y, d[2] = v.z, d[3] = v.w;
			}
		};
#pragma unroll
		for (int p = 0; p < 2; ++p)
#pragma unroll
			for (int i = 0; i < B; ++i) b[p][i] = 0;
#pragma unroll
		for (int k = 0; k < F / 2; k += 2) { // 128 activations at a time
			__syncwarp(); // the previous pieces have been read
			cols_split(buf, l.lane, f[2 * k], f[2 * k + 1]);
			cols_split(buf + 96, l.lane, f[2 * k + 2], f[2 * k + 3]);
			__syncwarp();
#pragma unroll
			for (int h = 0; h < 2; ++h) {
				if constexpr (DBITS == 16) { // both steps of 32 of a pair
					take(b[k + h], buf + 96 * h, 4 * which + l.t, true);
				} else { // a step of 64
#pragma unroll
					for (int q = 0; q < 2; ++q) take(b[k / 2] + 4 * q, buf + 96 * h, 2 * l.t + q, which == h);
				}
			}
		}
	}
};

// n steps of one stage's 8 rows; the stage is free for its next copy once they are in registers.  u: what sums in this lane's two columns are worth
template <int DBITS>
__device__ __forceinline__ void cols_multiply(ColsShared* sh, const unsigned char* ring, int slot, const ColsRun& r, const ColsLane& l, int n, const ColsFragments<DBITS>& x, float2 u, float (&acc)[4]) {
	const unsigned char* p = ring + slot * COLS_STAGE + l.g * COLS_PITCH + l.warp * r.own * 64 + l.t * 16;
	uint4 lo[2], up[2];
#pragma unroll
	for (int s = 0; s < 2; ++s) {
		lo[s] = 2 * s < n ? *reinterpret_cast<const uint4*>(p + 128 * s) : make_uint4(0, 0, 0, 0);
		up[s] = 2 * s + 1 < n ? *reinterpret_cast<const uint4*>(p + 128 * s + 64) : make_uint4(0, 0, 0, 0);
	}
	__syncwarp(); // every lane has its weights
	if (l.lane == 0) mbar_arrive(&sh->empty[slot]);
	float d[4] = {0.f, 0.f, 0.f, 0.f}; // a few products only add up in the tensor core, which truncates
	auto add = [&] { acc[0] = fmaf(d[0], u.x, acc[0]), acc[1] = fmaf(d[1], u.y, acc[1]), acc[2] = fmaf(d[2], u.x, acc[2]), acc[3] = fmaf(d[3], u.y, acc[3]); };
#pragma unroll
	for (int s = 0; s < 2; ++s) {
		if (2 * s >= n) break;
		const uint32_t wl[4] = {lo[s].x, lo[s].y, lo[s].z, lo[s].w}, wu[4] = {up[s].x, up[s].y, up[s].z, up[s].w};
		const uint32_t(&b)[ColsStep<DBITS>::B] = x.b[s];
		if constexpr (DBITS == 16) {
			d[0] = d[1] = d[2] = d[3] = 0.f;
			mma16816(d, wl[0], wu[0], wl[1], wu[1], b[0], b[1]);
			mma16816(d, wl[2], wu[2], wl[3], wu[3], b[2], b[3]);
			add();
		} else {
#pragma unroll
			for (int m = 0; m < 4; ++m)
				mma16816(d, __byte_perm(wl[m], 0, 0x1404), __byte_perm(wu[m], 0, 0x1404), __byte_perm(wl[m], 0, 0x3424), __byte_perm(wu[m], 0, 0x3424), b[2 * m], b[2 * m + 1]);
		}
	}
	if constexpr (DBITS != 16) add();
}

// this warp's sums of a tile's 8 rows: columns 0 - 2 of rows 0 - 7 and columns 3 - 5 of rows 8 - 15
__device__ __forceinline__ bool cols_hand_over(ColsShared* sh, const ColsRun& r, float* part, const ColsLane& l, int tile, const float (&acc)[4]) {
	float a = l.t == 2 ? acc[2] : acc[0], b = l.t == 0 ? acc[1] : acc[3];
	// An infinite weight: the sums of the first pieces (a of t = 0, b of t = 1) say which infinity, the other pieces may be zero or have the other sign.  (Where an activation is so far below
	// the largest beside it, 2^-39, that its first piece is zero too, the row stays a NaN.)
	// As a difference, since comparisons of a and b cost FFN up of 4096 x 14336 fp8 1.2 us and a vote of the warp 0.5.
	const float first = l.t == 0 ? a : l.t == 1 ? b : 0.f;
	float v = a + b;
	v = __fadd_rn(v, -v) == 0.f ? v : first;
	v += __shfl_xor_sync(0xffffffffu, v, 1);
	v += __shfl_xor_sync(0xffffffffu, v, 2);
	const int buf = tile % COLS_PARTS;
	if (tile >= COLS_PARTS && !cols_wait(sh, &sh->part_empty[buf], ((tile / COLS_PARTS) & 1) ^ 1, r, 9402)) return false;
	if (l.t == 0) part[(buf * COLS_WARPS + l.warp) * 8 + l.g] = v;
	__syncwarp();
	if (l.lane == 0) mbar_arrive(&sh->part_full[buf]);
	return true;
}

// The epilogue's warp: emit(tile, slot, v) with row slot lane % 8 and its sum in every eight lanes.
template <typename EmitFn>
__device__ __forceinline__ void cols_epilogue(ColsShared* sh, const ColsRun& r, const float* part, int tiles, EmitFn emit) {
	const int lane = threadIdx.x & 31, row = lane & 7, quarter = lane >> 3;
	for (int tile = 0; tile < tiles; ++tile) {
		const int buf = tile % COLS_PARTS;
		if (!cols_wait(sh, &sh->part_full[buf], (tile / COLS_PARTS) & 1, r, 9403)) return;
		const float* p = part + (buf * COLS_WARPS + quarter * (COLS_WARPS / 4)) * 8 + row;
		float v = p[0];
#pragma unroll
		for (int w = 1; w < COLS_WARPS / 4; ++w) v += p[w * 8];
		__syncwarp();
		if (lane == 0) mbar_arrive(&sh->part_empty[buf]);
		v += __shfl_xor_sync(0xffffffffu, v, 8);
		v += __shfl_xor_sync(0xffffffffu, v, 16);
		emit(tile, row, v);
	}
}
__device__ __forceinline__ float cols_rms(const ColsShared* sh, int n, float eps) { // after the first tile has arrived
	float ss = sh->ss[0];
#pragma unroll
	for (int w = 1; w < COLS_WARPS; ++w) ss += sh->ss[w];
	return 1.0f / sqrtf(ss / n + eps);
}

// Registers of a thread: two kernels of the chain share an SM's 65536 (2 x 352 threads x 88) unless rows are longer than usual.  Where 88 do not hold the vector's pieces they are kept in
// local memory, which costs more than the early start gives: FFN up 13824 x 5120 and 16384 x 6144 fp8 (three pieces of 16) 31.1 -> 26.5 us and 36.3 -> 31.9 with 168, 14336 x 5632 fp16
// (six of 8) 509 -> 500 us for a token of four layers.
constexpr int cols_regs(int pieces_and_sums) {
	return pieces_and_sums <= 40 ? 88 : 168;
}

// ---- first order: tile by tile, NC chunks a row, the vector's pieces in registers
template <int DBITS, int NC>
struct ColsTiles {
	static constexpr int F = ColsStep<DBITS>::F, REGS = cols_regs(2 * NC * ColsStep<DBITS>::B);
	ColsFragments<DBITS> x[NC];
	float f[NC * F];
	float2 u;

	// x (times the norm's weights, with the sum of its squares into sh->ss)
	__device__ __forceinline__ void load(ColsShared* sh, const ColsRun& r, const ColsLane& l, const float* __restrict__ xin, const float* __restrict__ normw) {
		float ss = 0.f;
#pragma unroll
		for (int c = 0; c < NC; ++c) {
			const int n = l.own(r, c) * ColsStep<DBITS>::K; // this warp's activations of the chunk
			const float2* p = reinterpret_cast<const float2*>(xin + l.at<DBITS>(r, c)) + l.lane;
#pragma unroll
			for (int k = 0; k < F / 2; ++k) {
				const float2 v = 64 * k < n ? __ldcg(p + 32 * k) : make_float2(0.f, 0.f);
				f[c * F + 2 * k] = v.x, f[c * F + 2 * k + 1] = v.y;
			}
		}
		if (normw) {
#pragma unroll
			for (int c = 0; c < NC; ++c) {
				const int n = l.own(r, c) * ColsStep<DBITS>::K;
				const float2* p = reinterpret_cast<const float2*>(normw + l.at<DBITS>(r, c)) + l.lane;
#pragma unroll
				for (int k = 0; k < F / 2; ++k) {
					const float2 w = 64 * k < n ? __ldg(p + 32 * k) : make_float2(0.f, 0.f);
					float &f0 = f[c * F + 2 * k], &f1 = f[c * F + 2 * k + 1];
					ss = fmaf(f0, f0, ss), ss = fmaf(f1, f1, ss);
					f0 *= w.x, f1 *= w.y;
				}
			}
			ss = warp_sum(ss);
			if (l.lane == 0) sh->ss[l.warp] = ss; // (read behind the first tile's barrier)
		}
		u = l.worth(cols_to_scale(f));
	}
	__device__ __forceinline__ void run(ColsShared* sh, const ColsRun& r, const ColsLane& l, uint32_t* buf, const unsigned char* ring, float* part, int tiles) {
		int slot = 0, parity = 0;
		const int whole = l.own(r, 0), rest = l.own(r, NC - 1);
		auto stage = [&](int c, float (&acc)[4]) {
			if (!cols_wait(sh, &sh->full[slot], parity, r, 9400)) return false;
			cols_multiply<DBITS>(sh, ring, slot, r, l, c < NC - 1 ? whole : rest, x[c], u, acc);
			if (++slot == COLS_STAGES) slot = 0, parity ^= 1;
			return true;
		};
		float acc[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
		for (int c = 0; c < NC; ++c) { // the first tile: a chunk's pieces are made when it is used, so that the first stages are free early
			x[c].make(buf, l, f + c * F);
			if (!stage(c, acc)) return;
		}
		if (!cols_hand_over(sh, r, part, l, 0, acc)) return;
		for (int tile = 1; tile < tiles; ++tile) {
			acc[0] = acc[1] = acc[2] = acc[3] = 0.f;
#pragma unroll
			for (int c = 0; c < NC; ++c)
				if (!stage(c, acc)) return;
			if (!cols_hand_over(sh, r, part, l, tile, acc)) return;
		}
	}
};

// ------------------------------------------------------------------------------------------------
// q/k/v: rows of the concatenation [wq; wk; wv], in pairs (RoPE)

template <int DBITS, int NC, typename KVT>
__global__ void __maxnreg__((ColsTiles<DBITS, NC>::REGS)) k_qkv_cols(const QkvArgs<KVT> a, const ColsRun r) {
	pdl_launch_next();
	extern __shared__ __align__(128) unsigned char smem_raw[];
	__shared__ __align__(16) ColsShared sh;
	float* part = reinterpret_cast<float*>(smem_raw + COLS_STAGES * COLS_STAGE);
	uint32_t* buf = reinterpret_cast<uint32_t*>(part + COLS_PARTS * COLS_WARPS * 8);
	const int nrows = a.q_dim + 2 * a.kv_dim;
	const int row0 = 2 * cols_share(nrows / 2, blockIdx.x), rows = 2 * cols_share(nrows / 2, blockIdx.x + 1) - row0, tiles = (rows + 7) / 8;
	const ColsLane l;
	cols_init(&sh);
	if (l.warp == COLS_WARPS || l.warp == COLS_WARPS + 1) {
		const size_t rowbytes = (size_t)r.steps * 64;
		cols_produce(&sh, r, smem_raw, tiles * NC, [&](int i, int& tile, int& chunk) { tile = i / NC, chunk = i % NC; },
		             [&](int tile, int slot) -> const unsigned char* {
			             const int j = row0 + 8 * tile + slot;
			             if (j >= row0 + rows) return nullptr;
			             if (j < a.q_dim) return (const unsigned char*)a.wq + j * rowbytes;
			             if (j < a.q_dim + a.kv_dim) return (const unsigned char*)a.wk + (j - a.q_dim) * rowbytes;
			             return (const unsigned char*)a.wv + (j - a.q_dim - a.kv_dim) * rowbytes;
		             });
	} else if (l.warp < COLS_WARPS) {
		ColsTiles<DBITS, NC> ct;
		cols_wait_prev(false);
		stamp_begin(a.stamp);
		ct.load(&sh, r, l, a.x, a.normw);
		ct.run(&sh, r, l, buf + l.warp * 192, smem_raw, part, tiles);
	} else {
		cols_wait_prev(false);
		auto pair_of = [&](int p) { // angle and bias of a row pair
			const int j = row0 + 2 * p;
			const float2 cs = j < a.q_dim + a.kv_dim ? a.rope_cs[(j % a.head_dim) >> 1] : make_float2(1.f, 0.f);
			return make_float4(cs.x, cs.y, a.bias ? a.bias[j] : 0.f, a.bias ? a.bias[j + 1] : 0.f);
		};
		for (int p = l.lane; p < min(rows / 2, COLS_PAIRS); p += 32) sh.pair[p] = pair_of(p);
		__syncwarp();
		const int kv_pos = a.tp->kv_pos;
		float post = 1.f;
		cols_epilogue(&sh, r, part, tiles, [&](int tile, int slot, float v) {
			if (tile == 0 && a.normw) post = cols_rms(&sh, a.dim, a.eps);
			v *= post;
			const float other = __shfl_xor_sync(0xffffffffu, v, 1);
			const int j = row0 + 8 * tile + slot;
			if (l.lane < 8 && !(slot & 1) && j < row0 + rows) {
				const int p = (8 * tile + slot) / 2;
				const float4 t = p < COLS_PAIRS ? sh.pair[p] : pair_of(p);
				float v0 = fminf(fmaxf(v + t.z, -a.clip), a.clip), v1 = fminf(fmaxf(other + t.w, -a.clip), a.clip);
				if (j < a.q_dim + a.kv_dim) { // rotate q and k (reference infer.c:223-236); angles from k_embed's table
					const float r0 = v0 * t.x - v1 * t.y, r1 = v0 * t.y + v1 * t.x;
					v0 = r0, v1 = r1;
				}
				if (j < a.q_dim) {
					*reinterpret_cast<float2*>(a.q_out + j) = make_float2(v0, v1);
				} else {
					const bool key = j < a.q_dim + a.kv_dim;
					const int k = j - a.q_dim - (key ? 0 : a.kv_dim), h = k / a.head_dim, d = k % a.head_dim;
					KVT* dst = (key ? a.kc : a.vc) + ((size_t)h * a.seq_len + kv_pos) * a.head_dim + d;
					kv_store(dst, v0);
					kv_store(dst + 1, v1);
				}
			}
		});
	}
	__syncthreads();
	if (a.xb_out && blockIdx.x == 0 && l.warp < COLS_WARPS) { // norm_par: the FFN reads the normalised vector
		const float post = a.normw ? cols_rms(&sh, a.dim, a.eps) : 1.f;
		for (int i = threadIdx.x; i < a.dim; i += 32 * COLS_WARPS) a.xb_out[i] = __ldcg(a.x + i) * (a.normw ? a.normw[i] : 1.f) * post;
	}
	if (threadIdx.x == 0 && sh.gave_up) *reinterpret_cast<volatile int*>(r.err) = sh.gave_up;
	stamp_end(a.stamp);
}

// ------------------------------------------------------------------------------------------------
// FFN up: hb[i] = act(w1[i] . xn) * (w3[i] . xn)  (reference infer.c:437-450).  Slots 0 - 3 of a tile are rows of w1, 4 - 7 the same rows of w3.

template <int DBITS, int NC>
__global__ void __maxnreg__((ColsTiles<DBITS, NC>::REGS)) k_ffn_up_cols(const FfnUpArgs a, const ColsRun r) {
	pdl_launch_next();
	extern __shared__ __align__(128) unsigned char smem_raw[];
	__shared__ __align__(16) ColsShared sh;
	float* part = reinterpret_cast<float*>(smem_raw + COLS_STAGES * COLS_STAGE);
	uint32_t* buf = reinterpret_cast<uint32_t*>(part + COLS_PARTS * COLS_WARPS * 8);
	const int i0 = cols_share(a.hidden, blockIdx.x), n = cols_share(a.hidden, blockIdx.x + 1) - i0, tiles = (n + 3) / 4;
	const ColsLane l;
	cols_init(&sh);
	if (l.warp == COLS_WARPS || l.warp == COLS_WARPS + 1) {
		const size_t rowbytes = (size_t)r.steps * 64;
		cols_produce(&sh, r, smem_raw, tiles * NC, [&](int i, int& tile, int& chunk) { tile = i / NC, chunk = i % NC; },
		             [&](int tile, int slot) -> const unsigned char* {
			             const int i = 4 * tile + (slot & 3);
			             return i >= n ? nullptr : (const unsigned char*)(slot < 4 ? a.w1 : a.w3) + (size_t)(i0 + i) * rowbytes;
		             });
	} else if (l.warp < COLS_WARPS) {
		ColsTiles<DBITS, NC> ct;
		cols_wait_prev(false);
		stamp_begin(a.stamp);
		ct.load(&sh, r, l, a.x, a.normw);
		ct.run(&sh, r, l, buf + l.warp * 192, smem_raw, part, tiles);
	} else {
		cols_wait_prev(false);
		float post = 1.f;
		cols_epilogue(&sh, r, part, tiles, [&](int tile, int slot, float v) {
			if (tile == 0 && a.normw) post = cols_rms(&sh, a.dim, a.eps);
			v *= post;
			const float u3 = __shfl_xor_sync(0xffffffffu, v, 4);
			const int i = 4 * tile + slot;
			if (l.lane < 4 && i < n) a.hb[i0 + i] = (a.gelu ? act_gelu(v) : act_silu(v)) * u3;
		});
	}
	__syncthreads();
	if (threadIdx.x == 0 && sh.gave_up) *reinterpret_cast<volatile int*>(r.err) = sh.gave_up;
	stamp_end(a.stamp);
}

// ------------------------------------------------------------------------------------------------
// y[row] (+)= W[row] . xin  (wo, w2; dense), the second order: T tiles

template <int DBITS, int T>
__global__ void __maxnreg__((cols_regs(2 * ColsStep<DBITS>::B + 4 * T))) k_matres_cols(const MatResArgs a, const ColsRun r) {
	pdl_launch_next();
	extern __shared__ __align__(128) unsigned char smem_raw[];
	__shared__ __align__(16) ColsShared sh;
	float* part = reinterpret_cast<float*>(smem_raw + COLS_STAGES * COLS_STAGE);
	uint32_t* buf = reinterpret_cast<uint32_t*>(part + COLS_PARTS * COLS_WARPS * 8);
	const int row0 = cols_share(a.d, blockIdx.x), rows = cols_share(a.d, blockIdx.x + 1) - row0;
	const int chunks = (r.steps + r.chunk_steps - 1) / r.chunk_steps;
	const ColsLane l;
	cols_init(&sh);
	if (l.warp == COLS_WARPS || l.warp == COLS_WARPS + 1) {
		const size_t rowbytes = (size_t)r.steps * 64;
		cols_produce(&sh, r, smem_raw, T * chunks, [&](int i, int& tile, int& chunk) { tile = i % T, chunk = i / T; },
		             [&](int tile, int slot) -> const unsigned char* {
			             const int j = 8 * tile + slot;
			             return j >= rows ? nullptr : (const unsigned char*)a.w + (size_t)(row0 + j) * rowbytes;
		             });
	} else if (l.warp < COLS_WARPS) {
		constexpr int F = ColsStep<DBITS>::F;
		float f[F], acc[T][4];
#pragma unroll
		for (int t = 0; t < T; ++t) acc[t][0] = acc[t][1] = acc[t][2] = acc[t][3] = 0.f;
		auto fetch = [&](int c) {
			const int n = c < chunks ? l.own(r, c) * ColsStep<DBITS>::K : 0;
			const float2* p = reinterpret_cast<const float2*>(a.xin + l.at<DBITS>(r, c)) + l.lane;
#pragma unroll
			for (int k = 0; k < F / 2; ++k) {
				const float2 v = 64 * k < n ? __ldcg(p + 32 * k) : make_float2(0.f, 0.f);
				f[2 * k] = v.x, f[2 * k + 1] = v.y;
			}
		};
		cols_wait_prev(false);
		stamp_begin(a.stamp);
		fetch(0);
		int slot = 0, parity = 0;
		bool ok = r.tries != 0;
		for (int c = 0; c < chunks && ok; ++c) {
			const float2 u = l.worth(cols_to_scale(f));
			ColsFragments<DBITS> x;
			x.make(buf + l.warp * 192, l, f);
			fetch(c + 1);
			const int n = l.own(r, c);
#pragma unroll
			for (int t = 0; t < T; ++t) {
				if (!mbar_wait_warp(&sh.full[slot], parity)) {
					ok = false;
					break;
				}
				cols_multiply<DBITS>(&sh, smem_raw, slot, r, l, n, x, u, acc[t]);
				if (++slot == COLS_STAGES) slot = 0, parity ^= 1;
			}
		}
#pragma unroll
		for (int t = 0; t < T; ++t)
			if (ok) ok = cols_hand_over(&sh, r, part, l, t, acc[t]);
		if (!ok && l.lane == 0) sh.gave_up = 9400;
	} else {
		cols_wait_prev(false);
		for (int j = l.lane; j < rows; j += 32) sh.rows[j] = a.accumulate && a.tpx.world <= 1 ? __ldcg(a.y + row0 + j) : 0.f;
		__syncwarp();
		cols_epilogue(&sh, r, part, T, [&](int tile, int slot, float v) {
			const int j = 8 * tile + slot;
			if (l.lane >= 8 || j >= rows) return;
			if (a.tpx.world > 1) sh.rows[j] = v;
			else a.y[row0 + j] = sh.rows[j] + v;
		});
	}
	__syncthreads();
	if (a.tpx.world > 1) { // the matvec -> all-reduce fusion of stages.cuh TpExchange
		tp_exchange_rows(a.tpx, sh.rows, row0, rows, a.y, a.d);
	}
	if (threadIdx.x == 0 && sh.gave_up) *reinterpret_cast<volatile int*>(r.err) = sh.gave_up;
	stamp_end(a.stamp);
}
