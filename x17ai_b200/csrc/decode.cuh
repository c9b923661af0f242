// int8 decode attention: one new token per sequence against an int8 KV cache. HBM-bound.
//
// The reference has no int8 decode kernel (its attn_incremental.cu:329-481 is a stale bf16
// header); the semantics here are those of row `kv_len` of the prefill kernel
// (cuda/attn_fwd_i8.cuh:368-619): keys kv_len-W' .. kv_len-1 plus the sink, temperature
// D^-1/2 / 64 * log2(min(W', kv_len) + 4) * temp_h, u8 probabilities in steps of 1/255,
// int32 P.V, out = rint(clamp(O / sum)), L = log2(sum) + max.
//
// Grid (head, batch, split). 256 threads; each group of D/16 lanes streams one key row
// (16 bytes per lane, 32 / (D/16) rows per warp instruction): q.k with dp4a + a butterfly
// inside the group, online softmax per group with lazy rescale (the int32 P.V accumulators
// are only flushed to f32 when the group's running maximum moves), P.V with dp4a after a 4x4
// byte transpose of four V rows. From three steps on the loads of the next step are in flight under the arithmetic of the
// current one.
// Groups, warps and (with n_splits > 1) splits are merged with
// the usual (max, sum, O) log-sum-exp combine; the sink token enters as one more partial.
// The splits of a (head, batch) form a cluster of up to 8 CTAs (a CTA takes every 8th split where there are more);
// their partials meet in the first CTA's shared memory: no scratch memory, no second launch. Beyond 64 splits
// the partials go through scratch memory and a second kernel merges them.
// Measured (32 heads x 128, one sequence, cache cold): 1500 keys 9.2 -> 6.9 us, 4096 keys 14.9 -> 11.0 us (with clusters
// of 16 instead of two splits per CTA 16.6); the allocation and release of scratch cost the host 8 us a call on top.
#pragma once

#include "ptx.cuh"

namespace x17 {

struct DecodeParams {
	i8 const *q;          // [B, H*D]
	u64 q_stride;
	i8 const *kv;         // [B, T, H*2*D], per head [K(D) | V(D)]
	u64 kv_stride, kv_batch_stride;
	u32 const *kv_lens;   // [B] or null (then kv_len); entries above kv_capacity are clamped to it
	u32 kv_len;
	u32 kv_capacity;      // rows of one sequence's cache
	u32 window;           // rounded up to 16; 0xFFFFFFFF = unbounded
	i8 const *sink_k, *sink_v;
	f32 const *temperature;
	i8 *out;              // [B, H*D]
	u64 o_stride;
	f32 *l;               // [B, H] or null
	u32 n_heads;
	u32 n_splits;
	f32 *scratch;         // [B][H][n_splits][D + 2] partials, or null: they meet in shared memory
};

namespace dec_cfg {
constexpr u32 WARPS = 8;
constexpr u32 THREADS = WARPS * 32;
constexpr u32 UNROLL = 4;  // key rows per lane group and step (also the dp4a depth of P.V)
constexpr u32 MAX_CLUSTER = 8;           // the portable size
constexpr u32 MAX_CLUSTER_SPLITS = 64;   // partials that the first CTA's shared memory takes
template <u32 D>
constexpr u32 partials_bytes(u32 n_splits) {
	return n_splits * (D + 2) * 4;
}
}  // namespace dec_cfg

// a: four signed bytes, b: four unsigned bytes
X17_DEV i32 dp4a_s8_u8(u32 a, u32 b, i32 c) {
	i32 d;
	asm("dp4a.s32.u32 %0, %1, %2, %3;" : "=r"(d) : "r"(a), "r"(b), "r"(c));
	return d;
}

X17_DEV void transpose4x4_bytes(u32 a, u32 b, u32 c, u32 d, u32 (&o)[4]) {
	u32 const t0 = __byte_perm(a, b, 0x5140);
	u32 const t1 = __byte_perm(c, d, 0x5140);
	u32 const t2 = __byte_perm(a, b, 0x7362);
	u32 const t3 = __byte_perm(c, d, 0x7362);
	o[0] = __byte_perm(t0, t1, 0x5410);
	o[1] = __byte_perm(t0, t1, 0x7632);
	o[2] = __byte_perm(t2, t3, 0x5410);
	o[3] = __byte_perm(t2, t3, 0x7632);
}

// combine partial (m, s, o[16]) <- with (m2, s2, o2[16])
X17_DEV void lse_merge(f32 &m, f32 &s, f32 (&o)[16], f32 m2, f32 s2, f32 const (&o2)[16]) {
	f32 const nm = fmaxf(m, m2);
	f32 const a = ex2_approx(m - nm);
	f32 const b = ex2_approx(m2 - nm);
	s = __fmaf_rn(s, a, s2 * b);
#pragma unroll
	for (u32 i = 0; i < 16; ++i) o[i] = __fmaf_rn(o[i], a, o2[i] * b);
	m = nm;
}

// The merged (m, s, o) of one output dim with the sink token (its score sink_s, weight 255, value 255 * sink_v).
template <u32 D>
X17_DEV void decode_finish(DecodeParams const &p, u32 batch, u32 head, u32 d, f32 fm, f32 fs, f32 fo, f32 sink_s, f32 sink_v) {
	f32 const nm = fmaxf(fm, sink_s);
	f32 const a = ex2_approx(fm - nm), b = ex2_approx(sink_s - nm);
	fs = __fmaf_rn(fs, a, 255.0f * b);
	fo = __fmaf_rn(fo, a, 255.0f * sink_v * b);
	p.out[u64(batch) * p.o_stride + head * D + d] = i8(f32_to_fixedi8(__fmul_rn(fo, rcp_approx(fs))));
	if (d == 0 && p.l != nullptr) p.l[u64(batch) * p.n_heads + head] = __fadd_rn(lg2_approx(fs), nm);
}
// Partials of n splits, [n][D + 2] = (o[D], m, s), merged in split order.
template <u32 D>
X17_DEV void merge_partials(f32 const *src, u32 n, u32 d, f32 &fm, f32 &fs, f32 &fo) {
	fm = src[D];
	fs = src[D + 1];
	fo = src[d];
	for (u32 s = 1; s < n; ++s) {
		f32 const *ps = src + u64(s) * (D + 2);
		f32 const m2 = ps[D];
		f32 const nm = fmaxf(fm, m2);
		f32 const a = ex2_approx(fm - nm), b = ex2_approx(m2 - nm);
		fs = __fmaf_rn(fs, a, ps[D + 1] * b);
		fo = __fmaf_rn(fo, a, ps[d] * b);
		fm = nm;
	}
}

// Key rows that a CTA takes at once.
template <u32 D>
constexpr u32 DECODE_STEP = dec_cfg::WARPS * (512 / D) * dec_cfg::UNROLL;

// Two CTAs per SM: 128 registers hold the rows in work and the rows on their way.
// CLUSTER: the splits of a (sequence, head) form a cluster and meet in shared memory; otherwise a CTA is one split.
// AHEAD: the next step's rows are loaded under the arithmetic of the current one: from three steps on (1639 keys a split at
// width 64 62.5 -> 59.7 us, 863 at width 128 59.1 -> 57.0). With one or two steps there is little to load ahead, and what it
// costs to hold the rows twice shows: 256 x 32 heads, 16 keys, 61.9 us without and 66.5 with it at width 32, 62.1 and 67.9
// at 128; 128 x 8 heads, 512 keys in two splits, width 64 30.0 and 31.1.
template <u32 D, bool CLUSTER, bool AHEAD>
__global__ void __launch_bounds__(dec_cfg::THREADS, 2)
attn_decode_kernel(const DecodeParams p) {
	using namespace dec_cfg;
	static_assert(D == 32 || D == 64 || D == 128);
	constexpr u32 LPR = D / 16;        // lanes per key row
	constexpr u32 RPI = 32 / LPR;      // key rows per warp instruction
	static_assert(DECODE_STEP<D> == WARPS * RPI * UNROLL);
	constexpr f32 NEG_BIG = -3.0e38f;

	u32 const head = blockIdx.x;
	u32 const batch = blockIdx.y;
	u32 const warp = threadIdx.x >> 5;
	u32 const lane = threadIdx.x & 31;
	u32 const grp = lane / LPR;        // which row of the instruction this lane works on
	u32 const sub = lane % LPR;        // which 16-byte chunk of the row

	if constexpr (CLUSTER) cluster_arrive();   // "this CTA runs"
	pdl_wait();
	u32 const kv_len = p.kv_lens ? min(p.kv_lens[batch], p.kv_capacity) : p.kv_len;
	u32 const w = p.window;
	u32 const k_lo = (w == 0xFFFFFFFFu || kv_len < w) ? 0u : kv_len - w;
	u32 const n_keys = kv_len - k_lo;
	u32 const per_split = ((n_keys + p.n_splits - 1) / p.n_splits + 15u) & ~15u;

	// this lane's 16 bytes of q
	uint4 const qv = *reinterpret_cast<uint4 const *>(p.q + u64(batch) * p.q_stride + head * D + sub * 16);
	u32 const qw[4] = {qv.x, qv.y, qv.z, qv.w};
	// the sink token's operands are read ahead of the stream of keys
	uint4 const sk = *reinterpret_cast<uint4 const *>(p.sink_k + head * D + sub * 16);
	f32 const sink_v = threadIdx.x < D ? f32(p.sink_v[head * D + threadIdx.x]) : 0.0f;

	u32 const n_att = (kv_len < w ? kv_len : w) + 4u;
	f32 const base_t = f32((1.0 / 64.0) * (D == 128 ? 0.08838834764831845 : D == 64 ? 0.125 : 0.17677669529663687));
	f32 const temp = __fmul_rn(__fmul_rn(base_t, lg2_approx(f32(n_att))), p.temperature[head]);

	i8 const *kv_base = p.kv + u64(batch) * p.kv_batch_stride + u64(head) * 2 * D + sub * 16;
	u32 const step = WARPS * RPI * UNROLL;

	__shared__ f32 sh_o[WARPS][D];
	__shared__ f32 sh_m[WARPS], sh_s[WARPS];
	extern __shared__ f32 partials[];   // first CTA of a cluster: [n_splits][D + 2]

	f32 fm = 0.0f, fs = 0.0f, fo = 0.0f;   // of the CTA's split, in the threads below D
	// Shared memory of another CTA may be written only once that CTA is known to run; being scheduled together is not enough,
	// and a split without keys gets to its store within a few hundred cycles. (Asked for at entry: 5.51 -> 5.54 us a call for
	// one sequence of 1500 keys.)
	if constexpr (CLUSTER) cluster_wait();
	#pragma unroll 1
	for (u32 split = blockIdx.z; split < p.n_splits; split += gridDim.z) {
		u32 const s_lo = k_lo + split * per_split;
		u32 const s_hi = min(kv_len, s_lo + per_split);
		f32 m = NEG_BIG, ssum = 0.0f;
		f32 o_f[16];
		i32 o_i[16];
#pragma unroll
		for (u32 i = 0; i < 16; ++i) {
			o_f[i] = 0.0f;
			o_i[i] = 0;
		}
		auto load = [&](u32 t0, uint4 (&kq)[UNROLL], uint4 (&vq)[UNROLL]) {
#pragma unroll
			for (u32 u = 0; u < UNROLL; ++u) {
				u32 const t = t0 + u * RPI + grp;
				i8 const *rowp = kv_base + u64(t < s_hi ? t : s_lo) * p.kv_stride;
				kq[u] = *reinterpret_cast<uint4 const *>(rowp);
				vq[u] = *reinterpret_cast<uint4 const *>(rowp + D);
			}
		};
		u32 since_flush = 0;  // an int32 accumulator takes at most 4 * 255 * 127 per step: flush long before 2^31
		u32 t0 = s_lo + (warp * UNROLL) * RPI;
		uint4 kn[UNROLL], vn[UNROLL];
		if (AHEAD && t0 < s_hi) load(t0, kn, vn);
		for (; t0 < s_hi; t0 += step) {
			uint4 kq[UNROLL], vq[UNROLL];
			if constexpr (AHEAD) {
#pragma unroll
				for (u32 u = 0; u < UNROLL; ++u) {
					kq[u] = kn[u];
					vq[u] = vn[u];
				}
				if (t0 + step < s_hi) load(t0 + step, kn, vn);
			} else {
				load(t0, kq, vq);
			}
			// ---- scores of UNROLL rows per group ----
			bool valid[UNROLL];
			f32 s[UNROLL];
			f32 smax = NEG_BIG;
#pragma unroll
			for (u32 u = 0; u < UNROLL; ++u) {
				valid[u] = t0 + u * RPI + grp < s_hi;
				i32 dot = __dp4a(i32(kq[u].x), i32(qw[0]), 0);
				dot = __dp4a(i32(kq[u].y), i32(qw[1]), dot);
				dot = __dp4a(i32(kq[u].z), i32(qw[2]), dot);
				dot = __dp4a(i32(kq[u].w), i32(qw[3]), dot);
#pragma unroll
				for (u32 mask = 1; mask < LPR; mask <<= 1) dot += __shfl_xor_sync(0xffffffffu, dot, mask);
				s[u] = valid[u] ? __fmul_rn(__int2float_rn(dot), temp) : NEG_BIG;
				smax = fmaxf(smax, s[u]);
			}
			// ---- online softmax with lazy flush of the int32 accumulators ----
			if (smax > m || ++since_flush >= 8192u) {
				since_flush = 0;
				smax = fmaxf(smax, m);
				f32 const a = ex2_approx(m - smax);
#pragma unroll
				for (u32 i = 0; i < 16; ++i) {
					o_f[i] = __fmul_rn(__fadd_rn(o_f[i], __int2float_rn(o_i[i])), a);
					o_i[i] = 0;
				}
				ssum = __fmul_rn(ssum, a);
				m = smax;
			}
			u32 pb[UNROLL];
#pragma unroll
			for (u32 u = 0; u < UNROLL; ++u) {
				f32 const e = valid[u] ? __fmul_rn(ex2_approx(__fsub_rn(s[u], m)), 255.0f) : 0.0f;
				ssum = __fadd_rn(ssum, e);
				pb[u] = u32(__float2int_rn(e));
			}
			static_assert(UNROLL == 4);
			u32 const p4 = pack4(pb[0], pb[1], pb[2], pb[3]);
			// ---- O += P . V for this lane's 16 dims ----
			u32 const va[4] = {vq[0].x, vq[0].y, vq[0].z, vq[0].w};
			u32 const vb[4] = {vq[1].x, vq[1].y, vq[1].z, vq[1].w};
			u32 const vc[4] = {vq[2].x, vq[2].y, vq[2].z, vq[2].w};
			u32 const vd[4] = {vq[3].x, vq[3].y, vq[3].z, vq[3].w};
#pragma unroll
			for (u32 wi = 0; wi < 4; ++wi) {
				u32 tr[4];
				transpose4x4_bytes(va[wi], vb[wi], vc[wi], vd[wi], tr);
#pragma unroll
				for (u32 j = 0; j < 4; ++j) o_i[4 * wi + j] = dp4a_s8_u8(tr[j], p4, o_i[4 * wi + j]);
			}
		}
#pragma unroll
		for (u32 i = 0; i < 16; ++i) o_f[i] = __fadd_rn(o_f[i], __int2float_rn(o_i[i]));

		// ---- merge the lane groups of the warp (lanes with equal `sub` hold the same dims) ----
#pragma unroll
		for (u32 mask = LPR; mask < 32; mask <<= 1) {
			f32 const m2 = __shfl_xor_sync(0xffffffffu, m, mask);
			f32 const s2 = __shfl_xor_sync(0xffffffffu, ssum, mask);
			f32 o2[16];
#pragma unroll
			for (u32 i = 0; i < 16; ++i) o2[i] = __shfl_xor_sync(0xffffffffu, o_f[i], mask);
			lse_merge(m, ssum, o_f, m2, s2, o2);
		}

		// ---- merge the warps through shared memory ----
		__syncthreads();   // the previous split's values have been read
		if (lane < LPR) {
#pragma unroll
			for (u32 i = 0; i < 16; ++i) sh_o[warp][lane * 16 + i] = o_f[i];
			if (lane == 0) {
				sh_m[warp] = m;
				sh_s[warp] = ssum;
			}
		}
		__syncthreads();
		if (threadIdx.x < D) {
			u32 const d = threadIdx.x;
			fm = sh_m[0];
			fs = sh_s[0];
			fo = sh_o[0][d];
#pragma unroll
			for (u32 wq = 1; wq < WARPS; ++wq) {
				f32 const nm = fmaxf(fm, sh_m[wq]);
				f32 const a = ex2_approx(fm - nm), b = ex2_approx(sh_m[wq] - nm);
				fs = __fmaf_rn(fs, a, sh_s[wq] * b);
				fo = __fmaf_rn(fo, a, sh_o[wq][d] * b);
				fm = nm;
			}
			if constexpr (CLUSTER) {
				u32 const dst = map_to_cta(smem_u32(partials + split * (D + 2)), 0);
				st_cluster_f32(dst + d * 4, fo);
				if (d == 0) {
					st_cluster_f32(dst + D * 4, fm);
					st_cluster_f32(dst + D * 4 + 4, fs);
				}
			} else if (p.n_splits > 1) {
				f32 *dst = p.scratch + ((u64(batch) * p.n_heads + head) * p.n_splits + split) * (D + 2);
				dst[d] = fo;
				if (d == 0) {
					dst[D] = fm;
					dst[D + 1] = fs;
				}
			}
		}
	}
	pdl_launch_dependents();   // not earlier: a next decode's clusters would be packed onto the few SMs with room
	if constexpr (CLUSTER) {
		__syncwarp();
		cluster_arrive();              // this CTA's partials are stored
		if (blockIdx.z != 0) return;   // its slot is free for the next CTA: only the first CTA waits
		cluster_wait();
	} else if (p.n_splits > 1) {
		return;
	}
	// ---- the sink token: exact int32 q . sink_k, from the lanes of one row ----
	i32 sdot = __dp4a(i32(sk.x), i32(qw[0]), 0);
	sdot = __dp4a(i32(sk.y), i32(qw[1]), sdot);
	sdot = __dp4a(i32(sk.z), i32(qw[2]), sdot);
	sdot = __dp4a(i32(sk.w), i32(qw[3]), sdot);
#pragma unroll
	for (u32 mask = 1; mask < LPR; mask <<= 1) sdot += __shfl_xor_sync(0xffffffffu, sdot, mask);
	f32 const sink_s = __fmul_rn(__int2float_rn(sdot), temp);
	if (threadIdx.x < D) {
		if constexpr (CLUSTER) merge_partials<D>(partials, p.n_splits, threadIdx.x, fm, fs, fo);
		decode_finish<D>(p, batch, head, threadIdx.x, fm, fs, fo, sink_s, sink_v);
	}
}

// Second kernel of the scratch path: one CTA per (head, batch), D threads.
template <u32 D>
__global__ void __launch_bounds__(D)
attn_decode_merge_kernel(const DecodeParams p) {
	u32 const head = blockIdx.x;
	u32 const batch = blockIdx.y;
	u32 const d = threadIdx.x;
	pdl_launch_dependents();
	pdl_wait();
	u32 const kv_len = p.kv_lens ? min(p.kv_lens[batch], p.kv_capacity) : p.kv_len;
	u32 const w = p.window;
	u32 const n_att = (kv_len < w ? kv_len : w) + 4u;
	f32 const base_t = f32((1.0 / 64.0) * (D == 128 ? 0.08838834764831845 : D == 64 ? 0.125 : 0.17677669529663687));
	f32 const temp = __fmul_rn(__fmul_rn(base_t, lg2_approx(f32(n_att))), p.temperature[head]);

	f32 fm, fs, fo;
	merge_partials<D>(p.scratch + (u64(batch) * p.n_heads + head) * p.n_splits * (D + 2), p.n_splits, d, fm, fs, fo);
	i32 sdot = 0;
	uint4 const *qh = reinterpret_cast<uint4 const *>(p.q + u64(batch) * p.q_stride + head * D);
	uint4 const *sk = reinterpret_cast<uint4 const *>(p.sink_k + head * D);
	for (u32 i = 0; i < D / 16; ++i) {
		uint4 a = qh[i], b = sk[i];
		sdot = __dp4a(i32(a.x), i32(b.x), sdot);
		sdot = __dp4a(i32(a.y), i32(b.y), sdot);
		sdot = __dp4a(i32(a.z), i32(b.z), sdot);
		sdot = __dp4a(i32(a.w), i32(b.w), sdot);
	}
	f32 const sink_s = __fmul_rn(__int2float_rn(sdot), temp);
	decode_finish<D>(p, batch, head, d, fm, fs, fo, sink_s, f32(p.sink_v[head * D + d]));
}

}  // namespace x17
