// Encoder kernels for sm_100a: fused forward CDF 9/7 level + quantiser + RD
// analysis, the rate-control resolve (one cluster of CTAs), and block packing.
//
// Reference behaviour followed (file:line in the reference tree):
//   forward level      shaders/dwt.comp:38-234 (tile + apron, H then V lifting)
//   quantiser / stats  shaders/wavelet_quant.comp:72-316
//   RD analysis        shaders/analyze_rate_control.comp:73-220
//   finalize/resolve   shaders/analyze_rate_control_finalize.comp:14-38,
//                      shaders/resolve_rate_control.comp:38-81, pyrowave_encoder.cpp:283-338
//   block packing      shaders/block_packing.comp:97-379
//   packetize layout   pyrowave_encoder.cpp:1048-1115
#include "pw_decode_body.cuh"

#include <algorithm>

namespace pw
{
namespace
{
// Reduction scratch of one 128-thread quantiser group (one 32x32 block).
struct QuantGroupShared
{
	float dist[4][16];
	uint32_t cost[4][16];
};

// ---------------------------------------------------------------------------
// Quantiser + RD analysis of a 32x32 block held in shared memory: one row of
// 8x8 blocks per warp (quant_analyze_row, four or eight warps per block), then
// the block's rate-control row from the four rows' sums (quant_finish_block, 16
// lanes). No barrier inside either; the caller puts one between them.
//
// A lane owns one 4x2 sub-block, sub = lane & 7 of 8x8 column lx = lane >> 3
// (the reference's mapping, wavelet_quant.comp:294-306). Every quantity is the
// reference's, computed in its order, with less work per quant level:
//   * the plane bytes at level q need no per-level reduction: with qp0 the Q
//     planes at level 0, a sub-block's planes at q are max(qp0 - q, 0) Q planes
//     plus max(code - max(q - qp0, 0), 0), and the sum over an 8x8's plane codes
//     is one population count of its code word (plane_code_sum);
//   * levels are evaluated in pairs (q, q + 1): the two squared errors share the
//     first exchange of the butterfly (each lane keeps the level of its own
//     parity), the two counts of significant values travel in one float;
//   * each lane ends with its own levels, sub and sub + 8, so the FP16 rounding
//     and the cost are computed once per lane, not once per level;
//   * a warp whose values all quantise to zero stores zeros and stops: a quarter
//     of the rows of a 1080p frame, half of a flat desktop's.
// Bound by instruction issue. Measured against one
// butterfly per level and sum on four-warp groups: encode of a 4K 4:4:4 frame
// (1.2 MB) 203 -> 183 us, of a 1080p 4:2:0 frame 51.2 -> 49.2 us.
//
// With S = 2, two warps share a row: warp r evaluates every other pair of
// levels. Each level is computed by exactly one warp, in the same order, so the
// results do not depend on S.
constexpr int kBandPitch = 36; // row pitch of a 32x32 band tile: 16-byte rows, conflict-free sub-block vectors

__device__ __forceinline__ float max3_nan(float a, float b, float c)
{
	float r;
	asm("max.NaN.f32 %0, %1, %2, %3;" : "=f"(r) : "f"(a), "f"(b), "f"(c));
	return r;
}

// Position of the highest set bit of int(x), x in [0, 32767] (-1: none), from the exponent.
__device__ __forceinline__ int float_msb(float x) { return max(int(__float_as_uint(x) >> 23) - 127, -1); }

// Per scale code, by k = code + 2: the 8x8 scale 8 / k and the squared inverse
// of the band's quantiser with it, computed once per band tile (k is at most 14
// below kQuantScaleFast). Threads 0..15 of a group fill it.
struct QuantScales
{
	float2 by_k[16];
};
__device__ __forceinline__ float2 quant_scale_entry(float scale, float quant_resolution)
{
	const float inv_quant = __frcp_rn(__fmul_rn(quant_resolution, scale));
	return make_float2(scale, __fmul_rn(inv_quant, inv_quant));
}
__device__ __forceinline__ void fill_quant_scales(QuantScales &sc, int k, float quant_resolution)
{
	sc.by_k[k] = quant_scale_entry(__frcp_rn(__fmul_rn(float(max(k, 1)), 0.125f)), quant_resolution);
}

template <int S>
__device__ __forceinline__ void quant_analyze_row(const float *tile, const int ly, const int r, QuantGroupShared &sh,
                                                  const QuantScales &scales, const LevelDesc &L, const BandParam &B,
                                                  const int bx32, const int by32, const EncodeBuffers &buf)
{
	const unsigned full = 0xffffffffu;
	const int lane = threadIdx.x & 31;
	const int sub = lane & 7, lx = lane >> 3;
	const int x8 = bx32 * 4 + lx, y8 = by32 * 4 + ly;
	const bool in_range = x8 < L.blocks8_x && y8 < L.blocks8_y;
	const float qres = B.quant_resolution;

	// Samples beyond the band are zeros in the tile.
	const float *src = tile + (ly * 8 + sub_y(sub)) * kBandPitch + lx * 8 + sub_x(sub);
	const ulonglong2 row0 = *reinterpret_cast<const ulonglong2 *>(src);
	const ulonglong2 row1 = *reinterpret_cast<const ulonglong2 *>(src + kBandPitch);
	// Coefficient i = 2 * column + row of the sub-block: pairs (0, 2), (4, 6) and
	// (1, 3), (5, 7) of the two rows.
	const f32x2 qres2 = f2_pack(qres, qres);
	const f32x2 vp[4] = {f2_mul_rn(row0.x, qres2), f2_mul_rn(row0.y, qres2), f2_mul_rn(row1.x, qres2),
	                     f2_mul_rn(row1.y, qres2)};
	float v[8];
	f2_unpack(vp[0], v[0], v[2]);
	f2_unpack(vp[1], v[4], v[6]);
	f2_unpack(vp[2], v[1], v[3]);
	f2_unpack(vp[3], v[5], v[7]);

	// 8x8 maximum and quant scale (wavelet_quant.comp:174-181).
	float max_sub = max3_nan(fabsf(v[0]), fabsf(v[1]), fabsf(v[2]));
	max_sub = max3_nan(max_sub, fabsf(v[3]), fabsf(v[4]));
	max_sub = max3_nan(max_sub, fabsf(v[5]), fabsf(v[6]));
	max_sub = max3_nan(max_sub, fabsf(v[7]), 0.0f);
	float max_wave = max_sub;
	max_wave = max3_nan(max_wave, __shfl_xor_sync(full, max_wave, 1), 0.0f);
	max_wave = max3_nan(max_wave, __shfl_xor_sync(full, max_wave, 2), 0.0f);
	max_wave = max3_nan(max_wave, __shfl_xor_sync(full, max_wave, 4), 0.0f);

	uint32_t qcode;
	float qs, iqs;
	if (__any_sync(full, !(max_wave < kQuantScaleFast)))
	{
		// A value too large for the short form of the scale, or NaN: the maximum
		// ignores NaN, and a NaN value is clamped to -32767 below.
		max_sub = 0.0f;
#pragma unroll
		for (int i = 0; i < 8; i++)
		{
			max_sub = fmaxf(max_sub, fabsf(v[i]));
			v[i] = v[i] != v[i] ? -3.0e38f : v[i];
		}
		max_wave = max_sub;
		max_wave = fmaxf(max_wave, __shfl_xor_sync(full, max_wave, 1));
		max_wave = fmaxf(max_wave, __shfl_xor_sync(full, max_wave, 2));
		max_wave = fmaxf(max_wave, __shfl_xor_sync(full, max_wave, 4));
		compute_quant_scale_any(max_wave, qcode, qs);
		iqs = quant_scale_entry(qs, qres).y;
	}
	else
	{
		const int k = quant_scale_step(max_wave);
		qcode = uint32_t(k - 2);
		const float2 e = scales.by_k[k];
		qs = e.x;
		iqs = e.y;
	}
	const f32x2 qs2 = f2_pack(qs, qs);
#pragma unroll
	for (int i = 0; i < 4; i++)
	{
		// Pairs (i, i + 4): adjacent as the two packed products leave them free.
		f32x2 p = f2_mul_rn(f2_pack(v[i], v[i + 4]), qs2);
		f2_unpack(p, v[i], v[i + 4]);
	}
	float av[8];
#pragma unroll
	for (int i = 0; i < 8; i++)
		av[i] = fminf(fabsf(v[i]), kMaxScaledMagnitude);
	max_sub = fminf(__fmul_rn(max_sub, qs), kMaxScaledMagnitude);
	max_wave = fminf(__fmul_rn(max_wave, qs), kMaxScaledMagnitude);
	const int msb = float_msb(max_wave);
	const int warp_msb = __reduce_max_sync(full, msb);
	uint32_t *const code_word = buf.code_words + B.block8_offset + y8 * B.block8_stride + x8;
	if (warp_msb < 0)
	{
		// Every value of the row quantises to zero: the packer does not look at its magnitudes.
		if (r == 0)
		{
			if (lane < 16)
			{
				sh.dist[ly][lane] = 0.0f;
				sh.cost[ly][lane] = 0u;
			}
			if (in_range && sub == 0)
				*code_word = 0u;
		}
		return;
	}

	// Magnitudes as pairs (i, i + 4): the two lanes of a pair accumulate the two
	// halves of the squared error, over i = 0..3 and i = 4..7, in the same order
	// as eight scalar steps would.
	f32x2 avp[4];
#pragma unroll
	for (int j = 0; j < 4; j++)
		avp[j] = f2_pack(av[j], av[j + 4]);

	// The packer's input: the scaled values as sign-magnitude (|int(v)| <= 32767),
	// one 16-byte store per sub-block, written by the first warp of each row.
	// int(|v|) is the low half of |v| + 2^23 rounded toward zero; the sign of a
	// magnitude of zero is not read.
	uint32_t mag[4];
	{
		uint32_t m[8];
#pragma unroll
		for (int j = 0; j < 4; j++)
		{
			float lo, hi;
			f2_unpack(f2_add_rz(avp[j], f2_pack(8388608.0f, 8388608.0f)), lo, hi);
			m[j] = __float_as_uint(lo);
			m[j + 4] = __float_as_uint(hi);
		}
#pragma unroll
		for (int j = 0; j < 4; j++)
			mag[j] = __byte_perm(m[2 * j], m[2 * j + 1], 0x5410);
	}
	if (r == 0 && buf.mag16)
	{
		uint32_t w[4];
#pragma unroll
		for (int j = 0; j < 4; j++)
			w[j] = mag[j] | (__byte_perm(__float_as_uint(v[2 * j]), __float_as_uint(v[2 * j + 1]), 0x7632) & 0x80008000u);
		const int blk = B.block32_offset + by32 * B.block32_stride + bx32;
		*reinterpret_cast<uint4 *>(buf.mag16 + int64_t(blk) * 1024 + 8 * (lane + 32 * ly)) =
		    make_uint4(w[0], w[1], w[2], w[3]);
	}
	const float rdo = B.rdo_scale;

	// Stats at q = 0 (wavelet_quant.comp:139-165,205-238): the 8x8's plane codes
	// (bits 0-15) and its number of significant values (from bit 16) in one sum.
	const int qp0 = max(msb - 2, 0);
	const uint32_t plane_code = uint32_t(max(float_msb(max_sub) + 1 - qp0, 0));
	uint32_t nz = 0; // one bit per value with int(|v|) != 0
#pragma unroll
	for (int j = 0; j < 4; j++)
		nz |= ((mag[j] + 0x7fff7fffu) & 0x80008000u) >> j;
	uint32_t codes = (plane_code << (2 * sub)) + (uint32_t(__popc(nz)) << 16);
	codes += __shfl_xor_sync(full, codes, 1);
	codes += __shfl_xor_sync(full, codes, 2);
	codes += __shfl_xor_sync(full, codes, 4);
	const uint32_t nsig0 = codes >> 16;

	// Distortion of dropping every plane (wavelet_quant.comp:253-256).
	float drop;
	{
		f32x2 e2 = f2_mul_rn(avp[0], avp[0]);
#pragma unroll
		for (int j = 1; j < 4; j++)
			e2 = f2_fma_rn(avp[j], avp[j], e2);
		float s0, s1;
		f2_unpack(e2, s0, s1);
		drop = __fmul_rn(__fadd_rn(s0, s1), iqs);
		drop = __fadd_rn(drop, __shfl_xor_sync(full, drop, 1));
		drop = __fadd_rn(drop, __shfl_xor_sync(full, drop, 2));
		drop = __fadd_rn(drop, __shfl_xor_sync(full, drop, 4));
	}

	// Lane `sub` ends with the 8x8's entries for quant levels sub and sub + 8:
	// the squared errors and the significant values of levels up to msb.
	float d_lo = drop, d_hi = drop;
	uint32_t n_lo = nsig0, n_hi = 0u;
	const bool odd = (sub & 1) != 0;
	for (int q = 1 + 2 * r; q <= warp_msb; q += 2 * S)
	{
		// compute_square_error + compute_quant_stats at q and q + 1
		// (wavelet_quant.comp:113-165). A value quantised at q is reconstructed
		// as trunc((floor(|v| / 2^q) + 0.5) * 2^q) when nonzero. R =
		// floor(|v| / 2^q) * 2^q in float arithmetic, exactly: adding M =
		// 2^(23+q) with round-toward-zero keeps the multiples of 2^q (the spacing
		// of floats in [M, 2M), and |v| < 2^15 < M), and subtracting M again is
		// exact. The reconstruction is R + min(R, 2^(q-1)), so the error is the
		// exact difference |v| - R - min(R, 2^(q-1)), and the sum of the minima
		// is the number of significant values times 2^(q-1).
		float se[2], ns[2];
#pragma unroll
		for (int h = 0; h < 2; h++)
		{
			const float hq = __int_as_float((126 + q + h) << 23);
			const float mq = __int_as_float((150 + q + h) << 23);
			const f32x2 mq2 = f2_pack(mq, mq);
			f32x2 ns2 = 0ull, e2 = 0ull;
#pragma unroll
			for (int j = 0; j < 4; j++)
			{
				const f32x2 R = f2_sub_rn(f2_add_rz(avp[j], mq2), mq2);
				float r_lo, r_hi;
				f2_unpack(R, r_lo, r_hi);
				const f32x2 half = f2_pack(fminf(r_lo, hq), fminf(r_hi, hq));
				ns2 = j == 0 ? half : f2_add_rn(ns2, half);
				const f32x2 err = f2_sub_rn(f2_sub_rn(avp[j], R), half);
				e2 = j == 0 ? f2_mul_rn(err, err) : f2_fma_rn(err, err, e2);
			}
			float e0, e1, n0, n1;
			f2_unpack(e2, e0, e1);
			f2_unpack(ns2, n0, n1);
			se[h] = __fmul_rn(__fmul_rn(__fadd_rn(e0, e1), rdo), iqs);
			ns[h] = __fadd_rn(n0, n1);
		}
		// Counts: n(q) + 1024 n(q + 1), exact. 2^(1-q) undoes the scale of ns[0].
		const float inv = __int_as_float((128 - q) << 23);
		float n = __fmaf_rn(ns[1], __fmul_rn(inv, 512.0f), __fmul_rn(ns[0], inv));
		// Odd lanes keep level q (odd), even lanes q + 1; the sums are those of a
		// butterfly over the eight lanes.
		float x = __fadd_rn(odd ? se[0] : se[1], __shfl_xor_sync(full, odd ? se[1] : se[0], 1));
		n = __fadd_rn(n, __shfl_xor_sync(full, n, 1));
		x = __fadd_rn(x, __shfl_xor_sync(full, x, 2));
		n = __fadd_rn(n, __shfl_xor_sync(full, n, 2));
		x = __fadd_rn(x, __shfl_xor_sync(full, x, 4));
		n = __fadd_rn(n, __shfl_xor_sync(full, n, 4));
		const int own = q + 1 - (sub & 1);
		const uint32_t both = uint32_t(int(n));
		const uint32_t cnt = odd ? (both & 1023u) : (both >> 10);
		if (own <= msb)
		{
			if (own == sub)
			{
				d_lo = x;
				n_lo = cnt;
			}
			if (own == sub + 8)
			{
				d_hi = x;
				n_hi = cnt;
			}
		}
	}
	d_lo = sub == 0 ? 0.0f : __half2float(__float2half_rn(fminf(d_lo, 60000.0f)));
	d_hi = __half2float(__float2half_rn(fminf(d_hi, 60000.0f)));

	// Bits per 8x8 at this lane's levels (wavelet_quant.comp:205-238), +24 per
	// coded 8x8 (analyze_rate_control.comp:169-215); levels sub + 8 in the high half.
	uint32_t c = 0;
	if (sub <= msb)
		c = uint32_t(8 * (8 * max(qp0 - sub, 0) + plane_code_sum(codes, sub - qp0)) + 24) + n_lo;
	if (sub + 8 <= msb)
		c += (uint32_t(8 * (8 * max(qp0 - sub - 8, 0) + plane_code_sum(codes, sub + 8 - qp0)) + 24) + n_hi) << 16;
	if (msb < 0)
		d_lo = d_hi = 0.0f;

	// Per-32x32 sums: butterfly over the 16 8x8 blocks in index order lx + 4 * ly
	// (the columns here, the rows in quant_finish_block). Lanes 0..7 end with
	// levels sub, lanes 8..15 with levels sub + 8.
	const bool hi = (lane & 8) != 0;
	float d = __fadd_rn(hi ? d_hi : d_lo, __shfl_xor_sync(full, hi ? d_lo : d_hi, 8));
	c += __shfl_xor_sync(full, c, 8);
	d = __fadd_rn(d, __shfl_xor_sync(full, d, 16));
	c += __shfl_xor_sync(full, c, 16);
	// The warp that computed a level stores it (level 0: warp 0).
	const int level = sub + (lane & 8);
	if (lane < 16 && (S == 1 || (level == 0 ? r == 0 : ((level - 1) >> 1) % S == r)))
	{
		sh.dist[ly][level] = d;
		sh.cost[ly][level] = hi ? c >> 16 : c & 0xffffu;
	}
	if (in_range && sub == 0 && r == 0)
		*code_word = msb < 0 ? 0u
		                     : (codes & 0xffffu) | (uint32_t(qp0) << kQPlanesOffset) | ((qcode & 0xfu) << kQuantScaleOffset);
}

// Rate-control row of a 32x32 block from its four rows' sums
// (analyze_rate_control.comp:101-220), by the 16 lanes of a half-warp; every lane of
// the warp calls it, `active` where its half has a block.
__device__ __forceinline__ void quant_finish_block(const bool active, const QuantGroupShared &sh, const BandParam &B,
                                                   const int subdivision_shift, const int bx32, const int by32,
                                                   const EncodeBuffers &buf)
{
	const int i = threadIdx.x & 15;
	const float d = __fadd_rn(__fadd_rn(sh.dist[0][i], sh.dist[1][i]), __fadd_rn(sh.dist[2][i], sh.dist[3][i]));
	uint32_t c = sh.cost[0][i] + sh.cost[1][i] + sh.cost[2][i] + sh.cost[3][i];
	if (c != 0)
		c += 64;
	const uint32_t rate = (c + 31) >> 5;
	const unsigned full = 0xffffffffu;
	const float d0 = __shfl_sync(full, d, 0, 16);
	const uint32_t r0 = __shfl_sync(full, rate, 0, 16);
	uint32_t bk = bucket_index(d, float(rate), d0, float(r0));
	if (i == 0)
		bk = 0;
	// inclusive_max_clustered16 (analyze_rate_control.comp:85-99)
	bk = min(bk, uint32_t(128 - 16 + i));
#pragma unroll
	for (int off = 1; off < 16; off *= 2)
	{
		const uint32_t up = __shfl_up_sync(full, bk, off, 16) + uint32_t(off);
		if (i >= off)
			bk = max(bk, up);
	}
	const uint32_t rate_prev = __shfl_up_sync(full, rate, 1, 16);
	if (!active)
		return;
	const uint32_t block_index = uint32_t(B.block32_offset + by32 * B.block32_stride + bx32);
	buf.rd_cost[block_index * 16 + i] = uint16_t(rate);
	buf.rd_bucket[block_index * 16 + i] = uint8_t(bk);
	buf.rd_dist[block_index * 16 + i] = d;
	if (i != 0)
	{
		const uint32_t saving = rate_prev - rate;
		if (saving != 0)
		{
			const uint32_t subdivision = block_index >> subdivision_shift;
			atomicAdd(&buf.rc->histogram[bk * kSubdivisions + subdivision], saving);
		}
	}
}

// Shared memory of one forward-level CTA of kThreads threads and kStripes
// stripes (DwtSplit below). The input tile is held as pairs of rows (r, r +
// kPairRows), column by column, so that the horizontal lifting loads packed
// pairs; after it, rows are plain, and pairs of adjacent columns are packed.
constexpr int kTileIn = 72;      // 64 input samples + 4-sample apron on each side
constexpr int kVecs = kTileIn / 4; // vectors of 4 samples per row
// A row pair's 72 columns as 36 chunks of two pairs, even chunks first: the
// loader's vector j is chunks 2j and 2j + 1, so lanes of consecutive j write
// consecutive 16 bytes. Rows of 37 * 16 bytes: lifting lanes (consecutive rows)
// read without bank conflicts.
constexpr int kInPitch = 148;
constexpr int kInOdd = 72;
constexpr int kHPitch = 68;      // 17 * 16 bytes, as above

template <int kRowsIn> struct DwtSharedT
{
	int xidx[kTileIn];
	int yidx[kTileIn];
	// The input tile, then (its horizontal lifting done) the four band tiles.
	union
	{
		alignas(16) float in[kRowsIn / 2][kInPitch];
		alignas(16) float bands[4][kRowsIn == kTileIn ? 32 : 1][kBandPitch];
	};
	alignas(16) float h[kRowsIn][kHPitch]; // after horizontal lifting: low in 0..31, high in 32..63
	QuantGroupShared q[4];
	QuantScales scales[4]; // of the bands the tile's quantiser codes
};

// Work split of the forward level for a CTA of kThreads threads. Whole tiles
// of large levels favour few instructions (long lifting segments: 24 samples
// lifted for 16 kept), stripes and the batch's 1024-thread CTAs a short chain.
template <int kThreads, int kStripes> struct DwtSplit
{
	static constexpr bool kShort = kThreads >= 1024 || kStripes > 1;
	static constexpr int kRowsIn = kStripes == 1 ? kTileIn : 64 / kStripes + 8; // input rows loaded and lifted
	static constexpr int kHPairs = kShort ? 2 : 8; // output pairs per horizontal lifting item
	static constexpr int kVPairs = kShort ? 2 : 8; // output pairs per vertical lifting item
	static constexpr int kQSplit = kThreads >= 1024 ? 2 : 1;    // warps per 8x8 row in the quantiser
	static constexpr int kGroupThreads = 128 * kQSplit;         // threads per quantised 32x32 block
	static constexpr int kGroups = kThreads / kGroupThreads;    // 32x32 blocks quantised at once
	static constexpr int kMinBlocks = kThreads >= 1024 ? 1 : 4; // CTAs per SM to fit
};
using DwtShared = DwtSharedT<kTileIn>;

// CTA size of the large levels (several CTAs per SM). 384-thread CTAs, which
// quantise the three high bands of a tile in one round, measured no faster.
constexpr int kLargeLevelThreads = 256;

// u / 255 - 0.5 and u / 65535 - 0.5, each operation rounded as the division and
// the subtraction are: the quotient is u * hi + (u * lo rounded), with 1 / n =
// hi + lo, fused, which equals the rounded quotient for every u in [0, n]
// (checked for all of them). Two samples at a time; bits holds 2^23 + u.
template <int kMax> __device__ __forceinline__ f32x2 unorm_centered2(uint32_t bits0, uint32_t bits1)
{
	static_assert(kMax == 255 || kMax == 65535, "8-bit or 16-bit samples");
	const float hi = kMax == 65535 ? 0x1.0001p-16f : 0x1.010102p-8f, lo = kMax == 65535 ? 0x1.0001p-48f : -0x1.fdfdfep-33f;
	const f32x2 u = f2_add_rn(f2_pack(__uint_as_float(bits0), __uint_as_float(bits1)), f2_pack(-8388608.0f, -8388608.0f));
	const f32x2 q = f2_fma_rn(u, f2_pack(hi, hi), f2_mul_rn(u, f2_pack(lo, lo)));
	return f2_add_rn(q, f2_pack(-0.5f, -0.5f));
}

// Four samples of a row as raw bits: 8-bit in .x (one byte each), 16-bit in .x
// and .y, FP32 in all four.
__device__ __forceinline__ uint32_t pack4_u8(const uint8_t *row, const int4 &x, int xs)
{
	const uint32_t a = row[size_t(x.x) * xs], b = row[size_t(x.y) * xs], c = row[size_t(x.z) * xs],
	               d = row[size_t(x.w) * xs];
	return __byte_perm(__byte_perm(a, b, 0x0040), __byte_perm(c, d, 0x0040), 0x5410);
}
__device__ __forceinline__ uint2 pack4_u16(const uint8_t *row, const int4 &x, int xs)
{
	const uint32_t a = *reinterpret_cast<const uint16_t *>(row + size_t(x.x) * xs),
	               b = *reinterpret_cast<const uint16_t *>(row + size_t(x.y) * xs),
	               c = *reinterpret_cast<const uint16_t *>(row + size_t(x.z) * xs),
	               d = *reinterpret_cast<const uint16_t *>(row + size_t(x.w) * xs);
	return make_uint2(__byte_perm(a, b, 0x5410), __byte_perm(c, d, 0x5410));
}

// Tile dataflow: waits (bounded) until every tile of the finer level whose LL
// samples this CTA reads has been stored: rows and columns of the input window,
// mirrored at the edges through the index tables, so at most 4 x 4 tiles.
// Called by every thread (after the index tables of an edge tile are built);
// ends with a CTA barrier.
template <int kRowsIn>
__device__ __forceinline__ void wait_finer_tiles(const int *xidx, const int *yidx, const bool interior, const int x0,
                                                 const int y0, const LevelParams &p, const EncodeBuffers &buf,
                                                 const int comp)
{
	if (threadIdx.x < 32)
	{
		const int lane = threadIdx.x;
		int ylo = y0, yhi = y0 + kRowsIn - 1, xlo = x0, xhi = x0 + kTileIn - 1;
		if (!interior)
		{
			ylo = xlo = 0x7fffffff;
			yhi = xhi = 0;
			for (int i = lane; i < kRowsIn; i += 32)
			{
				ylo = min(ylo, yidx[i]);
				yhi = max(yhi, yidx[i]);
			}
			for (int i = lane; i < kTileIn; i += 32)
			{
				xlo = min(xlo, xidx[i]);
				xhi = max(xhi, xidx[i]);
			}
			ylo = __reduce_min_sync(0xffffffffu, ylo);
			yhi = __reduce_max_sync(0xffffffffu, yhi);
			xlo = __reduce_min_sync(0xffffffffu, xlo);
			xhi = __reduce_max_sync(0xffffffffu, xhi);
		}
		const int ty0 = ylo >> 5, ty1 = yhi >> 5, tx0 = xlo >> 5, tx1 = xhi >> 5;
		const int w = tx1 - tx0 + 1, n = w * (ty1 - ty0 + 1);
		const uint32_t *base = buf.tile_done + p.prev_done_offset + comp * p.P.tiles_x * p.P.tiles_y;
		bool ok = true;
		for (int k = lane; k < n && ok; k += 32)
			ok = wait_counter(base + (ty0 + k / w) * p.P.tiles_x + tx0 + k % w, uint32_t(p.prev_parts));
		if (!__all_sync(0xffffffffu, ok) && lane == 0)
			atomicOr(&buf.rc->error, kErrorLevelWait);
	}
	__syncthreads();
}

// Quantises the transmitted bands of a transformed tile in shared memory.
template <int kThreads>
__device__ __forceinline__ void quant_tile(DwtShared &sh, const LevelParams &p, const EncodeBuffers &buf, const int level,
                                           const int comp, const int tx, const int ty)
{
	using Split = DwtSplit<kThreads, 1>;
	const LevelDesc &L = p.L;
	// Quantise the transmitted bands of this tile: HL, LH, HH (+ LL at the last
	// level), kGroups bands per round. (A last round on the whole CTA, two warps
	// per row, repeats the rows' fixed work: 1080p encode 42.25 against 41.0 us.)
	const int first_band = level == kLevels - 1 ? 0 : 1;
	const int nb = 4 - first_band;
	const int grp = threadIdx.x / Split::kGroupThreads, t = threadIdx.x % Split::kGroupThreads;
	const int ly = (t >> 5) & 3;
	for (int bi = grp; bi < nb; bi += Split::kGroups)
		quant_analyze_row<Split::kQSplit>(&sh.bands[first_band + bi][0][0], ly, t >> 7, sh.q[bi], sh.scales[bi], L,
		                                  p.band[comp][first_band + bi], tx, ty, buf);
	__syncthreads();
	// A half-warp per band finishes its block. Tile dataflow: the resolve waits for
	// the count of every CTA, released once after all of its bands' rows (with a
	// full fence and count per band, and one per stored tile, a 4K 4:4:4 frame's
	// encode took 148.5 instead of 144 us).
	const int bi = int(threadIdx.x) >> 4;
	if ((bi & ~1) >= nb)
		return;
	quant_finish_block(bi < nb, sh.q[min(bi, nb - 1)], p.band[comp][first_band + min(bi, nb - 1)], p.subdivision_shift, tx, ty,
	                   buf);
	if (buf.tile_done)
	{
		asm volatile("bar.sync 1, 64;" ::: "memory"); // the two finishing warps
		if (threadIdx.x == 0)
			red_release_add(&buf.rc->fused_done, 1u);
	}
}

// One forward level for one 32x32 band tile of one component (64x64 input
// samples): `tile` in row-major tile order, `comp_index` the component among
// those at this level. Run by every thread of a kThreads-thread CTA. With
// kStripes > 1 (transform only) the CTA computes one stripe of 32 / kStripes
// band rows of the tile: it loads and lifts horizontally only the input rows
// the stripe spans.
//
// Bound by instruction issue (large levels) or by the latency of one load, one
// store and the barriers between them (small levels), so each pass works on
// packed pairs of samples (two FP32 operations per instruction), which the
// shared-memory layouts keep in adjacent registers: rows (r, r + rows / 2) for
// the horizontal pass, adjacent columns for the vertical one. A loader thread
// keeps one group of four columns, so the mirrored column indices of an edge
// tile are read once; samples are converted as they are loaded (no table of
// 256 values, no tensor-map load whose rows would have to be paired again).
// Measured against scalar lifting with TMA loads and a table of converted
// samples: encode of a 720p 4:2:0 frame 37.9 -> 34.9 us, 1080p 49.2 -> 47.5 us,
// 4K 4:4:4 (1.2 MB) 183 -> 179 us.
//
// kHalf: the level or its input is stored in FP16 or staged through it; the
// all-FP32 form carries none of that code.
template <int kThreads, int kStripes, bool kHalf>
__device__ __forceinline__ void dwt_forward_body(DwtSharedT<DwtSplit<kThreads, kStripes>::kRowsIn> &sh,
                                                 const LevelParams &p, const PlaneInput &in, const EncodeBuffers &buf,
                                                 const int fused, const int tile, const int comp_index,
                                                 const int stripe = 0)
{
	using Split = DwtSplit<kThreads, kStripes>;
	constexpr int kRowsIn = Split::kRowsIn, kPairRows = kRowsIn / 2;
	pdl_trigger();
	const int level = p.level;
	const int comp = (level == 0 && !p.chroma444) ? 0 : comp_index;
	const LevelDesc &L = p.L;
	const int tx = tile % L.tiles_x, ty = tile / L.tiles_x;
	const bool from_plane = level == 0 || (level == 1 && comp != 0 && !p.chroma444);

	int res_w, res_h, al_w, al_h;
	if (from_plane)
	{
		res_w = p.plane_width[comp];
		res_h = p.plane_height[comp];
		al_w = level == 0 ? p.aligned_width : p.aligned_width >> 1;
		al_h = level == 0 ? p.aligned_height : p.aligned_height >> 1;
	}
	else
	{
		res_w = al_w = p.P.width;
		res_h = al_h = p.P.height;
	}

	// Input window of this CTA. Inside the source every sample maps to itself;
	// an edge tile goes through the mirrored index tables.
	const int x0 = tx * 64 - 4, y0 = ty * 64 - 4 + stripe * (64 / kStripes);
	const bool x_inside = x0 >= 0 && x0 + kTileIn <= res_w, y_inside = y0 >= 0 && y0 + kRowsIn <= res_h;
	const bool interior = x_inside && y_inside;
	if (!interior)
	{
		for (int k = threadIdx.x; k < kTileIn + kRowsIn; k += kThreads)
		{
			if (k < kTileIn)
				sh.xidx[k] = fwd_index(x0 + k, res_w, al_w);
			else
				sh.yidx[k - kTileIn] = fwd_index(y0 + (k - kTileIn), res_h, al_h);
		}
		__syncthreads();
	}
	// The input planes are complete before the frame's first kernel. With the
	// tile dataflow a finer level's LL is read once the tiles it comes from are
	// stored, else after the whole previous grid.
	if (buf.tile_done)
	{
		if (!from_plane)
			wait_finer_tiles<kRowsIn>(sh.xidx, sh.yidx, interior, x0, y0, p, buf, comp);
	}
	else if (!from_plane)
		pdl_wait();

	// Tile load: a thread takes rows r and r + kPairRows of its four columns,
	// every load of its iterations in flight at once. The few threads beyond
	// the last full row of vectors, and rows beyond the window, repeat others'
	// loads instead of branching.
	constexpr int kLoadRows = kThreads / kVecs; // row pairs per iteration
	constexpr int kIters = (kPairRows + kLoadRows - 1) / kLoadRows;
	{
		const int j = threadIdx.x % kVecs, pr0 = min(int(threadIdx.x) / kVecs, kPairRows - 1);
		// This thread's four columns are consecutive inside the source, or (edge) gathered.
		const int x = x0 + 4 * j;
		const bool inside = x >= 0 && x + 4 <= res_w;
		auto pair_row = [&](int u) {
			const int pr = pr0 + u * kLoadRows;
			return (u + 1) * kLoadRows <= kPairRows ? pr : min(pr, kPairRows - 1);
		};
		auto row_of = [&](int i) { return y_inside ? y0 + i : sh.yidx[i]; };
		auto put = [&](int u, const f32x2 (&v)[4]) {
			float *dst = &sh.in[pair_row(u)][4 * j];
			*reinterpret_cast<ulonglong2 *>(dst) = make_ulonglong2(v[0], v[1]);
			*reinterpret_cast<ulonglong2 *>(dst + kInOdd) = make_ulonglong2(v[2], v[3]);
		};
		auto half_stage = [&](f32x2 &v) {
			if (kHalf && L.stage16)
			{
				float lo, hi;
				f2_unpack(v, lo, hi);
				v = f2_pack(round_to_half(lo), round_to_half(hi));
			}
		};
		if (from_plane)
		{
			const uint8_t *src = comp == 0 ? in.data[0] : (comp == 1 ? in.data[1] : in.data[2]);
			const int pitch = comp == 0 ? in.pitch[0] : (comp == 1 ? in.pitch[1] : in.pitch[2]);
			const int xs = comp == 0 ? in.xstride[0] : (comp == 1 ? in.xstride[1] : in.xstride[2]);
			const uintptr_t align = reinterpret_cast<uintptr_t>(src) | uintptr_t(pitch);
			if (in.sample16)
			{
				uint2 raw[kIters][2];
				const bool vec = inside && xs == 2 && (align & 7u) == 0;
				int4 xi = make_int4(x, x + 1, x + 2, x + 3);
				if (!inside)
					xi = *reinterpret_cast<const int4 *>(&sh.xidx[4 * j]);
#pragma unroll
				for (int u = 0; u < kIters; u++)
#pragma unroll
					for (int h = 0; h < 2; h++)
					{
						const uint8_t *row = src + size_t(row_of(pair_row(u) + h * kPairRows)) * pitch;
						raw[u][h] = vec ? __ldg(reinterpret_cast<const uint2 *>(row + 2 * x)) : pack4_u16(row, xi, xs);
					}
#pragma unroll
				for (int u = 0; u < kIters; u++)
				{
					f32x2 v[4];
#pragma unroll
					for (int b = 0; b < 4; b++)
					{
						uint32_t bits[2]; // sample b of a row over the exponent of 2^23
#pragma unroll
						for (int h = 0; h < 2; h++)
							bits[h] = __byte_perm(b < 2 ? raw[u][h].x : raw[u][h].y, 0x4B000000u, (b & 1) ? 0x7432 : 0x7410);
						v[b] = unorm_centered2<65535>(bits[0], bits[1]);
						half_stage(v[b]);
					}
					put(u, v);
				}
			}
			else
			{
				uint32_t raw[kIters][2];
				if (x_inside && y_inside && xs == 1 && (align & 3u) == 0)
				{
					const uint8_t *at = src + size_t(y0 + pr0) * pitch + x;
#pragma unroll
					for (int u = 0; u < kIters; u++)
#pragma unroll
						for (int h = 0; h < 2; h++)
							raw[u][h] = __ldg(reinterpret_cast<const uint32_t *>(
							    at + size_t(uint32_t(pair_row(u) - pr0 + h * kPairRows)) * pitch));
				}
				else
				{
					const bool vec = inside && xs == 1 && (align & 3u) == 0;
					// Unaligned rows: two aligned words around the four bytes, where the
					// row has bytes on both sides of them.
					const bool vec_shift = !vec && inside && xs == 1 && x >= 4 && x + 8 <= res_w;
					int4 xi = make_int4(x, x + 1, x + 2, x + 3);
					if (!inside)
						xi = *reinterpret_cast<const int4 *>(&sh.xidx[4 * j]);
#pragma unroll
					for (int u = 0; u < kIters; u++)
#pragma unroll
						for (int h = 0; h < 2; h++)
						{
							const uint8_t *row = src + size_t(row_of(pair_row(u) + h * kPairRows)) * pitch;
							if (vec)
								raw[u][h] = __ldg(reinterpret_cast<const uint32_t *>(row + x));
							else if (vec_shift)
							{
								const uintptr_t a = reinterpret_cast<uintptr_t>(row + x);
								const uint32_t *w = reinterpret_cast<const uint32_t *>(a & ~uintptr_t(3));
								raw[u][h] = __funnelshift_r(__ldg(w), __ldg(w + 1), 8u * uint32_t(a & 3u));
							}
							else
								raw[u][h] = pack4_u8(row, xi, xs);
						}
				}
#pragma unroll
				for (int u = 0; u < kIters; u++)
				{
					f32x2 v[4];
#pragma unroll
					for (int b = 0; b < 4; b++)
					{
						v[b] = unorm_centered2<255>(__byte_perm(raw[u][0], 0x4B000000u, 0x7440 + b),
						                            __byte_perm(raw[u][1], 0x4B000000u, 0x7440 + b));
						half_stage(v[b]);
					}
					put(u, v);
				}
			}
			if (!buf.tile_done)
				pdl_wait(); // before this level's stores
		}
		else
		{
			const LevelDesc &P = p.P;
			const int64_t ll = comp == 0 ? p.prev_ll[0] : (comp == 1 ? p.prev_ll[1] : p.prev_ll[2]);
			const bool f16 = kHalf && P.fp16 != 0;
			float4 raw[kIters][2];
			if (interior && !f16)
			{
				const float *at = buf.coef32 + ll + int64_t(y0 + pr0) * P.pitch + x;
#pragma unroll
				for (int u = 0; u < kIters; u++)
#pragma unroll
					for (int h = 0; h < 2; h++)
						raw[u][h] = __ldcg(reinterpret_cast<const float4 *>(
						    at + (pair_row(u) - pr0 + h * kPairRows) * P.pitch));
			}
			else
			{
				int4 xi = make_int4(x, x + 1, x + 2, x + 3);
				if (!inside)
					xi = *reinterpret_cast<const int4 *>(&sh.xidx[4 * j]);
#pragma unroll
				for (int u = 0; u < kIters; u++)
#pragma unroll
					for (int h = 0; h < 2; h++)
					{
						const int64_t row = ll + int64_t(row_of(pair_row(u) + h * kPairRows)) * P.pitch;
						if (!inside)
							raw[u][h] = make_float4(load_coef(buf.coef32, buf.coef16, f16, row + xi.x),
							                        load_coef(buf.coef32, buf.coef16, f16, row + xi.y),
							                        load_coef(buf.coef32, buf.coef16, f16, row + xi.z),
							                        load_coef(buf.coef32, buf.coef16, f16, row + xi.w));
						else if (f16)
						{
							const uint2 hv = __ldcg(reinterpret_cast<const uint2 *>(buf.coef16 + row + x));
							const float2 a = __half22float2(*reinterpret_cast<const __half2 *>(&hv.x));
							const float2 b = __half22float2(*reinterpret_cast<const __half2 *>(&hv.y));
							raw[u][h] = make_float4(a.x, a.y, b.x, b.y);
						}
						else
							raw[u][h] = __ldcg(reinterpret_cast<const float4 *>(buf.coef32 + row + x));
					}
			}
#pragma unroll
			for (int u = 0; u < kIters; u++)
			{
				const f32x2 v[4] = {f2_pack(raw[u][0].x, raw[u][1].x), f2_pack(raw[u][0].y, raw[u][1].y),
				                    f2_pack(raw[u][0].z, raw[u][1].z), f2_pack(raw[u][0].w, raw[u][1].w)};
				put(u, v);
			}
		}
	}
	__syncthreads();

	if (kStripes == 1 && fused && threadIdx.x >= kThreads - 64)
	{
		// The last two warps have the lightest load below.
		const int i = int(threadIdx.x) - (kThreads - 64), first_band = level == kLevels - 1 ? 0 : 1;
		if (first_band + (i >> 4) < 4)
			fill_quant_scales(sh.scales[i >> 4], i & 15, p.band[comp][first_band + (i >> 4)].quant_resolution);
	}
	// Horizontal lifting of row pairs, segments of kHPairs output pairs. Items
	// start at another warp from tile to tile: they fill half the warps, and
	// warps of one index share an issue port.
	{
		constexpr int kPairs = Split::kHPairs, kSegs = 32 / kPairs, kWin = 2 * kPairs + 8;
		const int t0 = kStripes == 1 ? (threadIdx.x + 32 * (tile & 3)) & (kThreads - 1) : threadIdx.x;
		for (int item = t0; item < kPairRows * kSegs; item += kThreads)
		{
			const int pr = item % kPairRows, seg = item / kPairRows;
			f32x2 e[kWin];
#pragma unroll
			for (int j = 0; j < kWin; j += 2)
			{
				// Pairs j, j + 1 of the window: chunk seg * kPairs + j / 2.
				const int odd = ((j >> 1) & 1) ? kInOdd : 0;
				const ulonglong2 v =
				    *reinterpret_cast<const ulonglong2 *>(&sh.in[pr][odd + (seg * (kPairs / 2) + (j >> 2)) * 4]);
				e[j] = v.x;
				e[j + 1] = v.y;
			}
			lift_forward2(e);
			float *const row0 = &sh.h[pr][seg * kPairs], *const row1 = &sh.h[pr + kPairRows][seg * kPairs];
#pragma unroll
			for (int k = 0; k < kPairs; k += 2)
			{
				float lo0[2], lo1[2], hi0[2], hi1[2]; // [output pair], of rows pr and pr + kPairRows
#pragma unroll
				for (int m = 0; m < 2; m++)
				{
					float a, b;
					f2_unpack(e[4 + 2 * (k + m)], a, b);
					lo0[m] = __fmul_rn(a, kInvK);
					lo1[m] = __fmul_rn(b, kInvK);
					f2_unpack(e[5 + 2 * (k + m)], a, b);
					hi0[m] = __fmul_rn(a, kK);
					hi1[m] = __fmul_rn(b, kK);
					if (kHalf && L.stage16)
					{
						lo0[m] = round_to_half(lo0[m]);
						lo1[m] = round_to_half(lo1[m]);
						hi0[m] = round_to_half(hi0[m]);
						hi1[m] = round_to_half(hi1[m]);
					}
				}
				*reinterpret_cast<float2 *>(row0 + k) = make_float2(lo0[0], lo0[1]);
				*reinterpret_cast<float2 *>(row1 + k) = make_float2(lo1[0], lo1[1]);
				*reinterpret_cast<float2 *>(row0 + 32 + k) = make_float2(hi0[0], hi0[1]);
				*reinterpret_cast<float2 *>(row1 + 32 + k) = make_float2(hi1[0], hi1[1]);
			}
		}
	}
	__syncthreads();

	// Vertical lifting of column pairs. Columns 0..31 hold the horizontal low
	// band (-> LL, LH), 32..63 the high band (-> HL, HH). Outputs go to storage
	// and, for the quantiser, to the band tiles; samples beyond the band are
	// stored as zeros.
	{
		constexpr int kPairs = Split::kVPairs, kRows = 32 / kStripes, kSegs = kRows / kPairs, kWin = 2 * kPairs + 8;
		const bool whole = tx * 32 + 32 <= L.width && ty * 32 + 32 <= L.height;
		for (int item = threadIdx.x; item < 32 * kSegs; item += kThreads)
		{
			const int col = 2 * (item & 31), seg = item >> 5;
			f32x2 e[kWin];
#pragma unroll
			for (int j = 0; j < kWin; j++)
				e[j] = *reinterpret_cast<const f32x2 *>(&sh.h[seg * 2 * kPairs + j][col]);
			lift_forward2(e);
			const int c = col & 31, b_low = col >> 5;
			const int gx = tx * 32 + c, gy = ty * 32 + stripe * kRows + seg * kPairs;
			const int64_t at = int64_t(gy) * L.pitch + gx;
			const int64_t at_low = p.band[comp][b_low].offset + at, at_high = p.band[comp][b_low + 2].offset + at;
#pragma unroll
			for (int k = 0; k < kPairs; k++)
			{
				e[4 + 2 * k] = f2_mul_rn(e[4 + 2 * k], f2_pack(kInvK, kInvK));
				e[5 + 2 * k] = f2_mul_rn(e[5 + 2 * k], f2_pack(kK, kK));
			}
			if (kHalf && (L.fp16 || L.stage16))
			{
#pragma unroll
				for (int k = 0; k < 2 * kPairs; k++)
				{
					float lo, hi;
					f2_unpack(e[4 + k], lo, hi);
					e[4 + k] = f2_pack(round_to_half(lo), round_to_half(hi));
				}
			}
			if (!whole)
			{
				// By masks made once: compared sample by sample, these spilled in the batch's
				// persistent kernel, and a partial tile's pass took 5.1 K cycles instead of 2.1 K.
				const uint32_t m0 = gx < L.width ? ~0u : 0u, m1 = gx + 1 < L.width ? ~0u : 0u;
				const int rows = L.height - gy;
#pragma unroll
				for (int k = 0; k < 2 * kPairs; k++)
				{
					const bool inside = (k >> 1) < rows;
					float lo, hi;
					f2_unpack(e[4 + k], lo, hi);
					e[4 + k] = f2_pack(__uint_as_float(inside ? __float_as_uint(lo) & m0 : 0u),
					                   __uint_as_float(inside ? __float_as_uint(hi) & m1 : 0u));
				}
			}
			if (kHalf && L.fp16)
			{
#pragma unroll
				for (int k = 0; k < kPairs; k++)
				{
					float a[4];
					f2_unpack(e[4 + 2 * k], a[0], a[1]);
					f2_unpack(e[5 + 2 * k], a[2], a[3]);
					*reinterpret_cast<__half2 *>(buf.coef16 + at_low + k * L.pitch) = __floats2half2_rn(a[0], a[1]);
					*reinterpret_cast<__half2 *>(buf.coef16 + at_high + k * L.pitch) = __floats2half2_rn(a[2], a[3]);
				}
			}
			else
			{
				float *low = buf.coef32 + at_low, *high = buf.coef32 + at_high;
#pragma unroll
				for (int k = 0; k < kPairs; k++, low += L.pitch, high += L.pitch)
				{
					*reinterpret_cast<f32x2 *>(low) = e[4 + 2 * k];
					*reinterpret_cast<f32x2 *>(high) = e[5 + 2 * k];
				}
			}
			if constexpr (kStripes == 1)
			{
#pragma unroll
				for (int k = 0; k < kPairs; k++)
				{
					*reinterpret_cast<f32x2 *>(&sh.bands[b_low][seg * kPairs + k][c]) = e[4 + 2 * k];
					*reinterpret_cast<f32x2 *>(&sh.bands[b_low + 2][seg * kPairs + k][c]) = e[5 + 2 * k];
				}
			}
		}
	}

	if (buf.tile_done)
		cta_count_done(buf.tile_done + p.done_offset + comp * L.tiles_x * L.tiles_y + tile);
	if constexpr (kStripes == 1)
	{
		if (!fused)
			return;
		if (!buf.tile_done)
			__syncthreads();
		quant_tile<kThreads>(sh, p, buf, level, comp, tx, ty);
	}
}

template <int kThreads, bool kHalf>
__global__ void __launch_bounds__(kThreads, DwtSplit<kThreads, 1>::kMinBlocks)
    dwt_forward_kernel(const LevelParams p, const PlaneInput in, const EncodeBuffers buf, const int fused)
{
	__shared__ DwtShared sh;
	dwt_forward_body<kThreads, 1, kHalf>(sh, p, in, buf, fused, int(blockIdx.x), int(blockIdx.y));
}

// Small transform-only levels (fewer tiles than SMs): four 256-thread CTAs per
// tile, one per stripe of 8 band rows (blockIdx.x = tile * 4 + stripe). Same
// parameters as dwt_forward_kernel (graph nodes are updated with one argument
// list).
constexpr int kDwtStripes = kDwtStripeCtas;
template <bool kHalf>
__global__ void __launch_bounds__(kLargeLevelThreads, 4)
    dwt_stripes_kernel(const LevelParams p, const PlaneInput in, const EncodeBuffers buf, const int fused)
{
	(void)fused;
	__shared__ DwtSharedT<DwtSplit<kLargeLevelThreads, kDwtStripes>::kRowsIn> sh;
	dwt_forward_body<kLargeLevelThreads, kDwtStripes, kHalf>(sh, p, in, buf, 0, int(blockIdx.x) / kDwtStripes,
	                                                         int(blockIdx.y), int(blockIdx.x) % kDwtStripes);
}

// Batched form (FP32 storage): one CTA per (frame, component, tile) of this level.
template <int kThreads>
__global__ void __launch_bounds__(kThreads, DwtSplit<kThreads, 1>::kMinBlocks)
    dwt_forward_batch_kernel(const BatchFrame *frames, const BatchFrameIO *io, const uint32_t *cta_map, const int level,
                             const int fused)
{
	__shared__ LevelParams s_p;
	__shared__ PlaneInput s_in;
	__shared__ EncodeBuffers s_buf;
	int f, local;
	batch_item(cta_map, f, local);
	load_params(s_p, frames[f].lp[level]);
	load_params(s_in, io[f].in);
	load_params(s_buf, frames[f].eb);
	__syncthreads();
	const int ntiles = s_p.L.tiles_x * s_p.L.tiles_y;
	__shared__ DwtShared sh;
	dwt_forward_body<kThreads, 1, false>(sh, s_p, s_in, s_buf, fused, local % ntiles, local / ntiles);
}

// Quantiser over a pyramid already in storage (the reference's
// Encoder::encode_pre_transformed, pyrowave_encoder.cpp:1138-1151, and the
// small levels of a frame). G 32x32 blocks per CTA, 128 * S threads each:
// blocks first + item * G + group, those below `end`. `tile` holds G band
// tiles of 32 x kBandPitch floats, `q` G reduction scratches.
template <int S, int G>
__device__ __forceinline__ void quant_blocks_body(const BlockParams &p, const EncodeBuffers &buf, const int first,
                                                  const int end, const int item, float (*tile)[32][kBandPitch],
                                                  QuantGroupShared *q, QuantScales *scales)
{
	constexpr int kGroupThreads = 128 * S;
	pdl_trigger();
	const int grp = threadIdx.x / kGroupThreads, t = threadIdx.x % kGroupThreads;
	const int b = first + item * G + grp;
	const bool active = b < end;
	const int k = active ? find_band(p, b) : 0;
	const BandEntry &E = p.band[k];
	const LevelDesc &L = p.level[E.level];
	const int rel = b - E.block32_offset;
	const int by = rel / E.block32_stride, bx = rel - by * E.block32_stride;
	if (buf.tile_done)
	{
		// Tile dataflow: the block's transform tile is stored once its counter is complete.
		if (active && t == 0 && !wait_counter(buf.tile_done + E.done_index + rel, uint32_t(E.done_parts)))
			atomicOr(&buf.rc->error, kErrorLevelWait);
		__syncthreads();
	}
	else
		pdl_wait();
	if (active && t < 16)
		fill_quant_scales(scales[grp], t, E.quant_resolution);
	if (active)
	{
		// The block's 32 rows as 8 vectors of 4 each, every load in flight at once.
		for (int i = t; i < 256; i += kGroupThreads)
		{
			const int r = i >> 3, c4 = (i & 7) * 4;
			const int64_t idx = E.offset + int64_t(by * 32 + r) * L.pitch + bx * 32 + c4;
			float4 f;
			if (L.fp16)
			{
				const uint2 hv = __ldcg(reinterpret_cast<const uint2 *>(buf.coef16 + idx));
				const float2 a = __half22float2(*reinterpret_cast<const __half2 *>(&hv.x));
				const float2 c = __half22float2(*reinterpret_cast<const __half2 *>(&hv.y));
				f = make_float4(a.x, a.y, c.x, c.y);
			}
			else
				f = __ldcg(reinterpret_cast<const float4 *>(buf.coef32 + idx));
			// Beyond the band: zeros (storage written by the forward transform has them).
			const int x = bx * 32 + c4, left = by * 32 + r < L.height ? L.width - x : 0;
			if (left < 4)
			{
				f.x = left > 0 ? f.x : 0.0f;
				f.y = left > 1 ? f.y : 0.0f;
				f.z = left > 2 ? f.z : 0.0f;
				f.w = 0.0f;
			}
			*reinterpret_cast<float4 *>(&tile[grp][r][c4]) = f;
		}
	}
	__syncthreads();
	BandParam B;
	B.offset = E.offset;
	B.block8_offset = E.block8_offset;
	B.block8_stride = E.block8_stride;
	B.block32_offset = E.block32_offset;
	B.block32_stride = E.block32_stride;
	B.quant_resolution = E.quant_resolution;
	B.rdo_scale = E.rdo_scale;
	B.quant_code = E.quant_code;
	if (active)
		quant_analyze_row<S>(&tile[grp][0][0], (t >> 5) & 3, t >> 7, q[grp], scales[grp], L, B, bx, by, buf);
	__syncthreads();
	if (t < 32)
		quant_finish_block(active && t < 16, q[grp], B, p.subdivision_shift, bx, by, buf);
}

// One 32x32 block per CTA: the launch follows the last small-level transform
// on the critical path, and one block per CTA is the shortest CTA lifetime
// (the blocks of a frame's small levels fit one wave).
template <int S>
__global__ void __launch_bounds__(128 * S) quant_pretransformed_kernel(const BlockParams p, const EncodeBuffers buf,
                                                                       const int nblocks)
{
	__shared__ alignas(16) float tile[1][32][kBandPitch];
	__shared__ QuantGroupShared q[1];
	__shared__ QuantScales scales[1];
	quant_blocks_body<S, 1>(p, buf, 0, nblocks, int(blockIdx.x), tile, q, scales);
}

// Batched form: one CTA per pair of blocks among each frame's small-level blocks.
template <int S>
__global__ void __launch_bounds__(256 * S) quant_blocks_batch_kernel(const BatchFrame *frames, const uint32_t *cta_map)
{
	__shared__ BlockParams s_p;
	__shared__ EncodeBuffers s_buf;
	__shared__ alignas(16) float tile[2][32][kBandPitch];
	__shared__ QuantGroupShared q[2];
	__shared__ QuantScales scales[2];
	int f, local;
	batch_item(cta_map, f, local);
	load_params(s_p, frames[f].bp);
	load_params(s_buf, frames[f].eb);
	__syncthreads();
	quant_blocks_body<S, 2>(s_p, s_buf, 0, frames[f].small_blocks, local, tile, q, scales);
}

// ---------------------------------------------------------------------------
// Block-wide exclusive scan (blockDim.x a multiple of 32, at most 1024);
// returns the exclusive prefix and the block total. With kReuse it ends with a
// barrier, after which warp_sums may be used again.
template <bool kReuse = true, typename T> __device__ __forceinline__ T block_exclusive_scan(T v, T *warp_sums, T &total)
{
	const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nwarps = blockDim.x >> 5;
	T x = v;
#pragma unroll
	for (int off = 1; off < 32; off *= 2)
	{
		const T y = __shfl_up_sync(0xffffffffu, x, off);
		if (lane >= off)
			x += y;
	}
	if (lane == 31)
		warp_sums[warp] = x;
	__syncthreads();
	if (warp == 0)
	{
		T s = lane < nwarps ? warp_sums[lane] : T(0);
#pragma unroll
		for (int off = 1; off < 32; off *= 2)
		{
			const T y = __shfl_up_sync(0xffffffffu, s, off);
			if (lane >= off)
				s += y;
		}
		warp_sums[lane] = s;
	}
	__syncthreads();
	const T base = warp == 0 ? T(0) : warp_sums[warp - 1];
	total = warp_sums[nwarps - 1];
	if (kReuse)
		__syncthreads();
	return base + x - v;
}

// The RD row of one 32x32 block as stored: 16 u16 word counts (quant 0..15)
// and 16 u8 buckets, 48 bytes in three 16-byte loads.
struct RawRD
{
	uint4 c0, c1, bb;
};

__device__ __forceinline__ RawRD load_raw_rd(const EncodeBuffers &buf, int blk)
{
	RawRD r;
	r.c0 = __ldcg(reinterpret_cast<const uint4 *>(buf.rd_cost + size_t(blk) * 16));
	r.c1 = __ldcg(reinterpret_cast<const uint4 *>(buf.rd_cost + size_t(blk) * 16) + 1);
	r.bb = __ldcg(reinterpret_cast<const uint4 *>(buf.rd_bucket + size_t(blk) * 16));
	return r;
}

__device__ __forceinline__ uint32_t u4_word(const uint4 &v, int i)
{
	return i == 0 ? v.x : (i == 1 ? v.y : (i == 2 ? v.z : v.w));
}

// Word count at quant l (l is a compile-time index after unrolling).
__device__ __forceinline__ uint32_t rd_cost_at(const RawRD &r, int l)
{
	const uint32_t w = l < 8 ? u4_word(r.c0, l >> 1) : u4_word(r.c1, (l - 8) >> 1);
	return (w >> (16 * (l & 1))) & 0xffffu;
}

__device__ __forceinline__ uint32_t rd_bucket_at(const RawRD &r, int l)
{
	return (u4_word(r.bb, l >> 2) >> (8 * (l & 3))) & 0xffu;
}

// Saving of the block's RD operation in bucket bk (0 if none). Buckets of one
// block strictly increase with the step, so at most one step matches.
__device__ __forceinline__ uint32_t op_saving_at_bucket(const RawRD &r, uint32_t bk)
{
	uint32_t sv = 0;
#pragma unroll
	for (int l = 1; l < 16; l++)
		if (rd_bucket_at(r, l) == bk)
			sv = rd_cost_at(r, l - 1) - rd_cost_at(r, l);
	return sv;
}

// Quant of a block: its largest applied RD step. Steps are applied when their
// (bucket, subdivision) slot precedes x*, or equals it and the block precedes the cut.
__device__ __forceinline__ uint32_t block_words(const RawRD &r, int blk, int sdiv, int xstar, uint32_t cut, int &q)
{
	q = 0;
	uint32_t words = rd_cost_at(r, 0);
#pragma unroll
	for (int l = 1; l < 16; l++)
	{
		const uint32_t cost = rd_cost_at(r, l);
		const uint32_t saving = rd_cost_at(r, l - 1) - cost;
		const int x = int(rd_bucket_at(r, l)) * kSubdivisions + sdiv;
		if (saving != 0 && (x < xstar || (x == xstar && uint32_t(blk) < cut)))
		{
			q = l;
			words = cost;
		}
	}
	return words;
}

// Exact-rate resolve (analyze_rate_control_finalize.comp + resolve_rate_control.comp).
//
// The reference walks all 2048 (bucket, subdivision) slots; for each slot with
// savings it applies RD operations in block order while the running saving
// stays below need - savings_of_earlier_slots. Every slot before the first slot
// x* whose inclusive prefix reaches `need` is applied in full, slots after x*
// not at all, and x* up to the first operation whose exclusive prefix reaches
// its requirement (the cut).
//
// The blocks are split into slices of consecutive blocks, one 1024-thread CTA
// each. Every CTA scans the histogram for x* itself; a CTA whose slice meets
// the x* subdivision also finds the cut (from the savings of that subdivision
// up to the end of its slice). It then gives its blocks their quant (the
// largest applied step), word counts and offsets: the slice's own scan plus
// the totals the preceding slices publish.
constexpr int kOwnBatch = 2;           // RD rows per thread with their loads in flight together
constexpr int kSliceWaitSpins = 1 << 20; // bounded wait for one preceding slice's total

// Calls f(blk, row) for blocks [b0, b1) in order, the first kOwnBatch rows from
// `first`, the rest loaded kOwnBatch at a time.
template <typename F>
__device__ __forceinline__ void for_rows(const EncodeBuffers &buf, int b0, int b1, const RawRD (&first)[kOwnBatch],
                                         F f)
{
#pragma unroll
	for (int i = 0; i < kOwnBatch; i++)
		if (b0 + i < b1)
			f(b0 + i, first[i]);
	for (int base = b0 + kOwnBatch; base < b1; base += kOwnBatch)
	{
		RawRD r[kOwnBatch];
#pragma unroll
		for (int i = 0; i < kOwnBatch; i++)
			if (base + i < b1)
				r[i] = load_raw_rd(buf, base + i);
#pragma unroll
		for (int i = 0; i < kOwnBatch; i++)
			if (base + i < b1)
				f(base + i, r[i]);
	}
}

__device__ __forceinline__ void load_rows(const EncodeBuffers &buf, int b0, int b1, RawRD (&r)[kOwnBatch])
{
#pragma unroll
	for (int i = 0; i < kOwnBatch; i++)
		if (b0 + i < b1)
			r[i] = load_raw_rd(buf, b0 + i);
}

// Tile dataflow: the forward levels with a fused quantiser may still run when
// the resolve starts (its wait covers only the launch before it); wait, bounded,
// until each has counted its quantiser finished. Called by every thread.
__device__ __forceinline__ void wait_fused_quantisers(const ResolveParams &p, RateControlState *rc)
{
	if (p.fused_ctas == 0)
		return;
	if (threadIdx.x == 0 && !wait_counter(&rc->fused_done, p.fused_ctas))
		atomicOr(&rc->error, kErrorLevelWait);
	__syncthreads();
}

__device__ __forceinline__ void resolve_body(const ResolveParams &p, const EncodeBuffers &buf, const int slice,
                                             const int nslices)
{
	__shared__ uint32_t scan[kHistSize];
	__shared__ uint32_t warp_sums[32];
	__shared__ unsigned long long warp_sums64[32];
	__shared__ int s_xstar;
	__shared__ uint32_t s_cut;
	__shared__ unsigned long long s_base;
	RateControlState *rc = buf.rc;
	const int t = threadIdx.x, nthreads = blockDim.x;
	const int nblocks = p.block_count_32x32;
	// Slices are rate-control subdivisions, or 1024-block parts of larger
	// ones: only the slices of the x* subdivision depend on the cut.
	const int slice_blocks = resolve_slice_blocks(nblocks, p.blocks_per_subdivision);
	const int s0 = min(slice * slice_blocks, nblocks), s1 = min(s0 + slice_blocks, nblocks);
	const int per = (s1 - s0 + nthreads - 1) / nthreads;
	const int b0 = min(s0 + t * per, s1), b1 = min(b0 + per, s1);
	// Every quantiser has finished once the wait returns (with the tile dataflow,
	// the fused ones once their count is complete). The packer is released only
	// then, because it reads their output before its own wait.
	pdl_wait();
	wait_fused_quantisers(p, rc);
	pdl_trigger();

	RawRD own[kOwnBatch];
	load_rows(buf, b0, b1, own);
	// The histogram: kHistSize / nthreads consecutive slots per thread.
	const int hper = kHistSize / nthreads, h0 = t * hper;
	uint32_t hv[kHistSize / 256];
	uint32_t hsum = 0;
#pragma unroll
	for (int i = 0; i < kHistSize / 256; i++)
		if (i < hper)
		{
			hv[i] = __ldcg(&rc->histogram[h0 + i]);
			hsum += hv[i];
		}
	if (t == 0)
	{
		s_xstar = -1;
		s_cut = 0xffffffffu;
	}
	uint32_t total;
	uint32_t run = block_exclusive_scan(hsum, warp_sums, total);
#pragma unroll
	for (int i = 0; i < kHistSize / 256; i++)
		if (i < hper)
		{
			run += hv[i];
			scan[h0 + i] = run;
		}
	__syncthreads();

	// No block codes words at quant 15, so a block's savings add up to its words at quant 0.
	const int64_t need = int64_t(total) - int64_t(p.target_words);
	if (need > 0)
	{
		for (int x = h0; x < h0 + hper; x++)
			if (int64_t(scan[x]) >= need && (x == 0 || int64_t(scan[x - 1]) < need))
				s_xstar = x;
	}
	__syncthreads();
	const int xstar = s_xstar;

	const int start = xstar >= 0 ? (xstar & (kSubdivisions - 1)) * p.blocks_per_subdivision : 0;
	const int end = xstar >= 0 ? min(start + p.blocks_per_subdivision, nblocks) : 0;
	if (xstar >= 0 && s0 < end && s1 > start)
	{
		// The cut, as far as this slice needs it: scan the savings at bucket b*
		// of the x* subdivision's blocks up to the end of the slice.
		const int64_t required = need - (xstar > 0 ? int64_t(scan[xstar - 1]) : 0);
		const uint32_t bk = uint32_t(xstar >> 4);
		const int c1 = min(end, s1);
		const int cper = (c1 - start + nthreads - 1) / nthreads;
		const int c0 = min(start + t * cper, c1), c0e = min(c0 + cper, c1);
		RawRD r0[kOwnBatch];
		load_rows(buf, c0, c0e, r0);
		uint32_t local = 0;
		for_rows(buf, c0, c0e, r0, [&](int, const RawRD &r) { local += op_saving_at_bucket(r, bk); });
		uint32_t tot;
		uint32_t ex = block_exclusive_scan(local, warp_sums, tot);
		bool found = false;
		for_rows(buf, c0, c0e, r0, [&](int blk, const RawRD &r) {
			const uint32_t sv = op_saving_at_bucket(r, bk);
			if (!found && sv != 0 && int64_t(ex) >= required)
			{
				atomicMin(&s_cut, uint32_t(blk));
				found = true;
			}
			ex += sv;
		});
		__syncthreads();
	}
	const uint32_t cut = s_cut;

	// Word counts of this thread's run, the slice scan, then the slice's base
	// from the totals of the preceding slices.
	unsigned long long local = 0; // words << 32 | non-empty blocks << 1
	for_rows(buf, b0, b1, own, [&](int blk, const RawRD &r) {
		int q;
		const uint32_t w = block_words(r, blk, blk >> p.subdivision_shift, xstar, cut, q);
		local += (uint64_t(w) << 32) | (uint64_t(w != 0 ? 1 : 0) << 1);
	});
	unsigned long long slice_sum;
	const unsigned long long run_excl = block_exclusive_scan(local, warp_sums64, slice_sum);
	if (t == 0)
		st_release_u64(&rc->slice_total[slice], slice_sum | 1ull);
	unsigned long long pred = 0;
	if (t < slice)
	{
		// Every slice CTA is resident (the grid is at most kMaxResolveSlices
		// CTAs and the packer launches only after all of them started), so the
		// wait ends; it is bounded all the same.
		unsigned long long v;
		int spins = 0;
		while (((v = ld_acquire_u64(&rc->slice_total[t])) & 1ull) == 0ull)
		{
			if (++spins > kSliceWaitSpins)
			{
				atomicOr(&rc->error, kErrorSliceWait);
				v = 1ull;
				break;
			}
			__nanosleep(64);
		}
		pred = v & ~1ull;
	}
	unsigned long long base_total;
	(void)block_exclusive_scan(pred, warp_sums64, base_total);
	if (t == 0)
		s_base = base_total;
	__syncthreads();
	unsigned long long pos = s_base + run_excl;
	for_rows(buf, b0, b1, own, [&](int blk, const RawRD &r) {
		int q;
		const uint32_t w = block_words(r, blk, blk >> p.subdivision_shift, xstar, cut, q);
		buf.quant[blk] = q;
		*reinterpret_cast<uint2 *>(buf.block_meta + 2 * size_t(blk)) = make_uint2(uint32_t(pos >> 32), w);
		pos += uint64_t(w) << 32;
	});

	if (t == 0 && slice == nslices - 1)
	{
		const unsigned long long all = s_base + slice_sum;
		const uint32_t total_words = uint32_t(all >> 32);
		const uint32_t non_zero = uint32_t(all & 0xffffffffull) >> 1;
		rc->xstar = xstar;
		rc->consumed = total;
		rc->sequence = p.sequence & 7u;
		rc->total_words = total_words;
		rc->non_zero_blocks = non_zero;
		if (2 + uint64_t(total_words) > buf.stream_capacity_words)
			atomicOr(&rc->error, kErrorStreamCapacity);
		// Start-of-frame sequence header (bitstream.md:250-265).
		buf.stream[0] = uint32_t(p.width - 1) | (uint32_t(p.height - 1) << 14) | ((p.sequence & 7u) << 28) | (1u << 31);
		buf.stream[1] = (non_zero & 0xffffffu) | (uint32_t(p.chroma444 ? 1 : 0) << 26);
	}
}

template <int kThreads>
__global__ void __launch_bounds__(kThreads) resolve_kernel(const ResolveParams p, const EncodeBuffers buf)
{
	resolve_body(p, buf, int(blockIdx.x), int(gridDim.x));
}

// The same resolve on one thread-block cluster of C CTAs (C a power of two up
// to 16), for frames of at most C * 1024 * R blocks: thread g = rank * 1024 + t
// owns the run of at most R consecutive blocks from g * R', R' = ceil(blocks /
// (C * 1024)), its RD rows loaded once into registers. Every CTA scans the
// whole histogram itself (8 KB), so all of them find x* and the requirement
// with no exchange. The cut and the offsets need prefixes across CTAs: each
// CTA writes its totals into the shared memory of every higher-ranked CTA
// (distributed shared memory) and a hardware cluster barrier publishes them:
// once for the offsets, and once for the cut unless the x* subdivision lies
// inside one CTA. An operation at the x* slot is applied when the exclusive
// prefix of the x* subdivision's savings before its block is below the
// requirement, which is the same set as the blocks before the cut. Results are
// those of resolve_body.
constexpr int kClusterResolveThreads = 1024;
constexpr int kMaxResolveCluster = 16;

template <int R>
__global__ void __launch_bounds__(kClusterResolveThreads, 1)
    resolve_cluster_kernel(const ResolveParams p, const EncodeBuffers buf)
{
	__shared__ uint32_t warp_sums[2][32]; // one per scan: no barrier to reuse it
	__shared__ unsigned long long warp_sums64[32];
	__shared__ int s_xstar;
	__shared__ uint32_t s_before; // savings of the slots before x*
	__shared__ unsigned long long s_saving_totals[kMaxResolveCluster]; // [r]: savings total of rank r < this rank
	__shared__ unsigned long long s_word_totals[kMaxResolveCluster];   // [r]: words << 32 | non-empty << 1 of rank r
	// Peers write into this CTA's shared memory only after every CTA started.
	cluster_arrive_relaxed();
	RateControlState *rc = buf.rc;
	const int t = threadIdx.x;
	const uint32_t rank = cluster_rank(), ncta = cluster_size();
	const int n = p.block_count_32x32;
	const int per = (n + int(ncta) * kClusterResolveThreads - 1) / (int(ncta) * kClusterResolveThreads); // <= R
	const int b0 = min((int(rank) * kClusterResolveThreads + t) * per, n), b1 = min(b0 + per, n);
	pdl_wait();
	wait_fused_quantisers(p, rc);
	pdl_trigger();

	RawRD rows[R];
#pragma unroll
	for (int i = 0; i < R; i++)
		if (b0 + i < b1)
			rows[i] = load_raw_rd(buf, b0 + i);
	static_assert(kHistSize == 2 * kClusterResolveThreads, "two histogram slots per thread");
	const uint32_t h0 = __ldcg(&rc->histogram[2 * t]), h1 = __ldcg(&rc->histogram[2 * t + 1]);
	if (t == 0)
		s_xstar = -1;
	uint32_t total;
	const uint32_t run = block_exclusive_scan<false>(h0 + h1, warp_sums[0], total);

	// No block codes words at quant 15, so a block's savings add up to its words at quant 0.
	const int64_t need = int64_t(total) - int64_t(p.target_words);
	if (need > 0)
	{
		// The first slot whose inclusive prefix reaches the need (exactly one slot's does first).
		if (int64_t(run + h0) >= need && (t == 0 || int64_t(run) < need))
		{
			s_xstar = 2 * t;
			s_before = run;
		}
		if (int64_t(run + h0 + h1) >= need && int64_t(run + h0) < need)
		{
			s_xstar = 2 * t + 1;
			s_before = run + h0;
		}
	}
	__syncthreads();
	const int xstar = s_xstar; // the same in every CTA: each scanned the same histogram
	cluster_wait();

	// Which of this thread's blocks apply their operation at the x* slot.
	bool apply_x[R];
#pragma unroll
	for (int i = 0; i < R; i++)
		apply_x[i] = false;
	if (xstar >= 0)
	{
		const int start = (xstar & (kSubdivisions - 1)) * p.blocks_per_subdivision;
		const int end = min(start + p.blocks_per_subdivision, n);
		const int64_t required = need - int64_t(s_before);
		const uint32_t bk = uint32_t(xstar >> 4);
		uint32_t sv[R];
		uint32_t local = 0;
#pragma unroll
		for (int i = 0; i < R; i++)
		{
			const int blk = b0 + i;
			sv[i] = (blk < b1 && blk >= start && blk < end) ? op_saving_at_bucket(rows[i], bk) : 0u;
			local += sv[i];
		}
		uint32_t cta_total;
		uint32_t ex = block_exclusive_scan<false>(local, warp_sums[1], cta_total);
		// When the x* subdivision lies inside one CTA's blocks (every CTA sees
		// the same x*, so all take the same branch), the other CTAs hold none of
		// its savings and the prefix needs no exchange.
		const int cta_blocks = per * kClusterResolveThreads;
		uint64_t base = 0;
		if (start / cta_blocks != (end - 1) / cta_blocks)
		{
			if (t < int(ncta) && t > int(rank))
				st_cluster_u64(&s_saving_totals[rank], uint32_t(t), cta_total);
			cluster_sync();
			for (uint32_t r = 0; r < rank; r++)
				base += s_saving_totals[r];
		}
#pragma unroll
		for (int i = 0; i < R; i++)
		{
			apply_x[i] = sv[i] != 0 && int64_t(base + ex) < required;
			ex += sv[i];
		}
	}

	// Word counts, the cluster-wide scan of offsets, the per-block decisions.
	uint32_t w[R];
	int q[R];
	unsigned long long local = 0; // words << 32 | non-empty blocks << 1
#pragma unroll
	for (int i = 0; i < R; i++)
	{
		const int blk = b0 + i;
		w[i] = 0;
		q[i] = 0;
		if (blk < b1)
		{
			// Operations before the x* slot, plus the one at it where applied.
			w[i] = block_words(rows[i], blk, blk >> p.subdivision_shift, xstar, apply_x[i] ? 0xffffffffu : 0u, q[i]);
			local += (uint64_t(w[i]) << 32) | (uint64_t(w[i] != 0 ? 1 : 0) << 1);
		}
	}
	unsigned long long cta_words;
	unsigned long long pos = block_exclusive_scan<false>(local, warp_sums64, cta_words);
	if (t < int(ncta) && t > int(rank))
		st_cluster_u64(&s_word_totals[rank], uint32_t(t), cta_words);
	cluster_sync();
	unsigned long long base = 0;
	for (uint32_t r = 0; r < rank; r++)
		base += s_word_totals[r];
	pos += base;
#pragma unroll
	for (int i = 0; i < R; i++)
	{
		const int blk = b0 + i;
		if (blk < b1)
		{
			buf.quant[blk] = q[i];
			*reinterpret_cast<uint2 *>(buf.block_meta + 2 * size_t(blk)) = make_uint2(uint32_t(pos >> 32), w[i]);
			pos += uint64_t(w[i]) << 32;
		}
	}
	if (t == 0 && rank == ncta - 1)
	{
		const unsigned long long all = base + cta_words;
		const uint32_t total_words = uint32_t(all >> 32);
		const uint32_t non_zero = uint32_t(all & 0xffffffffull) >> 1;
		rc->xstar = xstar;
		rc->consumed = total;
		rc->sequence = p.sequence & 7u;
		rc->total_words = total_words;
		rc->non_zero_blocks = non_zero;
		if (2 + uint64_t(total_words) > buf.stream_capacity_words)
			atomicOr(&rc->error, kErrorStreamCapacity);
		// Start-of-frame sequence header (bitstream.md:250-265).
		buf.stream[0] = uint32_t(p.width - 1) | (uint32_t(p.height - 1) << 14) | ((p.sequence & 7u) << 28) | (1u << 31);
		buf.stream[1] = (non_zero & 0xffffffu) | (uint32_t(p.chroma444 ? 1 : 0) << 26);
	}
}

// Batched form: one CTA per (frame, slice).
__global__ void __launch_bounds__(kResolveBatchThreads) resolve_batch_kernel(const BatchFrame *frames, const BatchFrameIO *io,
                                                             const uint32_t *cta_map)
{
	__shared__ ResolveParams s_p;
	__shared__ EncodeBuffers s_buf;
	int f, local;
	batch_item(cta_map, f, local);
	load_params(s_p, io[f].rp);
	load_params(s_buf, frames[f].eb);
	__syncthreads();
	resolve_body(s_p, s_buf, local, frames[f].slices);
}

// ---------------------------------------------------------------------------
// Block packing: one 32x32 block per warp, four 4x2 sub-blocks per lane (8x8
// rows 0..3 of column lx = lane >> 3, sub-block lane & 7), assembled in the
// warp's own shared memory and written as whole words at its prefix-scanned
// offset. No CTA barrier: the block's prefixes are warp scans of the four rows'
// counts packed into fields of one or two registers, magnitudes stay two to a
// register (the quantiser's layout), the plane bytes come from one 8x8 bit
// transpose per sub-block, and the signs of the four rows are compacted
// together, a byte each. Bound by instruction issue at 4K, by latency at 1080p.
// Measured with the dequantiser against two sub-blocks per thread of a 64-thread
// CTA: encode of a 4K 4:4:4 frame (1.2 MB) 179 -> 168 us, 1080p 47.6 -> 46.2 us.

// Bits i of an 8-bit mask where the 16-bit field i of w (fields 2j and 2j + 1 in
// word j) has its top bit set.
__device__ __forceinline__ uint32_t top_bits8(const uint32_t (&w)[4])
{
	const uint32_t m = 0x80008000u;
	const uint32_t t = ((w[0] & m) >> 15) | ((w[1] & m) >> 13) | ((w[2] & m) >> 11) | ((w[3] & m) >> 9);
	return (t | (t >> 15)) & 0xffu;
}

// Per byte of m: the bits of x at the positions set in m, moved together to the
// low end in order (the parallel suffix method of Warren, Hacker's Delight 7-4,
// on four bytes at once).
__device__ __forceinline__ uint32_t compress_bytes(uint32_t x, uint32_t m)
{
	x &= m;
	uint32_t mk = (~m << 1) & 0xfefefefeu;
#pragma unroll
	for (int s = 1; s < 8; s *= 2)
	{
		uint32_t mp = mk ^ ((mk << 1) & 0xfefefefeu);
		mp ^= (mp << 2) & 0xfcfcfcfcu;
		mp ^= (mp << 4) & 0xf0f0f0f0u;
		const uint32_t mv = mp & m;
		m = (m ^ mv) | (mv >> s);
		const uint32_t t = x & mv;
		x = (x ^ t) | (t >> s);
		mk &= ~mp;
	}
	return x;
}

constexpr int kPackEarlyBlocks = 148 * 32; // about what 56 registers let reside
__device__ __forceinline__ void pack_body(uint32_t *const pkt, const BlockParams &p, const EncodeBuffers &buf, const int blk)
{
	const unsigned full = 0xffffffffu;
	pdl_trigger();
	const BandEntry &B = p.band[find_band(p, blk)];
	const LevelDesc &L = p.level[B.level];
	const int rel = blk - B.block32_offset;
	const int by32 = rel / B.block32_stride, bx32 = rel - by32 * B.block32_stride;
	const int lane = threadIdx.x & 31, sub = lane & 7, lx = lane >> 3;
	const int x8 = bx32 * 4 + lx;

	// The resolve kernel releases this grid only after every quantiser has
	// finished, so the quantised magnitudes and code words can be fetched before
	// the wait; only the rate-control decisions come from the resolve kernel itself.
	// That pays for frames whose blocks are all resident at once (kPackEarlyBlocks);
	// beyond, half the blocks of a frame code nothing, and only the rows that do are
	// read, once known.
	const bool early = p.block_count_32x32 <= kPackEarlyBlocks;
	const uint4 *const mags = reinterpret_cast<const uint4 *>(buf.mag16 + int64_t(blk) * 1024) + lane;
	uint32_t cw[4];
	uint4 sm[4];
#pragma unroll
	for (int h = 0; h < 4; h++)
	{
		const int y8 = by32 * 4 + h;
		const bool in_range = x8 < L.blocks8_x && y8 < L.blocks8_y;
		cw[h] = in_range ? __ldcg(&buf.code_words[B.block8_offset + y8 * B.block8_stride + x8]) : 0u;
		sm[h] = early ? __ldcg(mags + 32 * h) : make_uint4(0u, 0u, 0u, 0u);
	}
	pdl_wait();

	const uint2 meta = __ldcg(reinterpret_cast<const uint2 *>(buf.block_meta) + blk);
	const int quant = __ldcg(&buf.quant[blk]);
	const uint32_t words = meta.y;
	if (words == 0)
		return;
	const uint32_t offset = meta.x;
	for (int w = lane; w < int(words) && w < kMaxBlockWords; w += 32)
		pkt[w] = 0u;

	// Per row: the planes of this lane's sub-block, its significant coefficients,
	// the coded 8x8s and their plane bytes, in fields of packed words.
	uint32_t ballot = 0, planes4 = 0, sig4 = 0, neg4 = 0;
	uint32_t bytes01 = 0, bytes23 = 0;
#pragma unroll
	for (int h = 0; h < 4; h++)
	{
		cw[h] = quantize_code_word(cw[h], quant);
		const bool active = (cw[h] & 0xffffu) != 0;
		const uint32_t wb = __ballot_sync(full, active && sub == 0);
		ballot |= ((wb & 1u) | ((wb >> 7) & 2u) | ((wb >> 14) & 4u) | ((wb >> 21) & 8u)) << (4 * h);
		const uint32_t out_q = (cw[h] >> kQPlanesOffset) & 0xfu;
		const uint32_t pl = active ? ((cw[h] >> (2 * sub)) & 3u) + out_q : 0u;
		planes4 |= pl << (8 * h);
		const uint32_t nbytes = uint32_t(plane_code_sum(cw[h], 0)) + out_q * 8u;
		if (h < 2)
			bytes01 |= nbytes << (16 * h);
		else
			bytes23 |= nbytes << (16 * (h - 2));
		if (!early && wb != 0)
			sm[h] = __ldcg(mags + 32 * h);
	}
	const uint32_t threshold = (0x8000u - (1u << quant)) * 0x10001u;
#pragma unroll
	for (int h = 0; h < 4; h++)
	{
		const uint32_t pl = (planes4 >> (8 * h)) & 0xffu;
		// |int(v)| >> quant != 0, as a carry into the sign bit of each field.
		const uint32_t w[4] = {sm[h].x, sm[h].y, sm[h].z, sm[h].w};
		uint32_t ge[4];
#pragma unroll
		for (int j = 0; j < 4; j++)
			ge[j] = (w[j] & 0x7fff7fffu) + threshold;
		sig4 |= (pl != 0 ? top_bits8(ge) : 0u) << (8 * h);
		neg4 |= top_bits8(w) << (8 * h);
	}
	const uint32_t n = uint32_t(__popc(ballot));

	// Prefixes: plane bytes over the 16 8x8s, planes over the sub-blocks of an
	// 8x8 (at most 144 in all, four rows in one word), significant coefficients
	// over the 32 sub-blocks of a row (at most 256, two rows to a word).
	uint32_t bi01 = bytes01, bi23 = bytes23, pi = planes4;
	uint32_t si01 = uint32_t(__popc(sig4 & 0xffu)) | (uint32_t(__popc(sig4 & 0xff00u)) << 16),
	         si23 = uint32_t(__popc(sig4 & 0xff0000u)) | (uint32_t(__popc(sig4 & 0xff000000u)) << 16);
	const uint32_t s01 = si01, s23 = si23;
#pragma unroll
	for (int off = 1; off < 32; off *= 2)
	{
		const uint32_t a = __shfl_up_sync(full, si01, off), b = __shfl_up_sync(full, si23, off);
		if (lane >= off)
		{
			si01 += a;
			si23 += b;
		}
		if (off < 8)
		{
			const uint32_t c = __shfl_up_sync(full, pi, off);
			if (sub >= off)
				pi += c;
		}
		else
		{
			const uint32_t c = __shfl_up_sync(full, bi01, off), d = __shfl_up_sync(full, bi23, off);
			if (lane >= off)
			{
				bi01 += c;
				bi23 += d;
			}
		}
	}
	pi -= planes4;
	const uint32_t bt01 = __shfl_sync(full, bi01, 31), bt23 = __shfl_sync(full, bi23, 31);
	const uint32_t st01 = __shfl_sync(full, si01, 31), st23 = __shfl_sync(full, si23, 31);
	// Exclusive prefixes, first without the preceding rows.
	bi01 -= bytes01;
	bi23 -= bytes23;
	si01 -= s01;
	si23 -= s23;

	uint8_t *const bytes = reinterpret_cast<uint8_t *>(pkt);
	__syncwarp();
	if (lane == 0)
	{
		pkt[0] = (ballot & 0xffffu) | (words << 16) | ((__ldcg(&buf.rc->sequence) & 7u) << 28);
		pkt[1] = modify_quant_code(B.quant_code, quant) | (uint32_t(blk) << 8);
	}
	uint32_t row_bytes = 0;
#pragma unroll
	for (int h = 0; h < 4; h++)
	{
		if (((ballot >> (4 * h)) & 0xfu) == 0)
			continue; // no coded 8x8 in the row
		const int grp = 4 * h + lx;
		if (sub == 0 && ((ballot >> grp) & 1u))
		{
			const uint32_t compact = uint32_t(__popc(ballot & ((1u << grp) - 1u)));
			bytes[8 + 2 * compact + 0] = uint8_t(cw[h]);
			bytes[8 + 2 * compact + 1] = uint8_t(cw[h] >> 8);
			bytes[8 + 2 * n + compact] = uint8_t(cw[h] >> 16);
		}
		const uint32_t planes = (planes4 >> (8 * h)) & 0xffu;
		const uint32_t base = 8 + 3 * n + row_bytes + (((h < 2 ? bi01 : bi23) >> (16 * (h & 1))) & 0xffffu) +
		                      ((pi >> (8 * h)) & 0xffu);
		row_bytes += ((h < 2 ? bt01 : bt23) >> (16 * (h & 1))) & 0xffffu;
		// Bit plane k of the magnitudes (quant dropped) is byte k of the transposed
		// bit matrix whose byte i holds the magnitude of coefficient i; the most
		// significant plane comes first in the stream.
		const uint32_t keep = (0x7fffu >> quant) * 0x10001u;
		const uint32_t m0 = (sm[h].x >> quant) & keep, m1 = (sm[h].y >> quant) & keep, m2 = (sm[h].z >> quant) & keep,
		               m3 = (sm[h].w >> quant) & keep;
		unsigned long long lo = transpose8x8((unsigned long long)(__byte_perm(m2, m3, 0x6420)) << 32 |
		                                     __byte_perm(m0, m1, 0x6420));
		const uint32_t most = __reduce_max_sync(full, planes);
		if (most <= 8)
		{
			// The planes in stream order from byte 0 on.
			lo <<= 8 * (8 - planes) & 63;
			const uint32_t w0 = __byte_perm(uint32_t(lo >> 32), 0, 0x0123), w1 = __byte_perm(uint32_t(lo), 0, 0x0123);
#pragma unroll
			for (uint32_t k = 0; k < 8; k++)
			{
				if (k >= most)
					break;
				if (k < planes && base + k < uint32_t(kMaxBlockWords) * 4)
					bytes[base + k] = uint8_t((k < 4 ? w0 : w1) >> (8 * (k & 3)));
			}
		}
		else
		{
			const unsigned long long hi = transpose8x8((unsigned long long)(__byte_perm(m2, m3, 0x7531)) << 32 |
			                                           __byte_perm(m0, m1, 0x7531));
			for (uint32_t k = 0; k < planes; k++)
			{
				const uint32_t bit = planes - 1u - k;
				const uint32_t by = bit < 8 ? uint32_t(lo >> (8 * bit)) : (bit < 16 ? uint32_t(hi >> (8 * (bit - 8))) : 0u);
				if (base + k < uint32_t(kMaxBlockWords) * 4)
					bytes[base + k] = uint8_t(by);
			}
		}
	}
	const uint32_t total_bytes = row_bytes;
	__syncwarp();

	// Sign bits of significant coefficients, in coefficient order, after the
	// planes: a sub-block's are consecutive, OR-ed in with at most two updates.
	const uint32_t signs4 = compress_bytes(neg4, sig4);
	uint32_t bitpos = (8 + 3 * n + total_bytes) * 8;
#pragma unroll
	for (int h = 0; h < 4; h++)
	{
		const uint32_t bits = (signs4 >> (8 * h)) & 0xffu;
		const uint32_t at = bitpos + (((h < 2 ? si01 : si23) >> (16 * (h & 1))) & 0xffffu);
		bitpos += ((h < 2 ? st01 : st23) >> (16 * (h & 1))) & 0xffffu;
		const uint32_t w = at >> 5, shift = at & 31u;
		if (bits != 0 && w < uint32_t(kMaxBlockWords))
		{
			atomicOr(&pkt[w], bits << shift);
			if (shift > 24 && (bits >> (32u - shift)) != 0 && w + 1 < uint32_t(kMaxBlockWords))
				atomicOr(&pkt[w + 1], bits >> (32u - shift));
		}
	}
	__syncwarp();

	// The word count must match the rate-control estimate the offsets were built from.
	const uint32_t expect = (bitpos - 64 + 31) / 32 + 2;
	const bool fits = words <= uint32_t(kMaxBlockWords) && 2 + offset + words <= buf.stream_capacity_words;
	if (lane == 0 && (expect != words || !fits))
		atomicOr(&buf.rc->error, kErrorWordCount);
	if (!fits)
		return;
	uint32_t *dst = buf.stream + 2 + offset;
	for (int w = lane; w < int(words); w += 32)
		dst[w] = pkt[w];
}

// Two 32x32 blocks per CTA: a 1080p frame's 3261 blocks are resident in one wave.
constexpr int kPackThreads = 64;
__global__ void __launch_bounds__(kPackThreads) pack_kernel(const BlockParams p, const EncodeBuffers buf)
{
	__shared__ uint32_t pkt[kPackThreads / 32][kMaxBlockWords];
	const int warp = int(threadIdx.x) >> 5, blk = int(blockIdx.x) * (kPackThreads / 32) + warp;
	if (blk < p.block_count_32x32)
		pack_body(pkt[warp], p, buf, blk);
}

// Batched form: one 32-thread CTA per (frame, block).
__global__ void __launch_bounds__(32) pack_batch_kernel(const BatchFrame *frames, const uint32_t *cta_map)
{
	__shared__ BlockParams s_p;
	__shared__ EncodeBuffers s_buf;
	int f, local;
	batch_item(cta_map, f, local);
	load_params(s_p, frames[f].bp);
	load_params(s_buf, frames[f].eb);
	__syncthreads();
	__shared__ uint32_t pkt[kMaxBlockWords];
	pack_body(pkt, s_p, s_buf, local);
}

// ---------------------------------------------------------------------------
// The batched form as one persistent launch. Each CTA loops: take the next
// work item from the ticket counter, wait (bounded) until every item of the
// frame's gating stage has finished, copy the stage's parameters of that frame
// into shared memory, run the stage's body on the item, and count the item as
// finished. Items are taken in ticket order, so a CTA only ever waits for items
// that running CTAs took before it: the waits end whether or not every CTA of
// the grid is resident. Every stage body is the one the single-frame kernels
// run (at 256 threads; packing and dequantising run eight blocks per item, one
// per warp), so each frame's results are those of the single-frame path.
constexpr uint32_t kBatchWaitSpins = 1u << 22;

struct BatchQuantShared
{
	alignas(16) float tile[2][32][kBandPitch];
	QuantGroupShared q[2];
	QuantScales scales[2];
};

struct BatchShared
{
	union
	{
		DwtShared dwt;
		IdwtShared idwt;
		uint32_t pack[kBatchBlockItem][kMaxBlockWords];
		DequantShared deq[kBatchBlockItem];
		BatchQuantShared quant;
	} u;
	union
	{
		LevelParams lp;
		BlockParams bp;
		ResolveParams rp;
	} prm;
	EncodeBuffers eb;
	DecodeInput di;
	PlaneInput in;
	PlaneOutput out;
	int item;
};
// Four CTAs share an SM's 228 KB; each also has the resolve's static storage
// (8704 bytes) and 1 KB that the system reserves.
constexpr size_t kBatchStaticShared = 8704, kSmShared = 228 * 1024;
static_assert(4 * (sizeof(BatchShared) + kBatchStaticShared + 1024) <= kSmShared,
              "the persistent kernel's stage storage fits four CTAs per SM");

// The kernel's shared memory (dynamic: its stages' storage is a union larger
// than a static allocation may be).
extern __shared__ __align__(128) unsigned char batch_smem[];
__device__ __forceinline__ BatchShared &batch_shared() { return *reinterpret_cast<BatchShared *>(batch_smem); }

// Each stage body is its own function (not inlined into the loop), so that
// register allocation happens per stage, as in the single-frame kernels; each
// reaches the shared storage through the kernel's own symbol. The two kernels
// have functions of their own: with functions that both called, one kernel's
// decoded samples were off by one in places (nvcc 12.9).
template <bool kManyItems> __device__ __noinline__ void batch_forward_item(int level, int small_level, int local)
{
	BatchShared &sh = batch_shared();
	const int per_comp = sh.prm.lp.L.tiles_x * sh.prm.lp.L.tiles_y;
	dwt_forward_body<kBatchPersistentThreads, 1, false>(sh.u.dwt, sh.prm.lp, sh.in, sh.eb, level < small_level ? 1 : 0,
	                                                    local % per_comp, local / per_comp);
}

template <bool kManyItems> __device__ __noinline__ void batch_quant_item(int small_blocks, int local)
{
	BatchShared &sh = batch_shared();
	quant_blocks_body<1, 2>(sh.prm.bp, sh.eb, 0, small_blocks, local, sh.u.quant.tile, sh.u.quant.q, sh.u.quant.scales);
}

template <bool kManyItems> __device__ __noinline__ void batch_resolve_item(int slice, int slices)
{
	BatchShared &sh = batch_shared();
	resolve_body(sh.prm.rp, sh.eb, slice, slices);
}

template <bool kManyItems> __device__ __noinline__ void batch_pack_item(int blk, int warp)
{
	BatchShared &sh = batch_shared();
	pack_body(sh.u.pack[warp], sh.prm.bp, sh.eb, blk);
}

template <bool kManyItems> __device__ __noinline__ void batch_dequant_item(int blk, int warp)
{
	BatchShared &sh = batch_shared();
	dequant_body(sh.u.deq[warp], sh.prm.bp, sh.di, blk, blk == 0);
}

template <bool kManyItems> __device__ __noinline__ void batch_inverse_item(int local)
{
	BatchShared &sh = batch_shared();
	const int per_comp = sh.prm.lp.L.tiles_x * sh.prm.lp.L.tiles_y;
	idwt_body<kBatchPersistentThreads, 1, false>(sh.u.idwt, sh.prm.lp, sh.di, sh.out, nullptr, local % per_comp,
	                                   local / per_comp);
}

template <bool kManyItems>
__global__ void __launch_bounds__(kBatchPersistentThreads, 4) batch_persistent_kernel(const BatchRunParams rp)
{
	BatchShared &sh = batch_shared();
	// Thread 0 holds the CTA's next ticket, taken while the current item runs,
	// so the ticket's round trip overlaps the work. Without kManyItems a CTA that
	// waits at a gate takes it only once items of the gating stage have finished:
	// taken while idle, it would put two items of one stage on this CTA and none on
	// another (one 1080p frame, encode + decode: 247 us, now 202). With kManyItems,
	// two items per CTA and more in some stage, it is taken at once (twelve mixed
	// frames: 1702 us, 1733 waiting for the gate first). Tickets are still
	// processed in increasing order by every CTA, and an item only waits for items
	// with smaller tickets, so every wait still ends.
	int next = 0;
	if (threadIdx.x == 0)
		next = int(atomicAdd(rp.ticket, 1u));
	for (;;)
	{
		if (threadIdx.x == 0)
			sh.item = next;
		__syncthreads();
		const int item = sh.item;
		if (item >= rp.nwork)
			return;
		if (kManyItems && threadIdx.x == 0)
			next = int(atomicAdd(rp.ticket, 1u));
		const uint32_t w = __ldg(rp.work + item);
		const int f = int(w >> 24), stage = int((w >> kBatchLocalBits) & 31u);
		const int local = int(w & ((1u << kBatchLocalBits) - 1u));
		const BatchFrame &fr = rp.frames[f];
		if (threadIdx.x == 0)
		{
			bool taken = kManyItems;
			const uint32_t gate = __ldg(rp.gates + f * kBatchStages + stage);
			if (gate != kNoGate)
			{
				const uint32_t *count = rp.done + f * kBatchStages + (gate >> 24);
				const uint32_t target = gate & 0xffffffu;
				uint32_t spins = 0, finished;
				while ((finished = ld_acquire_u32(count)) < target)
				{
					if (finished != 0 && !taken)
					{
						next = int(atomicAdd(rp.ticket, 1u));
						taken = true;
					}
					if (++spins > kBatchWaitSpins)
					{
						atomicOr(&fr.eb.rc->error, kErrorLevelWait);
						break;
					}
					__nanosleep(64);
				}
			}
			if (!taken)
				next = int(atomicAdd(rp.ticket, 1u));
		}
		if (stage < kStageQuant)
		{
			load_params(sh.prm.lp, fr.lp[stage - kStageDwt0]);
			load_params(sh.in, rp.io[f].in);
			load_params(sh.eb, fr.eb);
		}
		else if (stage == kStageQuant || stage == kStagePack)
		{
			load_params(sh.prm.bp, fr.bp);
			load_params(sh.eb, fr.eb);
		}
		else if (stage == kStageResolve)
		{
			load_params(sh.prm.rp, rp.io[f].rp);
			load_params(sh.eb, fr.eb);
		}
		else if (stage == kStageDequant)
		{
			load_params(sh.prm.bp, fr.bp);
			load_params(sh.di, fr.di);
		}
		else
		{
			load_params(sh.prm.lp, fr.lp[kStageIdwt4 + 4 - stage]);
			load_params(sh.di, fr.di);
			load_params(sh.out, rp.io[f].out);
		}
		__syncthreads();
		const int warp = int(threadIdx.x) >> 5;
		if (stage < kStageQuant)
			batch_forward_item<kManyItems>(stage - kStageDwt0, rp.small_level, local);
		else if (stage == kStageQuant)
			batch_quant_item<kManyItems>(fr.small_blocks, local);
		else if (stage == kStageResolve)
			batch_resolve_item<kManyItems>(local, fr.slices);
		else if (stage == kStagePack)
		{
			const int blk = local * kBatchBlockItem + warp;
			if (blk < fr.block_count)
				batch_pack_item<kManyItems>(blk, warp);
		}
		else if (stage == kStageDequant)
		{
			const int blk = local * kBatchBlockItem + warp;
			if (blk < fr.block_count)
				batch_dequant_item<kManyItems>(blk, warp);
		}
		else
			batch_inverse_item<kManyItems>(local);
		__syncthreads();
		if (threadIdx.x == 0)
		{
			__threadfence();
			atomicAdd(rp.done + f * kBatchStages + stage, 1u);
		}
	}
}

} // namespace

namespace
{
template <bool kManyItems> int persistent_ctas_per_sm()
{
	cudaFuncSetAttribute(batch_persistent_kernel<kManyItems>, cudaFuncAttributeMaxDynamicSharedMemorySize,
	                     int(sizeof(BatchShared)));
	int n = 0;
	if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, batch_persistent_kernel<kManyItems>, kBatchPersistentThreads,
	                                                  sizeof(BatchShared)) != cudaSuccess ||
	    n < 1)
	{
		(void)cudaGetLastError();
		n = 1;
	}
	return n;
}
} // namespace

int batch_persistent_max_ctas_per_sm()
{
	static int cached = 0;
	if (!cached)
		cached = std::min(persistent_ctas_per_sm<false>(), persistent_ctas_per_sm<true>());
	return cached;
}

// The kernels' shared-memory attribute is set by batch_persistent_max_ctas_per_sm,
// which the batch calls before any launch (outside stream capture).
void launch_batch_persistent(const BatchRunParams &rp, bool many_items, int ctas, cudaStream_t stream)
{
	if (many_items)
		batch_persistent_kernel<true><<<ctas, kBatchPersistentThreads, sizeof(BatchShared), stream>>>(rp);
	else
		batch_persistent_kernel<false><<<ctas, kBatchPersistentThreads, sizeof(BatchShared), stream>>>(rp);
}

LaunchConfig::LaunchConfig(dim3 grid, dim3 block, cudaStream_t stream, bool programmatic)
{
	cfg = {};
	cfg.gridDim = grid;
	cfg.blockDim = block;
	cfg.dynamicSmemBytes = 0;
	cfg.stream = stream;
	attr.id = cudaLaunchAttributeProgrammaticStreamSerialization;
	attr.val.programmaticStreamSerializationAllowed = 1;
	cfg.attrs = programmatic ? &attr : nullptr;
	cfg.numAttrs = programmatic ? 1 : 0;
}

void launch_dwt_forward_level(const LevelParams &p, const PlaneInput &in, const EncodeBuffers &buf,
                              bool fused_quant, bool programmatic, cudaStream_t stream)
{
	const dim3 grid(p.L.tiles_x * p.L.tiles_y, (p.level == 0 && !p.chroma444) ? 1 : 3);
	const int f = fused_quant ? 1 : 0;
	const bool half = p.L.fp16 || p.L.stage16 || (p.level > 0 && p.P.fp16);
	if (int(grid.x * grid.y) < kSmallLevelTiles && f == 0)
	{
		LaunchConfig lc(dim3(grid.x * kDwtStripes, grid.y), dim3(kLargeLevelThreads), stream, programmatic);
		cudaLaunchKernelEx(&lc.cfg, half ? dwt_stripes_kernel<true> : dwt_stripes_kernel<false>, p, in, buf, f);
	}
	else
	{
		LaunchConfig lc(grid, dim3(kLargeLevelThreads), stream, programmatic);
		cudaLaunchKernelEx(&lc.cfg, half ? dwt_forward_kernel<kLargeLevelThreads, true> : dwt_forward_kernel<kLargeLevelThreads, false>,
		                   p, in, buf, f);
	}
}

// Two warps per row of 8x8 blocks halve the levels' serial loop, one warp does
// the row's fixed work once: measured, two are the faster below about two blocks
// per SM (256x144 encode + decode 39.6 against 40.3 us), one above (720p encode
// 32.75 -> 32.1 us, 12 mixed frames 857 -> 836 us; 1080p the same).
constexpr int kSplitRowsBlocks = 2 * 148;
void launch_quant_pretransformed(const BlockParams &p, const EncodeBuffers &buf, int nblocks, bool programmatic,
                                 cudaStream_t stream)
{
	const bool split = nblocks <= kSplitRowsBlocks;
	LaunchConfig lc(dim3(nblocks), dim3(split ? 256 : 128), stream, programmatic);
	cudaLaunchKernelEx(&lc.cfg, split ? quant_pretransformed_kernel<2> : quant_pretransformed_kernel<1>, p, buf, nblocks);
}

int resolve_cluster_max()
{
	static int cached = 0;
	if (cached == 0)
	{
		// Clusters of 16 CTAs are opt-in; use them where the device can place one.
		int n = 0;
		if (cudaFuncSetAttribute(resolve_cluster_kernel<1>, cudaFuncAttributeNonPortableClusterSizeAllowed, 1) ==
		        cudaSuccess &&
		    cudaFuncSetAttribute(resolve_cluster_kernel<2>, cudaFuncAttributeNonPortableClusterSizeAllowed, 1) ==
		        cudaSuccess &&
		    cudaFuncSetAttribute(resolve_cluster_kernel<4>, cudaFuncAttributeNonPortableClusterSizeAllowed, 1) ==
		        cudaSuccess)
		{
			cudaLaunchConfig_t cfg = {};
			cudaLaunchAttribute attr = {};
			cfg.gridDim = dim3(kMaxResolveCluster);
			cfg.blockDim = dim3(kClusterResolveThreads);
			attr.id = cudaLaunchAttributeClusterDimension;
			attr.val.clusterDim.x = kMaxResolveCluster;
			attr.val.clusterDim.y = 1;
			attr.val.clusterDim.z = 1;
			cfg.attrs = &attr;
			cfg.numAttrs = 1;
			if (cudaOccupancyMaxActiveClusters(&n, resolve_cluster_kernel<4>, &cfg) != cudaSuccess)
				n = 0;
		}
		(void)cudaGetLastError();
		cached = n > 0 ? kMaxResolveCluster : 8;
	}
	return cached;
}

bool resolve_cluster_shape(int blocks, int &ctas, int &rows)
{
	const int cmax = resolve_cluster_max();
	int c = 1;
	while (c < cmax && c * kClusterResolveThreads < blocks)
		c *= 2;
	const int r = (blocks + c * kClusterResolveThreads - 1) / (c * kClusterResolveThreads);
	if (r > 4)
		return false;
	ctas = c;
	rows = r <= 1 ? 1 : (r <= 2 ? 2 : 4);
	return true;
}

void launch_resolve(const ResolveParams &p, const EncodeBuffers &buf, cudaStream_t stream)
{
	int ctas = 0, rows = 0;
	if (resolve_cluster_shape(p.block_count_32x32, ctas, rows))
	{
		cudaLaunchConfig_t cfg = {};
		cudaLaunchAttribute attrs[2] = {};
		cfg.gridDim = dim3(ctas);
		cfg.blockDim = dim3(kClusterResolveThreads);
		cfg.stream = stream;
		attrs[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
		attrs[0].val.programmaticStreamSerializationAllowed = 1;
		attrs[1].id = cudaLaunchAttributeClusterDimension;
		attrs[1].val.clusterDim.x = unsigned(ctas);
		attrs[1].val.clusterDim.y = 1;
		attrs[1].val.clusterDim.z = 1;
		cfg.attrs = attrs;
		cfg.numAttrs = 2;
		if (rows == 1)
			cudaLaunchKernelEx(&cfg, resolve_cluster_kernel<1>, p, buf);
		else if (rows == 2)
			cudaLaunchKernelEx(&cfg, resolve_cluster_kernel<2>, p, buf);
		else
			cudaLaunchKernelEx(&cfg, resolve_cluster_kernel<4>, p, buf);
		return;
	}
	const int slices = resolve_slices(p.block_count_32x32, p.blocks_per_subdivision);
	// One thread per block of a slice, 256 to 1024 per CTA.
	if (p.blocks_per_subdivision >= 1024)
	{
		LaunchConfig lc(dim3(slices), dim3(1024), stream, true);
		cudaLaunchKernelEx(&lc.cfg, resolve_kernel<1024>, p, buf);
	}
	else if (p.blocks_per_subdivision >= 512)
	{
		LaunchConfig lc(dim3(slices), dim3(512), stream, true);
		cudaLaunchKernelEx(&lc.cfg, resolve_kernel<512>, p, buf);
	}
	else
	{
		LaunchConfig lc(dim3(slices), dim3(256), stream, true);
		cudaLaunchKernelEx(&lc.cfg, resolve_kernel<256>, p, buf);
	}
}

void launch_pack(const BlockParams &p, const EncodeBuffers &buf, cudaStream_t stream)
{
	constexpr int kBlocks = kPackThreads / 32;
	LaunchConfig lc(dim3((p.block_count_32x32 + kBlocks - 1) / kBlocks), dim3(kPackThreads), stream, true);
	cudaLaunchKernelEx(&lc.cfg, pack_kernel, p, buf);
}

void launch_dwt_forward_batch(const BatchFrame *frames, const BatchFrameIO *io, const uint32_t *cta_map, int nctas,
                              int level, bool fused_quant, bool large_ctas, bool programmatic, cudaStream_t stream)
{
	const int f = fused_quant ? 1 : 0;
	if (large_ctas)
	{
		LaunchConfig lc(dim3(nctas), dim3(1024), stream, programmatic);
		cudaLaunchKernelEx(&lc.cfg, dwt_forward_batch_kernel<1024>, frames, io, cta_map, level, f);
	}
	else
	{
		LaunchConfig lc(dim3(nctas), dim3(kLargeLevelThreads), stream, programmatic);
		cudaLaunchKernelEx(&lc.cfg, dwt_forward_batch_kernel<kLargeLevelThreads>, frames, io, cta_map, level, f);
	}
}

void launch_quant_blocks_batch(const BatchFrame *frames, const uint32_t *cta_map, int nctas, bool programmatic,
                               cudaStream_t stream)
{
	LaunchConfig lc(dim3(nctas), dim3(512), stream, programmatic);
	cudaLaunchKernelEx(&lc.cfg, quant_blocks_batch_kernel<2>, frames, cta_map);
}

void launch_resolve_batch(const BatchFrame *frames, const BatchFrameIO *io, const uint32_t *cta_map, int nctas,
                          cudaStream_t stream)
{
	LaunchConfig lc(dim3(nctas), dim3(kResolveBatchThreads), stream, true);
	cudaLaunchKernelEx(&lc.cfg, resolve_batch_kernel, frames, io, cta_map);
}

void launch_pack_batch(const BatchFrame *frames, const uint32_t *cta_map, int nctas, cudaStream_t stream)
{
	LaunchConfig lc(dim3(nctas), dim3(32), stream, true);
	cudaLaunchKernelEx(&lc.cfg, pack_batch_kernel, frames, cta_map);
}

} // namespace pw
