// Hashing kernels: per-slice MD5 + CRC32 (the IFSC entries) and per-file MD5,
// one independent hash stream per GPU thread.
//
// Semantics follow the reference's HasherInput (hasher/hasher_base.h:103-186,
// src/gf.cc:926-954, 1015-1039):
//   IFSC entry of a slice = MD5(slice bytes zero-padded to the slice size)
//                           ++ CRC32(same bytes) little-endian      (20 bytes)
//   file MD5 = MD5 of the file's bytes (no padding).
// MD5 is RFC 1321; CRC32 is the reflected IEEE polynomial 0xEDB88320.  The
// zero padding of the CRC is applied by multiplying the register by
// x^(8*pad) mod P (hasher/crc_zeropad.c:55-66); the MD5 must process the
// padding bytes.  The CRC is computed from shared-memory tables by other warps
// of the block, beside the MD5 chains.
#include "common.cuh"
#include "kernels.h"

namespace p2c {

// chains per warp of the IFSC's split form: the loads of 32 chains of a warp are
// 32 separate lines or rows of banks, and delay each other; one thread hashes
// 127.6 MB/s among 32 of a warp, 130.5 among 16 and 135.0 among 8 (while warps
// have a scheduler each: the other kernels choose by the number of chains)
#define P2C_MD5_LANES 8

// RFC 1321 round constants (a constexpr table: indexed by the unrolled step
// number, each becomes an immediate operand).
__device__ constexpr uint32_t c_md5K[64] = {
	0xd76aa478,0xe8c7b756,0x242070db,0xc1bdceee,0xf57c0faf,0x4787c62a,0xa8304613,0xfd469501,
	0x698098d8,0x8b44f7af,0xffff5bb1,0x895cd7be,0x6b901122,0xfd987193,0xa679438e,0x49b40821,
	0xf61e2562,0xc040b340,0x265e5a51,0xe9b6c7aa,0xd62f105d,0x02441453,0xd8a1e681,0xe7d3fbc8,
	0x21e1cde6,0xc33707d6,0xf4d50d87,0x455a14ed,0xa9e3e905,0xfcefa3f8,0x676f02d9,0x8d2a4c8a,
	0xfffa3942,0x8771f681,0x6d9d6122,0xfde5380c,0xa4beea44,0x4bdecfa9,0xf6bb4b60,0xbebfbc70,
	0x289b7ec6,0xeaa127fa,0xd4ef3085,0x04881d05,0xd9d4d039,0xe6db99e5,0x1fa27cf8,0xc4ac5665,
	0xf4292244,0x432aff97,0xab9423a7,0xfc93a039,0x655b59c3,0x8f0ccc92,0xffeff47d,0x85845dd1,
	0x6fa87e4f,0xfe2ce6e0,0xa3014314,0x4e0811a1,0xf7537e82,0xbd3af235,0x2ad7d2bb,0xeb86d391};

__device__ __forceinline__ uint32_t rotl(uint32_t x, int s) { return __funnelshift_l(x, x, s); }

// one 64-byte block; m[16] little-endian words
__device__ __forceinline__ void md5_block(uint32_t st[4], const uint32_t m[16]) {
	uint32_t a = st[0], b = st[1], c = st[2], d = st[3];
#pragma unroll
	for(int i = 0; i < 64; i++) {
		uint32_t f; int g, s;
		if(i < 16) { f = d ^ (b & (c ^ d)); g = i; s = (i & 3) == 0 ? 7 : (i & 3) == 1 ? 12 : (i & 3) == 2 ? 17 : 22; }
		else if(i < 32) { f = c ^ (d & (b ^ c)); g = (5 * i + 1) & 15; s = (i & 3) == 0 ? 5 : (i & 3) == 1 ? 9 : (i & 3) == 2 ? 14 : 20; }
		else if(i < 48) { f = b ^ c ^ d; g = (3 * i + 5) & 15; s = (i & 3) == 0 ? 4 : (i & 3) == 1 ? 11 : (i & 3) == 2 ? 16 : 23; }
		else { f = c ^ (b | ~d); g = (7 * i) & 15; s = (i & 3) == 0 ? 6 : (i & 3) == 1 ? 10 : (i & 3) == 2 ? 15 : 21; }
		// a + K + m does not depend on the previous step; the add of f is the
		// only add on the step's dependency chain (LOP3 -> add -> rotate-add).
		// It is written as its own PTX add so that the compiler cannot fold f
		// into the off-chain sum: with the four terms in one C expression the
		// step compiled to a second dependent add and ran ~21 cycles instead
		// of ~17 on GB300 with message words loaded from memory.
		const uint32_t pre = a + c_md5K[i] + m[g];
		uint32_t t;
		asm("add.u32 %0, %1, %2;" : "=r"(t) : "r"(f), "r"(pre));
		a = d; d = c; c = b;
		b = b + rotl(t, s);
	}
	st[0] += a; st[1] += b; st[2] += c; st[3] += d;
}

struct MsgBlock {
	uint32_t w[16];
	__device__ __forceinline__ explicit MsgBlock(const uint32_t (&m)[16]) {
#pragma unroll
		for(int q = 0; q < 16; q++) w[q] = m[q];
	}
};

// MD5 over `full` consecutive 64-byte blocks whose first word p lies C words
// (0..3) before a 16-byte boundary.  A single thread walks a long serial
// chain, so loads run two blocks ahead of it; each block's words stay where
// they were loaded (C > 0: the last C words of the load before it and the
// first 16 - C of its own), in three (four) buffers that the unrolled loop
// takes in turn, because copies and loads gathered between two blocks delay
// the chain: one thread hashes 144 MB/s this way and 138 with a copy per
// block (C = 0; 120 with a copy for C > 0).
// L2 prefetch distance (64-byte blocks) ahead of the register prefetch: the
// register loads then mostly hit L2, well inside their two-block lead
#define P2C_MD5_L2_AHEAD 48

// load k holds words C + 16 k ..; words the blocks do not need (the last C of
// the last load) are not read
template<int C>
__device__ __forceinline__ void md5_load(const uint32_t* p, size_t k, bool last, uint32_t (&m)[16]) {
	const uint4* p4 = reinterpret_cast<const uint4*>(p + C) + k * 4;
#pragma unroll
	for(int q = 0; q < 4; q++) {
		if(C == 0 || q < 3 || !last) {
			const uint4 v = __ldg(p4 + q);
			m[4 * q] = v.x; m[4 * q + 1] = v.y; m[4 * q + 2] = v.z; m[4 * q + 3] = v.w;
		} else {
#pragma unroll
			for(int e = 0; e < 4; e++) m[4 * q + e] = e < 4 - C ? __ldg(p + C + k * 16 + 4 * q + e) : 0u;
		}
	}
}
// one block from the load before it and its own
template<int C>
__device__ __forceinline__ void md5_joined(uint32_t st[4], const uint32_t (&prev)[16], const uint32_t (&cur)[16]) {
	uint32_t m[16];
#pragma unroll
	for(int q = 0; q < 16; q++) m[q] = q < C ? prev[(16 - C + q) & 15] : cur[q < C ? 0 : q - C];
	md5_block(st, m);
}
template<int C>
__device__ __forceinline__ void md5_blocks_at(uint32_t st[4], const uint32_t* p, size_t full) {
	if(!full) return;
	uint32_t X[16], Y[16], Z[16], W[16];
	// X: the load before the next block's, Y: its own, Z and W: the next two
#pragma unroll
	for(int q = 0; q < 16; q++) X[q] = q >= 16 - C ? __ldg(p + q - (16 - C)) : 0u;
	md5_load<C>(p, 0, full == 1, Y);
	if(full > 1) md5_load<C>(p, 1, full == 2, Z);
	size_t k = 0;
	auto ahead = [&](size_t b) {
		if(b + P2C_MD5_L2_AHEAD < full)
			asm volatile("prefetch.global.L2 [%0];" :: "l"(p + (b + P2C_MD5_L2_AHEAD) * 16));
	};
	if(C == 0) {
		for(; k + 5 <= full; k += 3) {
			ahead(k);
			ahead(k + 2);
			md5_load<C>(p, k + 2, false, X);
			md5_block(st, Y);
			md5_load<C>(p, k + 3, false, Y);
			md5_block(st, Z);
			md5_load<C>(p, k + 4, false, Z);
			md5_block(st, X);
			// block k + 3 is in Y, k + 4 in Z
		}
	} else {
		for(; k + 7 <= full; k += 4) {
			ahead(k);
			ahead(k + 2);
			md5_load<C>(p, k + 2, false, W);
			md5_joined<C>(st, X, Y);
			md5_load<C>(p, k + 3, false, X);
			md5_joined<C>(st, Y, Z);
			md5_load<C>(p, k + 4, false, Y);
			md5_joined<C>(st, Z, W);
			md5_load<C>(p, k + 5, false, Z);
			md5_joined<C>(st, W, X);
			// load k + 3 is in X, k + 4 in Y, k + 5 in Z
		}
	}
	for(; k < full; k++) {
		md5_joined<C>(st, X, Y);
#pragma unroll
		for(int q = 0; q < 16; q++) { X[q] = Y[q]; Y[q] = Z[q]; }
		if(k + 2 < full) md5_load<C>(p, k + 2, k + 3 == full, Z);
	}
}
__device__ __forceinline__ void md5_blocks(uint32_t st[4], const uint4* p4, size_t full) {
	md5_blocks_at<0>(st, reinterpret_cast<const uint32_t*>(p4), full);
}

// The same in two buffers with a copy per block: fewer registers and a shorter
// loop, for many chains per SM.  CRC: the words go through a CRC32 register too,
// in the bubbles of the MD5's dependency chain.
struct CrcTabs;
__device__ __forceinline__ uint32_t crc_word(const CrcTabs& T, uint32_t crc, uint32_t w);
template<bool CRC>
__device__ __forceinline__ void md5_blocks_pairs(uint32_t st[4], uint32_t& crc, const CrcTabs* T, const uint4* p4, size_t full) {
	const uint32_t* p = reinterpret_cast<const uint32_t*>(p4);
	uint32_t A[16], B[16];
	if(full > 0) md5_load<0>(p, 0, false, A);
	if(full > 1) md5_load<0>(p, 1, false, B);
	auto block = [&](uint32_t (&X)[16], size_t next) {
		uint32_t m[16];
#pragma unroll
		for(int q = 0; q < 16; q++) m[q] = X[q];
		if(next < full) md5_load<0>(p, next, false, X);
		if(CRC) {
#pragma unroll
			for(int q = 0; q < 16; q++) crc = crc_word(*T, crc, m[q]);
		}
		md5_block(st, m);
	};
	for(size_t b = 0; b < full; b += 2) {
		if(b + P2C_MD5_L2_AHEAD < full)
			asm volatile("prefetch.global.L2 [%0];" :: "l"(p4 + (b + P2C_MD5_L2_AHEAD) * 4));
		block(A, b + 2);
		if(b + 1 < full) block(B, b + 3);
	}
}

// The same from any 4-byte boundary with 32-bit loads: fewer registers, for
// blocks of many warps.
__device__ __forceinline__ void load_block32(const uint32_t* p, size_t b, uint32_t m[16]) {
#pragma unroll
	for(int q = 0; q < 16; q++) m[q] = __ldg(p + b * 16 + q);
}
__device__ __forceinline__ void md5_blocks32(uint32_t st[4], const uint32_t* p, size_t full) {
	uint32_t A[16];
	if(full > 0) load_block32(p, 0, A);
	for(size_t b = 0; b < full; b++) {
		if((b & 1) == 0 && b + P2C_MD5_L2_AHEAD < full)
			asm volatile("prefetch.global.L2 [%0];" :: "l"(p + (b + P2C_MD5_L2_AHEAD) * 16));
		const MsgBlock m(A);
		if(b + 1 < full) load_block32(p, b + 1, A);
		md5_block(st, m.w);
	}
}
// full 64-byte blocks from any 4-byte boundary
__device__ __forceinline__ void md5_blocks_words(uint32_t st[4], const uint32_t* p, size_t full) {
	switch((reinterpret_cast<uintptr_t>(p) >> 2) & 3) {
	case 0: md5_blocks_at<0>(st, p, full); break;
	case 1: md5_blocks_at<3>(st, p, full); break;
	case 2: md5_blocks_at<2>(st, p, full); break;
	default: md5_blocks_at<1>(st, p, full); break;
	}
}

// CRC32 slice-by-4 tables, built per CTA in shared memory
struct CrcTabs { uint32_t t[4][256]; };

__device__ void crc_tabs_build(CrcTabs& T) {
	for(int i = threadIdx.x; i < 256; i += blockDim.x) {
		uint32_t c = i;
		for(int k = 0; k < 8; k++) c = (c >> 1) ^ (0xEDB88320u & (0u - (c & 1)));
		T.t[0][i] = c;
	}
	__syncthreads();
	for(int i = threadIdx.x; i < 256; i += blockDim.x) {
		uint32_t c = T.t[0][i];
		for(int j = 1; j < 4; j++) { c = (c >> 8) ^ T.t[0][c & 255]; T.t[j][i] = c; }
	}
	__syncthreads();
}

__device__ __forceinline__ uint32_t crc_word(const CrcTabs& T, uint32_t crc, uint32_t w) {
	crc ^= w;
	return T.t[3][crc & 255] ^ T.t[2][(crc >> 8) & 255] ^ T.t[1][(crc >> 16) & 255] ^ T.t[0][crc >> 24];
}
__device__ __forceinline__ uint32_t crc_byte(const CrcTabs& T, uint32_t crc, uint32_t b) {
	return (crc >> 8) ^ T.t[0][(crc ^ b) & 255];
}
// a*b mod P, reflected bit order (bit 31 = x^0)
__device__ uint32_t crc_mulmod(uint32_t a, uint32_t b) {
	uint32_t r = 0;
	for(int i = 0; i < 32; i++) {
		r ^= (0u - (b >> 31)) & a;
		b <<= 1;
		a = (a >> 1) ^ (0xEDB88320u & (0u - (a & 1)));
	}
	return r;
}
// raw register after `n` more zero bytes: multiply by x^(8n)
__device__ uint32_t crc_zero_extend(uint32_t reg, uint64_t n) {
	uint32_t xn = 0x00800000u; // x^8
	while(n) {
		if(n & 1) reg = crc_mulmod(reg, xn);
		xn = crc_mulmod(xn, xn);
		n >>= 1;
	}
	return reg;
}

// MD5 finish for a stream whose unprocessed tail (< 64 bytes) is in `tail`
// (little-endian words, bytes beyond tailLen zero) with `zeros` zero bytes
// still to append, then the standard padding (md5_final_block semantics,
// hasher/md5-final.c:4-60).
__device__ void md5_finish(uint32_t st[4], uint32_t tail[16], uint32_t tailLen, uint64_t zeros, uint64_t total) {
	// zero padding: fill the current block, then whole zero blocks
	if(tailLen + zeros >= 64) {
		md5_block(st, tail); // bytes past tailLen are zero already
		zeros -= 64 - tailLen;
		uint32_t z[16];
#pragma unroll
		for(int i = 0; i < 16; i++) z[i] = 0;
		for(uint64_t b = zeros / 64; b; b--) md5_block(st, z);
		zeros %= 64;
#pragma unroll
		for(int i = 0; i < 16; i++) tail[i] = 0;
		tailLen = 0;
	}
	tailLen += (uint32_t)zeros;
	// 0x80 terminator
	tail[tailLen >> 2] |= 0x80u << (8 * (tailLen & 3));
	tailLen++;
	if(tailLen > 56) {
		md5_block(st, tail);
#pragma unroll
		for(int i = 0; i < 16; i++) tail[i] = 0;
	}
	const uint64_t bits = total << 3;
	tail[14] = (uint32_t)bits;
	tail[15] = (uint32_t)(bits >> 32);
	md5_block(st, tail);
}

__device__ __forceinline__ void md5_init(uint32_t st[4]) {
	st[0] = 0x67452301u; st[1] = 0xefcdab89u; st[2] = 0x98badcfeu; st[3] = 0x10325476u;
}

// ---- per-slice MD5 + CRC32 --------------------------------------------------
// Row i holds lens[i] bytes (or sliceBytes), hashed as if zero-padded to
// sliceBytes.  out: 20 bytes per row.
//
// The first blocks run the MD5s, P2C_IFSC_ROWS rows each, one row per thread:
// the kernel's time is that chain's latency.  The CRC is linear, so the other
// blocks compute it beside them, a row per warp: lane l takes the 16 bytes at
// 512 k + 16 l (coalesced 512-byte loads), four registers advance 512 bytes
// per step by table (x^4096), and the lanes' sums are joined by multiplying
// with x^128 per lane.  2000 slices of 256 KiB + 44, every tenth one shorter:
// 4.80 ms with the CRC in the MD5 thread, 3.26 with it in other warps of the
// MD5 blocks (and a branch between data and padding), 2.46 beside them, and
// 1.98 (132 MB/s a chain, of the 170 that the chain's own latency allows) with
// rows' partial blocks out of the loop (2.26) and 16 rows a block, so that two
// MD5 warps seldom share a scheduler (32 rows: 2.13).  10 000 slices of 64 KiB
// 1.01 -> 0.81 ms.
#define P2C_IFSC_ROWS 16
#define P2C_IFSC_THREADS (32 * P2C_IFSC_ROWS / P2C_MD5_LANES)
// tables of c x^4096 for the four bytes of a register
struct CrcStride { uint32_t t[4][256]; };
constexpr uint32_t crc_step_const(uint32_t c) { return (c >> 1) ^ (0xEDB88320u & (0u - (c & 1))); }
constexpr CrcStride crc_stride() {
	CrcStride r{};
	for(int k = 0; k < 4; k++) {
		uint32_t bit[8] = {};
		for(int b = 0; b < 8; b++) {
			uint32_t v = 1u << (8 * k + b);
			for(int i = 0; i < 4096; i++) v = crc_step_const(v);
			bit[b] = v;
		}
		for(int m = 0; m < 256; m++) {
			uint32_t v = 0;
			for(int b = 0; b < 8; b++) if(m >> b & 1) v ^= bit[b];
			r.t[k][m] = v;
		}
	}
	return r;
}
__device__ const CrcStride g_crc_stride = crc_stride();

__device__ __forceinline__ uint32_t crc_stride_mul(const CrcStride& S, uint32_t r) {
	return S.t[0][r & 255] ^ S.t[1][(r >> 8) & 255] ^ S.t[2][(r >> 16) & 255] ^ S.t[3][r >> 24];
}

// the raw CRC register of `len` bytes at the 16-byte aligned p, by one warp
__device__ uint32_t crc_row(const CrcTabs& T, const CrcStride& S, const uint8_t* p, size_t len, int lane) {
	const size_t steps = len / 512;
	const uint4* p4 = reinterpret_cast<const uint4*>(p) + lane;
	uint32_t a[4] = {0, 0, 0, 0};
	auto add = [&](const uint4& v) {
		a[0] = crc_stride_mul(S, a[0]) ^ v.x;
		a[1] = crc_stride_mul(S, a[1]) ^ v.y;
		a[2] = crc_stride_mul(S, a[2]) ^ v.z;
		a[3] = crc_stride_mul(S, a[3]) ^ v.w;
	};
	size_t k = 0;
	for(; k + 4 <= steps; k += 4) {
		uint4 v[4];
#pragma unroll
		for(int u = 0; u < 4; u++) v[u] = __ldg(p4 + (k + u) * 32);
#pragma unroll
		for(int u = 0; u < 4; u++) add(v[u]);
	}
	for(; k < steps; k++) add(__ldg(p4 + k * 32));
	// this lane's 16-byte column, then the lanes: sum over l of u_l x^(128 (31 - l))
	uint32_t u = 0;
#pragma unroll
	for(int q = 0; q < 4; q++) u = crc_word(T, u, a[q]);
	uint32_t r = 0;
	for(int l = 0; l < 32; l++) {
#pragma unroll
		for(int q = 0; q < 4; q++) r = crc_word(T, r, 0);
		r ^= __shfl_sync(0xFFFFFFFFu, u, l);
	}
	r ^= crc_zero_extend(0xFFFFFFFFu, steps * 512);
	for(size_t i = steps * 512; i < len; i++) r = crc_byte(T, r, p[i]);
	return r;
}

__device__ const uint4 g_md5_zero[4] = {};

__global__ void __launch_bounds__(P2C_IFSC_THREADS) k_slice_hash(const uint8_t* rows, size_t pitch, unsigned n, unsigned md5Blocks,
                                                   const uint32_t* lens, size_t sliceBytes, uint8_t* out)
{
	__shared__ CrcTabs T;
	__shared__ CrcStride S;
	const unsigned warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
	if(blockIdx.x >= md5Blocks) {
		for(int i = threadIdx.x; i < 1024; i += blockDim.x) S.t[i >> 8][i & 255] = g_crc_stride.t[i >> 8][i & 255];
		crc_tabs_build(T);
		const unsigned i = (blockIdx.x - md5Blocks) * (P2C_IFSC_THREADS / 32) + warp;
		if(i >= n) return;
		const size_t len = lens ? min((size_t)lens[i], sliceBytes) : sliceBytes;
		const uint32_t reg = crc_row(T, S, rows + (size_t)i * pitch, len, lane);
		if(lane == 0) {
			const uint32_t crc = ~crc_zero_extend(reg, sliceBytes - len);
			uint8_t* o = out + (size_t)i * 20;
			o[16] = (uint8_t)crc; o[17] = (uint8_t)(crc >> 8); o[18] = (uint8_t)(crc >> 16); o[19] = (uint8_t)(crc >> 24);
		}
		return;
	}
	const unsigned i = blockIdx.x * P2C_IFSC_ROWS + warp * P2C_MD5_LANES + lane;
	const uint32_t act = __ballot_sync(0xFFFFFFFFu, lane < P2C_MD5_LANES && i < n);
	if(lane >= P2C_MD5_LANES || i >= n) return;
	const size_t len = lens ? min((size_t)lens[i], sliceBytes) : sliceBytes;
	const uint8_t* p = rows + (size_t)i * pitch;
	const uint4* p4 = reinterpret_cast<const uint4*>(p);
	uint32_t st[4];
	md5_init(st);
	// Every row is sliceBytes / 64 blocks and a remainder, whatever its length:
	// blocks past its bytes are zero, taken in the same loop (from an address
	// of zeros), so that a short row does not make its warp run the padding
	// after the others' data.  A block that a row fills in part is put together
	// when it is used: the loop runs up to the pair of blocks that holds the
	// next one of any of the warp's rows, without a test per block.
	const uint32_t own = (uint32_t)(len / 64), all = (uint32_t)(sliceBytes / 64);
	const uint4* const zero = g_md5_zero;
	auto block = [&](uint32_t k, uint32_t (&m)[16]) {
		const uint4* src = k < own ? p4 + (size_t)k * 4 : zero;
#pragma unroll
		for(int q = 0; q < 4; q++) {
			const uint4 v = __ldg(src + q);
			m[4 * q] = v.x; m[4 * q + 1] = v.y; m[4 * q + 2] = v.z; m[4 * q + 3] = v.w;
		}
	};
	auto cut = [&](uint32_t k, uint32_t (&m)[16]) {
		if(k == own) {
			const uint32_t rem = (uint32_t)(len - (size_t)own * 64);
#pragma unroll
			for(int q = 0; q < 16; q++) {
				if((uint32_t)(4 * q + 4) <= rem) m[q] = __ldg(reinterpret_cast<const uint32_t*>(p4 + (size_t)own * 4) + q);
				else if((uint32_t)(4 * q) < rem)
					for(uint32_t e = 4 * q; e < rem; e++) m[q] |= (uint32_t)p[(size_t)own * 64 + e] << (8 * (e & 3));
			}
		}
	};
	uint32_t A[16], B[16];
	block(0, A);
	block(1, B);
	uint32_t k = 0;
	for(;;) {
		// the next block of which some lane has a part (or the last)
		const uint32_t mine = own >= k && own < all ? own : all;
		const uint32_t stop = __reduce_min_sync(act, mine) & ~1u;
		for(; k < stop; k += 2) {
			if(k + P2C_MD5_L2_AHEAD < own)
				asm volatile("prefetch.global.L2 [%0];" :: "l"(p4 + (size_t)(k + P2C_MD5_L2_AHEAD) * 4));
			{
				const MsgBlock m(A);
				block(k + 2, A);
				md5_block(st, m.w);
			}
			{
				const MsgBlock m(B);
				block(k + 3, B);
				md5_block(st, m.w);
			}
		}
		if(k >= all) break;
		{
			cut(k, A);
			const MsgBlock m(A);
			block(k + 2, A);
			md5_block(st, m.w);
		}
		if(k + 1 < all) {
			cut(k + 1, B);
			const MsgBlock m(B);
			block(k + 3, B);
			md5_block(st, m.w);
		}
		k += 2;
	}
	// the remainder of the slice (in A after an even number of blocks, else in B)
	uint32_t tail[16];
#pragma unroll
	for(int q = 0; q < 16; q++) tail[q] = (all & 1) ? B[q] : A[q];
	cut(all, tail);
	md5_finish(st, tail, (uint32_t)(sliceBytes - (size_t)all * 64), 0, sliceBytes);
	uint8_t* o = out + (size_t)i * 20;
#pragma unroll
	for(int w = 0; w < 4; w++) {
		o[4 * w] = (uint8_t)st[w]; o[4 * w + 1] = (uint8_t)(st[w] >> 8);
		o[4 * w + 2] = (uint8_t)(st[w] >> 16); o[4 * w + 3] = (uint8_t)(st[w] >> 24);
	}
}

// The same with one thread per row for both hashes: for short rows, where the
// CRC blocks' tables and joins cost more than the rows, and for many, where the
// MD5 chains of eight lanes a warp want more issue slots than there are.
__global__ void __launch_bounds__(128) k_slice_hash_rows(const uint8_t* rows, size_t pitch, unsigned n, const uint32_t* lens,
                                                         size_t sliceBytes, uint8_t* out)
{
	__shared__ CrcTabs T;
	crc_tabs_build(T);
	const unsigned i = blockIdx.x * blockDim.x + threadIdx.x;
	if(i >= n) return;
	const size_t len = lens ? min((size_t)lens[i], sliceBytes) : sliceBytes;
	const uint8_t* p = rows + (size_t)i * pitch;
	uint32_t st[4];
	md5_init(st);
	uint32_t crc = 0xFFFFFFFFu;
	const size_t full = len / 64;
	md5_blocks_pairs<true>(st, crc, &T, reinterpret_cast<const uint4*>(p), full);
	uint32_t tail[16];
#pragma unroll
	for(int q = 0; q < 16; q++) tail[q] = 0;
	const uint32_t rem = (uint32_t)(len - full * 64);
	for(uint32_t k = 0; k < rem; k++) {
		const uint32_t byte = p[full * 64 + k];
		tail[k >> 2] |= byte << (8 * (k & 3));
		crc = crc_byte(T, crc, byte);
	}
	md5_finish(st, tail, rem, sliceBytes - len, sliceBytes);
	crc = ~crc_zero_extend(crc, sliceBytes - len);
	uint8_t* o = out + (size_t)i * 20;
#pragma unroll
	for(int w = 0; w < 4; w++) {
		o[4 * w] = (uint8_t)st[w]; o[4 * w + 1] = (uint8_t)(st[w] >> 8);
		o[4 * w + 2] = (uint8_t)(st[w] >> 16); o[4 * w + 3] = (uint8_t)(st[w] >> 24);
	}
	o[16] = (uint8_t)crc; o[17] = (uint8_t)(crc >> 8); o[18] = (uint8_t)(crc >> 16); o[19] = (uint8_t)(crc >> 24);
}

int slice_hash(const void* rows, size_t pitchBytes, unsigned n, const uint32_t* dLens, size_t sliceBytes,
               uint8_t* dOut, cudaStream_t st)
{
	if(!n) return 0;
	if(pitchBytes % 16) { set_error("row pitch must be a multiple of 16 bytes"); return -1; }
	// Rows up to which the split form is the faster one.  The thread form takes
	// the time of one chain up to 16 000 rows; the split form takes less of it,
	// until its CRC blocks take more: a row costs them a fixed part, one per 512
	// bytes and one per byte past those (in the chain's bytes: 680, 42 and 1.3).
	// Times of the thread form over the split form's: 1024 bytes 1.11 at 1000 rows,
	// 0.84 at 2000; 1500 1.15 at 500, 0.83 at 1500; 3000 1.28 at 2000, 0.87 at 3000;
	// 4096 1.07 at 4000, 0.94 at 5000; 6000 1.16 at 3500, 0.95 at 4500; 12000 1.11 at
	// 6000, 0.92 at 7000; 16384 1.08 at 8000, 0.95 at 8200.  From there on the MD5
	// warps are too many: 32 KiB 1.19 at 8000, 0.98 at 10 000.  Below 1 KiB the
	// split form never wins (512 bytes 0.86 to 1.00).
	const size_t most = sliceBytes < 1024 ? 0 :
		std::min<size_t>(1000 * sliceBytes / (680 + 42 * (sliceBytes / 512) + 13 * (sliceBytes % 512) / 10), sliceBytes >= 32768 ? 9000 : 8192);
	// (and rows that are not 16-byte aligned: the thread form reads rows shorter
	// than a block by bytes)
	if(n > most || reinterpret_cast<uintptr_t>(rows) % 16) {
		k_slice_hash_rows<<<(n + 127) / 128, 128, 0, st>>>((const uint8_t*)rows, pitchBytes, n, dLens, sliceBytes, dOut);
		P2C_CUDA_TRY(cudaGetLastError());
		return 0;
	}
	const unsigned md5Blocks = (n + P2C_IFSC_ROWS - 1) / P2C_IFSC_ROWS, per = P2C_IFSC_THREADS / 32;
	k_slice_hash<<<md5Blocks + (n + per - 1) / per, P2C_IFSC_THREADS, 0, st>>>((const uint8_t*)rows, pitchBytes, n, md5Blocks, dLens,
	                                                                          sliceBytes, dOut);
	P2C_CUDA_TRY(cudaGetLastError());
	return 0;
}

// ---- calibration: the MD5 dependency-chain bound ------------------------------
// One MD5 stream on one GPU thread is bound by the latency of its serial
// step chain (3 dependent integer ops per step: the round function, the add
// of a + K + m, the rotate-and-add), not by memory.  This kernel runs that
// chain on register-resident data, one warp on one SM: the bytes/s of one
// lane is the ceiling for the per-file and per-slice hash kernels.  The state
// carries across blocks, so no block's work can be hoisted.
__global__ void __launch_bounds__(32) k_md5_chain(uint32_t* sink, unsigned blocks) {
	uint32_t st[4] = {0x67452301u ^ threadIdx.x, 0xefcdab89u, 0x98badcfeu, 0x10325476u};
	// the same message block every time, held in registers: each step's
	// a + K + m term has nothing to wait for, so the loop runs at the step
	// chain's own latency (LOP3 -> add -> rotate-add)
	uint32_t m[16];
#pragma unroll
	for(int q = 0; q < 16; q++) m[q] = (uint32_t)(q + 1) * 0x9E3779B9u ^ threadIdx.x;
	for(unsigned b = 0; b < blocks; b++) md5_block(st, m);
	if((st[0] ^ st[1] ^ st[2] ^ st[3]) == 0x5EEDF00Du && blocks == 0) sink[threadIdx.x] = st[0];
}

int md5_chain_rate(double* bytesPerSec, cudaStream_t st) {
	const unsigned blocks = 40000;   // ~25 ms at ~100 MB/s
	cudaEvent_t e0, e1;
	P2C_CUDA_TRY(cudaEventCreate(&e0));
	P2C_CUDA_TRY(cudaEventCreate(&e1));
	k_md5_chain<<<1, 32, 0, st>>>(nullptr, blocks / 8); // warm-up
	float best = 0.f;
	for(int rep = 0; rep < 3; rep++) {
		cudaEventRecord(e0, st);
		k_md5_chain<<<1, 32, 0, st>>>(nullptr, blocks);
		cudaEventRecord(e1, st);
		cudaError_t e = cudaEventSynchronize(e1);
		if(e != cudaSuccess) {
			cudaEventDestroy(e0); cudaEventDestroy(e1);
			set_error("md5 chain calibration: %s", cudaGetErrorString(e));
			return -1;
		}
		float ms = 0.f;
		cudaEventElapsedTime(&ms, e0, e1);
		if(rep == 0 || ms < best) best = ms;
	}
	cudaEventDestroy(e0);
	cudaEventDestroy(e1);
	P2C_CUDA_TRY(cudaGetLastError());
	*bytesPerSec = best > 0.f ? 64.0 * blocks / (best * 1e-3) : 0.0;
	return 0;
}

// ---- per-file MD5 -----------------------------------------------------------
// file f = rows first[f] .. first[f]+ceil(len[f]/sliceBytes)-1, each row
// contributing sliceBytes bytes except the last.  One thread per file.  MANY:
// for blocks of many warps, whose chains take turns at the schedulers: loops with
// fewer registers and instructions, an instantiation each for slices of whole
// blocks (WHOLE) and others, whose code is slower in one kernel (1000 files of 256 KiB,
// 64 a block: 2.18 against 2.52 ms; slices of 65 500 bytes 3.43 against 3.78).
template<int MAXT, bool MANY, bool WHOLE>
__global__ void __launch_bounds__(MAXT) k_file_md5(const uint8_t* rows, size_t pitch, unsigned nFiles,
                                                   const uint64_t* fileLen, const uint32_t* firstRow,
                                                   size_t sliceBytes, uint8_t* out)
{
	const unsigned f = blockIdx.x * blockDim.x + threadIdx.x;
	if(f >= nFiles) return;
	const uint64_t total = fileLen[f];
	// rows of whole words at 4-byte boundaries (the pitch is a multiple of 16);
	// any others are read by bytes
	const bool words = sliceBytes % 4 == 0 && reinterpret_cast<uintptr_t>(rows) % 4 == 0;
	uint32_t st[4];
	md5_init(st);
	uint32_t tail[16];
#pragma unroll
	for(int q = 0; q < 16; q++) tail[q] = 0;
	uint32_t tailLen = 0;
	uint64_t done = 0;
	size_t row = firstRow[f];
	while(done < total) {
		const size_t take = (size_t)min((uint64_t)sliceBytes, total - done);
		const uint8_t* p = rows + row * pitch;
		size_t pos = 0;
		if(MANY ? WHOLE : sliceBytes % 64 == 0) {
			// every row starts a block
			const size_t full = take / 64;
			uint32_t none = 0;
			if(MANY) md5_blocks_pairs<false>(st, none, nullptr, reinterpret_cast<const uint4*>(p), full);
			else md5_blocks(st, reinterpret_cast<const uint4*>(p), full);
			pos = full * 64;
		} else if(words && take >= 64) {
			// the words that complete the block the last
			// row began, then blocks from a 4-byte boundary; what is left
			// (whole words but in a file's last row) begins the next block
			const uint32_t* d32 = reinterpret_cast<const uint32_t*>(p);
			if(tailLen) {
				const uint32_t have = tailLen >> 2;
#pragma unroll
				for(uint32_t q = 0; q < 16; q++) if(q >= have) tail[q] = __ldg(d32 + q - have);
				md5_block(st, tail);
				pos = 64 - tailLen;
				tailLen = 0;
#pragma unroll
				for(int q = 0; q < 16; q++) tail[q] = 0;
			}
			const size_t full = (take - pos) / 64;
			if(MANY) md5_blocks32(st, d32 + pos / 4, full);
			else md5_blocks_words(st, d32 + pos / 4, full);
			pos += full * 64;
			const uint32_t left = (uint32_t)(take - pos) / 4;
#pragma unroll
			for(uint32_t q = 0; q < 16; q++) if(q < left) tail[q] = __ldg(d32 + pos / 4 + q);
			tailLen = 4 * left;
			pos += tailLen;
		}
		for(; pos < take; pos++) {
			tail[tailLen >> 2] |= (uint32_t)p[pos] << (8 * (tailLen & 3));
			if(++tailLen == 64) {
				md5_block(st, tail);
#pragma unroll
				for(int q = 0; q < 16; q++) tail[q] = 0;
				tailLen = 0;
			}
		}
		done += take;
		row++;
	}
	md5_finish(st, tail, tailLen, 0, total);
	uint8_t* o = out + (size_t)f * 16;
#pragma unroll
	for(int w = 0; w < 4; w++) {
		o[4 * w] = (uint8_t)st[w]; o[4 * w + 1] = (uint8_t)(st[w] >> 8);
		o[4 * w + 2] = (uint8_t)(st[w] >> 16); o[4 * w + 3] = (uint8_t)(st[w] >> 24);
	}
}

int file_md5(const void* rows, size_t pitchBytes, unsigned nFiles, const uint64_t* dFileLen, const uint32_t* dFirstRow,
             size_t sliceBytes, uint8_t* dOut, cudaStream_t st, unsigned filesPerBlock)
{
	if(!nFiles) return 0;
	if(pitchBytes % 16) { set_error("row pitch must be a multiple of 16 bytes"); return -1; }
	// one thread per file.  filesPerBlock 1 (default): one file per block,
	// spread over SMs (the fastest chains: 144 MB/s).  32: one warp of files
	// per block, ~6 % slower per chain but ceil(nFiles/32) blocks instead of
	// nFiles, each of which keeps a full-register-file CTA of other work off
	// its SM while the chains run.  Up to 512: the files of several jobs on
	// as few SMs as possible (a warp issues one instruction per ~4-cycle
	// dependency step, so a few warps per scheduler do not slow each other).
	if(filesPerBlock == 1) {
		k_file_md5<32, false, false><<<nFiles, 1, 0, st>>>((const uint8_t*)rows, pitchBytes, nFiles, dFileLen, dFirstRow, sliceBytes, dOut);
	} else if(filesPerBlock == 32) {
		k_file_md5<32, false, false><<<(nFiles + 31) / 32, 32, 0, st>>>((const uint8_t*)rows, pitchBytes, nFiles, dFileLen, dFirstRow,
		                                                   sliceBytes, dOut);
	} else {
		if(filesPerBlock % 32 || filesPerBlock > 512) {
			set_error("files per block %u must be 1 or a multiple of 32 up to 512", filesPerBlock);
			return -1;
		}
		const unsigned per = min(filesPerBlock, (nFiles + 31) / 32 * 32);
		(sliceBytes % 64 ? k_file_md5<512, true, false> : k_file_md5<512, true, true>)<<<(nFiles + per - 1) / per, per, 0, st>>>(
			(const uint8_t*)rows, pitchBytes, nFiles, dFileLen, dFirstRow, sliceBytes, dOut);
	}
	P2C_CUDA_TRY(cudaGetLastError());
	return 0;
}

// ---- per-file MD5 with the bytes staged through shared memory --------------
// One thread per file, as above, but the thread does not load its bytes from
// global memory itself: it keeps P2C_STG_NS bulk asynchronous copies
// (cp.async.bulk, the TMA engine) of P2C_STG_CH-byte chunks of its file in
// flight into its own ring of shared memory, each completing on an mbarrier
// of the ring, and hashes from shared memory.  The chain then never waits on
// an L2 miss, whatever else the GPU runs (another job's contraction streaming
// gigabytes through L2 evicted the prefetched lines of the register-loading
// kernel).  Needs sliceBytes % 64 == 0 (chunks never split an MD5 block) and
// 16-byte aligned rows; every wait is bounded (on timeout the error flag is
// set and the chain stops; its digest is then not valid).
#define P2C_STG_CH 1024
#define P2C_STG_NS 3
#define P2C_STG_STRIDE (P2C_STG_CH * P2C_STG_NS + 16)
#define P2C_STG_WAIT (1u << 24)
__device__ unsigned g_hash_error;

__device__ __forceinline__ uint32_t hs_saddr(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }

__device__ __forceinline__ bool hs_wait(uint32_t bar, uint32_t parity) {
	for(unsigned i = 0; i < P2C_STG_WAIT; i++) {
		uint32_t ok;
		asm volatile("{\n\t.reg .pred p;\n\tmbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\tselp.u32 %0, 1, 0, p;\n\t}"
		             : "=r"(ok) : "r"(bar), "r"(parity) : "memory");
		if(ok) return true;
	}
	return false;
}

// NT files per block, LANES of each warp's threads have one.
template<int NT, int LANES>
__global__ void __launch_bounds__(NT * 32 / LANES) k_file_md5_staged(const uint8_t* __restrict__ rows, size_t pitch, unsigned nFiles,
                                                        const uint64_t* __restrict__ fileLen,
                                                        const uint32_t* __restrict__ firstRow, size_t sliceBytes,
                                                        uint8_t* __restrict__ out, const uint32_t* __restrict__ outIndex)
{
	extern __shared__ __align__(128) uint8_t smem[];
	const unsigned t = (threadIdx.x >> 5) * LANES + (threadIdx.x & 31);
	const bool mine = (threadIdx.x & 31) < LANES;
	const unsigned f = blockIdx.x * NT + t;
	uint8_t* ring = smem + (size_t)t * P2C_STG_STRIDE;
	uint64_t* bars = reinterpret_cast<uint64_t*>(smem + (size_t)NT * P2C_STG_STRIDE) + t * P2C_STG_NS;
	const uint32_t ringA = hs_saddr(ring), barA = hs_saddr(bars);
	if(mine) for(int k = 0; k < P2C_STG_NS; k++)
		asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" :: "r"(barA + 8 * k) : "memory");
	asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
	__syncthreads();
	if(!mine || f >= nFiles) return;

	const uint64_t total = fileLen[f];
	const uint8_t* base = rows + (size_t)firstRow[f] * pitch;
	// chunk cursor: row r of the file, byte offset `off` inside it
	size_t issR = 0, issOff = 0;
	uint64_t issLeft = total;          // file bytes from the issue cursor on
	auto issue = [&](int slot) -> uint32_t {
		const uint64_t rowBytes = issLeft + issOff < sliceBytes ? issLeft + issOff : sliceBytes;
		const uint32_t size = (uint32_t)min((uint64_t)P2C_STG_CH, rowBytes - issOff);
		const uint32_t csize = (size + 15u) & ~15u;
		const uint8_t* src = base + issR * pitch + issOff;
		const uint32_t bar = barA + 8 * slot;
		asm volatile("{\n\t.reg .b64 st;\n\tmbarrier.arrive.expect_tx.shared::cta.b64 st, [%0], %1;\n\t}"
		             :: "r"(bar), "r"(csize) : "memory");
		asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];"
		             :: "r"(ringA + slot * P2C_STG_CH), "l"(src), "r"(csize), "r"(bar) : "memory");
		issLeft -= size;
		issOff += size;
		if(issOff == rowBytes) { issR++; issOff = 0; }
		return size;
	};
	uint32_t sizes[P2C_STG_NS];
	uint32_t phase = 0;                // bit k: parity of slot k's next completion
	uint32_t pend = 0;                 // bit k: slot k has a copy in flight
	int inflight = 0;
#pragma unroll
	for(int k = 0; k < P2C_STG_NS; k++) {
		sizes[k] = 0;
		if(issLeft) { sizes[k] = issue(k); inflight++; pend |= 1u << k; }
	}
	uint32_t st[4];
	md5_init(st);
	uint32_t tail[16];
#pragma unroll
	for(int q = 0; q < 16; q++) tail[q] = 0;
	uint32_t tailLen = 0;
	bool ok = true;
	for(int slot = 0; inflight > 0; slot = slot + 1 == P2C_STG_NS ? 0 : slot + 1) {
		if(!hs_wait(barA + 8 * slot, (phase >> slot) & 1u)) { ok = false; break; }
		phase ^= 1u << slot;
		pend &= ~(1u << slot);
		inflight--;
		uint32_t size = 0;
#pragma unroll
		for(int k = 0; k < P2C_STG_NS; k++) if(k == slot) size = sizes[k];
		const uint4* p4 = reinterpret_cast<const uint4*>(ring + slot * P2C_STG_CH);
		const uint32_t full = size / 64;
		uint32_t A[16];
		if(full) {
#pragma unroll
			for(int q = 0; q < 4; q++) { uint4 v = p4[q]; A[4 * q] = v.x; A[4 * q + 1] = v.y; A[4 * q + 2] = v.z; A[4 * q + 3] = v.w; }
		}
		for(uint32_t b = 0; b < full; b++) {
			uint32_t m[16];
#pragma unroll
			for(int q = 0; q < 16; q++) m[q] = A[q];
			if(b + 1 < full) {
#pragma unroll
				for(int q = 0; q < 4; q++) {
					uint4 v = p4[(b + 1) * 4 + q];
					A[4 * q] = v.x; A[4 * q + 1] = v.y; A[4 * q + 2] = v.z; A[4 * q + 3] = v.w;
				}
			}
			md5_block(st, m);
		}
		if(size % 64) {   // only the file's last chunk: its partial block goes to the finish
			const uint8_t* pb = ring + slot * P2C_STG_CH + full * 64;
			for(uint32_t k = 0; k < size % 64; k++) tail[k >> 2] |= (uint32_t)pb[k] << (8 * (k & 3));
			tailLen = size % 64;
		}
		if(issLeft) {
			// order this thread's reads of the slot before the copy that reuses it
			asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
#pragma unroll
			for(int k = 0; k < P2C_STG_NS; k++) if(k == slot) sizes[k] = issue(slot);
			inflight++;
			pend |= 1u << slot;
		}
	}
	if(!ok) {
		atomicExch(&g_hash_error, 1u);
		// let this chain's copies still in flight land before the block exits
		for(int k = 0; k < P2C_STG_NS; k++)
			if(pend >> k & 1u) hs_wait(barA + 8 * k, (phase >> k) & 1u);
		return;
	}
	md5_finish(st, tail, tailLen, 0, total);
	uint8_t* o = out + (size_t)(outIndex ? outIndex[f] : f) * 16;
#pragma unroll
	for(int w = 0; w < 4; w++) {
		o[4 * w] = (uint8_t)st[w]; o[4 * w + 1] = (uint8_t)(st[w] >> 8);
		o[4 * w + 2] = (uint8_t)(st[w] >> 16); o[4 * w + 3] = (uint8_t)(st[w] >> 24);
	}
}

int file_md5_staged(const void* rows, size_t pitchBytes, unsigned nFiles, const uint64_t* dFileLen,
                    const uint32_t* dFirstRow, size_t sliceBytes, uint8_t* dOut, unsigned filesPerBlock, cudaStream_t st,
                    const uint32_t* dOutIndex)
{
	if(!nFiles) return 0;
	if(pitchBytes % 16 || ((uintptr_t)rows & 15)) { set_error("staged file MD5: rows must be 16-byte aligned"); return -1; }
	if(sliceBytes % 64 || !sliceBytes) { set_error("staged file MD5: slice size must be a multiple of 64 bytes"); return -1; }
	if(filesPerBlock != 32 && filesPerBlock != 64) { set_error("staged file MD5: 32 or 64 files per block"); return -1; }
	const size_t smem = (size_t)filesPerBlock * (P2C_STG_STRIDE + 8 * P2C_STG_NS);
	auto launch = [&](auto kernel, unsigned lanes) -> int {
		P2C_CUDA_TRY(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
		kernel<<<(nFiles + filesPerBlock - 1) / filesPerBlock, filesPerBlock * 32 / lanes, smem, st>>>(
			(const uint8_t*)rows, pitchBytes, nFiles, dFileLen, dFirstRow, sliceBytes, dOut, dOutIndex);
		return 0;
	};
	// Four warps an SM, one per scheduler, are the most that do not delay each
	// other: 8 files a warp in blocks of 32 while every block has an SM to itself,
	// else 16 (times of 32 files a warp over those of 8 and of 16: 64 files a block 1.03
	// to 1.00 and 1.07; 32 a block 1.11 and 1.07 up to 4864 files, 0.94 and 1.07 at 5000).
	const int rc = filesPerBlock == 64 ? launch(k_file_md5_staged<64, 16>, 16)
	             : nFiles <= 152 * 32 ? launch(k_file_md5_staged<32, 8>, 8) : launch(k_file_md5_staged<32, 16>, 16);
	if(rc) return rc;
	P2C_CUDA_TRY(cudaGetLastError());
	return 0;
}

int hash_error_take() {
	unsigned v = 0, z = 0;
	if(cudaMemcpyFromSymbol(&v, g_hash_error, sizeof(v)) != cudaSuccess) return -1;
	if(v) cudaMemcpyToSymbol(g_hash_error, &z, sizeof(z));
	return (int)v;
}

// ---- MD5 of equal-length rows (recovery packets; MD5Multi, hasher/hasher.h:33-56)
// row i: prefix[i] (prefixLen bytes, host-assembled packet header) followed by
// dataLen bytes of row data.  One thread per row, LANES of a warp; WHOLE: the
// prefix is whole blocks (or none), so that the rows' blocks are the stream's.
// (An instantiation each: in one kernel the loops of both get slower code,
// 65 536 bytes of 1000 rows 0.53 instead of 0.46 ms.)
template<int LANES, bool WHOLE>
__global__ void __launch_bounds__(32 * 32 / LANES) k_rows_md5(const uint8_t* rows, size_t pitch, unsigned n, size_t dataLen,
                                                 const uint8_t* prefix, unsigned prefixLen, uint8_t* out)
{
	const unsigned lane = threadIdx.x & 31, i = blockIdx.x * 32 + (threadIdx.x >> 5) * LANES + lane;
	if(lane >= LANES || i >= n) return;
	uint32_t st[4];
	md5_init(st);
	uint32_t tail[16];
#pragma unroll
	for(int q = 0; q < 16; q++) tail[q] = 0;
	uint32_t tailLen = 0;
	const uint8_t* pre = prefix ? prefix + (size_t)i * prefixLen : nullptr;
	for(unsigned k = 0; k < prefixLen; k++) {
		tail[tailLen >> 2] |= (uint32_t)pre[k] << (8 * (tailLen & 3));
		if(++tailLen == 64) { md5_block(st, tail); for(int q = 0; q < 16; q++) tail[q] = 0; tailLen = 0; }
	}
	const uint8_t* p = rows + (size_t)i * pitch;
	size_t pos = 0;
	if(WHOLE) {
		md5_blocks_words(st, reinterpret_cast<const uint32_t*>(p), dataLen / 64);
		pos = dataLen / 64 * 64;
	} else if(tailLen % 4 == 0 && dataLen >= 64 - tailLen) {
		// a prefix of whole words (the 36-byte packet header): complete its
		// block with data words, then the data's blocks start 4-byte aligned
		const uint32_t* d32 = reinterpret_cast<const uint32_t*>(p);
		const unsigned need = (64 - tailLen) / 4;
		for(unsigned q = 0; q < need; q++) tail[(tailLen >> 2) + q] = __ldg(d32 + q);
		md5_block(st, tail);
#pragma unroll
		for(int q = 0; q < 16; q++) tail[q] = 0;
		tailLen = 0;
		pos = (size_t)need * 4;
		const size_t full = (dataLen - pos) / 64;
		md5_blocks_words(st, d32 + need, full);
		pos += full * 64;
	}
	for(; pos < dataLen; pos++) {
		tail[tailLen >> 2] |= (uint32_t)p[pos] << (8 * (tailLen & 3));
		if(++tailLen == 64) { md5_block(st, tail); for(int q = 0; q < 16; q++) tail[q] = 0; tailLen = 0; }
	}
	md5_finish(st, tail, tailLen, 0, prefixLen + dataLen);
	uint8_t* o = out + (size_t)i * 16;
#pragma unroll
	for(int w = 0; w < 4; w++) {
		o[4 * w] = (uint8_t)st[w]; o[4 * w + 1] = (uint8_t)(st[w] >> 8);
		o[4 * w + 2] = (uint8_t)(st[w] >> 16); o[4 * w + 3] = (uint8_t)(st[w] >> 24);
	}
}

int rows_md5(const void* rows, size_t pitchBytes, unsigned n, size_t dataLen, const uint8_t* dPrefix, unsigned prefixLen,
             uint8_t* dOut, cudaStream_t st)
{
	if(!n) return 0;
	if(pitchBytes % 16) { set_error("row pitch must be a multiple of 16 bytes"); return -1; }
	// 32 rows per block: a chain's latency is what counts, so the rows are
	// spread over the SMs, and a warp has as few chains as leave one warp to a
	// scheduler: two share it at a loss (prefix of 36 bytes, 65 536 bytes a row,
	// times at 8, 16 and 32 lanes: 4864 rows 0.50, 0.52, 0.54 ms; 5000 0.55, 0.52, 0.54;
	// 9728 0.54, 0.51, 0.52; 10 000 0.74, 0.55, 0.53; 32 768 1.61, 1.03, 0.72).
	const unsigned schedulers = 152 * 4;
	auto launch = [&](auto kernel, unsigned lanes) {
		kernel<<<(n + 31) / 32, 32 * 32 / lanes, 0, st>>>((const uint8_t*)rows, pitchBytes, n, dataLen, dPrefix, prefixLen, dOut);
	};
	const bool whole = prefixLen % 64 == 0;
	if(n <= 8 * schedulers) launch(whole ? k_rows_md5<8, true> : k_rows_md5<8, false>, 8);
	else if(n <= 16 * schedulers) launch(whole ? k_rows_md5<16, true> : k_rows_md5<16, false>, 16);
	else launch(whole ? k_rows_md5<32, true> : k_rows_md5<32, false>, 32);
	P2C_CUDA_TRY(cudaGetLastError());
	return 0;
}

} // namespace p2c
