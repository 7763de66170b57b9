// Row preparation kernels: zero padding, the internal GF checksum (compute on
// inputs, verify on outputs), PAR2 coefficient expansion into the
// combination-table index layout, and the seeded synthetic data generator.
//
// Checksum (same value as the reference's generic 8-byte checksum,
// gf16/gf16_checksum_generic.h:25-130 + gf16/gf16_cksum_base.h:32-60):
//   four 16-bit lanes; over the row's 8-byte blocks b = 0..nb-1 (data
//   zero-padded to Sp bytes), ck = sum_b 2^(nb-1-b) * block_b per lane
//   (Horner: ck = 2*ck ^ block).  The product is linear, so the recovery row's
//   carried checksum equals the checksum of its data iff nothing was corrupted.
#include "common.cuh"
#include "kernels.h"

namespace p2c {

// ---- per-row partial checksum + zero tail ----------------------------------
// grid: (rows, splits); each lane owns laneBytes (a multiple of 128) contiguous
// bytes of the row, folds their checksum, pre-multiplied by 2^(blocks after
// them), and the CTA's XOR goes into ckAcc[row] with one 64-bit atomic.  Bytes
// at or beyond lens[row] count as zero and, when zeroTail is set, are written as
// zero (each 16-byte unit is loaded by exactly one lane, so there is no race).
//
// Bound: memory.  The Horner chain wants a lane's bytes in order, but a warp
// that reads them so touches 32 lines per load, and the L1 takes one line per
// clock: 2.1 to 3.2 TB/s.  So the warp reads whole 128-byte lines, eight lanes
// to a line and four lines per load, and hands each lane its own line through
// shared memory (units rotated by the owner, so both sides are free of bank
// conflicts).  A lane's value is joined by one product with a power of 2 in
// shifts and XORs: four log and antilog look-ups are eight gathers of 32 lines.
// 2000 x 2 MiB: 1.05 -> 0.64 ms (6.55 TB/s); 300 x 1 MiB 0.097 -> 0.062;
// 2 x 100 MiB 0.101 -> 0.046; 4000 x 20 000 bytes 0.037 -> 0.033.
// Rows of up to 8 KiB have CTAs of one warp: the other warps would find little to
// do and hold registers that more rows could use (32768 x 4 KiB 0.268 -> 0.066 ms,
// 32768 x 64 bytes 0.113 -> 0.059).
constexpr unsigned CK_THREADS = 128, CK_CTAS = 5; // CTAs per SM: at 8 (64 registers) the eight loads spill, 5.87 TB/s
template<unsigned THREADS>
__global__ void __launch_bounds__(THREADS, CK_CTAS * CK_THREADS / THREADS) k_rows_cksum_partial(
	uint16_t* rows, size_t pitchWords, const uint32_t* lens, uint32_t fixedLen,
	size_t sliceBytes, unsigned laneBytes, unsigned long long* ckAcc, int zeroTail, GfTables gt)
{
	__shared__ uint4 stage[THREADS * 8];
	const unsigned row = blockIdx.x, lane = threadIdx.x & 31;
	const size_t Sp = round_up_dev(sliceBytes, 8);
	const size_t end = round_up_dev(Sp, 16);
	const size_t len = min((size_t)(lens ? lens[row] : fixedLen), Sp);
	uint8_t* base = reinterpret_cast<uint8_t*>(rows + (size_t)row * pitchWords);
	uint4* w = stage + (threadIdx.x & ~31u) * 8;
	const size_t warp0 = ((size_t)blockIdx.y * THREADS + (threadIdx.x & ~31u)) * laneBytes;
	const size_t load0 = warp0 + (size_t)(lane >> 3) * laneBytes + (lane & 7) * 16;

	uint32_t hLo = 0, hHi = 0; // lanes 0-1 and 2-3 of the running Horner value
	if(warp0 < end) {
		for(unsigned s = 0; s < laneBytes; s += 128) {
			uint4 v[8];
#pragma unroll
			for(int j = 0; j < 8; j++) {
				const size_t at = load0 + (size_t)(4 * j) * laneBytes + s;
				v[j] = make_uint4(0, 0, 0, 0);
				if(at < len) v[j] = *reinterpret_cast<const uint4*>(base + at);
			}
#pragma unroll
			for(int j = 0; j < 8; j++) {
				const size_t at = load0 + (size_t)(4 * j) * laneBytes + s;
				if(at + 16 > len) {
					if(at < len) { // mask bytes >= len to zero
						uint32_t* q = reinterpret_cast<uint32_t*>(&v[j]);
						const unsigned left = (unsigned)(len - at);
#pragma unroll
						for(unsigned k = 0; k < 4; k++)
							q[k] &= left >= 4 * k + 4 ? 0xFFFFFFFFu : left > 4 * k ? 0xFFFFFFFFu >> (8 * (4 * k + 4 - left)) : 0u;
					}
					if(zeroTail && at < end) *reinterpret_cast<uint4*>(base + at) = v[j];
				}
				const unsigned owner = 4 * j + (lane >> 3);
				w[owner * 8 + ((lane ^ owner) & 7)] = v[j];
			}
			__syncwarp();
#pragma unroll
			for(int k = 0; k < 8; k++) {
				const uint4 a = w[lane * 8 + ((k ^ lane) & 7)];
				hLo = mul2x2(hLo) ^ a.x;
				hHi = mul2x2(hHi) ^ a.y;
				hLo = mul2x2(hLo) ^ a.z;
				hHi = mul2x2(hHi) ^ a.w;
			}
			__syncwarp();
		}
	}
	uint64_t h = 0;
	if(hLo | hHi) {
		// blocks from the lane's last one to the row's: negative where the lane's
		// bytes pass the row's end (they were zero), and 2 has order 65535
		const long long after = (long long)(Sp / 8) - (long long)((warp0 + (size_t)(lane + 1) * laneBytes) / 8);
		const long long e = after % 65535;
		const uint32_t c = gt.exp[e < 0 ? e + 65535 : e];
		uint32_t pLo = 0, pHi = 0;
#pragma unroll
		for(int b = 15; b >= 0; b--) {
			const uint32_t m = 0u - ((c >> b) & 1u);
			pLo = mul2x2(pLo) ^ (hLo & m);
			pHi = mul2x2(pHi) ^ (hHi & m);
		}
		h = ((uint64_t)pHi << 32) | pLo;
	}
	// CTA-wide XOR reduction
#pragma unroll
	for(int off = 16; off; off >>= 1) h ^= __shfl_xor_sync(0xFFFFFFFFu, h, off);
	__shared__ uint64_t red[32];
	if((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = h;
	__syncthreads();
	if(threadIdx.x < 32) {
		h = threadIdx.x < (blockDim.x >> 5) ? red[threadIdx.x] : 0;
#pragma unroll
		for(int off = 16; off; off >>= 1) h ^= __shfl_xor_sync(0xFFFFFFFFu, h, off);
		if(threadIdx.x == 0 && h) atomicXor(ckAcc + row, (unsigned long long)h);
	}
}

// writes the accumulated checksum into the row's checksum block and zeroes the
// pitch padding after it; or (verify) compares it with the carried block
__global__ void k_rows_cksum_finish(uint16_t* rows, size_t pitchWords, unsigned nRows, size_t sliceBytes,
                                    const unsigned long long* ckAcc, int verify, uint8_t* flags)
{
	const unsigned row = blockIdx.x;
	if(row >= nRows) return;
	const size_t Sp = round_up_dev(sliceBytes, 8);
	uint16_t* r = rows + (size_t)row * pitchWords;
	const size_t ckWord = Sp / 2;
	if(verify) {
		if(threadIdx.x == 0) {
			uint64_t carried = 0;
			for(int l = 0; l < 4; l++) carried |= (uint64_t)r[ckWord + l] << (16 * l);
			flags[row] = carried == ckAcc[row] ? 1 : 0;
		}
		return;
	}
	for(size_t w = ckWord + threadIdx.x; w < pitchWords; w += blockDim.x) {
		uint16_t v = 0;
		if(w < ckWord + 4) v = (uint16_t)(ckAcc[row] >> (16 * (w - ckWord)));
		r[w] = v;
	}
}

int rows_cksum(uint16_t* rows, size_t pitchWords, unsigned nRows, const uint32_t* dLens, size_t sliceBytes,
               unsigned long long* dCkAcc, int verify, uint8_t* dFlags, const GfTables& gt, cudaStream_t st)
{
	if(!nRows) return 0;
	P2C_CUDA_TRY(cudaMemsetAsync(dCkAcc, 0, sizeof(unsigned long long) * nRows, st));
	const size_t Sp = round_up(sliceBytes, 8);
	// bytes per lane: the more, the fewer joins (512 against 256: 5.6 and 4.9 TB/s
	// at 2000 x 2 MiB; 1024 gives no more there and less at 200 rows), but a few
	// rows have to fill the chip: two CTAs for each that it holds (six: 3.4
	// against 4.4 TB/s at 300 x 1 MiB), and a row its CTA
	const bool warp = Sp <= 32 * 256;
	const unsigned threads = warp ? 32 : CK_THREADS;
	const size_t fill = std::min((size_t)nRows * Sp / (152 * 2 * CK_CTAS * CK_THREADS), round_up((Sp + threads - 1) / threads, 128));
	// (and no more CTAs to a row than a grid's second axis holds)
	const size_t least = Sp / (65535ull * CK_THREADS) / 128 * 128 + 128;
	const unsigned laneBytes = (unsigned)std::max(least, std::min<size_t>(512, std::max<size_t>(128, fill / 128 * 128)));
	const size_t ctaBytes = (size_t)threads * laneBytes;
	dim3 grid(nRows, (unsigned)std::max<size_t>(1, (Sp + ctaBytes - 1) / ctaBytes));
	(warp ? k_rows_cksum_partial<32> : k_rows_cksum_partial<CK_THREADS>)<<<grid, threads, 0, st>>>(
		rows, pitchWords, dLens, (uint32_t)sliceBytes, sliceBytes, laneBytes, dCkAcc, verify ? 0 : 1, gt);
	P2C_CUDA_TRY(cudaGetLastError());
	k_rows_cksum_finish<<<nRows, 64, 0, st>>>(rows, pitchWords, nRows, sliceBytes, dCkAcc, verify, dFlags);
	P2C_CUDA_TRY(cudaGetLastError());
	return 0;
}

// ---- coefficient expansion ---------------------------------------------------
// For recovery row r and input group g (inputs 8g..8g+7) writes 16 index bytes:
// byte k = sum_t bit_k(c(r, 8g+t)) << t.  Coefficients come either from PAR2
// logs (c = 2^(log_i * e_r mod 65535), gf16/gfmat_coeff.c:60-77) or from an
// explicit [input][R] matrix (addInput with coefficients).
__global__ void k_make_idx(const uint16_t* inLogs, const uint16_t* custom, const uint16_t* outExp,
                           unsigned R, unsigned nIn, unsigned G, uint4* idx, uint16_t* coeffOut, GfTables gt)
{
	const size_t id = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
	if(id >= (size_t)R * G) return;
	const unsigned r = (unsigned)(id / G), g = (unsigned)(id % G);
	uint32_t q[4] = {0, 0, 0, 0};
#pragma unroll
	for(int t = 0; t < 8; t++) {
		unsigned i = g * 8 + t;
		uint32_t c = 0;
		if(i < nIn) {
			if(custom) c = custom[(size_t)i * R + r];
			else c = gt.exp[((uint32_t)inLogs[i] * outExp[r]) % 65535u];
			if(coeffOut) coeffOut[(size_t)r * nIn + i] = (uint16_t)c;
		}
#pragma unroll
		for(int k = 0; k < 16; k++) q[k >> 2] |= ((c >> k) & 1u) << (8 * (k & 3) + t);
	}
	idx[(size_t)r * G + g] = make_uint4(q[0], q[1], q[2], q[3]);
}

int make_idx(const uint16_t* dInLogs, const uint16_t* dCustom, const uint16_t* dOutExp, unsigned R, unsigned nIn,
             uint4* dIdx, uint16_t* dCoeffOut, const GfTables& gt, cudaStream_t st)
{
	unsigned G = (nIn + 7) / 8;
	size_t n = (size_t)R * G;
	if(!n) return 0;
	k_make_idx<<<(unsigned)((n + 255) / 256), 256, 0, st>>>(dInLogs, dCustom, dOutExp, R, nIn, G, dIdx, dCoeffOut, gt);
	P2C_CUDA_TRY(cudaGetLastError());
	return 0;
}

// PAR2 coefficients straight from input numbers and exponents -> index layout
// (no host coefficient matrix: c = 2^(log(num_i) * e_r mod 65535))
__global__ void k_par2_idx(const uint16_t* nums, const uint16_t* outExp, unsigned R, unsigned nIn, unsigned G, uint4* idx,
                           GfTables gt)
{
	const size_t id = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
	if(id >= (size_t)R * G) return;
	const unsigned r = (unsigned)(id / G), g = (unsigned)(id % G);
	const uint32_t e = outExp[r];
	uint32_t q[4] = {0, 0, 0, 0};
#pragma unroll
	for(int t = 0; t < 8; t++) {
		unsigned i = g * 8 + t;
		uint32_t c = i < nIn ? gt.exp[((uint32_t)gt.inLog[nums[i] & 32767] * e) % 65535u] : 0;
#pragma unroll
		for(int k = 0; k < 16; k++) q[k >> 2] |= ((c >> k) & 1u) << (8 * (k & 3) + t);
	}
	idx[(size_t)r * G + g] = make_uint4(q[0], q[1], q[2], q[3]);
}

int par2_idx(const uint16_t* dNums, const uint16_t* dExp, unsigned R, unsigned nIn, uint4* dIdx, const GfTables& gt,
             cudaStream_t st)
{
	unsigned G = (nIn + 7) / 8;
	size_t n = (size_t)R * G;
	if(!n) return 0;
	k_par2_idx<<<(unsigned)((n + 255) / 256), 256, 0, st>>>(dNums, dExp, R, nIn, G, dIdx, gt);
	P2C_CUDA_TRY(cudaGetLastError());
	return 0;
}

// the PAR2 coefficient matrix [R][nIn] itself, from input numbers and
// exponents (for the methods that read coefficients rather than index bytes)
__global__ void k_par2_coeffs(const uint16_t* nums, const uint16_t* outExp, unsigned R, unsigned nIn, uint16_t* coeff,
                              GfTables gt)
{
	const size_t id = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
	if(id >= (size_t)R * nIn) return;
	const unsigned r = (unsigned)(id / nIn), i = (unsigned)(id % nIn);
	coeff[id] = gt.exp[((uint32_t)gt.inLog[nums[i] & 32767] * outExp[r]) % 65535u];
}

int par2_coeffs(const uint16_t* dNums, const uint16_t* dExp, unsigned R, unsigned nIn, uint16_t* dCoeff,
                const GfTables& gt, cudaStream_t st)
{
	const size_t n = (size_t)R * nIn;
	if(!n) return 0;
	k_par2_coeffs<<<(unsigned)((n + 255) / 256), 256, 0, st>>>(dNums, dExp, R, nIn, dCoeff, gt);
	P2C_CUDA_TRY(cudaGetLastError());
	return 0;
}

// coefficient matrix [R][nIn] -> index layout (used by the device-level entry point)
__global__ void k_coeff_to_idx(const uint16_t* coeff, unsigned R, unsigned nIn, unsigned G, uint4* idx)
{
	const size_t id = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
	if(id >= (size_t)R * G) return;
	const unsigned r = (unsigned)(id / G), g = (unsigned)(id % G);
	uint32_t q[4] = {0, 0, 0, 0};
#pragma unroll
	for(int t = 0; t < 8; t++) {
		unsigned i = g * 8 + t;
		uint32_t c = i < nIn ? coeff[(size_t)r * nIn + i] : 0;
#pragma unroll
		for(int k = 0; k < 16; k++) q[k >> 2] |= ((c >> k) & 1u) << (8 * (k & 3) + t);
	}
	idx[(size_t)r * G + g] = make_uint4(q[0], q[1], q[2], q[3]);
}

int coeff_to_idx(const uint16_t* dCoeff, unsigned R, unsigned nIn, uint4* dIdx, cudaStream_t st)
{
	unsigned G = (nIn + 7) / 8;
	size_t n = (size_t)R * G;
	if(!n) return 0;
	k_coeff_to_idx<<<(unsigned)((n + 255) / 256), 256, 0, st>>>(dCoeff, R, nIn, G, dIdx);
	P2C_CUDA_TRY(cudaGetLastError());
	return 0;
}

// ---- seeded synthetic data (same bytes as parpar_gb300/synth.py) -------------
__device__ __forceinline__ uint64_t splitmix_mix(uint64_t z) {
	z ^= z >> 30; z *= 0xBF58476D1CE4E5B9ull;
	z ^= z >> 27; z *= 0x94D049BB133111EBull;
	return z ^ (z >> 31);
}
// Two 8-byte units per thread, rows on the grid's second axis: a unit's row and
// place from one index cost a 64-bit division each, more than its bytes.  A
// block takes 256 >> shift rows, so that short ones fill it too (32768 rows of 64
// bytes 21 -> 7 us).
__global__ void __launch_bounds__(256) k_synth(uint8_t* dst, size_t pitchBytes, unsigned nRows, size_t rowBytes, uint64_t seed,
                                               uint64_t first, uint64_t unitOffset, unsigned shift)
{
	const size_t u = 2 * (((size_t)blockIdx.x << shift) + (threadIdx.x & ((1u << shift) - 1)));
	if(u * 8 >= rowBytes) return;
	const unsigned rows = 256u >> shift;
	for(size_t row = (size_t)blockIdx.y * rows + (threadIdx.x >> shift); row < nRows; row += (size_t)gridDim.y * rows) {
		const uint64_t base = seed * 0xD1342543DE82EF95ull + (first + row) * 0x9E3779B97F4A7C15ull + unitOffset + u;
		const uint64_t z[2] = {splitmix_mix(base), splitmix_mix(base + 1)};
		uint8_t* p = dst + row * pitchBytes + u * 8;
		if(u * 8 + 16 <= rowBytes && (reinterpret_cast<uintptr_t>(p) & 15) == 0) {
			*reinterpret_cast<ulonglong2*>(p) = make_ulonglong2(z[0], z[1]);
			continue;
		}
#pragma unroll
		for(int h = 0; h < 2; h++, p += 8) {
			const size_t at = (u + h) * 8;
			if(at + 8 <= rowBytes && (reinterpret_cast<uintptr_t>(p) & 7) == 0) *reinterpret_cast<uint64_t*>(p) = z[h];
			else
				for(size_t b = 0; b < 8 && at + b < rowBytes; b++) p[b] = (uint8_t)(z[h] >> (8 * b));
		}
	}
}

int synth_fill(void* dst, size_t pitchBytes, unsigned nRows, size_t rowBytes, uint64_t seed, uint64_t first, cudaStream_t st,
               uint64_t byteOffset)
{
	if(byteOffset % 8) { set_error("synthetic window offset must be a multiple of 8"); return -1; }
	if(!rowBytes || !nRows) return 0;
	unsigned shift = 0;
	while(shift < 8 && ((size_t)16 << shift) < rowBytes) shift++;
	const unsigned rows = 256u >> shift;
	const dim3 grid((unsigned)((rowBytes + ((size_t)16 << shift) - 1) >> (4 + shift)), std::min((nRows - 1) / rows + 1, 65535u));
	k_synth<<<grid, 256, 0, st>>>((uint8_t*)dst, pitchBytes, nRows, rowBytes, seed, first, byteOffset / 8, shift);
	P2C_CUDA_TRY(cudaGetLastError());
	return 0;
}

} // namespace p2c
