// The GF(2^16) contraction on the 4-bit tensor cores (tcgen05 kind::mxf4).
//
// Algebra.  GF(2^16) is the degree-4 extension of GF(16) by an element y.  With
// x = sum_b X_b y^b (X_b in GF(16)), the product of two elements is a product of
// two cubic polynomials over GF(16), fixed by its values at 6 points of GF(16)
// and at infinity:
//     c x = sum_{q<7} L_q ( E_q(c) E_q(x) ),    E_q(x) = X(alpha_q) in GF(16)
// with linear maps L_q back into GF(2^16).  Summing over the inputs commutes
// with L_q, so a recovery word is the sum over q of L_q of seven contractions
// over GF(16).  Against the product of 16x16 bit matrices (256 binary
// multiply-accumulates per word multiply-add) the two forms here need
//   form 4:  7 passes x 4x4 bit matrices                        = 112
//   form 1:  7 x 9 passes (each GF(16) product by two levels of
//            Karatsuba over its 4 bits) of single bits          =  63
// binary multiply-accumulates, exact in both cases.  Every pass is a product
//     D_p[w][c] = sum_k A_p[w][k] B_p[c][k]     (0/1 operands)
// and the parity of D_p[w][c], times a constant 16-bit mask of (p, c), is added
// to the recovery word: form 4 has 4 columns per recovery slice and 4 values of
// k per input, form 1 one column and one value of k per input.
//
// Operands.  A and B are e2m1 values, two per byte.  In memory A is compact:
// a 32-bit word holds 32 of its 0/1 values (form 4: 8 inputs x 4 bits of
// E_q(x); form 1: one bit of 32 inputs), and the GEMM expands it 4x in shared
// memory as it goes: the four bit positions of a nibble are masked out as
// e2m1 codes 1, 2, 4 and (shifted) 4, i.e. 0.5, 1, 2 and 2, and B holds 2, 1,
// 0.5 and 0.5 there, so that every product is 0 or 1 and the fp32 sums are
// exact integers (< 2^23).  Block scales are all 1.0.  Compact A is 3.5
// (form 4) or 7.9 (form 1) bytes per input word against 8 for expanded bit
// planes of the 16-bit matrix form, B 56 or 32 bytes per coefficient against 128.
//
// GEMM.  Persistent CTA pairs (cta_group::2, M = 256 words, N up to 240
// columns, K = 96 per MMA): each CTA of a pair stages its 128 words of A and
// half of the columns of B, and the pair's MMAs read B from both.  Measured on
// GB300 with resident operands: 14.5 PFLOP/s for the pair at K = 96, 12.9 for
// one CTA at K = 96 (shared-memory reads at 120 B/clk bound it), 9.7 at K = 64
// either way.  Operands lie in shared memory as 8-row x 16-byte core matrices
// without swizzle, which is also their order in global memory: a stage is one
// contiguous bulk copy (no tensor maps).  Two TMEM accumulators of up to 240
// columns (up to eight narrower ones) take the passes in turn, so that
// reading one out overlaps the next passes' MMAs.
// Every wait is bounded (error flag g_tc4_error, no hang).
#include "common.cuh"
#include "kernels.h"

#include <atomic>

namespace p2c {

#define T4_ROWS 128            // words per CTA tile (a pair takes 256)
#define T4_UNIT_A 6144         // expanded A of one MMA: [3 chunks][128 rows][16 bytes]
#define T4_UNIT_Q 1536         // compact A of one MMA: [3 words][128 rows][4 bytes]
#define T4_SU 5                // MMAs (units of K = 96) per stage
#define T4_MAXS 8              // slots of a ring at most (t4_rings)
#define T4_MAXN 240            // columns per tile: two accumulators + the scale factors fill TMEM
#define T4_NACC 8              // groups of accumulators at most
#define T4_TR 4                // ring of published tile numbers
#define T4_NO_TILE 0xFFFFFFFFu
#define T4_SF_COL 480          // TMEM columns of the scale factors (all 1.0, shared by A and B)
#define T4_WAIT (1u << 20)     // polls of a wait before it gives up: some 6 us each, so a few seconds
#define T4_THREADS 768
#define T4_EG 3                // groups of four expander warps
#define T4_EXP_WARPS (4 * T4_EG)
#define T4_EPI_WARPS 8
#define T4_REGS_LOW 64         // registers a thread after the split: 512 x 64 + 256 x 112 = 768 x 80
#define T4_REGS_EPI 112
#define T4_A_CHUNK_BYTES (1ull << 30)

// mbarriers (the same offsets in both CTAs of a pair; L = the leader's is used)
enum {
	T4B_QFULL = 0,                       // compact A landed (local)
	T4B_QEMPTY = T4B_QFULL + T4_MAXS,      // the expander warps have read it (local)
	T4B_BFULL = T4B_QEMPTY + T4_MAXS,      // B landed (local)
	T4B_READY = T4B_BFULL + T4_MAXS,     // L: A expanded and B landed in both CTAs (4 + 1 arrivals each); by B slot
	T4B_EMPTY = T4B_READY + T4_MAXS,       // the stage's MMAs completed (commit, both CTAs); by B slot
	T4B_TFULL = T4B_EMPTY + T4_MAXS,      // an accumulator holds a finished pass (commit, both CTAs)
	T4B_TEMPTY = T4B_TFULL + T4_NACC,    // L: both CTAs' epilogues have read it (16 arrivals)
	T4B_IDFULL = T4B_TEMPTY + T4_NACC,         // a tile number was published (to both CTAs)
	T4B_IDEMPTY = T4B_IDFULL + T4_TR,    // L: its readers have read it
	T4B_DRAIN = T4B_IDEMPTY + T4_TR,     // L: every MMA completed
	T4B_COUNT = T4B_DRAIN + 1
};
#define T4_RING_BYTES (227 * 1024 - 1024 - T4B_COUNT * 8 - (T4_TR + 2) * 4)   // of the dynamic shared memory
#define T4_SMEM (227 * 1024)
static_assert(2 * T4_MAXN <= T4_SF_COL, "accumulators overlap the scale factors");

__device__ unsigned g_tc4_error;

// ------------------------------------------------------------------ algebra
// GF(2^16) modulo 0x1100B; GF(16) = polynomials in z modulo z^4 + z + 1,
// embedded by z -> W with W^4 = W + 1; the extension element y is x itself.
constexpr uint32_t t4_mul(uint32_t a, uint32_t b) {
	uint32_t r = 0;
	for(int i = 0; i < 16; i++) {
		if(b >> i & 1) r ^= a;
		a <<= 1;
		if(a & 0x10000u) a ^= P2C_POLY;
	}
	return r;
}
constexpr uint32_t t4_pow(uint32_t a, uint32_t e) {
	uint32_t r = 1;
	for(; e; e >>= 1) { if(e & 1) r = t4_mul(r, a); a = t4_mul(a, a); }
	return r;
}
constexpr uint32_t t4_mul16(uint32_t a, uint32_t b) {
	uint32_t r = 0;
	for(int i = 0; i < 4; i++) if(b >> i & 1) r ^= a << i;
	for(int i = 6; i >= 4; i--) if(r >> i & 1) r ^= 0x13u << (i - 4);
	return r;
}
// a root of z^4 + z + 1: a power of the element of order 15
constexpr uint32_t t4_root() {
	uint32_t h = t4_pow(2, 65535 / 15), w = h;
	for(int k = 1; k < 15; k++) {
		if((t4_pow(w, 4) ^ w ^ 1u) == 0) return w;
		w = t4_mul(w, h);
	}
	return 0;
}
constexpr uint32_t T4_W = t4_root();
static_assert(T4_W != 0, "GF(16) not found");
constexpr uint32_t t4_embed(uint32_t v) {
	uint32_t r = 0;
	for(int j = 0; j < 4; j++) if(v >> j & 1) r ^= t4_pow(T4_W, j);
	return r;
}

struct T4Algebra {
	uint32_t ebit[16];         // 7 nibbles E_0..E_6 of x^b
	uint32_t eval[2][256];     // the same of the low / high byte of a word
	uint16_t mask4[7][4];      // what bit j of pass q adds to a recovery word
	uint16_t mask1[63];        // what pass 9q + m adds to a recovery word
	bool ok;
};
constexpr T4Algebra t4_algebra() {
	T4Algebra t{};
	// basis W^a y^b of GF(2^16) over GF(2): coordinates of the powers of x by elimination
	uint32_t row[16] = {}, coord[16] = {};
	for(int i = 0; i < 16; i++) { row[i] = t4_mul(t4_pow(T4_W, i & 3), t4_pow(2, i >> 2)); coord[i] = 1u << i; }
	t.ok = true;
	for(int bit = 0; bit < 16; bit++) {
		int p = -1;
		for(int i = bit; i < 16; i++) if(row[i] >> bit & 1) { p = i; break; }
		if(p < 0) { t.ok = false; return t; }
		uint32_t a = row[p], c = coord[p];
		row[p] = row[bit]; coord[p] = coord[bit];
		row[bit] = a; coord[bit] = c;
		for(int i = 0; i < 16; i++) if(i != bit && (row[i] >> bit & 1)) { row[i] ^= a; coord[i] ^= c; }
	}
	// coord[b]: coordinates of x^b; E of each single bit, then of every byte
	uint32_t* ebit = t.ebit;
	for(int b = 0; b < 16; b++) {
		for(int q = 0; q < 6; q++) {
			uint32_t v = 0;
			for(int j = 3; j >= 0; j--) v = t4_mul16(v, q) ^ (coord[b] >> (4 * j) & 15u);
			ebit[b] |= v << (4 * q);
		}
		ebit[b] |= (coord[b] >> 12 & 15u) << 24;
	}
	for(int h = 0; h < 2; h++)
		for(int v = 0; v < 256; v++)
			for(int b = 0; b < 8; b++) if(v >> b & 1) t.eval[h][v] ^= ebit[8 * h + b];
	// interpolation: Lagrange polynomials of the points 0..5 at y, and the
	// product of (y - point) for the value at infinity
	for(int q = 0; q < 7; q++) {
		uint32_t num = 1, den = 1;
		for(int b = 0; b < 6; b++) {
			if(b == q) continue;
			num = t4_mul(num, 2u ^ t4_embed(b));
			if(q < 6) den = t4_mul(den, t4_embed(q ^ b));
		}
		const uint32_t lam = t4_mul(num, t4_pow(den, 65534));
		for(int j = 0; j < 4; j++) t.mask4[q][j] = (uint16_t)t4_mul(t4_pow(T4_W, j), lam);
		// two levels of Karatsuba over the 4 bits: products of b0, b1, b2, b3,
		// b0+b1, b2+b3, b0+b2, b1+b3, b0+b1+b2+b3; contribution of each as a
		// polynomial in z (bit n = z^n)
		const uint32_t contrib[9] = {0x0F, 0x1E, 0x3C, 0x78, 0x0A, 0x28, 0x0C, 0x18, 0x08};
		for(int m = 0; m < 9; m++) {
			uint32_t v = contrib[m];
			for(int i = 6; i >= 4; i--) if(v >> i & 1) v ^= 0x13u << (i - 4);
			uint32_t w = 0;
			for(int j = 0; j < 4; j++) if(v >> j & 1) w ^= t.mask4[q][j];
			t.mask1[9 * q + m] = (uint16_t)w;
		}
	}
	return t;
}
static constexpr T4Algebra T4_ALG = t4_algebra();
static_assert(T4_ALG.ok, "basis of GF(2^16) over GF(16)");
struct T4Masks { uint16_t m4[7][4]; uint16_t m1[63]; };
constexpr T4Masks t4_masks() {
	T4Masks m{};
	for(int q = 0; q < 7; q++) for(int j = 0; j < 4; j++) m.m4[q][j] = T4_ALG.mask4[q][j];
	for(int p = 0; p < 63; p++) m.m1[p] = T4_ALG.mask1[p];
	return m;
}
struct T4Eval { uint32_t t[2][256]; };
constexpr T4Eval t4_eval() {
	T4Eval e{};
	for(int h = 0; h < 2; h++) for(int v = 0; v < 256; v++) e.t[h][v] = T4_ALG.eval[h][v];
	return e;
}
__constant__ T4Masks c_t4_masks = t4_masks();
__device__ const T4Eval g_t4_eval = t4_eval();

// ------------------------------------------------------------------ operands
// Launches of one call follow each other with programmatic dependent launch:
// a kernel starts while the one before it drains, and waits here until that
// one has completed and its writes are visible.  A grid lets the next one
// start once all its blocks have.
__device__ __forceinline__ void t4_pdl_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
__device__ __forceinline__ void t4_pdl_go() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }

// nibble q of v[t] -> nibble t of Q[q] (8 x 8 nibbles)
__device__ __forceinline__ void t4_nibbles(const uint32_t (&v)[8], uint32_t (&Q)[8]) {
	uint32_t a[2][4];      // nibbles 0-3 (or 4-7) of v[t] low, of v[t + 4] high
#pragma unroll
	for(int t = 0; t < 4; t++) {
		a[0][t] = __byte_perm(v[t], v[t + 4], 0x5410);
		a[1][t] = __byte_perm(v[t], v[t + 4], 0x7632);
	}
#pragma unroll
	for(int h = 0; h < 2; h++) {
#pragma unroll
		for(int b = 0; b < 2; b++) {
			const unsigned sel = b ? 0x7351 : 0x6240;
			const uint32_t c0 = __byte_perm(a[h][0], a[h][2], sel), c1 = __byte_perm(a[h][1], a[h][3], sel);
			Q[4 * h + 2 * b] = (c0 & 0x0F0F0F0Fu) | ((c1 << 4) & 0xF0F0F0F0u);
			Q[4 * h + 2 * b + 1] = ((c0 >> 4) & 0x0F0F0F0Fu) | (c1 & 0xF0F0F0F0u);
		}
	}
}
// bit b of nibble t of x[g] -> bit g of nibble t of T[b] (4 x 4 bits in every nibble)
__device__ __forceinline__ void t4_bits(const uint32_t (&x)[4], uint32_t (&T)[4]) {
	uint32_t y[4];
#pragma unroll
	for(int g = 0; g < 2; g++) {
		y[g] = (x[g] & 0x33333333u) | ((x[g + 2] << 2) & 0xCCCCCCCCu);
		y[g + 2] = ((x[g] >> 2) & 0x33333333u) | (x[g + 2] & 0xCCCCCCCCu);
	}
#pragma unroll
	for(int h = 0; h < 4; h += 2) {
		T[h] = (y[h] & 0x55555555u) | ((y[h + 1] << 1) & 0xAAAAAAAAu);
		T[h + 1] = ((y[h] >> 1) & 0x55555555u) | (y[h + 1] & 0xAAAAAAAAu);
	}
}
// the 9 Karatsuba planes of the 4 bits of a GF(16) value
__device__ __forceinline__ void t4_planes(const uint32_t (&T)[4], uint32_t (&m)[9]) {
	m[0] = T[0]; m[1] = T[1]; m[2] = T[2]; m[3] = T[3];
	m[4] = T[0] ^ T[1]; m[5] = T[2] ^ T[3]; m[6] = T[0] ^ T[2]; m[7] = T[1] ^ T[3];
	m[8] = m[4] ^ m[5];
}

// the 16 bit planes of 32 words (x[i]: a 16-bit word): word 8 g + t at bit 4 t + g
__device__ __forceinline__ void t4_word_planes(const uint32_t (&x)[32], uint32_t (&T)[16]) {
	uint32_t n[4][4];      // [nibble][group of 8 words], word t in nibble t
#pragma unroll
	for(int g = 0; g < 4; g++) {
		uint32_t a[4];
#pragma unroll
		for(int t = 0; t < 4; t++) a[t] = __byte_perm(x[8 * g + t], x[8 * g + t + 4], 0x5410);
#pragma unroll
		for(int b = 0; b < 2; b++) {
			const unsigned sel = b ? 0x7351 : 0x6240;
			const uint32_t c0 = __byte_perm(a[0], a[2], sel), c1 = __byte_perm(a[1], a[3], sel);
			n[2 * b][g] = (c0 & 0x0F0F0F0Fu) | ((c1 << 4) & 0xF0F0F0F0u);
			n[2 * b + 1][g] = ((c0 >> 4) & 0x0F0F0F0Fu) | (c1 & 0xF0F0F0F0u);
		}
	}
#pragma unroll
	for(int j = 0; j < 4; j++) {
		uint32_t t[4];
		t4_bits(n[j], t);
#pragma unroll
		for(int b = 0; b < 4; b++) T[4 * j + b] = t[b];
	}
}
// output bit O of E (of 28) from the bit planes of the words; bit b of V: plane b counts
constexpr uint32_t t4_eval_row(int o) {
	uint32_t v = 0;
	for(int b = 0; b < 16; b++) v |= (T4_ALG.ebit[b] >> o & 1u) << b;
	return v;
}
template<int O> struct T4EvalRow { static constexpr uint32_t V = t4_eval_row(O); };
template<int O> __device__ __forceinline__ uint32_t t4_eval_plane(const uint32_t (&T)[16]) {
	uint32_t v = 0;
#pragma unroll
	for(int b = 0; b < 16; b++) if(T4EvalRow<O>::V >> b & 1) v ^= T[b];
	return v;
}

// Compact A of a chunk: [128-word tile][pass][unit][3 words][128 rows] 32-bit
// words, for rows w0 .. w0 + 128 tiles - 1 (zero past nWords).  Words with no
// input below nIn are not written: B is zero there, and every bit pattern
// expands to finite codes.  Word j of a unit holds, in form 4, E_q of inputs 24 u + 8 j
// + t in nibble t; in form 1, one bit of inputs 96 u + 32 j + 8 g + t in bit
// 4 t + g.  Memory-bound: a thread takes one word of 32 inputs as 16 bit
// planes in registers, where E is XORs of planes (about 10 operations per
// word in all); every store of a warp is 128 contiguous bytes.
#define T4_PREP_THREADS 256
template<int FORM>
__global__ void __launch_bounds__(T4_PREP_THREADS) k_tc4_prep_in(
	const uint16_t* __restrict__ in, size_t inPitch, unsigned nIn, size_t nWords, size_t w0, unsigned items, unsigned groups,
	uint32_t* __restrict__ A, unsigned U, int first)
{
	t4_pdl_go();
	// a later chunk's planes replace those the launch before this one reads
	if(!first) t4_pdl_wait();
	const unsigned it = blockIdx.x * (T4_PREP_THREADS / 128) + (threadIdx.x >> 7);
	if(it >= items) {
		if(first) t4_pdl_wait();
		return;
	}
	const unsigned row = threadIdx.x & 127;
	const unsigned mt = it / groups, grp = it - mt * groups, i0 = 32 * grp;
	const size_t w = w0 + (size_t)mt * T4_ROWS + row;
	uint32_t x[32];
	const uint16_t* src = in + (size_t)i0 * inPitch + w;
	if(i0 + 32 <= nIn && w < nWords) {
#pragma unroll
		for(int t = 0; t < 32; t++) x[t] = __ldg(src + (size_t)t * inPitch);
	} else {
#pragma unroll
		for(int t = 0; t < 32; t++) x[t] = (i0 + t < nIn && w < nWords) ? __ldg(src + (size_t)t * inPitch) : 0u;
	}
	uint32_t T[16];
	t4_word_planes(x, T);
	auto pass_group = [&](int q, const uint32_t (&e)[4]) {
		if(FORM == 4) {
			uint32_t Q[4];
			t4_bits(e, Q);      // back to 8 inputs x 4 bits a word
#pragma unroll
			for(int g = 0; g < 4; g++) {
				const unsigned G = 4 * grp + g;
				if(8 * G < nIn) A[(((size_t)mt * 7 + q) * U * 3 + G) * 128 + row] = Q[g];
			}
		} else {
			uint32_t m[9];
			t4_planes(e, m);
#pragma unroll
			for(int k = 0; k < 9; k++) A[(((size_t)mt * 63 + 9 * q + k) * U * 3 + grp) * 128 + row] = m[k];
		}
	};
	{ const uint32_t e[4] = {t4_eval_plane<0>(T), t4_eval_plane<1>(T), t4_eval_plane<2>(T), t4_eval_plane<3>(T)}; pass_group(0, e); }
	{ const uint32_t e[4] = {t4_eval_plane<4>(T), t4_eval_plane<5>(T), t4_eval_plane<6>(T), t4_eval_plane<7>(T)}; pass_group(1, e); }
	{ const uint32_t e[4] = {t4_eval_plane<8>(T), t4_eval_plane<9>(T), t4_eval_plane<10>(T), t4_eval_plane<11>(T)}; pass_group(2, e); }
	{ const uint32_t e[4] = {t4_eval_plane<12>(T), t4_eval_plane<13>(T), t4_eval_plane<14>(T), t4_eval_plane<15>(T)}; pass_group(3, e); }
	{ const uint32_t e[4] = {t4_eval_plane<16>(T), t4_eval_plane<17>(T), t4_eval_plane<18>(T), t4_eval_plane<19>(T)}; pass_group(4, e); }
	{ const uint32_t e[4] = {t4_eval_plane<20>(T), t4_eval_plane<21>(T), t4_eval_plane<22>(T), t4_eval_plane<23>(T)}; pass_group(5, e); }
	{ const uint32_t e[4] = {t4_eval_plane<24>(T), t4_eval_plane<25>(T), t4_eval_plane<26>(T), t4_eval_plane<27>(T)}; pass_group(6, e); }
	// this grid completes only after the coefficients' launch before it, so
	// that a launch that waits for this one has waited for both
	if(first) t4_pdl_wait();
}

// 32 compact values -> 16 bytes of e2m1 codes: A's (1, 2, 4, 4 = 0.5, 1, 2, 2)
// and B's with the inverse values (4, 2, 1, 1)
__device__ __forceinline__ uint4 t4_codes_a(uint32_t q) {
	return make_uint4(q & 0x11111111u, q & 0x22222222u, q & 0x44444444u, (q >> 1) & 0x44444444u);
}
__device__ __forceinline__ uint4 t4_codes_b(uint32_t q) {
	return make_uint4((q << 2) & 0x44444444u, q & 0x22222222u, (q >> 2) & 0x11111111u, (q >> 3) & 0x11111111u);
}

// B: [column tile][half][pass][unit][3 chunks][BN / 2 columns][16 bytes], zero
// for recovery slices past R and inputs past nIn.  Thread: one recovery slice
// x one word of a unit (form 4: 8 inputs, 4 columns; form 1: 32 inputs).
template<int FORM>
__global__ void __launch_bounds__(256) k_tc4_prep_coeff(const uint16_t* __restrict__ coeff, unsigned R, unsigned nIn,
                                                      unsigned slots, unsigned BN, unsigned U, uint8_t* __restrict__ B,
                                                      unsigned* __restrict__ counter)
{
	t4_pdl_go();
	if(blockIdx.x == 0 && threadIdx.x == 0) *counter = 0u;   // the tile counter starts at 0 for this call
	__shared__ uint32_t tab[512];
	for(unsigned e = threadIdx.x; e < 512; e += 256) tab[e] = g_t4_eval.t[e >> 8][e & 255];
	__syncthreads();
	constexpr int P = FORM == 4 ? 7 : 63, CPR = FORM == 4 ? 4 : 1, NG = FORM == 4 ? 1 : 4;
	const size_t id = (size_t)blockIdx.x * 256 + threadIdx.x;
	const unsigned words = 3 * U;
	if(id >= (size_t)slots * words) return;
	const unsigned r = (unsigned)(id % slots), word = (unsigned)(id / slots);
	const unsigned unit = word / 3, j = word - unit * 3;
	uint32_t Qg[NG][8];
#pragma unroll
	for(int g = 0; g < NG; g++) {
		uint32_t v[8];
#pragma unroll
		for(int t = 0; t < 8; t++) {
			const size_t i = ((size_t)word * NG + g) * 8 + t;
			const uint32_t c = (r < R && i < nIn) ? __ldg(coeff + (size_t)r * nIn + i) : 0u;
			v[t] = tab[c & 255u] ^ tab[256 + (c >> 8)];
		}
		t4_nibbles(v, Qg[g]);
	}
	const unsigned rpt = BN / CPR, nt = r / rpt, col = (r - nt * rpt) * CPR;
	const unsigned half = col / (BN / 2), row = col - half * (BN / 2);
	const size_t passBytes = (size_t)U * BN * 24;
	uint8_t* base = B + ((size_t)nt * 2 + half) * P * passBytes +
	                (((size_t)unit * 3 + j) * (BN / 2) + row) * 16;
#pragma unroll
	for(int q = 0; q < 7; q++) {
		if(FORM == 4) {
			// columns n: bit n of c_q z^b at k-plane b (4x4 bit matrix of c_q)
			uint32_t Pb[4];
			Pb[0] = Qg[0][q];
#pragma unroll
			for(int b = 1; b < 4; b++) {
				const uint32_t top = (Pb[b - 1] >> 3) & 0x11111111u;
				Pb[b] = ((Pb[b - 1] << 1) & 0xEEEEEEEEu) ^ top ^ (top << 1);
			}
#pragma unroll
			for(int n = 0; n < 4; n++) {
				const uint4 c = make_uint4(((Pb[0] >> n) & 0x11111111u) << 2, ((Pb[1] >> n) & 0x11111111u) << 1,
				                           (Pb[2] >> n) & 0x11111111u, (Pb[3] >> n) & 0x11111111u);
				*reinterpret_cast<uint4*>(base + q * passBytes + n * 16) = c;
			}
		} else {
			const uint32_t xq[4] = {Qg[0][q], Qg[NG > 1 ? 1 : 0][q], Qg[NG > 2 ? 2 : 0][q], Qg[NG > 3 ? 3 : 0][q]};
			uint32_t T[4], m[9];
			t4_bits(xq, T);
			t4_planes(T, m);
#pragma unroll
			for(int k = 0; k < 9; k++) *reinterpret_cast<uint4*>(base + (size_t)(9 * q + k) * passBytes) = t4_codes_b(m[k]);
		}
	}
}

// ------------------------------------------------------------------ GEMM
__device__ __forceinline__ uint32_t t4_saddr(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }
// the same shared-memory offset in CTA `rank` of the cluster
__device__ __forceinline__ uint32_t t4_mapa(uint32_t a, uint32_t rank) {
	uint32_t r;
	asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(a), "r"(rank));
	return r;
}
// Memory order.  What a barrier's signals order, by who gives them:
//   T4_CTA   threads and copies of its own CTA (QFULL, QEMPTY, BFULL): CTA
//            scope, the default of arrivals and waits.
//   T4_PAIR  threads of either CTA, or MMAs that read both CTAs' shared memory
//            (READY, EMPTY, IDFULL, IDEMPTY): cluster scope.  An arrival is a
//            release fence and a relaxed arrival, a wait a relaxed wait and an
//            acquire fence, both restricted to shared memory, which is all that
//            these signals guard.
//   T4_TMEM  accumulators of the pair (TFULL, TEMPTY): cluster scope, relaxed;
//            the tcgen05 fences beside arrival and wait order TMEM.
// CTA scope would order nothing between the CTAs.  An unrestricted release or
// acquire at cluster scope waits ~2000 clocks for whatever the SM has in
// flight: 4096 x 4096 x 256 KiB takes 28.5 ms with the restricted fences, 49.6
// without the restriction, 100 x 10 x 1 MiB 0.200 and 0.228.
enum { T4_CTA, T4_PAIR, T4_TMEM };
__device__ __forceinline__ void t4_acquire_pair() {
	asm volatile("fence.acquire.sync_restrict::shared::cluster.cluster;" ::: "memory");
}
template<int BY = T4_CTA>
__device__ __forceinline__ bool t4_try(uint32_t bar, uint32_t parity) {
	uint32_t ok;
	if(BY != T4_CTA)
		asm volatile("{\n\t.reg .pred p;\n\tmbarrier.try_wait.parity.relaxed.cluster.shared::cta.b64 p, [%1], %2;\n\tselp.u32 %0, 1, 0, p;\n\t}"
		             : "=r"(ok) : "r"(bar), "r"(parity) : "memory");
	else
		asm volatile("{\n\t.reg .pred p;\n\tmbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\tselp.u32 %0, 1, 0, p;\n\t}"
		             : "=r"(ok) : "r"(bar), "r"(parity) : "memory");
	return ok != 0;
}
// a look at a barrier of the pair, without waiting; the acquire fence is the caller's
__device__ __forceinline__ uint32_t t4_test_pair(uint32_t bar, uint32_t parity) {
	uint32_t ok;
	asm volatile("{\n\t.reg .pred p;\n\tmbarrier.test_wait.parity.relaxed.cluster.shared::cta.b64 p, [%1], %2;\n\tselp.u32 %0, 1, 0, p;\n\t}"
	             : "=r"(ok) : "r"(bar), "r"(parity) : "memory");
	return ok;
}
__device__ __forceinline__ bool t4_wait(uint32_t bar, uint32_t parity) {
	for(unsigned i = 0; i < T4_WAIT; i++) if(t4_try(bar, parity)) return true;
	atomicExch(&g_tc4_error, 1u);
	return false;
}
// bounded wait that also gives up when another role of the pair has given up
// (flags in both CTAs' shared memory), so that one failed wait ends the pair quickly
template<int BY = T4_CTA>
__device__ __forceinline__ bool t4_wait_ab(uint32_t bar, uint32_t parity, volatile uint32_t* abortFlag) {
	for(unsigned i = 0; i < T4_WAIT; i++) {
		if(t4_try<BY>(bar, parity)) {
			if(BY == T4_PAIR) t4_acquire_pair();
			return true;
		}
		if((i & 1023u) == 1023u && *abortFlag) return false;
	}
	atomicExch(&g_tc4_error, 1u);
	const uint32_t a = t4_saddr(const_cast<uint32_t*>(abortFlag));
	asm volatile("st.shared::cluster.u32 [%0], 1;" :: "r"(t4_mapa(a, 0)) : "memory");
	asm volatile("st.shared::cluster.u32 [%0], 1;" :: "r"(t4_mapa(a, 1)) : "memory");
	return false;
}
__device__ __forceinline__ void t4_arrive(uint32_t bar) {
	asm volatile("{\n\t.reg .b64 st;\n\tmbarrier.arrive.shared::cta.b64 st, [%0];\n\t}" :: "r"(bar) : "memory");
}
// arrive on a barrier of either CTA (shared::cluster address)
__device__ __forceinline__ void t4_arrive_pair(uint32_t bar) {
	asm volatile("fence.release.sync_restrict::shared::cta.cluster;\n\t"
	             "mbarrier.arrive.relaxed.cluster.shared::cluster.b64 _, [%0];" :: "r"(bar) : "memory");
}
__device__ __forceinline__ void t4_cluster_sync() {
	asm volatile("barrier.cluster.arrive.aligned;\n\tbarrier.cluster.wait.aligned;" ::: "memory");
}
__device__ __forceinline__ void t4_expect(uint32_t bar, uint32_t bytes) {
	asm volatile("{\n\t.reg .b64 st;\n\tmbarrier.arrive.expect_tx.shared::cta.b64 st, [%0], %1;\n\t}"
	             :: "r"(bar), "r"(bytes) : "memory");
}
__device__ __forceinline__ void t4_bulk(uint32_t dst, const void* src, uint32_t bytes, uint32_t bar) {
	t4_expect(bar, bytes);
	asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];"
	             :: "r"(dst), "l"(src), "r"(bytes), "r"(bar) : "memory");
}
// K-major operand without swizzle: 8-row x 16-byte core matrices, `lbo` bytes
// between 16-byte steps of K, 128 bytes between 8-row groups
__device__ __forceinline__ uint64_t t4_desc(uint32_t saddr, uint32_t lbo) {
	return (uint64_t)((saddr >> 4) & 0x3FFFu) | ((uint64_t)(lbo >> 4) << 16) | ((uint64_t)(128 >> 4) << 32) | ((uint64_t)1 << 46);
}
// instruction descriptor of the block-scaled kinds: A and B e2m1 (mxf4 code
// 1), K-major, N >> 3, ue8m0 scale factors, M >> 4, scale-factor ids 0, K = 96
__device__ __forceinline__ uint32_t t4_idesc(uint32_t m, uint32_t n) {
	return (1u << 7) | (1u << 10) | ((n >> 3) << 17) | (1u << 23) | ((m >> 4) << 24) | (1u << 31);
}
__device__ __forceinline__ void t4_mma(uint32_t d, uint64_t a, uint64_t b, uint32_t idesc, uint32_t sf, uint32_t acc) {
	asm volatile("{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %5, 0;\n\t"
	             "tcgen05.mma.cta_group::2.kind::mxf4.block_scale.block32 [%0], %1, %2, %3, [%4], [%4], p;\n\t}"
	             :: "r"(d), "l"(a), "l"(b), "r"(idesc), "r"(sf), "r"(acc) : "memory");
}
// true in one thread of a converged warp
__device__ __forceinline__ bool t4_elect() {
	uint32_t r;
	asm volatile("{\n\t.reg .pred p;\n\telect.sync _|p, 0xffffffff;\n\tselp.u32 %0, 1, 0, p;\n\t}" : "=r"(r));
	return r != 0;
}
// arrives on the barrier in both CTAs when the MMAs issued so far have completed
__device__ __forceinline__ void t4_commit(uint32_t bar) {
	asm volatile("tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.multicast::cluster.b64 [%0], %1;"
	             :: "r"(bar), "h"((uint16_t)3) : "memory");
}

// tile t -> (pair tile mt, column tile nt): groups of groupM pair tiles walk
// the column tiles together
__device__ __forceinline__ void t4_tile(unsigned t, unsigned mTiles, unsigned nTiles, unsigned groupM, unsigned& mt,
                                        unsigned& nt) {
	const unsigned grp = t / (groupM * nTiles);
	const unsigned gm = min(groupM, mTiles - grp * groupM);
	const unsigned within = t - grp * groupM * nTiles;
	mt = grp * groupM + within % gm;
	nt = within / gm;
}

__device__ __forceinline__ void t4_fill_sf(uint32_t taddr) {
	asm volatile("tcgen05.st.sync.aligned.32x32b.x32.b32 [%0], "
	             "{%1,%1,%1,%1,%1,%1,%1,%1,%1,%1,%1,%1,%1,%1,%1,%1,%1,%1,%1,%1,%1,%1,%1,%1,%1,%1,%1,%1,%1,%1,%1,%1};"
	             :: "r"(taddr), "r"(0x7F7F7F7Fu) : "memory");
	asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
}
__device__ __forceinline__ void t4_ld16(uint32_t taddr, uint32_t (&v)[16]) {
	asm volatile("tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];"
	             : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]), "=r"(v[7]),
	               "=r"(v[8]), "=r"(v[9]), "=r"(v[10]), "=r"(v[11]), "=r"(v[12]), "=r"(v[13]), "=r"(v[14]), "=r"(v[15])
	             : "r"(taddr));
}
// waits for this thread's tcgen05.ld; the registers pass through it so that
// no use of them can move ahead of the wait
__device__ __forceinline__ void t4_wait_ld(uint32_t (&v)[16]) {
	asm volatile("tcgen05.wait::ld.sync.aligned;"
	             : "+r"(v[0]), "+r"(v[1]), "+r"(v[2]), "+r"(v[3]), "+r"(v[4]), "+r"(v[5]), "+r"(v[6]), "+r"(v[7]),
	               "+r"(v[8]), "+r"(v[9]), "+r"(v[10]), "+r"(v[11]), "+r"(v[12]), "+r"(v[13]), "+r"(v[14]), "+r"(v[15])
	             :: "memory");
}
// parities of two sums (exact integers < 2^23 in fp32) in bits 0 and 16:
// adding 2^23 gives unit ulp, so bit 0 of the encoding is bit 0 of the sum
__device__ __forceinline__ uint32_t t4_parity2(uint32_t a, uint32_t b) {
	return __byte_perm(__float_as_uint(__fadd_rn(__uint_as_float(a), 8388608.0f)),
	                   __float_as_uint(__fadd_rn(__uint_as_float(b), 8388608.0f)), 0x5410) & 0x00010001u;
}

// Persistent GEMM: a pair of CTAs per two SMs.  Roles in each CTA:
//   warp 0  B copies (in the leader also: takes pair tiles from a global
//           counter, so a pair that starts late simply takes fewer, and
//           publishes them to both CTAs)
//   warp 1  leader: issues the pair's MMAs
//   warp 2  compact A copies
//   warp 3  tells the leader that a stage's B has landed in this CTA
//   warps 4-15  expand compact A into e2m1 codes (thread: one word)
//   warps 16-23 read accumulators out (TMEM lane quarter warp % 4, every other
//           16 columns), keep the tile's recovery words in registers over the
//           passes and write them after the last
// Each pair does exactly one counter fetch beyond its last tile (the one that
// ends it), so a launch advances the counter by tiles + pairs.
// UC > 0: passes of UC < T4_SU units, as many whole passes per stage as fit;
// UC = 0: a pass is one or more stages (the last with its remainder).
// Passes accumulate beside each other in groups of PG, signalled as one.
// SPLIT: the passes of a tile of words and columns are those of S tiles, each of
// which adds its passes' share to the recovery words with 32-bit atomics, two words
// at a time.  (An instantiation: with S known only at run time the unsplit calls were
// 1 to 4 % slower.)
template<int FORM, unsigned UC, bool SPLIT>
__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(T4_THREADS, 1) k_tc4_gemm(
	const uint8_t* __restrict__ A, const uint8_t* __restrict__ B, uint16_t* __restrict__ rec, size_t recPitch, unsigned R,
	unsigned U_, unsigned BN, unsigned PG, unsigned rings, unsigned mTiles, unsigned nTiles, unsigned groupM, unsigned S_, size_t w0,
	size_t nWords, int accumulate, unsigned* __restrict__ tileCounter, unsigned tileBase)
{
	constexpr int P = FORM == 4 ? 7 : 63, CPR = FORM == 4 ? 4 : 1;
	constexpr bool SHORT = UC > 0;
	const unsigned U = SHORT ? UC : U_;
	extern __shared__ __align__(1024) uint8_t smem_raw[];
	const uint32_t raw = t4_saddr(smem_raw);
	const uint32_t pad = (1024u - (raw & 1023u)) & 1023u;
	uint8_t* sm = smem_raw + pad;
	const uint32_t sbase = raw + pad;
	const uint32_t barBase = sbase + T4_RING_BYTES / 8 * 8;
	auto bar = [&](int k) -> uint32_t { return barBase + 8u * (uint32_t)k; };
	volatile uint32_t* tileIds = reinterpret_cast<volatile uint32_t*>(sm + (barBase - sbase) + T4B_COUNT * 8);
	uint32_t* tslot = const_cast<uint32_t*>(tileIds) + T4_TR;
	volatile uint32_t* abortFlag = tslot + 1;
	const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
	const unsigned S = SPLIT ? S_ : 1u;
	const unsigned nAll = mTiles * nTiles * S;
	// a tile is a sequence of runs of stages (UC > 0: one run, of whole passes
	// per stage; else one run per pass); all stages of a run but the last
	// have `full` units
	constexpr unsigned pps = SHORT ? T4_SU / (SHORT ? UC : 1) : 1;
	const unsigned units = P * U;
	const unsigned spr = SHORT ? (P + pps - 1) / pps : (U + T4_SU - 1) / T4_SU;
	const unsigned full = SHORT ? pps * U : T4_SU, tail = (SHORT ? units : U) - (spr - 1) * full;
	// the first pass of a split, and the stages of split `part`
	auto pass0 = [&](unsigned part) -> unsigned { return part * P / S; };
	auto stages_of = [&](unsigned part) -> unsigned { return SHORT ? spr : (pass0(part + 1) - pass0(part)) * spr; };
	const uint32_t szA = full * T4_UNIT_A, szB = full * BN * 24, szQ = full * T4_UNIT_Q;
	const uint32_t aBase = sbase;
	const uint32_t nA = rings & 15u, nB = rings >> 4 & 15u, nQ = rings >> 8 & 15u;
	const uint32_t bBase = aBase + nA * szA, qBase = bBase + nB * szB;
	const unsigned nGrp = min((unsigned)T4_NACC, T4_SF_COL / (PG * BN));
	uint32_t rank;
	asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(rank));

	if(threadIdx.x < T4B_COUNT) {
		const int k = threadIdx.x;
		unsigned count = 1;
		if(k >= T4B_QEMPTY && k < T4B_BFULL) count = 4;
		if(k >= T4B_READY && k < T4B_EMPTY) count = 10;
		if(k >= T4B_TEMPTY && k < T4B_IDFULL) count = 2 * T4_EPI_WARPS;
		if(k >= T4B_IDEMPTY && k < T4B_DRAIN) count = 2 * (T4_EPI_WARPS + T4_EXP_WARPS + 3) + 1;
		asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" :: "r"(bar(k)), "r"(count) : "memory");
		*abortFlag = 0u;
		asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
	}
	if(warp == 1) {
		asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;" :: "r"(t4_saddr(tslot)), "r"(512u) : "memory");
		asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
	}
	asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
	__syncthreads();
	asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
	const uint32_t tmem = *tslot;
	if(warp >= 4 && warp < 8) t4_fill_sf(tmem + ((uint32_t)(32 * (warp & 3)) << 16) + T4_SF_COL);
	asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
	__syncthreads();
	t4_cluster_sync();      // both CTAs' barriers and scale factors are set up
	t4_pdl_wait();          // the operands (and what earlier launches did) are in memory
	asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");

	// the leader's barriers, from either CTA
	auto lead = [&](int k) -> uint32_t { return t4_mapa(bar(k), 0); };
	// next tile number of the pair (every role but the scheduler reads them in order)
	auto next_tile = [&](uint32_t j, unsigned& t) -> bool {
		const unsigned slot = j % T4_TR;
		if(!t4_wait_ab<T4_PAIR>(bar(T4B_IDFULL + slot), (j / T4_TR) & 1, abortFlag)) return false;
		t = tileIds[slot];
		return true;
	};

	// registers move from the other warpgroups to the epilogue's (768 threads
	// start with 80 each: 61440 >= 512 x 64 + 256 x 112)
	if(warp < 4 + T4_EXP_WARPS) {
		asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" :: "n"(T4_REGS_LOW));
		const bool el = t4_elect();      // these warps stay together; one thread issues
		if(warp == 0) {
			// B: stage g into slot g % NB.  The leader also takes the tiles:
			// one ahead of the copies, with the next counter fetch under way
			const uint32_t unitBytes = BN * 24;              // this CTA's half
			uint32_t s = 0, ph = 1, g = 0;                   // slot, parity of its previous stage's completion
			unsigned ahead = 0;
			bool ok = true;
			auto publish = [&](uint32_t j) -> bool {
				const unsigned slot = j % T4_TR;
				if(j >= T4_TR && !__all_sync(0xffffffffu, t4_wait_ab<T4_PAIR>(bar(T4B_IDEMPTY + slot), ((j / T4_TR) - 1) & 1, abortFlag))) return false;
				if(el) {
					const uint32_t idAddr = t4_saddr(const_cast<uint32_t*>(tileIds + slot));
					// subtracted here, not where it is fetched: there the warp would
					// wait for the counter's round trip (10 x 1 x 1 MiB 110 -> 104 us)
					ahead -= tileBase;
					if(ahead >= nAll) ahead = T4_NO_TILE;
					// stores that complete on each CTA's barrier (a release at
					// cluster scope would wait ~2000 clocks for the SM's traffic)
#pragma unroll
					for(uint32_t c = 0; c < 2; c++)
						asm volatile("st.async.weak.shared::cluster.mbarrier::complete_tx::bytes.u32 [%0], %1, [%2];"
						             :: "r"(t4_mapa(idAddr, c)), "r"(ahead), "r"(t4_mapa(bar(T4B_IDFULL + slot), c)) : "memory");
					if(ahead != T4_NO_TILE) ahead = atomicAdd(tileCounter, 1u);
				}
				__syncwarp();
				return true;
			};
			if(rank == 0) {
				if(el) ahead = atomicAdd(tileCounter, 1u);
				__syncwarp();
				ok = publish(0);
			}
			for(uint32_t j = 0; ok; j++) {
				unsigned t = T4_NO_TILE;
				if(el) t4_expect(bar(T4B_IDFULL + j % T4_TR), 4);
				if(!__all_sync(0xffffffffu, next_tile(j, t))) break;
				__syncwarp();
				if(el) t4_arrive_pair(lead(T4B_IDEMPTY + j % T4_TR));
				if(t == T4_NO_TILE) break;
				if(rank == 0 && !publish(j + 1)) break;
				unsigned mt, nt;
				t4_tile(t / S, mTiles, nTiles, groupM, mt, nt);
				const uint8_t* src = B + (((size_t)nt * 2 + rank) * units + pass0(t % S) * U) * unitBytes;
				unsigned left = spr;
				for(unsigned e = stages_of(t % S); e; e--, g++) {
					const uint32_t bytes = (left > 1 ? full : tail) * unitBytes;
					if(--left == 0) left = spr;
					if(g >= nB && !__all_sync(0xffffffffu, t4_wait_ab<T4_PAIR>(barBase + 8 * (T4B_EMPTY + s), ph, abortFlag))) { ok = false; break; }
					if(el) t4_bulk(bBase + s * szB, src, bytes, barBase + 8 * (T4B_BFULL + s));
					src += bytes;
					if(++s == nB) { s = 0; ph ^= 1; }
				}
			}
			// the last stages' MMAs have completed (and signalled this CTA)
			// before it ends; after a wait that gave up, at least the copies
			// still in flight land
			const bool gone = *abortFlag != 0;
			for(uint32_t h = g > nB ? g - nB : 0; h < g; h++)
				if(gone || !t4_wait_ab<T4_PAIR>(bar(T4B_EMPTY + h % nB), (h / nB) & 1, abortFlag))
					t4_wait(bar(T4B_BFULL + h % nB), (h / nB) & 1);
		} else if(warp == 1) {
			if(rank == 0) {
				// The warp stays together and one elected thread issues: measured
				// with resident operands, a warp that diverges to one thread pays
				// ~170 clocks for each wait on a barrier that is ready and ~40 for
				// each commit (4 MMAs per wait: 11.9 PFLOP/s), a converged one
				// nothing (14.5).  Ring slots and phases are counted along and the
				// descriptors' constant parts made once.
				const uint32_t idesc = t4_idesc(2 * T4_ROWS, BN);
				const uint32_t sf = tmem + T4_SF_COL;
				const uint64_t aDesc = t4_desc(aBase, 2048), bDesc = t4_desc(bBase, BN * 8);
				const uint32_t bUnit = BN * 24 / 16;             // descriptor address steps
				uint32_t sb = 0, phB = 0, saOff = 0, sbOff = 0;
				uint32_t grp = 0, phT = 1, kg = 0, np = 0;         // accumulator group, parity of its previous read-out, pass in it
				uint32_t dacc = tmem;
				bool ok = true, seen = false;
				// before a pass: its group's accumulators have been read out
				auto begin_pass = [&]() -> bool {
					if(kg) return true;
					if(np < nGrp) { np++; return true; }
					if(!__all_sync(0xffffffffu, t4_wait_ab<T4_TMEM>(barBase + 8 * (T4B_TEMPTY + grp), phT, abortFlag))) return false;
					asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
					return true;
				};
				auto end_pass = [&](bool last) {
					dacc += BN;
					if(++kg < PG && !last) return;
					if(el) t4_commit(barBase + 8 * (T4B_TFULL + grp));
					kg = 0;
					if(++grp == nGrp) { grp = 0; phT ^= 1; }
					dacc = tmem + grp * PG * BN;
				};
				for(uint32_t j = 0; ok; j++) {
					unsigned t = T4_NO_TILE;
					if(!__all_sync(0xffffffffu, next_tile(j, t))) break;
					__syncwarp();
					if(el) t4_arrive_pair(lead(T4B_IDEMPTY + j % T4_TR));
					if(t == T4_NO_TILE) break;
					if constexpr(!SHORT) {
						const unsigned n = pass0(t % S + 1) - pass0(t % S);
						for(unsigned p = 0; p < n && ok; p++) {
							if(!begin_pass()) { ok = false; break; }
							uint32_t acc = 0;
							for(unsigned left = spr; left; left--) {
								if(!__all_sync(0xffffffffu, t4_wait_ab<T4_PAIR>(barBase + 8 * (T4B_READY + sb), phB, abortFlag))) { ok = false; break; }
								asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
								const uint64_t ad = aDesc + saOff, bd = bDesc + sbOff;
								const uint32_t nu = left > 1 ? (uint32_t)T4_SU : tail;
#pragma unroll
								for(uint32_t u = 0; u < T4_SU; u++) {
									if(u < nu && el) t4_mma(dacc, ad + u * (T4_UNIT_A / 16), bd + u * bUnit, idesc, sf, acc);
									acc = 1;
								}
								if(el) t4_commit(barBase + 8 * (T4B_EMPTY + sb));
								saOff = saOff == (nA - 1) * (szA / 16) ? 0 : saOff + szA / 16;
								sbOff += szB / 16;
								if(++sb == nB) { sb = 0; sbOff = 0; phB ^= 1; }
							}
							if(ok) end_pass(p == n - 1);
						}
					} else {
						int p = 0;
						for(unsigned e = spr; e; e--) {
							if(seen) t4_acquire_pair();
							else if(!__all_sync(0xffffffffu, t4_wait_ab<T4_PAIR>(barBase + 8 * (T4B_READY + sb), phB, abortFlag))) { ok = false; break; }
							asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
							const uint64_t ad = aDesc + saOff, bd = bDesc + sbOff;
							const uint32_t empty = barBase + 8 * (T4B_EMPTY + sb);
							saOff = saOff == (nA - 1) * (szA / 16) ? 0 : saOff + szA / 16;
							sbOff += szB / 16;
							if(++sb == nB) { sb = 0; sbOff = 0; phB ^= 1; }
							// a look at the next stage while this one is issued
							const uint32_t peek = t4_test_pair(barBase + 8 * (T4B_READY + sb), phB);
#pragma unroll
							for(uint32_t k = 0; k < pps; k++) {
								if(p < P) {
									if(!begin_pass()) { ok = false; break; }
#pragma unroll
									for(uint32_t u = 0; u < UC; u++)
										if(el) t4_mma(dacc, ad + (k * UC + u) * (T4_UNIT_A / 16), bd + (k * UC + u) * bUnit, idesc, sf, u ? 1u : 0u);
									end_pass(++p == P);
								}
							}
							if(!ok) break;
							if(el) t4_commit(empty);
							seen = __all_sync(0xffffffffu, peek != 0);
						}
					}
				}
				// every MMA this warp issued has completed before TMEM is freed
				if(el)
					asm volatile("tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.b64 [%0];" :: "r"(bar(T4B_DRAIN)) : "memory");
				t4_wait(bar(T4B_DRAIN), 0);
			}
		} else if(warp == 2) {
			// compact A: stage g into slot g % NQ
			uint32_t s = 0, ph = 1, g = 0;
			bool ok = true;
			for(uint32_t j = 0; ok; j++) {
				unsigned t = T4_NO_TILE;
				if(!__all_sync(0xffffffffu, next_tile(j, t))) break;
				__syncwarp();
				if(el) t4_arrive_pair(lead(T4B_IDEMPTY + j % T4_TR));
				if(t == T4_NO_TILE) break;
				unsigned mt, nt;
				t4_tile(t / S, mTiles, nTiles, groupM, mt, nt);
				const uint8_t* src = A + (((size_t)mt * 2 + rank) * units + pass0(t % S) * U) * T4_UNIT_Q;
				unsigned left = spr;
				for(unsigned e = stages_of(t % S); e; e--, g++) {
					const uint32_t bytes = (left > 1 ? full : tail) * T4_UNIT_Q;
					if(--left == 0) left = spr;
					if(g >= nQ && !__all_sync(0xffffffffu, t4_wait_ab(barBase + 8 * (T4B_QEMPTY + s), ph, abortFlag))) { ok = false; break; }
					if(el) t4_bulk(qBase + s * szQ, src, bytes, barBase + 8 * (T4B_QFULL + s));
					src += bytes;
					if(++s == nQ) { s = 0; ph ^= 1; }
				}
			}
			for(uint32_t h = g > nQ ? g - nQ : 0; h < g; h++)
				t4_wait(bar(T4B_QFULL + h % nQ), (h / nQ) & 1);
		} else if(warp == 3) {
			// B is written by copies, which signal their own CTA's barrier: passed
			// on to the leader, who waits for A and B of both CTAs at one barrier
			// (READY).  The expanders arrive there themselves: each thread fences
			// its writes to the async proxy, the warp joins, and one thread
			// arrives for it, ordered across the pair as described at t4_try.
			const uint32_t ready = lead(T4B_READY);
			uint32_t s = 0, ph = 0;
			bool ok = true;
			for(uint32_t j = 0; ok; j++) {
				unsigned t = T4_NO_TILE;
				if(!__all_sync(0xffffffffu, next_tile(j, t))) break;
				__syncwarp();
				if(el) t4_arrive_pair(lead(T4B_IDEMPTY + j % T4_TR));
				if(t == T4_NO_TILE) break;
				for(unsigned e = stages_of(t % S); e; e--) {
					if(!__all_sync(0xffffffffu, t4_wait_ab(barBase + 8 * (T4B_BFULL + s), ph, abortFlag))) { ok = false; break; }
					if(el) t4_arrive_pair(ready + 8 * s);
					if(++s == nB) { s = 0; ph ^= 1; }
				}
			}
		} else if(warp < 4 + T4_EXP_WARPS) {
			// Groups of four warps take the stages in turn (thread: one word);
			// ring slots and phases are counted along.
			const unsigned row = threadIdx.x & 127, grp = (unsigned)(warp - 4) >> 2;
			const uint32_t* qBuf = reinterpret_cast<const uint32_t*>(sm + (qBase - sbase)) + row;
			uint4* aBuf = reinterpret_cast<uint4*>(sm + (aBase - sbase)) + row;
			const uint32_t ready = lead(T4B_READY);
			uint32_t turn = 0;                                   // whose turn the tile's first stage is
			uint32_t qs = grp % T4_MAXS, qph = 0, sa = grp % nA, sb = grp % nB;      // slots of this group's next stage
			uint32_t seq = grp, eb = 0, eph = 0;                 // its place in the CTA's sequence; the stage that used its A slot before
			bool ok = true;
			for(uint32_t j = 0; ok; j++) {
				unsigned t = T4_NO_TILE;
				if(!__all_sync(0xffffffffu, next_tile(j, t))) break;
				__syncwarp();
				if(el) t4_arrive_pair(lead(T4B_IDEMPTY + j % T4_TR));
				if(t == T4_NO_TILE) break;
				uint32_t e = grp >= turn ? grp - turn : grp + T4_EG - turn;
				const uint32_t stages = stages_of(t % S);
				turn = (turn + stages) % T4_EG;
				uint32_t pos = e;                                    // in its run
				for(; e < stages; e += T4_EG) {
					while(pos >= spr) pos -= spr;
					const uint32_t n = pos + 1 == spr ? tail : full;
					pos += T4_EG;
					if(!__all_sync(0xffffffffu, t4_wait_ab(barBase + 8 * (T4B_QFULL + qs), qph, abortFlag))) { ok = false; break; }
					const uint32_t* qp = qBuf + qs * (szQ / 4);
					uint32_t q[3 * T4_SU];
#pragma unroll
					for(int k = 0; k < 3 * T4_SU; k++) if(k < 3 * (int)n) q[k] = qp[k * 128];
					// reads of the slot before the bulk copy that refills it: ordered
					// across the proxies (without the fence a copy overtook them
					// now and then)
					asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
					__syncwarp();
					if(el) t4_arrive(barBase + 8 * (T4B_QEMPTY + qs));
					qs += T4_EG;
					if(qs >= nQ) { qs -= nQ; qph ^= 1; }
					// the MMAs of the slot's previous stage (nA stages before) have
					// completed.  A group waits for every third stage only, so it
					// has not waited for this barrier's phase before: that one had
					// completed when its last wait was over, as the stages complete,
					// and their commits signal, in the order of issue (nB > 3 stages
					// back is before its last one, and nB >= nA keeps this phase
					// the last one completed)
					if(seq >= nA) {
						if(!__all_sync(0xffffffffu, t4_wait_ab<T4_PAIR>(barBase + 8 * (T4B_EMPTY + eb), eph, abortFlag))) { ok = false; break; }
						eb += T4_EG;
						if(eb >= nB) { eb -= nB; eph ^= 1; }
					} else {
						seq += T4_EG;
						if(seq >= nA) eb = seq - nA;
					}
					uint4* ap = aBuf + sa * (szA / 16);
#pragma unroll
					for(int k = 0; k < 3 * T4_SU; k++) if(k < 3 * (int)n) ap[k * 128] = t4_codes_a(q[k]);
					asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
					__syncwarp();
					if(el) t4_arrive_pair(ready + 8 * sb);
					sa += T4_EG;
					if(sa >= nA) sa -= nA;
					sb += T4_EG;
					if(sb >= nB) sb -= nB;
				}
			}
		}
	} else {
		asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;" :: "n"(T4_REGS_EPI));
		const unsigned quarter = warp & 3, half = (unsigned)(warp - 4 - T4_EXP_WARPS) >> 2;
		const uint32_t tq = tmem + ((uint32_t)(32 * quarter) << 16);
		const unsigned rpt = BN / CPR;
		constexpr int CH = T4_MAXN / 16;                 // 16-column chunks, every other one is this warp's
		constexpr int MY = (CH + 1) / 2, PAIRS = 8 / CPR, NV = FORM == 4 ? 4 : 1;
		const bool el = t4_elect();
		const uint32_t tempty = lead(T4B_TEMPTY);
		uint32_t grp = 0, phT = 0;
		bool ok = true;
		for(uint32_t j = 0; ok; j++) {
			unsigned t = T4_NO_TILE;
			if(!__all_sync(0xffffffffu, next_tile(j, t))) break;
			__syncwarp();
			if(el) t4_arrive_pair(lead(T4B_IDEMPTY + j % T4_TR));
			if(t == T4_NO_TILE) break;
			unsigned mt, nt;
			t4_tile(t / S, mTiles, nTiles, groupM, mt, nt);
			uint32_t st[MY][PAIRS];                          // two recovery words each
#pragma unroll
			for(int i = 0; i < MY; i++)
#pragma unroll
				for(int e = 0; e < PAIRS; e++) st[i][e] = 0;
			const int pLast = (int)pass0(t % S + 1);
			for(int p = (int)pass0(t % S); p < pLast;) {
				if(!__all_sync(0xffffffffu, t4_wait_ab<T4_TMEM>(barBase + 8 * (T4B_TFULL + grp), phT, abortFlag))) { ok = false; break; }
				asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
				const int pEnd = min(pLast, p + (int)PG);
				uint32_t col = tq + grp * PG * BN + 16 * half;
				for(; p < pEnd; p++, col += BN) {
					if(16 * half >= BN) continue;
					uint32_t m[CPR];
#pragma unroll
					for(int b = 0; b < CPR; b++) m[b] = FORM == 4 ? c_t4_masks.m4[p][b] : c_t4_masks.m1[p];
					// as many columns in flight as registers allow (form 1 keeps 60
					// words of results, form 4 15): a read-out waits for TMEM once
					// per NV chunks
#pragma unroll
					for(int i = 0; i < MY; i += NV) {
						if(16 * half + 32 * i >= BN) break;
						uint32_t v[NV][16];
#pragma unroll
						for(int h = 0; h < NV; h++)
							if(i + h < MY && 16 * half + 32 * (i + h) < BN) t4_ld16(col + 32 * (i + h), v[h]);
#pragma unroll
						for(int h = 0; h < NV; h++) t4_wait_ld(v[h]);
#pragma unroll
						for(int h = 0; h < NV; h++)
							if(i + h < MY && 16 * half + 32 * (i + h) < BN) {
#pragma unroll
								for(int e = 0; e < PAIRS; e++)
#pragma unroll
									for(int b = 0; b < CPR; b++)
										st[i + h < MY ? i + h : 0][e] ^= t4_parity2(v[h][2 * e * CPR + b], v[h][(2 * e + 1) * CPR + b]) * m[b];
							}
					}
				}
				// this warp's TMEM reads are done: the accumulators may take new passes
				asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
				__syncwarp();
				if(el) t4_arrive_pair(tempty + 8 * grp);
				if(++grp == nGrp) { grp = 0; phT ^= 1; }
			}
			if(!ok) break;
			const size_t w = w0 + ((size_t)mt * 2 + rank) * T4_ROWS + 32 * quarter + lane;
			// recovery slices of this warp's columns that exist
			const unsigned r0 = nt * rpt + half * (16 / CPR), rows = min(R - nt * rpt, rpt);
			uint16_t* d = rec + (size_t)r0 * recPitch + w;
			if constexpr(SPLIT) {
				// an even lane adds its word and the next lane's (whose word is past
				// the row's only if its own is: an even number of words)
#pragma unroll
				for(int i = 0; i < MY; i++) {
					const unsigned rr = (2 * i + half) * (16 / CPR);
					if(rr >= rows) break;
#pragma unroll
					for(int e = 0; e < 2 * PAIRS; e++) {
						if(rr + e < rows) {
							const uint32_t v = st[i][e >> 1] >> (16 * (e & 1)) & 0xFFFFu;
							const uint32_t next = __shfl_down_sync(0xffffffffu, v, 1);
							if((lane & 1) == 0 && w < nWords) atomicXor(reinterpret_cast<uint32_t*>(d + (size_t)e * recPitch), v | next << 16);
						}
					}
					d += (size_t)(2 * 16 / CPR) * recPitch;
				}
			} else if(w < nWords) {
#pragma unroll
				for(int i = 0; i < MY; i++) {
					const unsigned rr = (2 * i + half) * (16 / CPR);
					if(rr >= rows) break;
#pragma unroll
					for(int e = 0; e < 2 * PAIRS; e++) {
						if(rr + e < rows) {
							const uint16_t v = (uint16_t)(st[i][e >> 1] >> (16 * (e & 1)));
							uint16_t* q = d + (size_t)e * recPitch;
							*q = accumulate ? (uint16_t)(*q ^ v) : v;
						}
					}
					d += (size_t)(2 * 16 / CPR) * recPitch;
				}
			}
		}
	}
	__syncwarp();
	if(*abortFlag) __nanosleep(20000);   // signals of the pair's last commits are on their way
	asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
	__syncthreads();
	t4_cluster_sync();      // no CTA leaves while the other may still signal or read it
	asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
	if(warp == 1)
		asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" :: "r"(tmem), "r"(512u) : "memory");
}

// ------------------------------------------------------------------ host
// scratch: [tile counter, 1 KiB] [B] [compact A of a word chunk].  The sizes
// asked of callers are those of plain 4-bit bit planes (128 bytes per
// coefficient of recovery slices padded to 48, 8 bytes per input word of
// inputs padded to 16): form 4 always fits in them, and form 1 is taken only
// where it does.
#define T4_HDR_BYTES 1024
static size_t t4_kbytes(unsigned nIn) { return (size_t)round_up(nIn ? nIn : 1, 16) * 8; }
static size_t t4_bbytes(unsigned R, unsigned nIn) {
	return round_up(round_up(R ? R : 1, 48) * 16 * t4_kbytes(nIn), 1024);
}
size_t tc4_scratch_bytes(unsigned R, unsigned nIn, size_t nWords) {
	const size_t aFull = round_up(nWords ? nWords : 1, T4_ROWS) * t4_kbytes(nIn);
	const size_t aMax = std::max<size_t>(T4_A_CHUNK_BYTES, (size_t)T4_ROWS * t4_kbytes(nIn));
	return T4_HDR_BYTES + t4_bbytes(R, nIn) + round_up(std::min(aFull, aMax), 1024);
}
size_t tc4_scratch_chunked_bytes(unsigned R, unsigned nIn, size_t nWords, size_t aChunkBytes) {
	const size_t aMin = std::max<size_t>(aChunkBytes, (size_t)T4_ROWS * t4_kbytes(nIn));
	return std::min(tc4_scratch_bytes(R, nIn, nWords), T4_HDR_BYTES + t4_bbytes(R, nIn) + round_up(aMin, 1024));
}

static std::atomic<int> g_tc4_shape{0};
int set_tc4_shape(int shape) { return g_tc4_shape.exchange(shape); }
static std::atomic<int> g_tc4_group{0};
int set_tc4_group(int groupM) { return g_tc4_group.exchange(groupM); }
// tile shape: 1 = up to 240 columns per tile, 2 = up to 128
int tc4_shape_for(unsigned kBlocks) {
	(void)kBlocks;
	return g_tc4_shape.load() == 2 ? 2 : 1;
}

struct T4Plan {
	int form;              // 4 or 1
	unsigned P, U;         // passes, K = 96 units per pass
	unsigned BN, nTiles;   // columns per tile, column tiles
	size_t bBytes;         // prepared coefficients
	size_t pairBytes;      // compact A of 256 words
	unsigned chunks;       // chunks of words, one preparation and one GEMM launch each
	unsigned splits;       // tiles that share the passes of one
	unsigned nBig;         // the first nBig hold bigWords, the others restWords, the last what is left
	size_t bigWords, restWords;
	bool fits;             // in the scratch
	double cost;           // modelled clocks of a CTA pair for the whole call
};

// Sizes of the chunks.  A launch takes whole waves of the grid, however few
// tiles the last one has, and as many chunks of one size often end just past a
// wave: 2000 x 200 x 2 MiB, 16 chunks of 3.4 waves cost 64.  Where two sizes,
// one of whole waves and one above it, come to fewer waves for as many chunks,
// they are taken (58 there: 11.39 -> 10.66 ms; 4096 x 4096 x 256 KiB, 125 -> 122
// waves, 28.08 -> 27.63; 4096 x 240 x 256 KiB 3.05 -> 2.77; 1 to 3 % more on either
// side since the pair's signals have cluster scope).
static unsigned t4_chunks(T4Plan& pl, size_t nWords, size_t cw, size_t capPairs, unsigned nPairsSM) {
	const size_t pairWords = 2 * T4_ROWS;
	auto waves = [&](size_t pairs) { return (pairs * pl.nTiles + nPairsSM - 1) / nPairsSM; };
	pl.chunks = pl.nBig = (unsigned)((nWords + cw - 1) / cw);
	pl.bigWords = pl.restWords = cw;
	const size_t lastWords = nWords - (size_t)(pl.chunks - 1) * cw;
	const size_t even = (pl.chunks - 1) * waves((cw + pairWords - 1) / pairWords) + waves((lastWords + pairWords - 1) / pairWords);
	const size_t total = (nWords + pairWords - 1) / pairWords, n = pl.chunks;
	const size_t lo = total / n * pl.nTiles / nPairsSM;      // whole waves of an average chunk
	if(n < 2 || !lo) return (unsigned)even;
	const size_t a = lo * nPairsSM / pl.nTiles, b = std::min((lo + 1) * nPairsSM / pl.nTiles, capPairs);
	if(!a || b <= a) return (unsigned)even;
	const size_t big = a * n >= total ? 0 : (total - a * n + b - a - 1) / (b - a);
	if(big > n) return (unsigned)even;
	const size_t mixed = big * waves(b) + (n - big) * waves(a), spare = big * b + (n - big) * a - total;
	if(mixed >= even || spare >= (big < n ? a : b)) return (unsigned)even;
	pl.nBig = (unsigned)big;
	pl.bigWords = b * pairWords;
	pl.restWords = a * pairWords;
	return (unsigned)mixed;
}

static T4Plan t4_form(int form, unsigned R, unsigned nIn, size_t nWords, size_t cw, size_t scratchBytes, unsigned nPairsSM,
                      bool maySplit) {
	T4Plan pl;
	pl.splits = 1;
	const unsigned cpr = form == 4 ? 4 : 1;
	const unsigned cap = tc4_shape_for(0) == 2 ? 128 : T4_MAXN;
	pl.form = form;
	pl.P = form == 4 ? 7 : 63;
	pl.U = (nIn + (form == 4 ? 23 : 95)) / (form == 4 ? 24 : 96);
	const size_t cols = (size_t)R * cpr;
	const size_t nt = (cols + cap - 1) / cap;
	pl.BN = (unsigned)round_up((cols + nt - 1) / nt, 16);
	pl.nTiles = (unsigned)((cols + pl.BN - 1) / pl.BN);
	pl.bBytes = round_up((size_t)pl.nTiles * pl.P * pl.U * pl.BN * 48, 1024);
	pl.pairBytes = (size_t)2 * pl.P * pl.U * T4_UNIT_Q;
	const size_t fixed = T4_HDR_BYTES + pl.bBytes, needed = (cw + 2 * T4_ROWS - 1) / (2 * T4_ROWS) * pl.pairBytes;
	pl.fits = scratchBytes >= fixed + needed;
	if(!pl.fits) return pl;
	const double waves = t4_chunks(pl, nWords, cw, (scratchBytes - fixed) / pl.pairBytes, nPairsSM);
	// Fitted to GB300 times: a pass costs ~1000 clocks (its signals between
	// the roles), ~100 per stage and the MMAs (0.5 per column, at least 68);
	// a launch takes whole waves of the grid; preparing an input word moves
	// 2 + 3.5 (form 4) or 2 + 7.9 bytes at 6.7 clocks of the grid per byte
	// and pair tile.  Form 1 wins where the passes are long and the columns
	// fill its tiles (ms, form 1 against form 4): 4096 x 4096 x 256 KiB 28.5
	// and 45.2, 2000 x 200 x 2 MiB 10.8 and 12.4, 777 x 133 x 1400012 bytes 3.3 and
	// 2.8, 1000 x 100 x 1 MiB 3.1 and 2.0; before the pair's signals had cluster
	// scope (1 to 3 % more since, on either side) 1000 x 480 x 1 MiB 5.7 and
	// 6.0; form 4 for 1000 x 300 x 1 MiB 5.4 and 3.9, 2000 x 100 x 2 MiB 10.1
	// and 7.2, 500 x 480 x 1 MiB 4.4 and 3.6.
	const double stages = (pl.U + T4_SU - 1) / T4_SU;
	const double pass = 1000 + 100 * stages + pl.U * std::max(0.5 * pl.BN, 68.0);
	const double pairs = (double)((nWords + 2 * T4_ROWS - 1) / (2 * T4_ROWS));
	double best = waves * pl.P;
	// Passes split over tiles that keep idle pairs busy: few words, long passes.
	// Worth the zeroed rows and atomics where a pair is left with two passes at most
	// and they are 13 units or more (times whole over split: 500 x 30 x 4 KiB 2.1,
	// 1000 x 16 x 4 KiB 1.35, 3000 x 60 x 4 KiB 2.25, 3000 x 16 x 256 bytes 2.45; 200 inputs 0.90
	// to 1.18; with two splits 500 to 10 000 x 16 x 16 KiB 0.91 to 1.00).
	const unsigned splits = (unsigned)std::min<double>(pl.P, nPairsSM / (pairs * pl.nTiles));
	if(maySplit && form == 4 && pl.U >= 13 && pl.chunks == 1 && splits >= 4) {
		pl.splits = splits;
		best = (pl.P + splits - 1) / splits;
	}
	pl.cost = best * pass + 6.7 * nIn * (2 + (form == 4 ? 3.5 : 7.9)) * pairs / nPairsSM;
	return pl;
}

// Slots of the three rings (nA | nB << 4 | nQ << 8) for stages of `full`
// units: as many of expanded A (3 to 6, the ring whose refill goes round the
// most roles) as leave B at least as many; six slots of compact A where they
// fit, else three.  A multiple of three, so that a slot always belongs to the
// same expander group (whose waits would otherwise skip phases), and more
// than three slots of B, by which the groups' waits for free slots of A go.
static unsigned t4_rings(unsigned full, unsigned BN) {
	const size_t a = (size_t)full * T4_UNIT_A, b = (size_t)full * BN * 24, q = (size_t)full * T4_UNIT_Q;
	for(unsigned nQ = 6; nQ >= 3; nQ -= 3)
		for(unsigned nA = 6; nA >= 3; nA--) {
			if(nA * a + nQ * q > T4_RING_BYTES) continue;
			const unsigned nB = (unsigned)std::min<size_t>(T4_MAXS, (T4_RING_BYTES - nA * a - nQ * q) / b);
			if(nB > T4_EG && nB >= nA) return nA | nB << 4 | nQ << 8;
		}
	return 0;
}

static size_t t4_min_scratch(unsigned R, unsigned nIn) {
	return T4_HDR_BYTES + t4_bbytes(R, nIn) + (size_t)T4_ROWS * t4_kbytes(nIn);
}

// false: too little scratch.  The number of word chunks is that of expanded
// planes of 8 bytes per word and (padded) input in the given scratch, the
// launch count callers are told; t4_chunks lays them out within that number.
static bool t4_plan(T4Plan& pl, unsigned R, unsigned nIn, size_t nWords, size_t scratchBytes, unsigned nPairsSM,
                    bool maySplit) {
	if(scratchBytes < t4_min_scratch(R, nIn)) return false;
	size_t cw = (scratchBytes - T4_HDR_BYTES - t4_bbytes(R, nIn)) / t4_kbytes(nIn) / T4_ROWS * T4_ROWS;
	cw = std::min(cw, round_up(nWords, T4_ROWS));
	const size_t chunks = (nWords + cw - 1) / cw;
	const size_t even = round_up((nWords + chunks - 1) / chunks, 2 * T4_ROWS);
	if(even <= cw && (nWords + even - 1) / even == chunks) cw = even;
	bool have = false;
	for(int form : {4, 1}) {
		const T4Plan c = t4_form(form, R, nIn, nWords, cw, scratchBytes, nPairsSM, maySplit);
		if(form == 1 && c.U < T4_SU) continue;       // its passes are single stages or more
		if(!c.fits) continue;
		if(!have || c.cost < pl.cost) pl = c;
		have = true;
	}
	return have;
}

// what t4_run makes of a plan: passes per accumulator group (at least two groups
// fit TMEM beside each other), and the rings
static unsigned t4_group_passes(const T4Plan& pl) { return std::max(1u, std::min(pl.P, (T4_SF_COL / pl.BN) / 2)); }
static unsigned t4_stage_units(const T4Plan& pl) { return pl.U < T4_SU ? T4_SU / pl.U * pl.U : T4_SU; }

static int t4_pairs_on_device(unsigned* out) {
	int dev = 0, nSM = 0;
	P2C_CUDA_TRY(cudaGetDevice(&dev));
	P2C_CUDA_TRY(cudaDeviceGetAttribute(&nSM, cudaDevAttrMultiProcessorCount, dev));
	*out = (unsigned)std::max(nSM / 2, 1);
	return 0;
}

int tc4_plan_info(unsigned R, unsigned nIn, size_t nWords, size_t scratchBytes, unsigned nPairsSM, unsigned out[13]) {
	T4Plan pl;
	if(!R || !nWords || !nIn || !nPairsSM || !t4_plan(pl, R, nIn, nWords, scratchBytes, nPairsSM, nWords % 2 == 0)) {
		set_error("tensor method (mxf4): no plan for %u x %u x %zu words in %zu bytes of scratch", nIn, R, nWords, scratchBytes);
		return -1;
	}
	const unsigned rings = t4_rings(t4_stage_units(pl), pl.BN);
	const unsigned v[13] = {(unsigned)pl.form, pl.P, pl.U, pl.BN, pl.nTiles, t4_stage_units(pl), t4_group_passes(pl),
	                        rings & 15u, rings >> 4 & 15u, rings >> 8 & 15u, pl.chunks, pl.nBig, pl.splits};
	std::copy(v, v + 13, out);
	return 0;
}

unsigned tc4_launches(unsigned R, unsigned nIn, size_t nWords, size_t scratchBytes) {
	T4Plan pl;
	if(!R || !nWords || !nIn || !t4_plan(pl, R, nIn, nWords, scratchBytes, 76, true)) return 0;
	return 1 + 2 * pl.chunks;   // coefficients, then per chunk: inputs + GEMM
}

typedef decltype(&k_tc4_gemm<4, 0, false>) T4Gemm;
template<int FORM> static T4Gemm t4_short_gemm(unsigned U) {
	if(FORM != 4) return nullptr;       // form 1 is chosen for long passes only
	return U == 1 ? k_tc4_gemm<4, 1, false> : U == 2 ? k_tc4_gemm<4, 2, false> : U == 3 ? k_tc4_gemm<4, 3, false> : k_tc4_gemm<4, 4, false>;
}

template<int FORM>
static int t4_run(const T4Plan& pl, const uint16_t* in, size_t inPitch, unsigned nIn, const uint16_t* coeff, uint16_t* rec,
                  size_t recPitch, unsigned R, size_t nWords, int accumulate, uint8_t* scratch, unsigned nPairsSM,
                  cudaStream_t st)
{
	constexpr int CPR = FORM == 4 ? 4 : 1;
	// the epilogue's setmaxnreg.inc waits for registers that the other
	// warpgroups gave up: never launched unless the block's own cover the split
	cudaFuncAttributes fa;
	const bool isShort = pl.U < T4_SU;
	T4Gemm gemm = k_tc4_gemm<FORM, 0, false>;
	if(isShort) gemm = t4_short_gemm<FORM>(pl.U);
	if constexpr(FORM == 4) if(pl.splits > 1) gemm = k_tc4_gemm<4, 0, true>;
	P2C_CUDA_TRY(cudaFuncGetAttributes(&fa, gemm));
	if(fa.numRegs * T4_THREADS < (T4_THREADS - 32 * T4_EPI_WARPS) * T4_REGS_LOW + 32 * T4_EPI_WARPS * T4_REGS_EPI) {
		set_error("tensor method (mxf4): %d registers a thread do not cover the kernel's split", fa.numRegs);
		return -1;
	}
	P2C_CUDA_TRY(cudaFuncSetAttribute(gemm, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)T4_SMEM));
	unsigned* counter = reinterpret_cast<unsigned*>(scratch);
	uint8_t* B = scratch + T4_HDR_BYTES;
	uint8_t* A = B + pl.bBytes;
	const unsigned slots = pl.nTiles * (pl.BN / CPR);
	const size_t nB = (size_t)slots * 3 * pl.U;
	if(pl.splits > 1 && !accumulate) P2C_CUDA_TRY(cudaMemset2DAsync(rec, recPitch * 2, 0, nWords * 2, R, st));
	k_tc4_prep_coeff<FORM><<<(unsigned)((nB + 255) / 256), 256, 0, st>>>(coeff, R, nIn, slots, pl.BN, pl.U, B, counter);
	P2C_CUDA_TRY(cudaGetLastError());
	// pair tiles per raster group: a wave of CTA pairs then reads about as
	// many bytes of A as of B
	unsigned groupM = 34;
	if(g_tc4_group.load() > 0) groupM = (unsigned)g_tc4_group.load();
	// each launch advances the tile counter by its tiles + pairs (every pair's
	// last fetch finds no tile)
	const unsigned PG = t4_group_passes(pl), rings = t4_rings(t4_stage_units(pl), pl.BN);
	if(!rings) { set_error("tensor method (mxf4): no stage layout for %u columns", pl.BN); return -1; }
	unsigned base = 0;
	size_t w0 = 0, wEnd;
	for(unsigned chunk = 0; chunk < pl.chunks; chunk++, w0 = wEnd) {
		wEnd = std::min(nWords, w0 + (chunk < pl.nBig ? pl.bigWords : pl.restWords));
		const unsigned mTiles = (unsigned)((wEnd - w0 + 2 * T4_ROWS - 1) / (2 * T4_ROWS));
		const unsigned groups = (nIn + 31) / 32;
		const size_t items = (size_t)mTiles * 2 * groups;
		constexpr unsigned PER = T4_PREP_THREADS / 128;
		cudaLaunchAttribute pdl;
		pdl.id = cudaLaunchAttributeProgrammaticStreamSerialization;
		pdl.val.programmaticStreamSerializationAllowed = 1;
		cudaLaunchConfig_t cfg = {};
		cfg.stream = st;
		cfg.attrs = &pdl;
		cfg.numAttrs = 1;
		cfg.gridDim = dim3((unsigned)((items + PER - 1) / PER));
		cfg.blockDim = dim3(T4_PREP_THREADS);
		P2C_CUDA_TRY(cudaLaunchKernelEx(&cfg, k_tc4_prep_in<FORM>, in, inPitch, nIn, wEnd, w0, (unsigned)items, groups,
		                                reinterpret_cast<uint32_t*>(A), pl.U, (int)(w0 == 0)));
		const unsigned nAll = mTiles * pl.nTiles * pl.splits;
		const unsigned grid = std::min(nAll, nPairsSM);
		cfg.gridDim = dim3(2 * grid);
		cfg.blockDim = dim3(T4_THREADS);
		cfg.dynamicSmemBytes = T4_SMEM;
		P2C_CUDA_TRY(cudaLaunchKernelEx(&cfg, gemm, (const uint8_t*)A, (const uint8_t*)B, rec, recPitch, R, pl.U, pl.BN, PG, rings,
		                                mTiles, pl.nTiles, groupM, pl.splits, w0, wEnd, accumulate, counter, base));
		base += nAll + grid;
	}
	return 0;
}

int tc4_muladd(const uint16_t* in, size_t inPitch, unsigned nIn, const uint16_t* coeff, uint16_t* rec, size_t recPitch,
               unsigned R, size_t nWords, int accumulate, void* scratch, size_t scratchBytes, cudaStream_t st)
{
	if(!R || !nWords) return 0;
	if(!nIn) {
		if(!accumulate) P2C_CUDA_TRY(cudaMemset2DAsync(rec, recPitch * 2, 0, nWords * 2, R, st));
		return 0;
	}
	if(nIn >= (1u << 19)) {
		// a column sums up to 4 x nIn ones; the parity read needs the sum below 2^23
		set_error("tensor method (mxf4): %u inputs in one call, at most %u", nIn, (1u << 19) - 1);
		return -1;
	}
	const size_t minBytes = t4_min_scratch(R, nIn);
	if(!scratch || scratchBytes < minBytes) {
		set_error("tensor method (mxf4) needs at least %zu bytes of scratch, %zu given", minBytes, scratchBytes);
		return -1;
	}
	if(reinterpret_cast<uintptr_t>(scratch) & 15) {
		set_error("tensor method (mxf4): the scratch must be 16-byte aligned");
		return -1;
	}
	unsigned nPairsSM = 0;
	if(t4_pairs_on_device(&nPairsSM)) return -1;
	// split passes are added by pairs of words: whole 32-bit words of the rows
	const bool maySplit = reinterpret_cast<uintptr_t>(rec) % 4 == 0 && recPitch % 2 == 0 && nWords % 2 == 0;
	T4Plan pl;
	if(!t4_plan(pl, R, nIn, nWords, scratchBytes, nPairsSM, maySplit)) {
		set_error("tensor method (mxf4): no plan fits %zu bytes of scratch", scratchBytes);
		return -1;
	}
	uint8_t* sp = reinterpret_cast<uint8_t*>(scratch);
	return pl.form == 4 ? t4_run<4>(pl, in, inPitch, nIn, coeff, rec, recPitch, R, nWords, accumulate, sp, nPairsSM, st)
	                    : t4_run<1>(pl, in, inPitch, nIn, coeff, rec, recPitch, R, nWords, accumulate, sp, nPairsSM, st);
}

// ------------------------------------------------------------------ peak
// Calibration of the roofline denominator: pairs of CTAs issue `iters` MMAs
// of the GEMM's shape (M = 256, N = 240, K = 96, kind::mxf4, unit scales) on
// operands resident in shared memory, back to back into one accumulator, and
// wait (bounded) for their completion.  No global memory traffic: the rate
// is the tensor pipe's for this instruction.
__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(128, 1) k_tc4_mma_rate(unsigned iters)
{
	extern __shared__ __align__(1024) uint8_t smem_raw[];
	const uint32_t raw = t4_saddr(smem_raw);
	const uint32_t pad = (1024u - (raw & 1023u)) & 1023u;
	uint8_t* sm = smem_raw + pad;
	const uint32_t sbase = raw + pad;
	constexpr int STAGE = T4_SU * (T4_UNIT_A + T4_MAXN * 24);
	const uint32_t doneBar = sbase + STAGE;
	uint32_t* tslot = reinterpret_cast<uint32_t*>(sm + STAGE + 8);
	const int warp = threadIdx.x >> 5;
	uint32_t rank;
	asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(rank));
	for(int e = threadIdx.x; e < STAGE / 16; e += 128) reinterpret_cast<uint4*>(sm)[e] = make_uint4(0, 0, 0, 0);
	if(threadIdx.x == 0) {
		asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" :: "r"(doneBar) : "memory");
		asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
	}
	asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
	if(warp == 0) {
		asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;" :: "r"(t4_saddr(tslot)), "r"(512u) : "memory");
		asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
	}
	asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
	__syncthreads();
	asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
	const uint32_t tmem = *tslot;
	t4_fill_sf(tmem + ((uint32_t)(32 * warp) << 16) + T4_SF_COL);
	asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
	__syncthreads();
	t4_cluster_sync();
	asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
	if(threadIdx.x == 0 && rank == 0) {
		const uint32_t idesc = t4_idesc(2 * T4_ROWS, T4_MAXN);
		for(unsigned it = 0; it < iters; it++) {
			const uint32_t u = it % T4_SU;
			t4_mma(tmem, t4_desc(sbase + u * T4_UNIT_A, 2048), t4_desc(sbase + T4_SU * T4_UNIT_A + u * T4_MAXN * 24, T4_MAXN * 8), idesc,
			       tmem + T4_SF_COL, it != 0);
		}
		t4_commit(doneBar);
	}
	__syncwarp();
	t4_wait(doneBar, 0);
	asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
	__syncthreads();
	t4_cluster_sync();
	if(warp == 0)
		asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" :: "r"(tmem), "r"(512u) : "memory");
}

int tc4_mma_rate(double* macsPerSec, cudaStream_t st) {
	unsigned pairs = 0;
	if(t4_pairs_on_device(&pairs)) return -1;
	const size_t smem = T4_SU * (T4_UNIT_A + T4_MAXN * 24) + 8 + 16 + 1024;
	P2C_CUDA_TRY(cudaFuncSetAttribute(k_tc4_mma_rate, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
	const unsigned iters = 20000;
	cudaEvent_t e0, e1;
	P2C_CUDA_TRY(cudaEventCreate(&e0));
	P2C_CUDA_TRY(cudaEventCreate(&e1));
	float best = 0.f;
	for(int rep = 0; rep < 3; rep++) {
		cudaEventRecord(e0, st);
		k_tc4_mma_rate<<<2 * pairs, 128, smem, st>>>(iters);
		cudaEventRecord(e1, st);
		cudaEventSynchronize(e1);
		float ms = 0.f;
		cudaEventElapsedTime(&ms, e0, e1);
		if(rep == 0 || ms < best) best = ms;
	}
	cudaEventDestroy(e0);
	cudaEventDestroy(e1);
	P2C_CUDA_TRY(cudaGetLastError());
	*macsPerSec = best > 0.f ? (double)iters * pairs * (2 * T4_ROWS) * T4_MAXN * 96 / (best * 1e-3) : 0.0;
	return 0;
}

int tc4_error_take() {
	unsigned v = 0, z = 0;
	if(cudaMemcpyFromSymbol(&v, g_tc4_error, sizeof(v)) != cudaSuccess) return -1;
	if(v) cudaMemcpyToSymbol(g_tc4_error, &z, sizeof(z));
	return (int)v;
}

} // namespace p2c
