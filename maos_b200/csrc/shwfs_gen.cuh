// Imaging stages (b)-(e) for the larger FFT sizes, n_f = n_w = N in {64, 128,
// 256} (the NGS and tip-tilt sensors of an uneven batch, large-sampling LGS):
// a chain of batched 1-D FFT passes over a per-powfs scratch image in global
// memory (L2-resident for the small batches), each pass a kernel over tiles of
// rows or columns of an image, with the element-wise step of the chain fused in:
//
//   pass 1  columns x in [pad, pad+n_o): field E = amp exp(i 2 pi opd / lambda), FFT along y
//   pass 2  rows ky:                     FFT along x (columns outside the pupil are zero),
//                                        |.|^2 * scale, FFT along x (the PSF's transform)
//   pass 3  columns fx:                  FFT along ky (the OTF), x conj(uplink OTF) x ETF / DTF
//                                        nominal, inverse FFT along fy
//   pass 4  rows y:                      inverse FFT along fx, real part
//   pixels  a thread per pixel:          bilinear pixel map, noise, CoG / matched filter
//
// The two-dimensional transforms are separable, so each pass takes its lines
// through two of them where the chain allows (the PSF's rows right after the
// field's, the inverse's columns right after the OTF's): four passes over the
// image instead of six, with the same transforms and element-wise steps
// as maos/wfsints.c:233-286 (cembed_wvf with pad (n_w - n_o)/2, cfft2 with
// FFTW's sign and no normalisation, cabs2toreal, ccwmc with the uplink OTF,
// apply_dtf_etf, cfft2 inverse, dspmulcreal).  For the LLT pupil, passes 1-3
// up to the OTF give the uplink OTF (maos/wfsints.c:149-199).
// Transfer functions are stored transposed per subaperture ([fy + N fx]), as
// in the 32-point path; the scratch image is row-major ([row][column]).
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>
#include "shwfs_kernels.cuh"

namespace shwfs {

// FFT lines per tile: what GEN_THREADS threads of 16 points hold
__host__ __device__ constexpr int gen_lines(int n) { return 2048 / n; }
constexpr int GEN_THREADS = 128;

enum GenPass { GEN_FIELD_COLS = 1, GEN_PSF_ROWS, GEN_OTF_COLS, GEN_INV_ROWS };
constexpr int GEN_NPASS = 4;

// Line stride of a tile in the exchange (float2): the 16 (N / 16 + 1) slots of a
// line, padded so that the lanes of a half warp fall on distinct banks where
// they run along the lines' elements (row passes) or across the lines.
__host__ __device__ constexpr int gen_ls(int n, bool rows) {
	return n == 64 ? (rows ? 84 : 81) : n == 128 ? (rows ? 152 : 153) : (rows ? 272 : 274);
}

// FFT of a line of N points by its T = N / 16 threads of 16 points each:
// thread t brings v[i] = x[T i + t] and leaves with v[i] = X[t + T i] (natural
// order, unnormalised; DIR -1 forward, +1 inverse).  A 16-point transform in
// registers, the twiddles w_N^(t k1), one exchange through the line's slots
// ex[k1 (T + 1) + t], then the 16 / T T-point transforms of k1 = t + T m:
//   X[k1 + 16 k2] = sum_t w_T^(t k2) w_N^(t k1) sum_i w_16^(i k1) x[T i + t].
// The outputs sit where the next transform of the line takes its inputs, so a
// pass that transforms its lines twice stays in registers in between: one
// shared-memory round trip a transform, where radix-2 stages taken two at a
// time made four with a block barrier each.  52 images of 128 x 128 points, the
// four passes one after the other with cold caches: 8 + 17 + 18 + 11 -> 8 + 6 +
// 13 + 8 us; images and gradients in one call 36 -> 15.5 us where calls overlap
// (its five launches now set the rate), 56 -> 34 back to back on one stream.  ROWS: a line's threads are lanes of one warp.
// tw[k] = exp(-2 pi i k / N), k < N.
template <int N, int DIR, bool ROWS>
__device__ __forceinline__ void gen_fft(float2 (&v)[16], float2* ex, int t, const float2* __restrict__ tw) {
	constexpr int T = N / 16, M = 16 / T;
	fft_reg<DIR, 16>(v);
#pragma unroll
	for (int k = 1; k < 16; k++) {
		const float2 w = __ldg(tw + t * k);
		v[k] = DIR > 0 ? cmulc(v[k], w) : cmul(v[k], w);
	}
#pragma unroll
	for (int k = 0; k < 16; k++) ex[k * (T + 1) + t] = v[k];
	if (ROWS) __syncwarp();
	else __syncthreads();
#pragma unroll
	for (int m = 0; m < M; m++) {
		float2 u[T];
#pragma unroll
		for (int j = 0; j < T; j++) u[j] = ex[(t + T * m) * (T + 1) + j];
		fft_reg<DIR, T>(u);
#pragma unroll
		for (int k2 = 0; k2 < T; k2++) v[m + M * k2] = u[k2];
	}
	if (ROWS) __syncwarp();  // the slots may be written again
	else __syncthreads();
}

// A launch covers nitem images.  WFS mode: image i is subaperture i / nw of
// wfs[i % nw] (the order of the 32-point launches).  Uplink mode: image i is
// the LLT pupil of wfs[i] (opd = LLT OPD, amp = LLT amplitude), and pass 3
// stores its OTF, transposed, into wfs[i].lotfT instead of applying it.
struct GenParams {
	int nitem, nw, nopd, pad;
	int uplink;
	float scale;                 // factor on |.|^2: 1 for WFS images, 1/N^2 for LLT pupils
	float twoinvwvl;
	float2* buf;                 // nitem * N * N scratch, row-major per image
	const float2* tw;            // N twiddles exp(-2 pi i k / N)
	const WfsDev* wfs;
	const float2* etfT1;         // nsa * N^2 transposed, or null
	const float2* etfT2;
	float etfwt1, etfwt2;
	const float* nominalT;       // N^2 (or nsa * N^2) transposed, or null
	int nominal_per_sa;
};

// Shared memory of one pass tile: the exchange, and the tile's transfer
// functions (or uplink OTF) by line and frequency (line stride N + 1).
__host__ __device__ constexpr int gen_tile_smem(int n) {
	return gen_lines(n) * ((gen_ls(n, true) > gen_ls(n, false) ? gen_ls(n, true) : gen_ls(n, false)) + n + 1) *
		(int)sizeof(float2);
}

// Reads of the scratch image: through L1, or from L2 only (L2ONLY) where other
// blocks of the same launch wrote it (L1 is not coherent between SMs).
template <bool L2ONLY>
__device__ __forceinline__ float2 gen_ld(const float2* p) {
	if constexpr (L2ONLY) return __ldcg(p);
	else return *p;
}

// One pass over tile `tile` of image i by a block of GEN_THREADS threads; gen_s
// is the tile's shared memory (gen_tile_smem(N) bytes).  The scratch image
// goes straight between global memory and registers: consecutive lanes take
// consecutive elements of a row, or consecutive columns.
template <int N, int PASS, int NT, bool L2ONLY>
__device__ __forceinline__ void gen_pass_tile(const GenParams& G, int i, int tile, float2* gen_s) {
	constexpr int L = gen_lines(N), T = N / 16;
	constexpr bool ROWS = PASS == GEN_PSF_ROWS || PASS == GEN_INV_ROWS;
	constexpr int LS = gen_ls(N, ROWS), TLS = N + 1;
	static_assert(NT == L * T && NT == GEN_THREADS, "a thread per 16 points of the tile");
	const int isa = G.uplink ? 0 : i / G.nw;
	const WfsDev& W = G.wfs[G.uplink ? i : i % G.nw];
	float2* im = G.buf + (size_t)i * N * N;
	const int tid = threadIdx.x;
	const int line = ROWS ? tid / T : tid % L, t = ROWS ? tid % T : tid / L;
	float2* ex = gen_s + line * LS;
	float2* tfs = gen_s + L * (gen_ls(N, true) > gen_ls(N, false) ? gen_ls(N, true) : gen_ls(N, false));
	int l0 = tile * L, nl = L;  // first line and lines of the tile
	if (PASS == GEN_FIELD_COLS) {  // only the pupil's columns
		nl = min(L, G.nopd - l0);
		l0 += G.pad;
	}
	const size_t at0 = ROWS ? (size_t)(l0 + line) * N + t : (size_t)t * N + l0 + line;
	constexpr size_t STEP = ROWS ? T : (size_t)T * N;
	float2 v[16];
	if (PASS == GEN_FIELD_COLS) {
		float o[16], a[16];
		const int x = l0 + line - G.pad;
#pragma unroll
		for (int k = 0; k < 16; k++) {
			const int y = T * k + t - G.pad;
			const bool in = line < nl && y >= 0 && y < G.nopd;
			const size_t e = (size_t)isa * G.nopd * G.nopd + (size_t)y * G.nopd + x;
			o[k] = in ? __ldg(W.opd + e) : 0.f;
			a[k] = in ? __ldg(W.amp + e) : 0.f;
		}
#pragma unroll
		for (int k = 0; k < 16; k++) {
			const int y = T * k + t - G.pad;
			v[k] = make_float2(0.f, 0.f);
			if (line < nl && y >= 0 && y < G.nopd) {
				float sn, cs;
				sincospif(G.twoinvwvl * o[k], &sn, &cs);
				v[k] = make_float2(a[k] * cs, a[k] * sn);
			}
		}
	} else {
#pragma unroll
		for (int k = 0; k < 16; k++) {
			const int n = T * k + t;  // rows of pass 2: columns outside the pupil are zero
			v[k] = PASS != GEN_PSF_ROWS || (n >= G.pad && n < G.pad + G.nopd) ? gen_ld<L2ONLY>(im + at0 + STEP * k)
																				: make_float2(0.f, 0.f);
		}
	}
	if (PASS == GEN_OTF_COLS && !G.uplink) {
		// the tile's transfer functions ([fy + N fx], fy fastest) in runs of fy: conj(uplink OTF) x ETF / nominal
		const size_t f0 = (size_t)N * l0;
		const float2* e1 = G.etfT1 ? G.etfT1 + (size_t)isa * N * N + f0 : nullptr;
		const float2* e2 = G.etfT2 ? G.etfT2 + (size_t)isa * N * N + f0 : nullptr;
		const float* nm = G.nominalT ? G.nominalT + (G.nominal_per_sa ? (size_t)isa * N * N : 0) + f0 : nullptr;
		const float2* up = W.lotfT ? W.lotfT + f0 : nullptr;
#pragma unroll 4
		for (int k = 0; k < 16; k++) {
			const int idx = tid + k * NT;
			float2 w = make_float2(1.f, 0.f);
			if (e1) {
				w = __ldg(e1 + idx);
				if (e2) {
					const float2 b = __ldg(e2 + idx);
					w = make_float2(w.x * G.etfwt1 + b.x * G.etfwt2, w.y * G.etfwt1 + b.y * G.etfwt2);
				}
			} else if (nm) {
				w.x = __ldg(nm + idx);
			}
			if (up) w = cmulc(w, __ldg(up + idx));
			tfs[(idx / N) * TLS + idx % N] = w;
		}
	}
	gen_fft<N, PASS == GEN_INV_ROWS ? 1 : -1, ROWS>(v, ex, t, G.tw);
	// ---- element-wise steps of the chain, and a pass's second transform
	if (PASS == GEN_PSF_ROWS) {
		// |.|^2 * scale: the PSF row, then its own transform along x (the OTF's)
#pragma unroll
		for (int k = 0; k < 16; k++) v[k] = make_float2((v[k].x * v[k].x + v[k].y * v[k].y) * G.scale, 0.f);
		gen_fft<N, -1, ROWS>(v, ex, t, G.tw);
	}
	if (PASS == GEN_OTF_COLS) {
		// line = fx - l0, element fy = t + T k: the OTF
		if (G.uplink) {
#pragma unroll
			for (int k = 0; k < 16; k++) tfs[line * TLS + t + T * k] = v[k];
			__syncthreads();
#pragma unroll 4
			for (int k = 0; k < 16; k++) {
				const int idx = tid + k * NT;
				const_cast<float2*>(W.lotfT)[(size_t)N * l0 + idx] = tfs[(idx / N) * TLS + idx % N];  // the uplink OTF
			}
			return;
		}
		// gen_fft's barriers lie between the stores to tfs and these reads
#pragma unroll
		for (int k = 0; k < 16; k++) v[k] = cmul(v[k], tfs[line * TLS + t + T * k]);
		gen_fft<N, 1, ROWS>(v, ex, t, G.tw);  // the inverse along fy
	}
	// ---- store (natural order; the last pass keeps the real part)
	if (line < nl) {
#pragma unroll
		for (int k = 0; k < 16; k++) {
			if (PASS == GEN_INV_ROWS) v[k].y = 0.f;
			im[at0 + STEP * k] = v[k];
		}
	}
}

// One pass over one tile (blockIdx.y) of one image (blockIdx.x).
template <int N, int PASS>
__global__ void __launch_bounds__(GEN_THREADS) gen_pass_kernel(GenParams G) {
	extern __shared__ float2 gen_s[];
	gen_pass_tile<N, PASS, GEN_THREADS, false>(G, blockIdx.x, blockIdx.y, gen_s);
}

// Pixels, noise and gradients of generic-size images: one warp per work item
// (item = isa * nw + k as in the imaging launch), image item of buf (n2 = N^2
// elements each), real part.
template <int NPQ, bool L2ONLY>
__device__ __forceinline__ void gen_pixels_item(const PowfsDev& P, const WfsDev* __restrict__ wfs, int nw, int item,
	const float2* __restrict__ buf, int n2, int lane) {
	const int isa = item / nw;
	const WfsDev& W = wfs[item % nw];
	const float2* im = buf + (size_t)item * n2;
	const int npix = P.npix;
	// a pixel's 4 map entries are one 16-byte row (cudaMalloc'd, 4 entries per pixel)
	const int4* sidx = reinterpret_cast<const int4*>(P.simap_idx) + (P.simap_per_sa ? (size_t)isa * npix : 0);
	const float4* swt = reinterpret_cast<const float4*>(P.simap_wt) + (P.simap_per_sa ? (size_t)isa * npix : 0);
	// Few warps run these images, so every load latency is exposed: the map
	// rows, then the image taps, are each issued as one independent wave.  A
	// missing tap (index < 0) reads as 0, and fmaf(w, 0, v) = v, so the sums
	// equal those that skip it.
	float x[NPQ][4];
#pragma unroll
	for (int q = 0; q < NPQ; q++) {
		const int p = lane + 32 * q;
		const int4 id = p < npix ? __ldg(sidx + p) : make_int4(-1, -1, -1, -1);
		x[q][0] = id.x >= 0 ? gen_ld<L2ONLY>(im + id.x).x : 0.f;
		x[q][1] = id.y >= 0 ? gen_ld<L2ONLY>(im + id.y).x : 0.f;
		x[q][2] = id.z >= 0 ? gen_ld<L2ONLY>(im + id.z).x : 0.f;
		x[q][3] = id.w >= 0 ? gen_ld<L2ONLY>(im + id.w).x : 0.f;
	}
	float pix[NPQ];
#pragma unroll
	for (int q = 0; q < NPQ; q++) {
		const int p = lane + 32 * q;
		float v = 0.f;
		if (p < npix) {
			const float4 w = __ldg(swt + p);
			v = fmaf(w.x, x[q][0], v);
			v = fmaf(w.y, x[q][1], v);
			v = fmaf(w.z, x[q][2], v);
			v = fmaf(w.w, x[q][3], v);
			v *= W.alpha;
			if (P.accum) v += W.ints[(size_t)isa * npix + p];  // dtrat > 1: the frames so far
		}
		pix[q] = v;
	}
	if (W.noisy) {
#pragma unroll
		for (int q = 0; q < NPQ; q++) {
			const int p = lane + 32 * q;
			if (p < npix) {
				PixelRng rng(W.seed, (uint32_t)(isa * npix + p), W.wfs_id, (uint32_t)P.isim);
				pix[q] = poisson_draw(rng, pix[q] + P.bkgrnd) + P.rne * rng.normal() - P.bkgrndc;
			}
		}
	}
	if (W.ints) {
#pragma unroll
		for (int q = 0; q < NPQ; q++) {
			const int p = lane + 32 * q;
			if (p < npix) W.ints[(size_t)isa * npix + p] = pix[q];
		}
	}
	if (W.grad)
		grad_from_pixels<NPQ>(pix, npix, P.pixpsax, P.pixpsay, P, W.mtche + (size_t)isa * 2 * npix, W.i0sum, isa, lane,
			W.grad, P.nsa);
}
// The same step with one block per image (blockIdx.x = item), a thread per
// pixel (npix rounded up to whole warps): the launches of these sizes often
// hold a few images, where a warp walking 8 pixels' noise draws in turn set
// their latency.  The
// image's first warp then forms the gradients from the pixels in shared
// memory, in gen_pixels_item's lane order (pixel p = lane + 32 q), so
// intensities, noise and gradients equal those of gen_pixels_item.
constexpr int GEN_PIX_THREADS = 256;  // the largest pixel count of these sizes
__global__ void __launch_bounds__(GEN_PIX_THREADS) gen_pixels_block_kernel(PowfsDev P,
	const WfsDev* __restrict__ wfs, int nw, const float2* __restrict__ buf, int n2) {
	__shared__ float spix[GEN_PIX_THREADS];
	const int item = blockIdx.x, p = threadIdx.x;
	const int isa = item / nw;
	const WfsDev& W = wfs[item % nw];
	const int npix = P.npix;
	float v = 0.f;
	if (p < npix) {
		const float2* im = buf + (size_t)item * n2;
		const size_t m = (P.simap_per_sa ? (size_t)isa * npix : 0) + p;
		const int4 id = __ldg(reinterpret_cast<const int4*>(P.simap_idx) + m);
		const float4 w = __ldg(reinterpret_cast<const float4*>(P.simap_wt) + m);
		v = fmaf(w.x, id.x >= 0 ? im[id.x].x : 0.f, v);
		v = fmaf(w.y, id.y >= 0 ? im[id.y].x : 0.f, v);
		v = fmaf(w.z, id.z >= 0 ? im[id.z].x : 0.f, v);
		v = fmaf(w.w, id.w >= 0 ? im[id.w].x : 0.f, v);
		v *= W.alpha;
		if (P.accum) v += W.ints[(size_t)isa * npix + p];  // dtrat > 1: the frames so far
		if (W.noisy) {
			PixelRng rng(W.seed, (uint32_t)(isa * npix + p), W.wfs_id, (uint32_t)P.isim);
			v = poisson_draw(rng, v + P.bkgrnd) + P.rne * rng.normal() - P.bkgrndc;
		}
		if (W.ints) W.ints[(size_t)isa * npix + p] = v;
	}
	spix[p] = v;
	__syncthreads();
	if (p < 32 && W.grad) {
		float pix[GEN_PIX_THREADS / 32];
#pragma unroll
		for (int q = 0; q < GEN_PIX_THREADS / 32; q++) pix[q] = p + 32 * q < npix ? spix[p + 32 * q] : 0.f;
		grad_from_pixels<GEN_PIX_THREADS / 32>(pix, npix, P.pixpsax, P.pixpsay, P, W.mtche + (size_t)isa * 2 * npix,
			W.i0sum, isa, p, W.grad, P.nsa);
	}
}

// ---------------------------------------------------------------------------
// n_f = n_w = 64 fused per image: one block of 128 threads holds the 64x64
// image in shared memory; every 64-point line transform is 8 x 8: n = 8 n1 +
// n2, k = k1 + 8 k2, X[k] = sum_n2 w64^(n2 k1) w8^(n2 k2) sum_n1 x[n] w8^(n1 k1),
// with the 8-point transforms in registers, so each line costs two passes
// through shared memory.  Form F takes the line in natural order and leaves
// X[k] at the digit-reversed position r(k) = 8 (k mod 8) + k / 8; form G takes
// the line in digit-reversed order and leaves it natural.  The chain uses F
// for the field and the inverse transforms and G for the PSF -> OTF transform,
// so the OTF is in natural order where the transfer functions multiply it, and
// the final image sits at digit-reversed rows and columns.
// ---------------------------------------------------------------------------
constexpr int N64_LS = 65;  // line stride of the shared image (float2): row, column and
                            // transfer-function accesses all at the 2-wavefront minimum

__device__ __forceinline__ int digrev8(int k) { return ((k & 7) << 3) | (k >> 3); }

// 8-point DFT in registers, natural order in and out; dir -1 forward, +1
// inverse.  dft8_tail: what follows the radix-2 stage on the pairs (j, j+4).
__device__ __forceinline__ void dft8_tail(float2 (&b)[8], float2 (&a)[8], float dir) {
	const float h = 0.70710678118654752f;
	// twiddles w8^j on b[4..7]: w8 = exp(dir i pi/4)
	{
		float2 t = b[5];
		b[5] = make_float2(h * (t.x - dir * t.y), h * (t.y + dir * t.x));
		t = b[6];
		b[6] = make_float2(-dir * t.y, dir * t.x);
		t = b[7];
		b[7] = make_float2(h * (-t.x - dir * t.y), h * (-t.y + dir * t.x));
	}
	// two 4-point DFTs: (b0..b3) -> even outputs, (b4..b7) -> odd outputs
#pragma unroll
	for (int g = 0; g < 2; g++) {
		const float2 c0 = b[4 * g], c1 = b[4 * g + 1], c2 = b[4 * g + 2], c3 = b[4 * g + 3];
		const float2 s0 = cadd(c0, c2), d0 = csub(c0, c2), s1 = cadd(c1, c3), d1 = csub(c1, c3);
		const float2 d1r = make_float2(-dir * d1.y, dir * d1.x);  // d1 * (dir i)
		a[g] = cadd(s0, s1);                                  // X[0] / X[1]
		a[g + 2] = make_float2(d0.x + d1r.x, d0.y + d1r.y);  // X[2] / X[3]
		a[g + 4] = csub(s0, s1);                              // X[4] / X[5]
		a[g + 6] = make_float2(d0.x - d1r.x, d0.y - d1r.y);  // X[6] / X[7]
	}
}
__device__ __forceinline__ void dft8(float2 (&a)[8], float dir) {
	float2 b[8];
#pragma unroll
	for (int j = 0; j < 4; j++) {
		b[j] = cadd(a[j], a[j + 4]);
		b[j + 4] = csub(a[j], a[j + 4]);
	}
	dft8_tail(b, a, dir);
}
// the same with a[0], a[1], a[6] and a[7] zero (not read)
__device__ __forceinline__ void dft8_mid(float2 (&a)[8], float dir) {
	float2 b[8] = {a[4], a[5], a[2], a[3], make_float2(-a[4].x, -a[4].y), make_float2(-a[5].x, -a[5].y), a[2], a[3]};
	dft8_tail(b, a, dir);
}
// a[i] *= exp(DIR 2 pi i t i / 64); tw[N64_TS t + i] = exp(-2 pi i t i / 64), read in pairs
// (rows 80 bytes apart, so that the rows of a quarter warp fall on distinct banks)
constexpr int N64_TS = 10;
template <int DIR>
__device__ __forceinline__ void n64_twiddle(float2 (&a)[8], const float2* tw, int t) {
	const float4* w4 = reinterpret_cast<const float4*>(tw + N64_TS * t);
#pragma unroll
	for (int q = 0; q < 4; q++) {
		const float4 w = w4[q];
		if (q) a[2 * q] = DIR > 0 ? cmulc(a[2 * q], make_float2(w.x, w.y)) : cmul(a[2 * q], make_float2(w.x, w.y));
		a[2 * q + 1] = DIR > 0 ? cmulc(a[2 * q + 1], make_float2(w.z, w.w)) : cmul(a[2 * q + 1], make_float2(w.z, w.w));
	}
}
// elements at p[es (8 t + i)] (group t) or p[es (8 i + t)] (stride t) of a line
template <int ES>
__device__ __forceinline__ void n64_get(float2 (&a)[8], const float2* p) {
#pragma unroll
	for (int i = 0; i < 8; i++) a[i] = p[ES * i];
}
template <int ES>
__device__ __forceinline__ void n64_put(float2* p, const float2 (&a)[8]) {
#pragma unroll
	for (int i = 0; i < 8; i++) p[ES * i] = a[i];
}

// (b)-(e) fused for n_f = n_w = 64: one block of N64_THREADS threads per work
// item (item = isa * nw + k as in the other imaging launches).  Dynamic shared
// memory N64_SMEM_BYTES.  tw64[k] = exp(-2 pi i k / 64), k < 64.
//
// The kernel is bound by the shared-memory wavefronts of its eleven passes
// over the image, so every element-wise step rides on a pass that holds its
// operands in registers: the field on the first row transforms' loads (from
// the OPD itself), |.|^2 and the packing of two PSF rows into one complex row
// on the last column transforms (a thread takes rows 8t + i and 8t + i + 32 of
// a column), the unpacking of the half spectrum on the loads of the OTF's
// columns, the transfer functions between the OTF's last pass and the
// inverse's first one (both on elements 8i + t of a column: no pass between
// them), the packing of two image rows on the loads of the inverse's rows (a
// thread takes the residues t and 8 - t, which hold each other's mirrored
// frequencies).  Lanes take consecutive lines, so accesses are free of bank
// conflicts (line stride 65) and a warp shares its twiddles; the pass with the
// transfer functions takes 8 consecutive frequencies of 4 columns 8 apart
// instead, so that they are read in 64-byte runs.  Against the 16-pass form
// with 256 threads (6725 -> 4425 wavefronts an image): 6 WFS of 2820 images
// 464 -> 334 us, 3 WFS of 808 images 71 -> 52 us.
constexpr int N64_THREADS = 128;
constexpr int N64_SMEM_BYTES = (64 * N64_LS + 8 * N64_TS) * 8 + 256 * 4;
// NOPD > 0 fixes the pupil size at compile time (nopd is then ignored).
template <int NOPD>
__global__ void __launch_bounds__(N64_THREADS, 6) ints_n64_kernel(PowfsDev P, const WfsDev* __restrict__ wfs, int nw,
	int nitem, int nopd_rt, float twoinvwvl, const float2* __restrict__ tw64) {
	static_assert(NOPD == 0 || NOPD == 32, "fixed pupil sizes: 32");
	constexpr int LS = N64_LS;
	const int nopd = NOPD > 0 ? NOPD : nopd_rt;
	extern __shared__ __align__(16) float2 n64_s[];
	float2* img = n64_s;
	float2* tw = n64_s + 64 * LS;
	float* spix = reinterpret_cast<float*>(tw + 8 * N64_TS);
	const int item = blockIdx.x, tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
	if (item >= nitem) return;
	const int isa = item / nw;
	const WfsDev& W = wfs[item % nw];
	const int pad = (64 - nopd) / 2, no2 = nopd * nopd;
	if (tid < 64) tw[N64_TS * (tid >> 3) + (tid & 7)] = tw64[(tid >> 3) * (tid & 7)];
	__syncthreads();
	float2 a[8], b[8];
	// (b) field, zero-padded (cembed_wvf, maos/wfsints.c:233), and (c) PSF: forward along x on the pupil rows
	{
		const float* opd = W.opd + (size_t)isa * no2;
		const float* amp = W.amp + (size_t)isa * no2;
		for (int task = tid; task < nopd * 8; task += N64_THREADS) {
			const int y = task >> 3, t = task & 7;
			float o[8], m[8];
#pragma unroll
			for (int i = 0; i < 8; i++) {
				const int x = 8 * i + t - pad;
				const bool in = NOPD ? i >= 2 && i < 6 : x >= 0 && x < nopd;
				o[i] = in ? __ldg(opd + y * nopd + x) : 0.f;
				m[i] = in ? __ldg(amp + y * nopd + x) : 0.f;
			}
#pragma unroll
			for (int i = 0; i < 8; i++) {
				if (NOPD && (i < 2 || i >= 6)) continue;
				float sn, cs;
				sincospif(twoinvwvl * o[i], &sn, &cs);
				a[i] = make_float2(m[i] * cs, m[i] * sn);
			}
			if (NOPD) dft8_mid(a, -1.f);
			else dft8(a, -1.f);
			n64_twiddle<-1>(a, tw, t);
			n64_put<8>(img + (y + pad) * LS + t, a);
		}
	}
	__syncthreads();
	for (int task = tid; task < nopd * 8; task += N64_THREADS) {
		const int L = task % nopd, t = task / nopd;
		float2* p = img + (pad + L) * LS + 8 * t;
		n64_get<1>(a, p);
		dft8(a, -1.f);
		n64_put<1>(p, a);
	}
	__syncthreads();
	// forward along y, the rows outside the pupil being zero
#pragma unroll 1
	for (int t = tid >> 6; t < 8; t += 2) {
		float2* p = img + (tid & 63) + t * LS;
		if (NOPD) {
#pragma unroll
			for (int i = 2; i < 6; i++) a[i] = p[8 * LS * i];
			dft8_mid(a, -1.f);
		} else {
#pragma unroll
			for (int i = 0; i < 8; i++) {
				const int y = 8 * i + t;
				a[i] = y >= pad && y < pad + nopd ? p[8 * LS * i] : make_float2(0.f, 0.f);
			}
			dft8(a, -1.f);
		}
		n64_twiddle<-1>(a, tw, t);
		n64_put<8 * LS>(p, a);
	}
	__syncthreads();
	// |.|^2, two real PSF rows per complex row: row r <- (PSF row r) + i (PSF row r + 32)
#pragma unroll 1
	for (int t = tid >> 6; t < 4; t += 2) {
		float2* p = img + (tid & 63) + 8 * t * LS;
		n64_get<LS>(a, p);
		n64_get<LS>(b, p + 32 * LS);
		dft8(a, -1.f);
		dft8(b, -1.f);
#pragma unroll
		for (int i = 0; i < 8; i++)
			p[LS * i] = make_float2(a[i].x * a[i].x + a[i].y * a[i].y, b[i].x * b[i].x + b[i].y * b[i].y);
	}
	__syncthreads();
	// OTF, half spectrum kx = 0..32 (the PSF is real, so OTF(-k) = conj OTF(k)):
	// forward along kx on the 32 packed rows (digit-reversed inputs)
#pragma unroll 1
	for (int t = warp; t < 8; t += 4) {
		float2* p = img + lane * LS + 8 * t;
		n64_get<1>(a, p);
		dft8(a, -1.f);
		n64_twiddle<-1>(a, tw, t);
		n64_put<1>(p, a);
	}
	__syncthreads();
#pragma unroll 1
	for (int t = warp; t < 8; t += 4) {
		float2* p = img + lane * LS + t;
		n64_get<8>(a, p);
		dft8(a, -1.f);
		n64_put<8>(p, a);
	}
	__syncthreads();
	// forward along ky on columns kx = 0..31 (digit-reversed inputs), unpacking
	// the pairs: row r's spectrum Z = H_r + i H_{r+32}, H_r(kx) = (Z(kx) + conj
	// Z(-kx)) / 2, H_{r+32}(kx) = (Z(kx) - conj Z(-kx)) / 2i.  H(0) and H(32) are
	// real, so column 0 carries H(0) + i H(32).
	{
		const int t = warp, kx = lane;
		float2* p = img + 8 * t * LS + kx;
		const float2* pm = img + 8 * t * LS + (kx ? 64 - kx : 32);
#pragma unroll
		for (int i = 0; i < 8; i++) {
			const float2 z = p[LS * i], zm = pm[LS * i];
			a[i] = kx ? make_float2(0.5f * (z.x + zm.x), 0.5f * (z.y - zm.y)) : make_float2(z.x, zm.x);
			b[i] = kx ? make_float2(0.5f * (z.y + zm.y), 0.5f * (zm.x - z.x)) : make_float2(z.y, zm.y);
		}
		dft8(a, -1.f);
		n64_twiddle<-1>(a, tw, t);
		n64_put<LS>(p, a);
		dft8(b, -1.f);
		n64_twiddle<-1>(b, tw, t + 4);
		n64_put<LS>(p + 32 * LS, b);
	}
	__syncthreads();
	// the columns' second half: natural OTF at fy = 8 i + t, x conj(uplink OTF) x
	// ETF / nominal (transfer functions are [fy + 64 fx]), then the first half
	// of the inverse along fy on the same elements.  The transfer functions are
	// transforms of real kernels (uplink PSF, elongated spot, pixel response),
	// Hermitian to rounding, so each half-spectrum element takes TF itself: the
	// image is then the real part of the full inverse up to rounding.  Column 0
	// holds Y = O(.,0) + i O(.,32) with O(.,0), O(.,32) the transforms of real
	// columns; it goes on as X(.,0) + i X(.,32).
	{
		const float2* e1 = P.etfT1 ? P.etfT1 + (size_t)isa * 4096 : nullptr;
		const float2* e2 = P.etfT2 ? P.etfT2 + (size_t)isa * 4096 : nullptr;
		const float* nm = P.nominalT ? P.nominalT + (P.nominal_per_sa ? (size_t)isa * 4096 : 0) : nullptr;
		const int t = lane & 7;
		auto tf1 = [&](int k) {  // transfer function at element k
			float2 o = make_float2(1.f, 0.f);
			if (e1) {
				o = __ldg(e1 + k);
				if (e2) {
					const float2 f = __ldg(e2 + k);
					o = make_float2(o.x * P.etfwt1 + f.x * P.etfwt2, o.y * P.etfwt1 + f.y * P.etfwt2);
				}
			} else if (nm) {
				o.x = __ldg(nm + k);
			}
			return W.lotfT ? cmulc(o, __ldg(W.lotfT + k)) : o;
		};
		// the same at elements t0 + 8 i, the loads together
		auto tf = [&](float2 (&o)[8], int t0) {
			if (e1) {
#pragma unroll
				for (int i = 0; i < 8; i++) o[i] = __ldg(e1 + t0 + 8 * i);
				if (e2) {
#pragma unroll
					for (int i = 0; i < 8; i++) {
						const float2 f = __ldg(e2 + t0 + 8 * i);
						o[i] = make_float2(o[i].x * P.etfwt1 + f.x * P.etfwt2, o[i].y * P.etfwt1 + f.y * P.etfwt2);
					}
				}
			} else {
#pragma unroll
				for (int i = 0; i < 8; i++) o[i] = make_float2(nm ? __ldg(nm + t0 + 8 * i) : 1.f, 0.f);
			}
			if (W.lotfT) {
#pragma unroll
				for (int i = 0; i < 8; i++) o[i] = cmulc(o[i], __ldg(W.lotfT + t0 + 8 * i));
			}
		};
#pragma unroll 1
		for (int c = warp; c < 8; c += 4) {
			const int fx = c + (lane & 24);
			float2* p = img + t * LS + fx;
			n64_get<8 * LS>(a, p);
			tf(b, t + 64 * fx);
			dft8(a, -1.f);
			if (c == 0) {  // column 0 is lanes 0..7's: fy's mirror 64 - fy is element 7 - i of lane 8 - t (t = 0: its own 8 - i)
				float2 ym[8];
#pragma unroll
				for (int i = 0; i < 8; i++) {
					const int src = (lane & 24) | ((8 - t) & 7);
					const float2 m = make_float2(__shfl_sync(0xffffffffu, a[7 - i].x, src), __shfl_sync(0xffffffffu, a[7 - i].y, src));
					ym[i] = t ? m : a[(8 - i) & 7];
				}
				if (fx == 0) {
#pragma unroll
					for (int i = 0; i < 8; i++) {
						const float2 y = a[i], m = ym[i];
						const float2 o0 = make_float2(0.5f * (y.x + m.x), 0.5f * (y.y - m.y));
						const float2 o32 = make_float2(0.5f * (y.y + m.y), 0.5f * (m.x - y.x));
						const float2 x0 = cmul(o0, b[i]), x32 = cmul(o32, tf1(t + 8 * i + 64 * 32));
						a[i] = make_float2(x0.x - x32.y, x0.y + x32.x);
					}
				} else {
#pragma unroll
					for (int i = 0; i < 8; i++) a[i] = cmul(a[i], b[i]);
				}
			} else {
#pragma unroll
				for (int i = 0; i < 8; i++) a[i] = cmul(a[i], b[i]);
			}
			dft8(a, 1.f);
			n64_twiddle<1>(a, tw, t);
			n64_put<8 * LS>(p, a);
		}
	}
	__syncthreads();
	// G(y, kx) at digit-reversed rows, column 0 holding G(., 0) + i G(., 32) (both real)
#pragma unroll 1
	for (int t = warp; t < 8; t += 4) {
		float2* p = img + lane + 8 * t * LS;
		n64_get<LS>(a, p);
		dft8(a, 1.f);
		n64_put<LS>(p, a);
	}
	__syncthreads();
	// inverse along fx on 32 complex rows of two real image rows each: row r is
	// A + i B over the full kx range, A and B the Hermitian extensions of rows r
	// and r + 32: at kx < 32 A + i B, at 64 - kx conj A + i conj B
	{
		float2* row = img + lane * LS;
		const int t1 = warp, t2 = warp ? 8 - warp : 4;
		float2 A1[4], B1[4], A2[4], B2[4];
#pragma unroll
		for (int i = 0; i < 4; i++) {
			A1[i] = row[8 * i + t1];
			B1[i] = row[32 * LS + 8 * i + t1];
			A2[i] = row[8 * i + t2];
			B2[i] = row[32 * LS + 8 * i + t2];
		}
		auto lower = [](float2 u, float2 v) { return make_float2(u.x - v.y, u.y + v.x); };
		auto upper = [](float2 u, float2 v) { return make_float2(u.x + v.y, v.x - u.y); };
#pragma unroll
		for (int i = 0; i < 4; i++) {
			a[i] = lower(A1[i], B1[i]);
			b[i] = lower(A2[i], B2[i]);
		}
		if (warp) {  // 64 - (8 i + t1) = 8 (7 - i) + t2 and the reverse
#pragma unroll
			for (int i = 4; i < 8; i++) {
				a[i] = upper(A2[7 - i], B2[7 - i]);
				b[i] = upper(A1[7 - i], B1[7 - i]);
			}
		} else {  // 64 - 8 i = 8 (8 - i), kx = 0 and 32 packed; 64 - (8 i + 4) = 8 (7 - i) + 4
			a[0] = make_float2(A1[0].x, B1[0].x);
			a[4] = make_float2(A1[0].y, B1[0].y);
#pragma unroll
			for (int i = 5; i < 8; i++) a[i] = upper(A1[8 - i], B1[8 - i]);
#pragma unroll
			for (int i = 4; i < 8; i++) b[i] = upper(A2[7 - i], B2[7 - i]);
		}
		dft8(a, 1.f);
		n64_twiddle<1>(a, tw, t1);
		n64_put<8>(row + t1, a);
		dft8(b, 1.f);
		n64_twiddle<1>(b, tw, t2);
		n64_put<8>(row + t2, b);
	}
	__syncthreads();
	// image row s (digit-reversed) is the real part of row s for s < 32, the
	// imaginary part of row s - 32 otherwise
#pragma unroll 1
	for (int t = warp; t < 8; t += 4) {
		float2* p = img + lane * LS + 8 * t;
		n64_get<1>(a, p);
		dft8(a, 1.f);
		n64_put<1>(p, a);
	}
	__syncthreads();
	// (d) pixels (bilinear map) and noise, one thread per pixel
	const int npix = P.npix;
	const int* sidx = P.simap_idx + (P.simap_per_sa ? (size_t)isa * npix * 4 : 0);
	const float* swt = P.simap_wt + (P.simap_per_sa ? (size_t)isa * npix * 4 : 0);
	for (int p = tid; p < npix; p += N64_THREADS) {
		float v = 0.f;
#pragma unroll
		for (int c = 0; c < 4; c++) {
			const int id = __ldg(sidx + 4 * p + c);
			if (id >= 0) {
				const int sr = digrev8(id >> 6);
				const float2 q = img[(sr & 31) * N64_LS + digrev8(id & 63)];
				v = fmaf(__ldg(swt + 4 * p + c), sr < 32 ? q.x : q.y, v);
			}
		}
		v *= W.alpha;
		if (P.accum) v += W.ints[(size_t)isa * npix + p];  // dtrat > 1: the frames so far
		if (W.noisy) {
			PixelRng rng(W.seed, (uint32_t)(isa * npix + p), W.wfs_id, (uint32_t)P.isim);
			v = poisson_draw(rng, v + P.bkgrnd) + P.rne * rng.normal() - P.bkgrndc;
		}
		if (W.ints) W.ints[(size_t)isa * npix + p] = v;
		spix[p] = v;
	}
	__syncthreads();
	// (e) gradients
	if (tid < 32 && W.grad) {
		float pix[8];
#pragma unroll
		for (int q = 0; q < 8; q++) {
			const int p = tid + 32 * q;
			pix[q] = p < npix ? spix[p] : 0.f;
		}
		grad_from_pixels<8>(pix, npix, P.pixpsax, P.pixpsay, P, W.mtche + (size_t)isa * 2 * npix, W.i0sum, isa, tid,
			W.grad, P.nsa);
	}
}

}  // namespace shwfs
