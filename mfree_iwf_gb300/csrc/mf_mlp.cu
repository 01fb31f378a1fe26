// MLP surrogate: an ensemble of small fully connected ReLU networks with BF16 weights
// and activations and FP32 accumulation, trained with Adam on FP32 master weights.
// It maps ring-impact parameters to the solver's rebound velocity, peak von Mises
// stress and contact-force history (mfree_iwf_gb300/surrogate.py).  No counterpart in
// the reference: this is a learned screen placed in front of the solver.
//
// Inference runs the whole network in one tcgen05 kernel (namespace fz).  Per-layer
// forward products run on tcgen05 (namespace tc) where K is a multiple of 64, else on a
// pipelined mma.sync kernel (k_gemm_nt).  The backward products of a training step, a few
// hundred rows per member and a few microseconds each, are 64x64 mma.sync tiles
// (namespace tr) that fill the SMs with small blocks; a layer's weight gradient, its bias
// gradient and the gradient of its input (with the ReLU mask) share one launch.
//
// Training keeps the whole data set on the device.  One training step -- bootstrap
// minibatch gather (each member draws its own rows), forward, MSE, backward, Adam --
// is captured once as a CUDA graph and replayed; the step counter, learning-rate
// schedule and loss history live in device memory, so replays need no host work.
#include <algorithm>
#include <cmath>
#include <cstdint>
#include <cstring>
#include <string>
#include <vector>

#include <unistd.h>

#include <cuda.h>  // CUtensorMap and its enums; the encoder is fetched from the driver at run time
#include <cuda_bf16.h>
#include <cuda_runtime.h>

#include "../../include/mfree_gb300.h"
#include "mf_launch.cuh"

namespace {

typedef __nv_bfloat16 bf16;

struct GemmArgs {
	int M, N, K;
	const bf16* A;
	int lda;
	long long sA;  // member strides, elements
	const bf16* B;
	int ldb;
	long long sB;
	float* C;  // FP32 output, optional
	int ldc;
	long long sC;
	bf16* Cb;  // BF16 output, optional
	int ldcb;
	long long sCb;
	const float* bias;  // per output column, optional
	long long sBias;
	int relu;
	int n_store;  // tcgen05 path: FP32 output columns stored (0: all N), any ldc
	int n_slice;  // tcgen05 path: columns per block when N is split over gridDim.z
};

// The forward product Z = H W^T (A row-major [M][K], B = W row-major [N][K], both
// contiguous in k) as a pipelined kernel: 128x64 output tiles, 8 warps of 32x32,
// K in slices of 32 double-buffered in shared memory by 16-byte cp.async (zero-filled
// past M and K), fragments by ldmatrix, mma.sync m16n8k16 BF16 -> FP32.  Needs K, lda
// and ldb multiples of 8 (the padded widths are multiples of 16).
constexpr int NT_BM = 128, NT_BN = 64, NT_BK = 32, NT_LD = NT_BK + 8;  // 80-byte rows: ldmatrix conflict-free

__device__ __forceinline__ void cp16z(void* smem, const void* gmem, uint32_t bytes) {
	uint32_t sa = (uint32_t)__cvta_generic_to_shared(smem);
	asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;\n" ::"r"(sa), "l"(gmem), "r"(bytes) : "memory");
}
__device__ __forceinline__ void ldsm_x4(uint32_t& r0, uint32_t& r1, uint32_t& r2, uint32_t& r3, const void* p) {
	uint32_t a = (uint32_t)__cvta_generic_to_shared(p);
	asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0,%1,%2,%3}, [%4];\n"
	             : "=r"(r0), "=r"(r1), "=r"(r2), "=r"(r3)
	             : "r"(a));
}

// The training step is a chain of small launches (a dozen of 2 to 8 us), each launched by
// launch_after: 50 steps of 5 members 4.15 -> 3.93 ms.  (Started already when the previous
// kernel's blocks had passed their own wait, 4.54 ms: they take its blocks' places.)
__global__ void __launch_bounds__(256) k_gemm_nt(GemmArgs g) {
	after_previous();
	__shared__ __align__(128) bf16 As[2][NT_BM][NT_LD];
	__shared__ __align__(128) bf16 Bs[2][NT_BN][NT_LD];
	const int z = blockIdx.z;
	const bf16* A = g.A + z * g.sA;
	const bf16* B = g.B + z * g.sB;
	const int m0 = blockIdx.y * NT_BM, n0 = blockIdx.x * NT_BN;
	const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
	const int wm = warp >> 1, wn = warp & 1;  // 4 x 2 warps
	const int gid = lane >> 2, tig = lane & 3;
	auto load = [&](int st, int k0) {
		// A: 128 rows x 4 chunks of 8 elements; B: 64 rows x 4 chunks
#pragma unroll
		for (int r = 0; r < 2; r++) {
			const int e = tid + 256 * r, row = e >> 2, ch = e & 3;
			const int m = m0 + row, k = k0 + ch * 8;
			const bool ok = m < g.M && k < g.K;
			cp16z(&As[st][row][ch * 8], ok ? (const void*)(A + (long long)m * g.lda + k) : (const void*)A, ok ? 16u : 0u);
		}
		{
			const int row = tid >> 2, ch = tid & 3;
			const int n = n0 + row, k = k0 + ch * 8;
			const bool ok = n < g.N && k < g.K;
			cp16z(&Bs[st][row][ch * 8], ok ? (const void*)(B + (long long)n * g.ldb + k) : (const void*)B, ok ? 16u : 0u);
		}
		asm volatile("cp.async.commit_group;\n" ::: "memory");
	};
	float acc[2][4][4];
#pragma unroll
	for (int a = 0; a < 2; a++)
#pragma unroll
		for (int b = 0; b < 4; b++)
#pragma unroll
			for (int c = 0; c < 4; c++) acc[a][b][c] = 0.f;
	const int nk = (g.K + NT_BK - 1) / NT_BK;
	load(0, 0);
	for (int kt = 0; kt < nk; kt++) {
		if (kt + 1 < nk) {
			load((kt + 1) & 1, (kt + 1) * NT_BK);
			asm volatile("cp.async.wait_group 1;\n" ::: "memory");
		} else {
			asm volatile("cp.async.wait_group 0;\n" ::: "memory");
		}
		__syncthreads();
		const int st = kt & 1;
#pragma unroll
		for (int ks = 0; ks < NT_BK; ks += 16) {
			uint32_t af[2][4], bfr[4][2];
#pragma unroll
			for (int mt = 0; mt < 2; mt++) {
				const int r = wm * 32 + mt * 16 + (lane & 15), c = ks + (lane >> 4) * 8;
				ldsm_x4(af[mt][0], af[mt][1], af[mt][2], af[mt][3], &As[st][r][c]);
			}
#pragma unroll
			for (int np = 0; np < 2; np++) {  // two n-tiles of 8 per ldmatrix.x4
				const int r = wn * 32 + np * 16 + (lane & 7) + ((lane >> 4) << 3), c = ks + ((lane >> 3) & 1) * 8;
				ldsm_x4(bfr[2 * np][0], bfr[2 * np][1], bfr[2 * np + 1][0], bfr[2 * np + 1][1], &Bs[st][r][c]);
			}
#pragma unroll
			for (int mt = 0; mt < 2; mt++)
#pragma unroll
				for (int nt = 0; nt < 4; nt++) {
					float* d = acc[mt][nt];
					asm volatile(
					    "mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, "
					    "{%0,%1,%2,%3};\n"
					    : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
					    : "r"(af[mt][0]), "r"(af[mt][1]), "r"(af[mt][2]), "r"(af[mt][3]), "r"(bfr[nt][0]),
					      "r"(bfr[nt][1]));
				}
		}
		__syncthreads();
	}
	// epilogue: each thread holds column pairs (n, n+1) -- stored as one float2 / bf16x2
	// (N, ldc and ldcb are even: the padded widths are multiples of 16)
	float* C = g.C ? g.C + z * g.sC : nullptr;
	bf16* Cb = g.Cb ? g.Cb + z * g.sCb : nullptr;
	const float* bias = g.bias ? g.bias + z * g.sBias : nullptr;
#pragma unroll
	for (int mt = 0; mt < 2; mt++)
#pragma unroll
		for (int nt = 0; nt < 4; nt++)
#pragma unroll
			for (int h = 0; h < 2; h++) {
				const int m = m0 + wm * 32 + mt * 16 + gid + 8 * h;
				const int n = n0 + wn * 32 + nt * 8 + tig * 2;
				if (m >= g.M || n >= g.N) continue;
				float v0 = acc[mt][nt][2 * h], v1 = acc[mt][nt][2 * h + 1];
				if (bias) {
					v0 += bias[n];
					v1 += bias[n + 1];
				}
				if (g.relu) {
					v0 = fmaxf(v0, 0.f);
					v1 = fmaxf(v1, 0.f);
				}
				if (C) *reinterpret_cast<float2*>(C + (long long)m * g.ldc + n) = make_float2(v0, v1);
				if (Cb) *reinterpret_cast<__nv_bfloat162*>(Cb + (long long)m * g.ldcb + n) = __floats2bfloat162_rn(v0, v1);
			}
}

// ---- The forward products on Blackwell's tensor cores: tcgen05.mma with the FP32
// accumulators in tensor memory (TMEM), operands staged by TMA.  Z = H W^T for K a
// multiple of 64 and N <= 256 (the 256-wide layers and the output layer).
//
// One persistent CTA per (slice of the row tiles, member); 10 warps with fixed roles:
//   warp 0     one thread issues the TMA copies: the member's whole W once (N x K,
//              K-major, 128-byte swizzled, resident for all of the CTA's tiles), then
//              128-row x 64-column slices of H through a 3-stage ring;
//   warp 1     allocates TMEM (two accumulators of N columns, so that a tile's
//              epilogue overlaps the next tile's products); one thread issues
//              tcgen05.mma (M = 128, N, K = 16, BF16 x BF16 -> FP32) and tcgen05.commit,
//              which releases each H stage and, after a tile's last slice, hands the
//              accumulator to the epilogue;
//   warps 2-9  the epilogue: warp w reads TMEM lanes 32 (w mod 4) .. +31 -- one tile row
//              per thread -- 32 columns at a time (tcgen05.ld; warps 2-5 the even
//              32-column chunks, warps 6-9 the odd ones), adds the bias, applies ReLU
//              and stores FP32 and/or BF16 rows.  Two warps per scheduler in the
//              epilogue hide each other's TMEM-load and store latencies.
// Every mbarrier wait is bounded: past the limit the thread sets the error word and
// leaves its loop; all threads meet at the end, where warp 1 frees the TMEM.
namespace tc {

constexpr int BM = 128;      // tile rows: one TMEM lane each
constexpr int BK = 64;       // K per stage: 64 BF16 = 128 bytes, one 128-byte swizzle span
constexpr int STAGES = 3;
constexpr int EPI = 8;  // epilogue warps: two per TMEM lane quarter, splitting the columns
constexpr int THREADS = 64 + 32 * EPI;
constexpr uint32_t SPIN_LIMIT = 1u << 24;

__device__ __forceinline__ uint32_t saddr(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }

__device__ __forceinline__ void mbar_init(uint64_t* b, uint32_t count) {
	asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;\n" ::"r"(saddr(b)), "r"(count) : "memory");
}
__device__ __forceinline__ void mbar_expect_tx(uint64_t* b, uint32_t bytes) {
	asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;\n" ::"r"(saddr(b)), "r"(bytes) : "memory");
}
__device__ __forceinline__ void mbar_arrive(uint64_t* b) {
	asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];\n" ::"r"(saddr(b)) : "memory");
}
// Wait until the phase of parity `ph` has completed; false after SPIN_LIMIT tries.
__device__ __forceinline__ bool mbar_wait(uint64_t* b, uint32_t ph) {
	const uint32_t a = saddr(b);
	for (uint32_t it = 0; it < SPIN_LIMIT; it++) {
		uint32_t done;
		asm volatile(
		    "{\n.reg .pred p;\nmbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\nselp.u32 %0, 1, 0, p;\n}\n"
		    : "=r"(done)
		    : "r"(a), "r"(ph)
		    : "memory");
		if (done) return true;
	}
	return false;
}

__device__ __forceinline__ void tma_load_2d(void* dst, const CUtensorMap* tm, int x, int y, uint64_t* bar) {
	asm volatile(
	    "cp.async.bulk.tensor.2d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3}], [%4];\n" ::"r"(
	        saddr(dst)),
	    "l"(reinterpret_cast<uint64_t>(tm)), "r"(x), "r"(y), "r"(saddr(bar))
	    : "memory");
}
__device__ __forceinline__ void tma_load_3d(void* dst, const CUtensorMap* tm, int x, int y, int z, uint64_t* bar) {
	asm volatile(
	    "cp.async.bulk.tensor.3d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3, %4}], [%5];\n" ::"r"(
	        saddr(dst)),
	    "l"(reinterpret_cast<uint64_t>(tm)), "r"(x), "r"(y), "r"(z), "r"(saddr(bar))
	    : "memory");
}

__device__ __forceinline__ void fence_before() { asm volatile("tcgen05.fence::before_thread_sync;\n" ::: "memory"); }
__device__ __forceinline__ void fence_after() { asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory"); }

// Shared-memory matrix descriptor of a K-major operand in the 128-byte-swizzled layout
// that TMA writes: rows of 128 bytes, 8-row groups 1024 bytes apart (stride byte
// offset), descriptor version 1, swizzle mode 2 (128 bytes).
__device__ __forceinline__ uint64_t sw128_desc(uint32_t a) {
	return (uint64_t)((a >> 4) & 0x3FFFu) | ((uint64_t)1 << 16) | ((uint64_t)(1024 >> 4) << 32) | ((uint64_t)1 << 46) |
	       ((uint64_t)2 << 61);
}
// Instruction descriptor of kind::f16: FP32 accumulator, BF16 A and B, both K-major,
// N >> 3 at bit 17, M >> 4 at bit 24.
__host__ __device__ constexpr uint32_t idesc_bf16(int M, int N) {
	return (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(N >> 3) << 17) | ((uint32_t)(M >> 4) << 24);
}

__device__ __forceinline__ void mma_bf16(uint32_t d, uint64_t ad, uint64_t bd, uint32_t idesc, uint32_t acc) {
	asm volatile(
	    "{\n.reg .pred p;\nsetp.ne.b32 p, %4, 0;\ntcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n}\n" ::"r"(d),
	    "l"(ad), "l"(bd), "r"(idesc), "r"(acc)
	    : "memory");
}
__device__ __forceinline__ void mma_commit(uint64_t* bar) {
	asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];\n" ::"r"(saddr(bar))
	             : "memory");
}
__device__ __forceinline__ void tmem_ld32(uint32_t taddr, uint32_t (&r)[32]) {
	asm volatile("tcgen05.ld.sync.aligned.32x32b.x32.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16,%17,%18,%19,%20,%21,%22,%23,%24,%25,%26,%27,%28,%29,%30,%31}, [%32];\n"
	             : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15]), "=r"(r[16]), "=r"(r[17]), "=r"(r[18]), "=r"(r[19]), "=r"(r[20]), "=r"(r[21]), "=r"(r[22]), "=r"(r[23]), "=r"(r[24]), "=r"(r[25]), "=r"(r[26]), "=r"(r[27]), "=r"(r[28]), "=r"(r[29]), "=r"(r[30]), "=r"(r[31])
	             : "r"(taddr));
	asm volatile("tcgen05.wait::ld.sync.aligned;\n" ::: "memory");
}

// dynamic shared memory: the member's W (K/64 blocks of N rows x 128 B), the H stages
// (128 rows x 128 B each), the mbarriers and the TMEM address; +1 KB for the 1 KB
// alignment that the 128-byte swizzle needs
constexpr int STG_ROW = 144;  // epilogue staging row: 32 FP32 (or 32 BF16) + 16 bytes of padding
__host__ __device__ constexpr size_t smem_bytes(int N, int K) {
	return 1024 + (size_t)(K / BK) * N * 128 + (size_t)STAGES * BM * 128 + EPI * 32 * STG_ROW + 8 * (1 + 2 * STAGES + 4) + 16;
}
__host__ __device__ constexpr uint32_t tmem_cols(int N) { return N <= 128 ? 256u : 512u; }

__global__ void __launch_bounds__(THREADS, 1)
    k_gemm_tc(const __grid_constant__ CUtensorMap tmA, const __grid_constant__ CUtensorMap tmW, GemmArgs g,
              int rows_per_member, uint32_t* err) {
	after_previous();
	extern __shared__ uint8_t smem_raw[];
	// gridDim.z > 1: each block takes n_slice of the N columns (rows of W past N are zero)
	const int n0 = blockIdx.z * g.n_slice, N = gridDim.z > 1 ? g.n_slice : g.N;
	const int KB = g.K / BK, G = gridDim.x, z = blockIdx.y;
	const uint32_t raw = saddr(smem_raw);
	uint8_t* sW = smem_raw + (((raw + 1023u) & ~1023u) - raw);
	uint8_t* sA = sW + (size_t)KB * N * 128;
	uint8_t* sStg = sA + (size_t)STAGES * BM * 128;  // EPI epilogue warps x 32 rows x STG_ROW
	uint64_t* w_full = reinterpret_cast<uint64_t*>(sStg + EPI * 32 * STG_ROW);
	uint64_t* a_full = w_full + 1;
	uint64_t* a_empty = a_full + STAGES;
	uint64_t* acc_full = a_empty + STAGES;
	uint64_t* acc_empty = acc_full + 2;
	uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(acc_empty + 2);
	const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
	const int tiles = (g.M + BM - 1) / BM;
	const uint32_t ncols = tmem_cols(N), acc_stride = ncols / 2;

	if (threadIdx.x == 0) {
		mbar_init(w_full, 1);
		for (int s = 0; s < STAGES; s++) {
			mbar_init(a_full + s, 1);
			mbar_init(a_empty + s, 1);
		}
		for (int b = 0; b < 2; b++) {
			mbar_init(acc_full + b, 1);
			mbar_init(acc_empty + b, EPI);  // one arrival per epilogue warp
		}
		asm volatile("fence.mbarrier_init.release.cluster;\n" ::: "memory");
	}
	if (warp == 1) {
		asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;\n" ::"r"(saddr(tmem_slot)),
		             "r"(ncols)
		             : "memory");
		asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;\n" ::: "memory");
	}
	fence_before();
	__syncthreads();
	fence_after();
	const uint32_t tmem = *tmem_slot;
	bool ok = true;

	if (warp == 0) {
		if (lane == 0) {  // TMA producer
			mbar_expect_tx(w_full, (uint32_t)(KB * N * 128));
			for (int kb = 0; kb < KB; kb++) tma_load_3d(sW + (size_t)kb * N * 128, &tmW, kb * BK, n0, z, w_full);
			uint32_t it = 0;
			for (int t = blockIdx.x; t < tiles && ok; t += G)
				for (int kb = 0; kb < KB; kb++, it++) {
					const int s = (int)(it % STAGES);
					const uint32_t use = it / STAGES;
					if (use > 0 && !(ok = mbar_wait(a_empty + s, (use - 1) & 1u))) break;
					mbar_expect_tx(a_full + s, BM * 128);
					tma_load_2d(sA + (size_t)s * BM * 128, &tmA, kb * BK, z * rows_per_member + t * BM, a_full + s);
				}
		}
	} else if (warp == 1) {
		if (lane == 0) {  // MMA issuer
			const uint32_t idesc = idesc_bf16(BM, N);
			ok = mbar_wait(w_full, 0);
			uint32_t it = 0, i = 0;
			for (int t = blockIdx.x; t < tiles && ok; t += G, i++) {
				const uint32_t ab = i & 1u, use = i >> 1;
				if (use > 0 && !(ok = mbar_wait(acc_empty + ab, (use - 1) & 1u))) break;
				fence_after();
				const uint32_t d = tmem + ab * acc_stride;
				for (int kb = 0; kb < KB; kb++, it++) {
					const int s = (int)(it % STAGES);
					if (!(ok = mbar_wait(a_full + s, (it / STAGES) & 1u))) break;
					fence_after();
					const uint32_t a0 = saddr(sA + (size_t)s * BM * 128), b0 = saddr(sW + (size_t)kb * N * 128);
#pragma unroll
					for (int k = 0; k < BK / 16; k++)  // K = 16 per instruction: 32 bytes along the swizzled row
						mma_bf16(d, sw128_desc(a0 + 32u * k), sw128_desc(b0 + 32u * k), idesc, (kb | k) != 0);
					mma_commit(a_empty + s);  // the stage is free once these products are done
				}
				if (ok) mma_commit(acc_full + ab);
			}
		}
	} else {  // epilogue
		// each warp stages its 32 rows x 32 columns in shared memory (rows padded to
		// 144 bytes: the 16-byte accesses of 8 lanes hit distinct banks) and writes
		// them out coalesced -- BF16: 16-byte chunks, 8 rows of 64 bytes per
		// instruction; FP32: one row of up to 128 bytes per instruction, any ldc
		const int q = warp & 3, grp = (warp - 2) >> 2;  // lane quarter; column group (chunks grp, grp + 2, ...)
		uint8_t* stg = sStg + (size_t)(warp - 2) * 32 * STG_ROW;
		const float* bias = g.bias ? g.bias + z * g.sBias + n0 : nullptr;
		float* C = g.C ? g.C + z * g.sC + n0 : nullptr;
		bf16* Cb = g.Cb ? g.Cb + z * g.sCb + n0 : nullptr;
		const int n_end = g.N - n0;  // columns of this block that exist
		const int nst = (g.n_store > 0 ? g.n_store : g.N) - n0;
		uint32_t i = 0;
		for (int t = blockIdx.x; t < tiles && ok; t += G, i++) {
			const uint32_t ab = i & 1u;
			if (!(ok = mbar_wait(acc_full + ab, (i >> 1) & 1u))) break;
			fence_after();
			const int row0 = t * BM + 32 * q;  // this warp's first row
			const uint32_t taddr = tmem + ((uint32_t)(32 * q) << 16) + ab * acc_stride;
			for (int c0 = 32 * grp; c0 < N; c0 += 64) {
				uint32_t r[32];
				tmem_ld32(taddr + (uint32_t)c0, r);  // row 32q + lane, columns c0..c0+31
				float v[32];
#pragma unroll
				for (int j = 0; j < 32; j++) {
					float x = __uint_as_float(r[j]);
					if (bias && c0 + j < n_end) x += bias[c0 + j];
					if (g.relu) x = fmaxf(x, 0.f);
					v[j] = x;
				}
				if (Cb) {
					uint4* srow = reinterpret_cast<uint4*>(stg + lane * STG_ROW);
#pragma unroll
					for (int j = 0; j < 4; j++) {
						__nv_bfloat162 h0 = __floats2bfloat162_rn(v[8 * j], v[8 * j + 1]);
						__nv_bfloat162 h1 = __floats2bfloat162_rn(v[8 * j + 2], v[8 * j + 3]);
						__nv_bfloat162 h2 = __floats2bfloat162_rn(v[8 * j + 4], v[8 * j + 5]);
						__nv_bfloat162 h3 = __floats2bfloat162_rn(v[8 * j + 6], v[8 * j + 7]);
						srow[j] = make_uint4(*reinterpret_cast<uint32_t*>(&h0), *reinterpret_cast<uint32_t*>(&h1),
						                     *reinterpret_cast<uint32_t*>(&h2), *reinterpret_cast<uint32_t*>(&h3));
					}
					__syncwarp();
#pragma unroll
					for (int k = 0; k < 4; k++) {
						const int e = lane + 32 * k, rr = e >> 2, ch = e & 3, m = row0 + rr;
						if (m < g.M && c0 + 8 * ch < n_end)
							*reinterpret_cast<uint4*>(Cb + (long long)m * g.ldcb + c0 + 8 * ch) =
							    *reinterpret_cast<const uint4*>(stg + rr * STG_ROW + 16 * ch);
					}
					__syncwarp();
				}
				if (C) {
					float4* srow = reinterpret_cast<float4*>(stg + lane * STG_ROW);
#pragma unroll
					for (int j = 0; j < 8; j++) srow[j] = make_float4(v[4 * j], v[4 * j + 1], v[4 * j + 2], v[4 * j + 3]);
					__syncwarp();
					if (c0 + lane < nst)
						for (int rr = 0; rr < 32; rr++) {
							const int m = row0 + rr;
							if (m < g.M) C[(long long)m * g.ldc + c0 + lane] = reinterpret_cast<const float*>(stg + rr * STG_ROW)[lane];
						}
					__syncwarp();
				}
			}
			fence_before();
			__syncwarp();
			if (lane == 0) mbar_arrive(acc_empty + ab);
		}
	}
	if (!ok) atomicOr(err, 1u);
	fence_before();
	__syncthreads();
	fence_after();
	if (warp == 1) asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;\n" ::"r"(tmem), "r"(ncols) : "memory");
}

}  // namespace tc

// Fused inference: the whole forward pass of every member in one persistent kernel,
// the hidden activations never leaving the SM.  A pair of CTAs (a cluster, on two SMs)
// takes tiles of 512 rows of one member, two halves of 256 rows, 128 of a half's in each
// CTA (one TMEM accumulator of up to 256 FP32 columns per half and CTA), and runs them
// through all layers:
//   - the epilogue warps write the tile's input rows (FP32 -> BF16, zero padded to the
//     first layer's K) into shared memory in the 128-byte-swizzled K-major layout that
//     a TMA load would produce, so the tensor core reads them as an operand: per 64-wide
//     K chunk the CTA's 256 rows in order (half 0's 128, then half 1's);
//   - the producers (warp 0 of each CTA) stream each layer's BF16 weights, 64-wide K
//     chunks, through a ring of shared-memory stages with TMA, half of the chunk's N rows
//     to each CTA, both reporting to the first CTA's barrier;
//   - the MMA issuer (warp 1 of the first CTA) multiplies with cta_group::2: A = a half's
//     256 rows, B = the chunk's N weight rows, each CTA holding half of both (N padded by
//     zeros to a multiple of 32, the widths that published code uses with M = 256).  A layer's
//     chunks stay in the ring for both halves: half 0's epilogue runs under half 1's
//     products, and half 0's next products under half 1's epilogue;
//   - the epilogue warps (16 in each CTA: four TMEM lane quarters x two halves x two
//     column sets) read their half's accumulator, add the bias, apply ReLU, round to BF16
//     and write the next layer's operand over the current one (whose products are complete
//     by then); the output layer's rows go through shared memory, 16 outputs at a time, for
//     coalesced stores, the next tile's input having been handed on before the last of them.
// Why pairs: the products of a 256 x 256 layer of 256 rows take an SM about 4,500 clocks
// and the epilogue as long, so one has to run under the other.  A CTA by itself has 96 KB
// left for weights beside its activations, less than the 128 KB of one such layer, and
// its halves could be no more than a chunk or two apart; half the weights in each CTA
// make room for a layer and a chunk, and are read from L2 half as often.  262,140 rows,
// 5 members, 6-256-256-256-66: 626 us with single CTAs and both halves in step; 575 with
// the issuer's ring divisions out and 16 epilogue warps; 510 with pairs and an elected
// issuing lane; 422 with 16-column TMEM loads ahead of the conversions and two bias
// copies, 403 with the half loops spelled out (the products alone: 196 us).  What is
// left is each half's own chain: products, epilogue, handing over.
// Only the inputs (in FP32), the weights (from L2: every pair on a member reads the same
// ones) and the outputs move through memory.  The products are the per-layer path's --
// BF16 operands, FP32 accumulation in K order, the bias added in FP32 -- with K padded
// to 64 by zeros.  Every wait is bounded; on a timeout the kernel sets the error word,
// waits (bounded) for its own copies and products in flight, frees the TMEM and returns.
namespace fz {

constexpr int HALF = 128;            // rows of a half in one CTA
constexpr int TILE = 4 * HALF;       // two halves, two CTAs
constexpr int CHUNK = HALF * 128;    // one 64-wide K chunk of a half's rows: 128 rows x 128 bytes
constexpr int EPI = 16;              // epilogue warps: two per half and TMEM lane quarter
constexpr int THREADS = 64 + 32 * EPI;
constexpr int HALF_WARPS = EPI / 2;
constexpr int STAGES = 5;            // weight chunks in shared memory: a layer's (K <= 256) and one more
constexpr uint32_t TMEM_COLS = 512;  // two accumulators of up to 256 columns

struct Maps {
	CUtensorMap w[MF_MLP_MAX_LAYERS];  // per layer: [members][N2][K] BF16, boxes of 64 K x N2 / 2 rows
};
struct Args {
	int L, in, out, rows, kc_max, n_max;
	int N[MF_MLP_MAX_LAYERS], KC[MF_MLP_MAX_LAYERS];  // width (padded to 16); K / 64 (K padded to 64)
	int N2[MF_MLP_MAX_LAYERS];                        // MMA width: N padded to 32
	int b_off[MF_MLP_MAX_LAYERS];
	const float* bias;
	long long b_per;
	const float* x;  // x[z * sx + r * in + c] (sx = 0: one input shared by the members)
	long long sx;
	float* y;  // y[z * sy + r * ldy + c]
	long long sy;
	int ldy;
	int members;
};

// the mbarriers (2 per weight stage, 2 x 2 per half, 1 to drain) and the TMEM address,
// rounded up to 16 bytes
constexpr size_t BAR_BYTES = (8 * (2 * STAGES + 5) + 4 + 15) / 16 * 16;
// shared memory: the operand chunks of the tile, the weight stages, the barriers and each
// half's two copies of a layer's bias (the current one's and the next one's).  (The swizzled operands need 1 KB alignment,
// which the start of dynamic shared memory has; the kernel checks it.)
__host__ __device__ constexpr size_t smem_bytes(int kc_max, int n_max) {
	return (size_t)2 * kc_max * CHUNK + (size_t)STAGES * n_max * 64 + BAR_BYTES + (size_t)4 * n_max * 4;
}
static_assert(smem_bytes(4, 256) <= 227 * 1024, "the widest layers fit");

// the 16-byte unit holding columns col .. col + 7 (col a multiple of 8) of row r of half
// h: K chunk col / 64 (the chunk's 256 rows: half 0, then half 1), unit (col % 64) / 8
// XOR (r % 8) -- the 128-byte swizzle
__device__ __forceinline__ uint4* unit_at(uint8_t* act, int h, int r, int col) {
	const int kc = col >> 6, u = (col >> 3) & 7;
	return reinterpret_cast<uint4*>(act + (size_t)(2 * kc + h) * CHUNK + r * 128 + ((u ^ (r & 7)) << 4));
}
__device__ __forceinline__ uint32_t pack2(float a, float b) {
	__nv_bfloat162 h = __floats2bfloat162_rn(a, b);
	return *reinterpret_cast<uint32_t*>(&h);
}
__device__ __forceinline__ void proxy_fence() { asm volatile("fence.proxy.async.shared::cta;\n" ::: "memory"); }
// max(a, 0) and max(b, 0) rounded to BF16, a in the low half
__device__ __forceinline__ uint32_t pack2_relu(float a, float b) {
	uint32_t d;
	asm("cvt.rn.relu.bf16x2.f32 %0, %1, %2;\n" : "=r"(d) : "f"(b), "f"(a));
	return d;
}
__device__ __forceinline__ void tmem_wait() { asm volatile("tcgen05.wait::ld.sync.aligned;\n" ::: "memory"); }
// 16 columns of the warp's 32 TMEM lanes without waiting (tmem_wait before use)
__device__ __forceinline__ void tmem_ld16_async(uint32_t taddr, uint32_t* r) {
	asm volatile("tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];\n"
	             : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
	             : "r"(taddr));
}

// ---- the pair of CTAs.  Rank 0 issues the products and holds their barriers.
__device__ __forceinline__ uint32_t cluster_rank() {
	uint32_t r;
	asm volatile("mov.u32 %0, %%cluster_ctarank;\n" : "=r"(r));
	return r;
}
__device__ __forceinline__ void cluster_sync() {
	asm volatile("barrier.cluster.arrive.release;\nbarrier.cluster.wait.acquire;\n" ::: "memory");
}
// the address of rank 0's copy of a shared-memory object
__device__ __forceinline__ uint32_t in_rank0(const void* p) {
	uint32_t a;
	asm volatile("mapa.shared::cluster.u32 %0, %1, 0;\n" : "=r"(a) : "r"(tc::saddr(p)));
	return a;
}
// An arrival at a barrier of either CTA, of the default (CTA) scope: what it vouches for --
// this CTA's operand, behind the writers' proxy fences, and its accumulators, behind
// tcgen05.fence -- is only touched again by this SM's own tensor core.  (A release at
// cluster scope waits for all earlier stores of the thread: 602 us instead of 529 for
// 262,140 rows and 5 members of 6-256-256-256-66 when pairs were first in use.)
__device__ __forceinline__ void arrive_cluster(uint32_t bar) {
	asm volatile("mbarrier.arrive.shared::cluster.b64 _, [%0];\n" ::"r"(bar) : "memory");
}
// one lane of the (converged) warp
__device__ __forceinline__ bool elect_one() {
	uint32_t r;
	asm volatile("{\n.reg .pred p;\nelect.sync _|p, 0xffffffff;\nselp.u32 %0, 1, 0, p;\n}\n" : "=r"(r)::"memory");
	return r != 0;
}
// tc::mbar_wait of a whole warp, which agrees on the outcome
__device__ __forceinline__ bool wait_warp(uint64_t* b, uint32_t ph) { return __all_sync(0xffffffffu, tc::mbar_wait(b, ph)); }
// a box to this CTA's shared memory, its bytes reported to `bar` of either CTA
__device__ __forceinline__ void tma_load_pair(void* dst, const CUtensorMap* tm, int x, int y, int z, uint32_t bar) {
	asm volatile(
	    "cp.async.bulk.tensor.3d.cta_group::2.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3, %4}], [%5];\n" ::"r"(
	        tc::saddr(dst)),
	    "l"(reinterpret_cast<uint64_t>(tm)), "r"(x), "r"(y), "r"(z), "r"(bar)
	    : "memory");
}
__device__ __forceinline__ void mma_pair(uint32_t d, uint64_t ad, uint64_t bd, uint32_t idesc, uint32_t acc) {
	asm volatile(
	    "{\n.reg .pred p;\nsetp.ne.b32 p, %4, 0;\ntcgen05.mma.cta_group::2.kind::f16 [%0], %1, %2, %3, p;\n}\n" ::"r"(d),
	    "l"(ad), "l"(bd), "r"(idesc), "r"(acc)
	    : "memory");
}
// the products issued so far -> one arrival at this barrier of both CTAs
__device__ __forceinline__ void commit_pair(uint64_t* bar) {
	asm volatile("tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.multicast::cluster.b64 [%0], %1;\n" ::"r"(
	                 tc::saddr(bar)),
	             "h"((uint16_t)3)
	             : "memory");
}

// barrier over the epilogue threads of half h (named barrier 1 + h); the AND of p over them
__device__ __forceinline__ bool half_all(int h, bool p) {
	uint32_t r;
	asm volatile("{\n.reg .pred q;\nsetp.ne.u32 q, %1, 0;\nbar.red.and.pred q, %2, %3, q;\nselp.u32 %0, 1, 0, q;\n}\n"
	             : "=r"(r)
	             : "r"((uint32_t)p), "r"(1 + h), "n"(32 * HALF_WARPS)
	             : "memory");
	return r != 0;
}

// (a + b, rounded as two FP32 additions)
__device__ __forceinline__ float2 add2(float2 a, float2 b) {
	float2 d;
	asm("{\n.reg .b64 x, y;\nmov.b64 x, {%2, %3};\nmov.b64 y, {%4, %5};\nadd.rn.f32x2 x, x, y;\nmov.b64 {%0, %1}, x;\n}\n"
	    : "=f"(d.x), "=f"(d.y)
	    : "f"(a.x), "f"(a.y), "f"(b.x), "f"(b.y));
	return d;
}
// 16 accumulator columns col0 .. col0 + 15 of row r (in v) -> bias (sb: the layer's in
// shared memory), ReLU, BF16 -> their two 16-byte units of the next operand; columns at or
// past N (the layer's width, a multiple of 16) become zeros up to the next layer's K
__device__ __forceinline__ void hidden_units(uint8_t* act, int h, int r, int col0, int N, const uint32_t* v, const float* sb) {
	uint32_t w[8] = {};
	if (col0 < N) {
		const float4* b4 = reinterpret_cast<const float4*>(sb + col0);
#pragma unroll
		for (int u = 0; u < 4; u++) {
			const float4 b = b4[u];
			const float2 f = add2(make_float2(__uint_as_float(v[4 * u]), __uint_as_float(v[4 * u + 1])), make_float2(b.x, b.y));
			const float2 g = add2(make_float2(__uint_as_float(v[4 * u + 2]), __uint_as_float(v[4 * u + 3])), make_float2(b.z, b.w));
			w[2 * u] = pack2_relu(f.x, f.y);
			w[2 * u + 1] = pack2_relu(g.x, g.y);
		}
	}
	*unit_at(act, h, r, col0) = make_uint4(w[0], w[1], w[2], w[3]);
	*unit_at(act, h, r, col0 + 8) = make_uint4(w[4], w[5], w[6], w[7]);
}

__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(THREADS, 1)
    k_mlp_fused(const __grid_constant__ Maps maps, const Args a, uint32_t* err) {
	using namespace tc;
	extern __shared__ __align__(1024) uint8_t smem_raw[];
	if (saddr(smem_raw) & 1023u) {  // (the driver's layout has always been aligned)
		atomicOr(err, 1u);
		return;
	}
	uint8_t* act = smem_raw;
	const size_t wst = (size_t)a.n_max * 64;  // half of a chunk's rows
	constexpr int S = STAGES;
	const int L = a.L;
	uint8_t* sW = act + (size_t)2 * a.kc_max * CHUNK;
	uint64_t* w_full = reinterpret_cast<uint64_t*>(sW + (size_t)S * wst);  // rank 0's: both CTAs' boxes have landed
	uint64_t* w_empty = w_full + S;
	uint64_t* acc_full = w_empty + S;    // per half: the layer's products are complete
	uint64_t* act_ready = acc_full + 2;  // rank 0's, per half: both CTAs have written the next layer's operand
	uint64_t* fin = act_ready + 2;
	uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(fin + 1);
	float* sbias = reinterpret_cast<float*>(sW + (size_t)S * wst + BAR_BYTES);  // per half and step parity: a layer's bias
	const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
	const uint32_t rank = cluster_rank();
	const int tpm = (a.rows + TILE - 1) / TILE, total = tpm * a.members;
	const int first = blockIdx.x >> 1, pairs = gridDim.x >> 1;

	if (threadIdx.x == 0) {
		for (int s = 0; s < S; s++) {
			mbar_init(w_full + s, 1);
			mbar_init(w_empty + s, 1);
		}
		for (int h = 0; h < 2; h++) {
			mbar_init(acc_full + h, 1);
			mbar_init(act_ready + h, 2 * HALF_WARPS);  // the half's warps of both CTAs
		}
		mbar_init(fin, 1);
		asm volatile("fence.mbarrier_init.release.cluster;\n" ::: "memory");
	}
	if (warp == 1) {
		asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;\n" ::"r"(saddr(tmem_slot)),
		             "r"(TMEM_COLS)
		             : "memory");
		asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;\n" ::: "memory");
	}
	fence_before();
	__syncthreads();
	cluster_sync();
	fence_after();
	const uint32_t tmem = *tmem_slot;  // (all columns: the same address in both CTAs)
	bool ok = true, good = true;

	if (warp == 0) {
		if (lane == 0) {  // weight producer
			// (ring positions are counted: the divisions of an index cost the issuer below more
			// than the products of a chunk)
			int st = 0, loads = 0;
			uint32_t ph = 1;  // parity of the phase that frees the stage (the first round waits for none)
			for (int t = first; t < total && ok; t += pairs) {
				const int z = t % a.members;
				for (int l = 0; l < L && ok; l++) {
					const int rows = a.N2[l] >> 1;
					for (int kc = 0; kc < a.KC[l]; kc++) {
						if (loads == S && !(ok = mbar_wait(w_empty + st, ph))) break;
						if (rank == 0) mbar_expect_tx(w_full + st, 2u * (uint32_t)rows * 128u);
						tma_load_pair(sW + (size_t)st * wst, &maps.w[l], kc * 64, (int)rank * rows, z, in_rank0(w_full + st));
						loads = min(loads + 1, S);
						if (++st == S) {
							st = 0;
							ph ^= 1u;
						}
					}
				}
			}
			// the loads still in flight land, and are used, before the CTA leaves: the last
			// `loads` stages, the newest just before st
			for (int k = 0; k < loads; k++) {
				if (--st < 0) {
					st = S - 1;
					ph ^= 1u;
				}
				if (rank == 0) mbar_wait(w_full + st, ph ^ 1u);
				mbar_wait(w_empty + st, ph ^ 1u);
			}
		}
	} else if (warp == 1) {
		if (rank == 0) {  // MMA issuer: the whole warp walks along, one elected lane issues
			// (issued from a branch of lane 0, a product took 150 clocks to issue whatever its N:
			// its operands are warp-uniform registers, which a divergent branch has to gather)
			uint32_t step = 0, ph = 0;
			int st = 0;  // ring stage of the layer's next chunk (ph: its phase)
			bool issued = false;
			const uint64_t act_d = sw128_desc(saddr(act)), w_d = sw128_desc(saddr(sW));
			const uint32_t w16 = (uint32_t)(wst >> 4);  // (descriptors count 16 bytes)
			for (int t = first; t < total && ok; t += pairs)
				for (int l = 0; l < L && ok; l++, step++) {
					const int KC = a.KC[l], layer_st = st;
					const uint32_t idesc = idesc_bf16(2 * HALF, a.N2[l]);
					for (int h = 0; h < 2 && ok; h++) {
						if (!(ok = wait_warp(act_ready + h, step & 1u))) break;
						st = layer_st;
						uint64_t ad = act_d + (uint32_t)(h * (CHUNK >> 4));
						for (int kc = 0; kc < KC; kc++, ad += 2 * (CHUNK >> 4)) {
							if (h == 0 && !(ok = wait_warp(w_full + st, st < layer_st ? ph ^ 1u : ph))) break;
							fence_after();
							issued = true;
							const uint64_t wd = w_d + (uint32_t)st * w16;
							if (elect_one()) {
#pragma unroll
								for (int k = 0; k < 4; k++)  // K = 16 per instruction: 32 bytes along the swizzled row
									mma_pair(tmem + (uint32_t)(h * 256), ad + 2 * k, wd + 2 * k, idesc, (kc | k) != 0);
								if (h == 1) commit_pair(w_empty + st);  // the stage is free once these products are done
								if (kc == KC - 1) commit_pair(acc_full + h);
							}
							__syncwarp();
							if (++st == STAGES) st = 0;
						}
					}
					if (st <= layer_st) ph ^= 1u;  // (a layer has at most STAGES - 1 chunks)
				}
			if (issued) {  // nothing of the pair's left in the tensor pipes before the TMEM is freed
				if (elect_one())
					asm volatile("tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.b64 [%0];\n" ::"r"(saddr(fin))
					             : "memory");
				__syncwarp();
				wait_warp(fin, 0);
			}
		}
	} else {  // epilogue: half h, TMEM lane quarter q, row r of the CTA's 128, column set `part`
		const int h = (warp - 2) / HALF_WARPS, part = (warp - 2) / 4 % 2, q = warp & 3, r = 32 * q + lane;
		const int et = (threadIdx.x - 64) % (32 * HALF_WARPS);  // thread of the half
		const uint32_t acc = tmem + ((uint32_t)(32 * q) << 16) + (uint32_t)(h * 256);  // this warp's lane quarter
		const uint32_t ready = in_rank0(act_ready + h);
		// tile tt: member tt % members (pairs running side by side read different members'
		// weights), rows (tt / members) * TILE + ...; the first 8 input columns of this
		// thread's row are fetched ahead into registers
		float xp[8];
		auto x_row = [&](int tt, bool& live) {
			const int grow = (tt / a.members) * TILE + (2 * h + (int)rank) * HALF + r;
			live = grow < a.rows;
			return a.x + (tt % a.members) * a.sx + (long long)(live ? grow : 0) * a.in;
		};
		auto x_fetch = [&](int tt) {
			bool live;
			const float* xr = x_row(tt, live);
#pragma unroll
			for (int j = 0; j < 8; j++) xp[j] = part == 0 && live && j < a.in ? xr[j] : 0.f;
		};
		auto x_write = [&](int tt) {  // the input row, BF16, zero padded to the first layer's K
			if (part == 0)
				*unit_at(act, h, r, 0) = make_uint4(pack2(xp[0], xp[1]), pack2(xp[2], xp[3]), pack2(xp[4], xp[5]), pack2(xp[6], xp[7]));
			bool live;
			const float* xr = x_row(tt, live);
			for (int col = part == 0 ? 16 : 8; col < a.KC[0] * 64; col += 16) {
				float f[8];
#pragma unroll
				for (int j = 0; j < 8; j++) f[j] = live && col + j < a.in ? xr[col + j] : 0.f;
				*unit_at(act, h, r, col) = make_uint4(pack2(f[0], f[1]), pack2(f[2], f[3]), pack2(f[4], f[5]), pack2(f[6], f[7]));
			}
			proxy_fence();  // generic-proxy writes, read next by the tensor core
			__syncwarp();
			if (lane == 0) arrive_cluster(ready);
		};
		int t = first;
		if (t < total) {
			x_fetch(t);
			x_write(t);
		}
		uint32_t step = 0;
		for (; t < total && ok; t += pairs) {
			const int z = t % a.members, tn = t + pairs;
			const int row0 = (t / a.members) * TILE + (2 * h + (int)rank) * HALF + 32 * q;  // of this warp
			for (int l = 0; l < L; l++, step++) {
				const bool last = l + 1 == L;
				const float* bias = a.bias + z * a.b_per + a.b_off[l];
				const int N = a.N[l];
				const float bv = et < N ? __ldg(bias + et) : 0.f;
				if (last && tn < total) x_fetch(tn);  // its latency hides under the products
				// the bias to shared memory while the products run; the half's threads agree here on
				// whether the last wait ended well (none waits alone at this barrier)
				float* sb = sbias + (2 * h + (int)(step & 1u)) * a.n_max;
				if (et < N) sb[et] = bv;
				__syncwarp();
				if (!(ok = half_all(h, good))) break;
				good = mbar_wait(acc_full + h, step & 1u);
				__syncwarp();
				fence_after();
				uint32_t va[16], vb[16];
				if (!last) {
					// 16 columns at a time, the half's two warps of a lane quarter in turn, the next
					// ones loading while these are converted
					const int Kn = 64 * a.KC[l + 1];
					if (16 * part < N) tmem_ld16_async(acc + (uint32_t)(16 * part), va);
					for (int c0 = 16 * part; c0 < Kn; c0 += 64) {
						tmem_wait();
						if (c0 + 32 < N) tmem_ld16_async(acc + (uint32_t)(c0 + 32), vb);
						hidden_units(act, h, r, c0, N, va, sb);
						tmem_wait();
						if (c0 + 64 < N) tmem_ld16_async(acc + (uint32_t)(c0 + 64), va);
						hidden_units(act, h, r, c0 + 32, N, vb, sb);
					}
					fence_before();
					proxy_fence();
					__syncwarp();
					if (lane == 0) arrive_cluster(ready);
				} else {
					// 16 outputs at a time through this warp's 2 KB of the last K chunk (free by
					// now): a thread writes its row's, 16-byte units XORed against bank conflicts,
					// and half a warp reads a row.  The next tile's input, handed on when the last
					// accumulators have been read, lies below that chunk, or waits until the half is
					// through with it
					float* stage = reinterpret_cast<float*>(act + (size_t)(2 * (a.kc_max - 1) + h) * CHUNK + (2 * q + part) * 2048);
					const bool early = a.kc_max > a.KC[0];
					bool handed = false;
					auto hand_on = [&] {
						fence_before();
						if (tn < total) x_write(tn);
						handed = true;
					};
					float* yz = a.y + z * a.sy;
					const int c = lane & 15;
					auto put = [&](int c0, const uint32_t* v) {
#pragma unroll
						for (int u = 0; u < 4; u++)
							*reinterpret_cast<uint4*>(stage + 16 * lane + 4 * (u ^ (lane >> 1 & 3))) =
							    make_uint4(v[4 * u], v[4 * u + 1], v[4 * u + 2], v[4 * u + 3]);
						const int f = c0 + c;
						const float b = f < N ? sb[f] : 0.f;
						__syncwarp();
						float* yp = yz + (long long)(row0 + (lane >> 4)) * a.ldy + f;
#pragma unroll
						for (int i = 0; i < 16; i++, yp += 2 * a.ldy) {
							const int rr = 2 * i + (lane >> 4);
							const float o = stage[16 * rr + 4 * ((c >> 2) ^ (i & 3)) + (c & 3)] + b;
							if (f < a.out && row0 + rr < a.rows) *yp = o;
						}
						__syncwarp();
					};
					if (16 * part < a.out) tmem_ld16_async(acc + (uint32_t)(16 * part), va);
					for (int c0 = 16 * part; c0 < a.out; c0 += 64) {
						const int c1 = c0 + 32, c2 = c0 + 64;
						tmem_wait();
						if (c1 < a.out) tmem_ld16_async(acc + (uint32_t)c1, vb);
						if (c2 >= a.out) {
							tmem_wait();
							if (early) hand_on();
						}
						put(c0, va);
						if (c1 < a.out) {
							tmem_wait();
							if (c2 < a.out) tmem_ld16_async(acc + (uint32_t)c2, va);
							put(c1, vb);
						}
					}
					if (!early) half_all(h, true);
					if (!handed) hand_on();
				}
			}
		}
	}
	ok = ok && good;
	if (!ok) atomicOr(err, 1u);
	fence_before();
	__syncthreads();
	cluster_sync();  // (neither CTA frees its TMEM or leaves while the other may still use its memory)
	fence_after();
	__syncwarp();
	if (warp == 1)
		asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;\n" ::"r"(tmem), "r"(TMEM_COLS) : "memory");
}

// weights of one layer for the fused kernel: [members][Np][Kp] BF16, N and K padded to Np (a
// multiple of 32) and Kp (of 64) by zeros
__global__ void k_pack_layer(int members, int N, int K, int Np, int Kp, const bf16* src, long long s_per, bf16* dst,
                             long long d_per) {
	const long long e = (long long)blockIdx.x * blockDim.x + threadIdx.x;
	const long long per = (long long)Np * Kp;
	if (e >= per * members) return;
	const int z = (int)(e / per);
	const long long w = e % per;
	const int o = (int)(w / Kp), i = (int)(w % Kp);
	dst[z * d_per + w] = o < N && i < K ? src[z * s_per + (long long)o * K + i] : __float2bfloat16(0.f);
}

}  // namespace fz

// ---- The backward products of a training step: 64x64 tiles of mma.sync m16n8k16 (BF16
// inputs, FP32 accumulators, K ascending in steps of 16), four warps of 32x32, K in slices
// of 64 through a 3-stage cp.async ring (zero-filled past M, N and K), fragments by
// ldmatrix (transposed where the operand's K does not run along its rows).  At 512 rows
// and five members a 256-wide layer is 80 + 160 tiles: one or two waves of small blocks,
// bound by the latency of their four to eight slices.  Per step of 512 rows and five
// members of 6-256-256-256-66: 428 us with element-wise staged tiles and a launch for
// each product, ReLU mask and bias gradient; 69 us now (this launch 54 + 19 + 19 + 4 -> 7.6 us a layer).
namespace tr {

constexpr int T = 64, LD = T + 8, STAGES = 3, THREADS = 128;  // 144-byte rows: ldmatrix conflict-free
constexpr size_t SMEM = (size_t)STAGES * 2 * T * LD * sizeof(bf16);

__device__ __forceinline__ void ldsm_x4_t(uint32_t& r0, uint32_t& r1, uint32_t& r2, uint32_t& r3, const void* p) {
	uint32_t a = (uint32_t)__cvta_generic_to_shared(p);
	asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0,%1,%2,%3}, [%4];\n"
	             : "=r"(r0), "=r"(r1), "=r"(r2), "=r"(r3)
	             : "r"(a));
}

// 64x64 elements from row r0, column c0 of a row-major matrix of R x C elements
__device__ __forceinline__ void load_tile(bf16* s, const bf16* g, int ld, int r0, int c0, int R, int C) {
#pragma unroll
	for (int e = threadIdx.x; e < T * T / 8; e += THREADS) {
		const int row = e >> 3, col = (e & 7) * 8;
		const bool ok = r0 + row < R && c0 + col < C;  // (C is a multiple of 8)
		cp16z(s + row * LD + col, ok ? (const void*)(g + (long long)(r0 + row) * ld + c0 + col) : (const void*)g, ok ? 16u : 0u);
	}
}

// acc += A(m0.., k) B(k, n0..) over k < K.  AT: A is stored [k][m], else [m][k];
// BT: B is stored [n][k], else [k][n].
template <bool AT, bool BT>
__device__ __forceinline__ void product(const bf16* A, int lda, const bf16* B, int ldb, int m0, int n0, int M, int N, int K,
                                        bf16* smem, float (&acc)[2][4][4]) {
	const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, wm = (warp >> 1) * 32, wn = (warp & 1) * 32;
	const int nk = (K + T - 1) / T;
	auto load = [&](int kt) {
		if (kt < nk) {
			bf16 *As = smem + (kt % STAGES) * 2 * T * LD, *Bs = As + T * LD;
			if (AT) load_tile(As, A, lda, kt * T, m0, K, M);
			else load_tile(As, A, lda, m0, kt * T, M, K);
			if (BT) load_tile(Bs, B, ldb, n0, kt * T, N, K);
			else load_tile(Bs, B, ldb, kt * T, n0, K, N);
		}
		asm volatile("cp.async.commit_group;\n" ::: "memory");  // (empty past the last slice: the waits count groups)
	};
#pragma unroll
	for (int mt = 0; mt < 2; mt++)
#pragma unroll
		for (int nt = 0; nt < 4; nt++)
#pragma unroll
			for (int c = 0; c < 4; c++) acc[mt][nt][c] = 0.f;
#pragma unroll
	for (int kt = 0; kt < STAGES - 1; kt++) load(kt);
	for (int kt = 0; kt < nk; kt++) {
		asm volatile("cp.async.wait_group %0;\n" ::"n"(STAGES - 2) : "memory");
		__syncthreads();  // slice kt has landed, and every warp is done with the slot the next load takes
		load(kt + STAGES - 1);
		const bf16 *As = smem + (kt % STAGES) * 2 * T * LD, *Bs = As + T * LD;
#pragma unroll
		for (int ks = 0; ks < T; ks += 16) {
			uint32_t af[2][4], bq[4][2];
#pragma unroll
			for (int mt = 0; mt < 2; mt++) {
				const int m = wm + mt * 16;
				if (AT)
					ldsm_x4_t(af[mt][0], af[mt][1], af[mt][2], af[mt][3],
					          As + (ks + (lane >> 4) * 8 + (lane & 7)) * LD + m + ((lane >> 3) & 1) * 8);
				else
					ldsm_x4(af[mt][0], af[mt][1], af[mt][2], af[mt][3], As + (m + (lane & 15)) * LD + ks + (lane >> 4) * 8);
			}
#pragma unroll
			for (int np = 0; np < 2; np++) {  // two n-tiles of 8 per ldmatrix.x4
				const int n = wn + np * 16;
				if (BT)
					ldsm_x4(bq[2 * np][0], bq[2 * np][1], bq[2 * np + 1][0], bq[2 * np + 1][1],
					        Bs + (n + (lane & 7) + ((lane >> 4) << 3)) * LD + ks + ((lane >> 3) & 1) * 8);
				else
					ldsm_x4_t(bq[2 * np][0], bq[2 * np][1], bq[2 * np + 1][0], bq[2 * np + 1][1],
					          Bs + (ks + ((lane >> 3) & 1) * 8 + (lane & 7)) * LD + n + (lane >> 4) * 8);
			}
#pragma unroll
			for (int mt = 0; mt < 2; mt++)
#pragma unroll
				for (int nt = 0; nt < 4; nt++) {
					float* d = acc[mt][nt];
					asm volatile(
					    "mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, "
					    "{%0,%1,%2,%3};\n"
					    : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
					    : "r"(af[mt][0]), "r"(af[mt][1]), "r"(af[mt][2]), "r"(af[mt][3]), "r"(bq[nt][0]), "r"(bq[nt][1]));
				}
		}
	}
}

// f(m, n, v0, v1) for every element pair (n, n + 1) that this thread holds
template <class F>
__device__ __forceinline__ void each_pair(int m0, int n0, const float (&acc)[2][4][4], F f) {
	const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
#pragma unroll
	for (int mt = 0; mt < 2; mt++)
#pragma unroll
		for (int nt = 0; nt < 4; nt++)
#pragma unroll
			for (int h = 0; h < 2; h++)
				f(m0 + (warp >> 1) * 32 + mt * 16 + (lane >> 2) + 8 * h, n0 + (warp & 1) * 32 + nt * 8 + (lane & 3) * 2,
				  acc[mt][nt][2 * h], acc[mt][nt][2 * h + 1]);
}

// Sums of 64 columns over `rows` rows of FP32, added row by row: 32-row tiles through a
// cp.async ring, one thread a column.
__device__ __forceinline__ void column_sums(const float* g, int ld, int n0, int N, int rows, float* smem, float* out) {
	constexpr int ROWS = 32;
	const int nt = (rows + ROWS - 1) / ROWS;
	auto load = [&](int t) {
		if (t < nt) {
			float* s = smem + (t % STAGES) * ROWS * T;
#pragma unroll
			for (int e = threadIdx.x; e < ROWS * T / 4; e += THREADS) {
				const int row = e / (T / 4), col = e % (T / 4) * 4;
				const bool ok = t * ROWS + row < rows && n0 + col < N;
				cp16z(s + row * T + col, ok ? (const void*)(g + (long long)(t * ROWS + row) * ld + n0 + col) : (const void*)g,
				      ok ? 16u : 0u);
			}
		}
		asm volatile("cp.async.commit_group;\n" ::: "memory");
	};
#pragma unroll
	for (int t = 0; t < STAGES - 1; t++) load(t);
	float sum = 0.f;
	for (int t = 0; t < nt; t++) {
		asm volatile("cp.async.wait_group %0;\n" ::"n"(STAGES - 2) : "memory");
		__syncthreads();
		load(t + STAGES - 1);
		if (threadIdx.x < T) {
			const float* s = smem + (t % STAGES) * ROWS * T + threadIdx.x;
			const int r1 = min(ROWS, rows - t * ROWS);
			if (r1 == ROWS) {
#pragma unroll
				for (int r = 0; r < ROWS; r++) sum += s[r * T];
			} else {
				for (int r = 0; r < r1; r++) sum += s[r * T];
			}
		}
	}
	if (threadIdx.x < T && n0 + (int)threadIdx.x < N) out[n0 + threadIdx.x] = sum;
}

// One layer backward over a batch, three roles by block: dW = dZ^T H (w_tiles blocks); the
// bias gradient, dZ's column sums (b_tiles blocks); the previous layer's dZ = dZ W where
// its ReLU output H > 0 (the rest).  dZ comes and goes as BF16 (the products' operand)
// and FP32 (the bias gradient's).
struct Bwd {
	int batch, out_p, in_p;
	const bf16 *dz, *H, *W;
	const float* dzf;
	long long sDz, sHin, sW;
	float *gW, *gB;
	long long sGw, sGb;
	bf16* dz_prev;
	float* dzf_prev;
	int w_tiles, b_tiles;
};
__global__ void __launch_bounds__(THREADS) k_backward(Bwd g) {
	after_previous();
	extern __shared__ __align__(16) bf16 smem[];
	const int z = blockIdx.y, nx = (g.in_p + T - 1) / T;
	const bf16 *dz = g.dz + z * g.sDz, *H = g.H + z * g.sHin;
	float acc[2][4][4];
	int t = blockIdx.x;
	if (t < g.w_tiles) {
		const int m0 = t / nx * T, n0 = t % nx * T;
		product<true, false>(dz, g.out_p, H, g.in_p, m0, n0, g.out_p, g.in_p, g.batch, smem, acc);
		float* gW = g.gW + z * g.sGw;
		each_pair(m0, n0, acc, [&](int m, int n, float v0, float v1) {
			if (m < g.out_p && n < g.in_p) *reinterpret_cast<float2*>(gW + (long long)m * g.in_p + n) = make_float2(v0, v1);
		});
		return;
	}
	t -= g.w_tiles;
	if (t < g.b_tiles) {
		column_sums(g.dzf + z * g.sDz, g.out_p, t * T, g.out_p, g.batch, reinterpret_cast<float*>(smem), g.gB + z * g.sGb);
		return;
	}
	t -= g.b_tiles;
	const int m0 = t / nx * T, n0 = t % nx * T;
	product<false, false>(dz, g.out_p, g.W + z * g.sW, g.in_p, m0, n0, g.batch, g.in_p, g.out_p, smem, acc);
	bf16* prev = g.dz_prev + z * g.sDz;
	float* prevf = g.dzf_prev + z * g.sDz;
	each_pair(m0, n0, acc, [&](int m, int n, float v0, float v1) {
		if (m < g.batch && n < g.in_p) {
			const long long e = (long long)m * g.in_p + n;
			const __nv_bfloat162 h = *reinterpret_cast<const __nv_bfloat162*>(H + e);
			v0 = __low2float(h) > 0.f ? v0 : 0.f;
			v1 = __high2float(h) > 0.f ? v1 : 0.f;
			*reinterpret_cast<__nv_bfloat162*>(prev + e) = __floats2bfloat162_rn(v0, v1);
			*reinterpret_cast<float2*>(prevf + e) = make_float2(v0, v1);
		}
	});
}

}  // namespace tr

// Training control block in device memory, read by the graph's kernels on every replay.
struct TrainCtl {
	uint32_t step;   // Adam steps taken so far (inside a step its number is step + 1)
	uint32_t t0;     // step count when the current mf_mlp_train call began
	uint32_t total;  // steps of the current call (cosine schedule length)
	uint32_t n_data;
	float lr0, lr1;
	float* hist;  // [total][members] loss history of the current call
	uint64_t seed;
};

__device__ __forceinline__ uint64_t splitmix64(uint64_t x) {
	x += 0x9E3779B97F4A7C15ull;
	x = (x ^ (x >> 30)) * 0xBF58476D1CE4E5B9ull;
	x = (x ^ (x >> 27)) * 0x94D049BB133111EBull;
	return x ^ (x >> 31);
}

// bootstrap minibatch: member z's row r takes data row splitmix(seed, step, z, r) mod n;
// a warp per row
__global__ void __launch_bounds__(128) k_gather(const TrainCtl* ctl, int rows, int in, int in_p, int out, long long sH0,
                                                long long sY, const float* X, const float* Y, bf16* H0, float* Yb) {
	after_previous();
	const int r = blockIdx.x * 4 + threadIdx.x / 32, z = blockIdx.y, lane = threadIdx.x % 32;
	if (r >= rows) return;
	const uint64_t key = ctl->seed ^ ((uint64_t)(ctl->step + 1) << 20) ^ ((uint64_t)z << 52) ^ (uint64_t)r;
	const uint32_t src = (uint32_t)(splitmix64(key) % ctl->n_data);
	for (int c = lane; c < in_p; c += 32)
		H0[z * sH0 + (long long)r * in_p + c] = __float2bfloat16(c < in ? X[(long long)src * in + c] : 0.f);
	for (int c = lane; c < out; c += 32) Yb[z * sY + (long long)r * out + c] = Y[(long long)src * out + c];
}

// x (FP32 [batch][in] per member, member stride sx; 0 = shared) -> BF16 [batch][in_p], zero padded
__global__ void k_input(int members, int batch, int in, int in_p, const float* x, long long sx, bf16* h, long long sh) {
	const long long e = (long long)blockIdx.x * blockDim.x + threadIdx.x;
	const long long per = (long long)batch * in_p;
	if (e >= per * members) return;
	const int z = (int)(e / per);
	const long long w = e % per;
	const int c = (int)(w % in_p);
	const long long r = w / in_p;
	h[z * sh + w] = __float2bfloat16(c < in ? x[z * sx + r * in + c] : 0.f);
}

// mean squared error of member z over batch x out; dZ = 2 (y_pred - y) / (batch * out)
__global__ void k_mse(int batch, int out, int out_p, const float* yp, long long syp, const float* y, long long sy,
                      float* dz, bf16* dzb, long long sdz, float* loss) {
	after_previous();
	const int z = blockIdx.y;
	float s = 0.f;
	const float inv = 1.f / (float)(batch * out);
	for (int e = blockIdx.x * blockDim.x + threadIdx.x; e < batch * out_p; e += gridDim.x * blockDim.x) {
		const int c = e % out_p, r = e / out_p;
		float d = 0.f;
		if (c < out) {
			const float diff = yp[z * syp + e] - y[z * sy + (long long)r * out + c];
			s += diff * diff;
			d = 2.f * diff * inv;
		}
		dz[z * sdz + e] = d;
		dzb[z * sdz + e] = __float2bfloat16(d);
	}
	__shared__ float red[256];
	red[threadIdx.x] = s;
	__syncthreads();
	for (int o = blockDim.x / 2; o > 0; o >>= 1) {
		if (threadIdx.x < o) red[threadIdx.x] += red[threadIdx.x + o];
		__syncthreads();
	}
	if (threadIdx.x == 0) atomicAdd(&loss[z], red[0] * inv);
}

// Adam (Kingma & Ba 2015) on FP32 master parameters with a cosine learning-rate
// schedule from lr0 to lr1 over the current call; refreshes the BF16 weight copy.  The
// weights' blocks first, then the biases' (one launch); the schedule once per block.
struct AdamSet {
	long long n;
	float* w;
	const float* g;
	float *m, *v;
	bf16* wb;  // optional
};
__global__ void __launch_bounds__(256) k_adam(const TrainCtl* ctl, AdamSet weights, AdamSet biases, unsigned w_blocks) {
	after_previous();
	__shared__ float s_lr, s_c1, s_c2;
	const float b1 = 0.9f, b2 = 0.999f, eps = 1e-8f;
	const bool wts = blockIdx.x < w_blocks;
	const AdamSet& p = wts ? weights : biases;
	const long long q = (long long)(wts ? blockIdx.x : blockIdx.x - w_blocks) * 256 + threadIdx.x;
	const bool in = 4 * q < p.n;  // (n is a multiple of 16, the arrays 16-byte aligned)
	float4 w{}, m{}, v{}, g{};
	if (in) {
		w = ((float4*)p.w)[q];
		m = ((float4*)p.m)[q];
		v = ((float4*)p.v)[q];
		g = ((const float4*)p.g)[q];
	}
	if (threadIdx.x == 0) {
		const uint32_t t = ctl->step + 1;
		const float frac = ctl->total > 1 ? (float)(t - 1 - ctl->t0) / (float)(ctl->total - 1) : 0.f;
		s_lr = ctl->lr1 + 0.5f * (ctl->lr0 - ctl->lr1) * (1.f + cospif(fminf(fmaxf(frac, 0.f), 1.f)));
		s_c1 = 1.f - powf(b1, (float)t);
		s_c2 = 1.f - powf(b2, (float)t);
	}
	__syncthreads();
	if (!in) return;
	const float lr = s_lr, c1 = s_c1, c2 = s_c2;
	auto one = [&](float& wi, float& mi, float& vi, float gi) {
		// (the two contractions spelled out: any other rounding of them, amplified by the
		// steps that follow, ends in other weights)
		mi = __fmaf_rn(1.f - b1, gi, __fmul_rn(b1, mi));
		vi = __fmaf_rn(__fmul_rn(1.f - b2, gi), gi, __fmul_rn(b2, vi));
		wi = wi - lr * (mi / c1) / (sqrtf(vi / c2) + eps);
	};
	one(w.x, m.x, v.x, g.x);
	one(w.y, m.y, v.y, g.y);
	one(w.z, m.z, v.z, g.z);
	one(w.w, m.w, v.w, g.w);
	((float4*)p.m)[q] = m;
	((float4*)p.v)[q] = v;
	((float4*)p.w)[q] = w;
	if (p.wb) {
		((__nv_bfloat162*)p.wb)[2 * q] = __floats2bfloat162_rn(w.x, w.y);
		((__nv_bfloat162*)p.wb)[2 * q + 1] = __floats2bfloat162_rn(w.z, w.w);
	}
}

// the step's losses into the history, and the counters ready for the next step
__global__ void k_step_end(TrainCtl* ctl, float* loss, int members) {
	after_previous();
	const uint32_t row = ctl->step - ctl->t0;
	for (int z = threadIdx.x; z < members; z += blockDim.x) {
		if (ctl->hist && row < ctl->total) ctl->hist[(size_t)row * members + z] = loss[z];
		loss[z] = 0.f;
	}
	__syncthreads();
	if (threadIdx.x == 0) ctl->step += 1;
}

__global__ void k_to_bf16(long long n, const float* a, bf16* b) {
	const long long e = (long long)blockIdx.x * blockDim.x + threadIdx.x;
	if (e < n) b[e] = __float2bfloat16(a[e]);
}

// unpadded outputs [members][rows][out] from the padded last layer [members][rows][out_p]
__global__ void k_output(int members, int rows, int out, int out_p, const float* yp, long long syp, float* y,
                         long long sy) {
	const long long e = (long long)blockIdx.x * blockDim.x + threadIdx.x;
	const long long per = (long long)rows * out;
	if (e >= per * members) return;
	const int z = (int)(e / per);
	const long long w = e % per;
	y[z * sy + w] = yp[z * syp + (w / out) * out_p + (w % out)];
}

inline int pad16(int v) { return (v + 15) / 16 * 16; }
inline int pad32(int v) { return (v + 31) / 32 * 32; }
inline unsigned nblk(long long n, int bs) { return (unsigned)((n + bs - 1) / bs); }

template <class T>
struct Buf {
	T* p = nullptr;
	size_t n = 0;
	cudaError_t alloc(size_t count) {
		free();
		n = count;
		return cudaMalloc(&p, std::max<size_t>(count, 1) * sizeof(T));
	}
	void free() {
		if (p) cudaFree(p);
		p = nullptr;
		n = 0;
	}
	~Buf() { free(); }
};

// portable seeded initialisation: splitmix64 -> uniform in [-1, 1)
struct HostRng {
	uint64_t s;
	uint64_t next() {
		uint64_t x = (s += 0x9E3779B97F4A7C15ull);
		x = (x ^ (x >> 30)) * 0xBF58476D1CE4E5B9ull;
		x = (x ^ (x >> 27)) * 0x94D049BB133111EBull;
		return x ^ (x >> 31);
	}
	float sym() { return (float)((double)(next() >> 11) * (1.0 / 9007199254740992.0) * 2.0 - 1.0); }
};

}  // namespace

struct mf_mlp {
	int members = 0, L = 0, rows = 0, device = 0;
	std::vector<int> dims, pd;            // true and padded widths, L + 1 each
	std::vector<long long> w_off, b_off;  // per-layer offsets inside one member's block
	long long w_per = 0, b_per = 0;       // parameters per member (padded)
	int widest = 0;
	Buf<float> W, Bias, gW, gB, mW, vW, mB, vB;
	Buf<bf16> Wb;
	std::vector<Buf<bf16>> H;  // H[l]: BF16 [members][rows][pd[l]], l = 0..L-1
	Buf<float> Yp;             // FP32 [members][rows][pd[L]]
	Buf<float> dz[2];          // FP32 and
	Buf<bf16> dzb[2];          // BF16 [members][rows][widest]: a layer's output gradient and the one before it
	Buf<float> loss;           // [members]
	Buf<float> Xin, Yin;       // batches from the host: [members][rows][in], [members][rows][out]
	Buf<float> Xst, Yst;       // inference from or to the host: staged rows, st_rows of them
	int st_rows = 0;
	Buf<float> Xd, Yd;         // training set [n][in], [n][out]
	Buf<float> hist;
	Buf<TrainCtl> ctl;
	TrainCtl h_ctl{};
	cudaStream_t stream = nullptr;
	cudaGraphExec_t graph = nullptr;
	uint64_t launches = 0, step_launches = 0;
	std::string err;
	bool tc = false;       // forward products with K % 64 == 0 on tcgen05 (else mma.sync)
	bool fused = true;     // with tc: inference through the fused whole-network kernel when it applies
	int sm_count = 1;
	// fused inference: the BF16 weights re-laid per layer as [members][N][K padded to 64],
	// their tensor maps, and the kernel's shared-memory plan
	Buf<bf16> Wf;
	std::vector<long long> wf_off;
	long long wf_per = 0;
	bool wf_dirty = true;  // Wb changed since Wf was packed
	fz::Maps maps{};
	int fz_kc = 1, fz_n = 16;
	bool fz_fits = false;
	Buf<uint32_t> dev_err; // set by a bounded wait of the tcgen05 GEMM that gave up
	~mf_mlp() {
		if (graph) cudaGraphExecDestroy(graph);
		if (stream) cudaStreamDestroy(stream);
	}
};

namespace {

mf_status mlp_fail(mf_mlp* m, const std::string& what, cudaError_t e) {
	m->err = what + ": " + cudaGetErrorString(e);
	return MF_ERR_CUDA;
}
#define MCK(call)                                             \
	do {                                                      \
		cudaError_t e_ = (call);                              \
		if (e_ != cudaSuccess) return mlp_fail(m, #call, e_); \
	} while (0)

typedef CUresult (*EncodeTiled)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*,
                                const cuuint64_t*, const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave,
                                CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

// cuTensorMapEncodeTiled from the driver (no link-time dependency on libcuda)
EncodeTiled tensor_map_encoder() {
	static EncodeTiled fn = [] {
		void* p = nullptr;
		cudaDriverEntryPointQueryResult q{};
		if (cudaGetDriverEntryPointByVersion("cuTensorMapEncodeTiled", &p, 12000, cudaEnableDefault, &q) != cudaSuccess ||
		    q != cudaDriverEntryPointSuccess)
			p = nullptr;
		return reinterpret_cast<EncodeTiled>(p);
	}();
	return fn;
}

constexpr size_t TC_SMEM_MAX = 227 * 1024;

// The tcgen05 path takes the forward products Z = H W^T whose operands are contiguous
// K-major rows with K a multiple of 64, N a multiple of 16 up to 256, and whose staged
// operands fit the shared memory; H is [members][rows][K], W [N][K] per member.
bool tc_eligible(const mf_mlp* m, const GemmArgs& g) {
	return m->tc && g.K % tc::BK == 0 && g.N % 16 == 0 && g.N <= 256 && g.lda == g.K && g.ldb == g.K &&
	       g.sA == (long long)m->rows * g.K && g.M <= m->rows && tc::smem_bytes(g.N, g.K) <= TC_SMEM_MAX &&
	       (!g.Cb || g.ldcb % 8 == 0) && g.sB % 8 == 0;
}

cudaError_t gemm_tc(mf_mlp* m, GemmArgs g) {
	// With few row tiles (a training batch: 4 a member) one block per tile leaves most SMs
	// idle and loads all of W first; 64-column slices put four times the blocks to work on
	// a quarter of W each (512 rows, 5 members, 256 x 256: 9.5 -> 6.1 us).  From half the
	// SMs on, whole tiles keep W resident and read H once.
	const int row_tiles = (g.M + tc::BM - 1) / tc::BM;
	g.n_slice = row_tiles * m->members <= m->sm_count / 2 && g.N > 64 ? 64 : g.N;
	const int slices = (g.N + g.n_slice - 1) / g.n_slice;
	EncodeTiled enc = tensor_map_encoder();
	CUtensorMap tA, tW;
	// H as [members * rows][K]; boxes of 64 K x 128 rows, 128-byte swizzle, zero fill past the end
	const cuuint64_t dA[2] = {(cuuint64_t)g.K, (cuuint64_t)m->members * m->rows};
	const cuuint64_t sA[1] = {(cuuint64_t)g.K * 2};
	const cuuint32_t bA[2] = {tc::BK, tc::BM}, e1[3] = {1, 1, 1};
	// W as [members][N][K] (member stride sB elements); boxes of 64 K x N rows x 1 member
	const cuuint64_t dW[3] = {(cuuint64_t)g.K, (cuuint64_t)g.N, (cuuint64_t)m->members};
	const cuuint64_t sW[2] = {(cuuint64_t)g.K * 2, (cuuint64_t)g.sB * 2};
	const cuuint32_t bW[3] = {tc::BK, (cuuint32_t)g.n_slice, 1};
	if (enc(&tA, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, const_cast<bf16*>(g.A), dA, sA, bA, e1,
	        CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
	        CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) != CUDA_SUCCESS ||
	    enc(&tW, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 3, const_cast<bf16*>(g.B), dW, sW, bW, e1,
	        CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
	        CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) != CUDA_SUCCESS)
		return cudaErrorInvalidValue;
	const int G = std::max(1, std::min(row_tiles, m->sm_count / m->members));
	launch_after(tc::k_gemm_tc, dim3(G, m->members, slices), tc::THREADS, tc::smem_bytes(g.n_slice, g.K), m->stream,
	                   tA, tW, g, m->rows, m->dev_err.p);
	m->launches++;
	return cudaGetLastError();
}

// Z = H W^T (the padded widths are multiples of 16, so k_gemm_nt takes what tcgen05 does not)
cudaError_t gemm(mf_mlp* m, const GemmArgs& g) {
	if (tc_eligible(m, g)) return gemm_tc(m, g);
	dim3 gnt((g.N + NT_BN - 1) / NT_BN, (g.M + NT_BM - 1) / NT_BM, m->members);
	launch_after(k_gemm_nt, gnt, 256, 0, m->stream, g);
	m->launches++;
	return cudaGetLastError();
}

long long sH(const mf_mlp* m, int l) { return (long long)m->rows * m->pd[l]; }

// The fused inference kernel takes models whose padded widths are all at most 256 (one
// accumulator per half tile, at most four K chunks).
void fused_plan(mf_mlp* m) {
	m->fz_kc = 1;
	m->fz_n = 32;
	bool fits = true;
	for (int l = 0; l < m->L; l++) {
		m->fz_kc = std::max(m->fz_kc, (m->pd[l] + 63) / 64);
		m->fz_n = std::max(m->fz_n, pad32(m->pd[l + 1]));
		fits = fits && m->pd[l] <= 256 && m->pd[l + 1] <= 256;
	}
	m->fz_fits = fits;
}

bool fused_eligible(const mf_mlp* m) { return m->tc && m->fused && m->fz_fits; }

// (re)packs the BF16 weights for the fused kernel and encodes one tensor map per layer:
// [members][Np][Kp] with member stride wf_per, boxes of 64 K x Np / 2 rows x 1 member
mf_status fused_prepare(mf_mlp* m) {
	if (!m->wf_dirty) return MF_OK;
	if (!m->Wf.p) {
		m->wf_off.clear();
		m->wf_per = 0;
		for (int l = 0; l < m->L; l++) {
			m->wf_off.push_back(m->wf_per);
			m->wf_per += (long long)pad32(m->pd[l + 1]) * ((m->pd[l] + 63) / 64 * 64);
		}
		MCK(m->Wf.alloc((size_t)m->wf_per * m->members));
	}
	EncodeTiled enc = tensor_map_encoder();
	for (int l = 0; l < m->L; l++) {
		const int N = m->pd[l + 1], K = m->pd[l], Np = pad32(N), Kp = (K + 63) / 64 * 64;
		const long long per = (long long)Np * Kp * m->members;
		fz::k_pack_layer<<<nblk(per, 256), 256, 0, m->stream>>>(m->members, N, K, Np, Kp, m->Wb.p + m->w_off[l], m->w_per,
		                                                      m->Wf.p + m->wf_off[l], m->wf_per);
		m->launches++;
		MCK(cudaGetLastError());
		const cuuint64_t dW[3] = {(cuuint64_t)Kp, (cuuint64_t)Np, (cuuint64_t)m->members};
		const cuuint64_t sW[2] = {(cuuint64_t)Kp * 2, (cuuint64_t)m->wf_per * 2};
		const cuuint32_t bW[3] = {64, (cuuint32_t)(Np / 2), 1}, e1[3] = {1, 1, 1};
		if (enc(&m->maps.w[l], CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 3, m->Wf.p + m->wf_off[l], dW, sW, bW, e1,
		        CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
		        CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) != CUDA_SUCCESS) {
			m->err = "fused inference: encoding a weight tensor map failed";
			return MF_ERR_CUDA;
		}
	}
	m->wf_dirty = false;
	return MF_OK;
}

// all members over `rows` rows: x[z * sx + r * in + c] -> y[z * sy + r * ldy + c]
cudaError_t fused_forward(mf_mlp* m, const float* x, long long sx, int rows, float* y, long long sy, int ldy) {
	if (rows <= 0) return cudaSuccess;
	fz::Args a{};
	a.L = m->L;
	a.in = m->dims[0];
	a.out = m->dims[m->L];
	a.rows = rows;
	a.kc_max = m->fz_kc;
	a.n_max = m->fz_n;
	for (int l = 0; l < m->L; l++) {
		a.N[l] = m->pd[l + 1];
		a.N2[l] = pad32(m->pd[l + 1]);
		a.KC[l] = (m->pd[l] + 63) / 64;
		a.b_off[l] = (int)m->b_off[l];
	}
	a.bias = m->Bias.p;
	a.b_per = m->b_per;
	a.x = x;
	a.sx = sx;
	a.y = y;
	a.sy = sy;
	a.ldy = ldy;
	a.members = m->members;
	const long long tiles = (long long)(rows + fz::TILE - 1) / fz::TILE * m->members;
	const int G = 2 * (int)std::min<long long>(tiles, std::max(1, m->sm_count / 2));  // pairs of CTAs
	fz::k_mlp_fused<<<G, fz::THREADS, fz::smem_bytes(a.kc_max, a.n_max), m->stream>>>(m->maps, a,
	                                                                                           m->dev_err.p);
	m->launches++;
	return cudaGetLastError();
}

bool device_pointer(const void* p) {
	cudaPointerAttributes at{};
	if (cudaPointerGetAttributes(&at, p) != cudaSuccess) {
		cudaGetLastError();
		return false;
	}
	return at.type == cudaMemoryTypeDevice || at.type == cudaMemoryTypeManaged;
}

// forward pass of all members over `batch` rows already in H[0], the padded outputs into Yp;
// with y: the unpadded ones into y[z * sy + r * out + c] instead, by the last layer itself
// where it runs on tcgen05
cudaError_t forward_layers(mf_mlp* m, int batch, float* y = nullptr, long long sy = 0) {
	const int out = m->dims[m->L];
	bool direct = false;
	for (int l = 0; l < m->L; l++) {
		GemmArgs g{};
		g.M = batch; g.N = m->pd[l + 1]; g.K = m->pd[l];
		g.A = m->H[l].p; g.lda = m->pd[l]; g.sA = sH(m, l);
		g.B = m->Wb.p + m->w_off[l]; g.ldb = m->pd[l]; g.sB = m->w_per;
		g.bias = m->Bias.p + m->b_off[l]; g.sBias = m->b_per;
		if (l + 1 < m->L) {
			g.Cb = m->H[l + 1].p; g.ldcb = m->pd[l + 1]; g.sCb = sH(m, l + 1);
			g.relu = 1;
		} else {
			g.C = m->Yp.p; g.ldc = m->pd[l + 1]; g.sC = sH(m, l + 1);
			if (y && tc_eligible(m, g)) {
				g.C = y; g.ldc = out; g.sC = sy;
				g.n_store = out;
				direct = true;
			}
		}
		cudaError_t e = gemm(m, g);
		if (e != cudaSuccess) return e;
	}
	if (y && !direct) {
		const long long per = (long long)batch * out;
		k_output<<<nblk(per * m->members, 256), 256, 0, m->stream>>>(m->members, batch, out, m->pd[m->L], m->Yp.p, sH(m, m->L), y, sy);
		m->launches++;
	}
	return cudaGetLastError();
}

// gradients of the mean squared error against y (FP32 [members][rows][out]) into gW,
// gB; the per-member losses accumulate into m->loss (zeroed beforehand)
cudaError_t backward_layers(mf_mlp* m, const float* y, int batch) {
	cudaStream_t s = m->stream;
	const int L = m->L;
	const long long sdz = (long long)m->rows * m->widest;  // member stride of dz, dzb
	auto tiles = [](int n) { return (n + tr::T - 1) / tr::T; };
	launch_after(k_mse, dim3(32, m->members), 256, 0, s, batch, m->dims[L], m->pd[L], m->Yp.p, sH(m, L), y,
	                   (long long)m->rows * m->dims[L], m->dz[L & 1].p, m->dzb[L & 1].p, sdz, m->loss.p);
	m->launches++;
	for (int l = L - 1; l >= 0; l--) {
		tr::Bwd g{};
		g.batch = batch; g.out_p = m->pd[l + 1]; g.in_p = m->pd[l];
		g.dz = m->dzb[(l + 1) & 1].p; g.dzf = m->dz[(l + 1) & 1].p; g.sDz = sdz;
		g.H = m->H[l].p; g.sHin = sH(m, l);
		g.W = m->Wb.p + m->w_off[l]; g.sW = m->w_per;
		g.gW = m->gW.p + m->w_off[l]; g.sGw = m->w_per;
		g.gB = m->gB.p + m->b_off[l]; g.sGb = m->b_per;
		g.dz_prev = m->dzb[l & 1].p; g.dzf_prev = m->dz[l & 1].p;
		g.w_tiles = tiles(g.out_p) * tiles(g.in_p);
		g.b_tiles = tiles(g.out_p);
		const int x_tiles = l > 0 ? tiles(batch) * tiles(g.in_p) : 0;
		launch_after(tr::k_backward, dim3(g.w_tiles + g.b_tiles + x_tiles, m->members), tr::THREADS, tr::SMEM, s, g);
		m->launches++;
	}
	return cudaGetLastError();
}

cudaError_t adam_update(mf_mlp* m) {
	const AdamSet w{m->w_per * m->members, m->W.p, m->gW.p, m->mW.p, m->vW.p, m->Wb.p};
	const AdamSet b{m->b_per * m->members, m->Bias.p, m->gB.p, m->mB.p, m->vB.p, nullptr};
	const unsigned wb = nblk(w.n, 1024);
	launch_after(k_adam, wb + nblk(b.n, 1024), 256, 0, m->stream, m->ctl.p, w, b, wb);
	m->launches++;
	return cudaGetLastError();
}

// one full training step on the stream (this sequence is what the graph captures)
cudaError_t train_step_launches(mf_mlp* m) {
	cudaStream_t s = m->stream;
	const int out = m->dims[m->L];
	launch_after(k_gather, dim3((m->rows + 3) / 4, m->members), 128, 0, s, m->ctl.p, m->rows, m->dims[0], m->pd[0],
	                   out, sH(m, 0), (long long)m->rows * out, m->Xd.p, m->Yd.p, m->H[0].p, m->Yin.p);
	m->launches++;
	cudaError_t e;
	if ((e = forward_layers(m, m->rows)) != cudaSuccess) return e;
	if ((e = backward_layers(m, m->Yin.p, m->rows)) != cudaSuccess) return e;
	if ((e = adam_update(m)) != cudaSuccess) return e;
	launch_after(k_step_end, 1, 64, 0, s, m->ctl.p, m->loss.p, m->members);
	m->launches++;
	return cudaGetLastError();
}

// MF_ERR_TIMEOUT (and the error word cleared) when a tcgen05 GEMM gave up a wait
mf_status tc_status(mf_mlp* m) {
	if (!m->tc) return MF_OK;
	uint32_t e = 0;
	MCK(cudaMemcpy(&e, m->dev_err.p, 4, cudaMemcpyDeviceToHost));
	if (!e) return MF_OK;
	MCK(cudaMemset(m->dev_err.p, 0, 4));
	m->err = "tcgen05 GEMM: a bounded wait gave up";
	return MF_ERR_TIMEOUT;
}

void drop_graph(mf_mlp* m) {
	if (m->graph) cudaGraphExecDestroy(m->graph);
	m->graph = nullptr;
}

// parameters of one member, unpadded, layer by layer: W_l [out][in] row-major, then b_l
enum class Walk { GetParams, GetGrads, SetParams };
mf_status param_walk(mf_mlp* m, int member, float* host, Walk mode) {
	size_t o = 0;
	float* Wsrc = mode == Walk::GetGrads ? m->gW.p : m->W.p;
	float* Bsrc = mode == Walk::GetGrads ? m->gB.p : m->Bias.p;
	const bool get = mode != Walk::SetParams;
	for (int l = 0; l < m->L; l++) {
		const size_t wdev = (size_t)member * m->w_per + m->w_off[l];
		const size_t wid = (size_t)m->dims[l] * 4, pitch = (size_t)m->pd[l] * 4;
		if (get) MCK(cudaMemcpy2D(host + o, wid, Wsrc + wdev, pitch, wid, m->dims[l + 1], cudaMemcpyDeviceToHost));
		else MCK(cudaMemcpy2D(Wsrc + wdev, pitch, host + o, wid, wid, m->dims[l + 1], cudaMemcpyHostToDevice));
		o += (size_t)m->dims[l] * m->dims[l + 1];
		const size_t bdev = (size_t)member * m->b_per + m->b_off[l];
		if (get) MCK(cudaMemcpy(host + o, Bsrc + bdev, m->dims[l + 1] * 4, cudaMemcpyDeviceToHost));
		else MCK(cudaMemcpy(Bsrc + bdev, host + o, m->dims[l + 1] * 4, cudaMemcpyHostToDevice));
		o += m->dims[l + 1];
	}
	return MF_OK;
}

}  // namespace

extern "C" {

MF_API mf_status mf_mlp_create(const mf_mlp_config* cfg, mf_mlp** out) {
	if (!cfg || !out) return MF_ERR_ARG;
	*out = nullptr;
	if (cfg->members < 1 || cfg->members > 64 || cfg->n_layers < 1 || cfg->n_layers > MF_MLP_MAX_LAYERS ||
	    cfg->max_batch < 1)
		return MF_ERR_ARG;
	if (cfg->max_batch > 65535) return MF_ERR_CAPACITY;  // gridDim.y of the GEMM tiles and the gather
	for (int l = 0; l <= cfg->n_layers; l++) {
		if (cfg->dims[l] < 1) return MF_ERR_ARG;
		if (cfg->dims[l] > MF_MLP_MAX_WIDTH) return MF_ERR_CAPACITY;
	}
	int ndev = 0;
	if (cudaGetDeviceCount(&ndev) != cudaSuccess || ndev == 0) return MF_ERR_NO_DEVICE;
	if (cfg->device < 0 || cfg->device >= ndev) return MF_ERR_ARG;
	if (cudaSetDevice(cfg->device) != cudaSuccess) return MF_ERR_NO_DEVICE;
	mf_mlp* m = new mf_mlp();
	m->members = cfg->members;
	m->L = cfg->n_layers;
	m->rows = cfg->max_batch;
	m->device = cfg->device;
	for (int l = 0; l <= m->L; l++) {
		m->dims.push_back(cfg->dims[l]);
		m->pd.push_back(pad16(cfg->dims[l]));
		m->widest = std::max(m->widest, m->pd.back());
	}
	for (int l = 0; l < m->L; l++) {
		m->w_off.push_back(m->w_per);
		m->b_off.push_back(m->b_per);
		m->w_per += (long long)m->pd[l + 1] * m->pd[l];
		m->b_per += m->pd[l + 1];
	}
	const long long nw = m->w_per * m->members, nb = m->b_per * m->members;
	// He-uniform weights U(-sqrt(6/fan_in), sqrt(6/fan_in)), zero biases, zero padding
	std::vector<float> hw(nw, 0.f);
	HostRng rng{cfg->seed};
	for (int z = 0; z < m->members; z++)
		for (int l = 0; l < m->L; l++) {
			const float lim = std::sqrt(6.f / (float)m->dims[l]);
			for (int o = 0; o < m->dims[l + 1]; o++)
				for (int i = 0; i < m->dims[l]; i++)
					hw[z * m->w_per + m->w_off[l] + (long long)o * m->pd[l] + i] = lim * rng.sym();
		}
	auto setup = [&]() -> mf_status {
		MCK(cudaStreamCreateWithFlags(&m->stream, cudaStreamNonBlocking));
		Buf<float>* wbufs[] = {&m->W, &m->gW, &m->mW, &m->vW};
		for (auto* b : wbufs) {
			MCK(b->alloc(nw));
			MCK(cudaMemset(b->p, 0, nw * 4));
		}
		Buf<float>* bbufs[] = {&m->Bias, &m->gB, &m->mB, &m->vB};
		for (auto* b : bbufs) {
			MCK(b->alloc(nb));
			MCK(cudaMemset(b->p, 0, nb * 4));
		}
		MCK(m->Wb.alloc(nw));
		MCK(cudaMemcpy(m->W.p, hw.data(), nw * 4, cudaMemcpyHostToDevice));
		k_to_bf16<<<nblk(nw, 256), 256, 0, m->stream>>>(nw, m->W.p, m->Wb.p);
		m->launches++;
		MCK(cudaGetLastError());
		m->H.resize(m->L);
		for (int l = 0; l < m->L; l++) MCK(m->H[l].alloc((size_t)m->members * sH(m, l)));
		const size_t act = (size_t)m->members * m->rows * m->widest;
		MCK(m->Yp.alloc((size_t)m->members * sH(m, m->L)));
		for (int k = 0; k < 2; k++) {
			MCK(m->dz[k].alloc(act));
			MCK(m->dzb[k].alloc(act));
		}
		MCK(cudaFuncSetAttribute(tr::k_backward, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)tr::SMEM));
		MCK(m->loss.alloc(m->members));
		MCK(m->Xin.alloc((size_t)m->members * m->rows * m->dims[0]));
		MCK(m->Yin.alloc((size_t)m->members * m->rows * m->dims[m->L]));
		MCK(m->ctl.alloc(1));
		MCK(m->dev_err.alloc(1));
		MCK(cudaMemset(m->dev_err.p, 0, 4));
		// the tcgen05 forward products on Blackwell (compute capability 10.x), where the
		// driver provides the tensor-map encoder
		int major = 0;
		MCK(cudaDeviceGetAttribute(&major, cudaDevAttrComputeCapabilityMajor, m->device));
		MCK(cudaDeviceGetAttribute(&m->sm_count, cudaDevAttrMultiProcessorCount, m->device));
		m->tc = major == 10 && tensor_map_encoder() != nullptr;
		fused_plan(m);
		if (m->tc) {
			MCK(cudaFuncSetAttribute(tc::k_gemm_tc, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)TC_SMEM_MAX));
			MCK(cudaFuncSetAttribute(fz::k_mlp_fused, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)TC_SMEM_MAX));
		}
		m->h_ctl = TrainCtl{};
		m->h_ctl.seed = cfg->seed * 0x2545F4914F6CDD1Dull + 1;
		MCK(cudaMemcpy(m->ctl.p, &m->h_ctl, sizeof(TrainCtl), cudaMemcpyHostToDevice));
		MCK(cudaStreamSynchronize(m->stream));
		return MF_OK;
	};
	mf_status st = setup();
	if (st != MF_OK) {
		delete m;
		return st;
	}
	*out = m;
	return MF_OK;
}

MF_API void mf_mlp_destroy(mf_mlp* m) {
	if (!m) return;
	cudaSetDevice(m->device);
	delete m;
}

MF_API const char* mf_mlp_last_error(const mf_mlp* m) { return m ? m->err.c_str() : "null model"; }

MF_API mf_status mf_mlp_num_params(const mf_mlp* m, uint64_t* n) {
	if (!m || !n) return MF_ERR_ARG;
	uint64_t t = 0;
	for (int l = 0; l < m->L; l++) t += (uint64_t)m->dims[l + 1] * m->dims[l] + m->dims[l + 1];
	*n = t;
	return MF_OK;
}

MF_API mf_status mf_mlp_get_params(mf_mlp* m, int32_t member, float* host) {
	if (!m || !host || member < 0 || member >= m->members) return MF_ERR_ARG;
	MCK(cudaSetDevice(m->device));
	MCK(cudaStreamSynchronize(m->stream));
	return param_walk(m, member, host, Walk::GetParams);
}

MF_API mf_status mf_mlp_get_grads(mf_mlp* m, int32_t member, float* host) {
	if (!m || !host || member < 0 || member >= m->members) return MF_ERR_ARG;
	MCK(cudaSetDevice(m->device));
	MCK(cudaStreamSynchronize(m->stream));
	return param_walk(m, member, host, Walk::GetGrads);
}

MF_API mf_status mf_mlp_set_params(mf_mlp* m, int32_t member, const float* host) {
	if (!m || !host || member < 0 || member >= m->members) return MF_ERR_ARG;
	MCK(cudaSetDevice(m->device));
	MCK(cudaStreamSynchronize(m->stream));
	mf_status st = param_walk(m, member, const_cast<float*>(host), Walk::SetParams);
	if (st != MF_OK) return st;
	const long long nw = m->w_per * m->members;
	k_to_bf16<<<nblk(nw, 256), 256, 0, m->stream>>>(nw, m->W.p, m->Wb.p);
	m->launches++;
	m->wf_dirty = true;
	MCK(cudaGetLastError());
	MCK(cudaStreamSynchronize(m->stream));
	return MF_OK;
}

MF_API mf_status mf_mlp_gradients(mf_mlp* m, const float* x, const float* y, int32_t batch, float* loss) {
	if (!m || !x || !y || batch < 1) return MF_ERR_ARG;
	if (batch > m->rows) return MF_ERR_CAPACITY;
	MCK(cudaSetDevice(m->device));
	cudaStream_t s = m->stream;
	const int in = m->dims[0], out = m->dims[m->L];
	// [members][batch][...] rows into the [members][rows][...] slots
	MCK(cudaMemcpy2DAsync(m->Xin.p, (size_t)m->rows * in * 4, x, (size_t)batch * in * 4, (size_t)batch * in * 4,
	                      m->members, cudaMemcpyDefault, s));
	MCK(cudaMemcpy2DAsync(m->Yin.p, (size_t)m->rows * out * 4, y, (size_t)batch * out * 4, (size_t)batch * out * 4,
	                      m->members, cudaMemcpyDefault, s));
	MCK(cudaMemsetAsync(m->loss.p, 0, m->members * 4, s));
	const long long per = (long long)batch * m->pd[0];
	k_input<<<nblk(per * m->members, 256), 256, 0, s>>>(m->members, batch, in, m->pd[0], m->Xin.p,
	                                                    (long long)m->rows * in, m->H[0].p, sH(m, 0));
	m->launches++;
	MCK(cudaGetLastError());
	MCK(forward_layers(m, batch));
	MCK(backward_layers(m, m->Yin.p, batch));
	if (loss) MCK(cudaMemcpyAsync(loss, m->loss.p, m->members * 4, cudaMemcpyDefault, s));
	MCK(cudaStreamSynchronize(s));
	return MF_OK;
}

MF_API mf_status mf_mlp_set_data(mf_mlp* m, const float* x, const float* y, int32_t n) {
	if (!m || !x || !y || n < 1) return MF_ERR_ARG;
	MCK(cudaSetDevice(m->device));
	MCK(cudaStreamSynchronize(m->stream));
	const int in = m->dims[0], out = m->dims[m->L];
	if (m->Xd.n < (size_t)n * in || m->Yd.n < (size_t)n * out) {
		drop_graph(m);  // the captured gather holds the data pointers
		MCK(m->Xd.alloc((size_t)n * in));
		MCK(m->Yd.alloc((size_t)n * out));
	}
	MCK(cudaMemcpy(m->Xd.p, x, (size_t)n * in * 4, cudaMemcpyDefault));
	MCK(cudaMemcpy(m->Yd.p, y, (size_t)n * out * 4, cudaMemcpyDefault));
	m->h_ctl.n_data = (uint32_t)n;
	return MF_OK;
}

MF_API mf_status mf_mlp_train(mf_mlp* m, int32_t steps, float lr0, float lr1, float* loss_history) {
	if (!m || steps < 0 || !(lr0 >= 0.f) || !(lr1 >= 0.f)) return MF_ERR_ARG;
	if (!m->h_ctl.n_data) {
		m->err = "mf_mlp_train: no training data (call mf_mlp_set_data first)";
		return MF_ERR_STATE;
	}
	if (!steps) return MF_OK;
	MCK(cudaSetDevice(m->device));
	cudaStream_t s = m->stream;
	MCK(cudaStreamSynchronize(s));
	if (m->hist.n < (size_t)steps * m->members) MCK(m->hist.alloc((size_t)steps * m->members));
	// the device step counter is authoritative; rewrite the schedule fields around it
	TrainCtl cur;
	MCK(cudaMemcpy(&cur, m->ctl.p, sizeof(TrainCtl), cudaMemcpyDeviceToHost));
	m->h_ctl.step = cur.step;
	m->h_ctl.t0 = cur.step;
	m->h_ctl.total = (uint32_t)steps;
	m->h_ctl.lr0 = lr0;
	m->h_ctl.lr1 = lr1;
	m->h_ctl.hist = m->hist.p;
	MCK(cudaMemcpy(m->ctl.p, &m->h_ctl, sizeof(TrainCtl), cudaMemcpyHostToDevice));
	if (!m->graph) {
		cudaGraph_t g = nullptr;
		MCK(cudaStreamBeginCapture(s, cudaStreamCaptureModeThreadLocal));
		const uint64_t before = m->launches;
		cudaError_t e = train_step_launches(m);
		cudaError_t e2 = cudaStreamEndCapture(s, &g);
		m->step_launches = m->launches - before;
		m->launches = before;
		if (e != cudaSuccess || e2 != cudaSuccess) {
			if (g) cudaGraphDestroy(g);
			return mlp_fail(m, "capturing the training step", e != cudaSuccess ? e : e2);
		}
		e = cudaGraphInstantiate(&m->graph, g, 0);
		cudaGraphDestroy(g);
		if (e != cudaSuccess) {
			m->graph = nullptr;
			return mlp_fail(m, "cudaGraphInstantiate", e);
		}
	}
	m->wf_dirty = true;
	MCK(cudaMemsetAsync(m->loss.p, 0, m->members * 4, s));  // (each step leaves it zero for the next)
	for (int t = 0; t < steps; t++) MCK(cudaGraphLaunch(m->graph, s));
	m->launches += m->step_launches * (uint64_t)steps;
	if (loss_history)
		MCK(cudaMemcpyAsync(loss_history, m->hist.p, (size_t)steps * m->members * 4, cudaMemcpyDefault, s));
	MCK(cudaStreamSynchronize(s));
	return tc_status(m);
}

// Rows of a chunk of inference between host arrays: as many as STAGE_BYTES of staging
// hold (kept with the model, grown as calls ask for it), never fewer than max_batch, whose
// buffers are there anyway and serve where the memory for more is not.  (A launch of 512
// rows for 5 members fills 10 of 152 SMs, and each chunk's copies wait for it: 10,000 rows
// in 20 chunks of 512 took 836 us, in one 137.)
constexpr size_t STAGE_BYTES = 64u << 20;
static int stage_chunk(mf_mlp* m, int n) {
	const size_t row = (size_t)(m->dims[0] + m->members * m->dims[m->L]) * 4;
	const int want = (int)std::min<size_t>((size_t)n, STAGE_BYTES / row);
	if (want <= m->rows) return m->rows;
	if (want > m->st_rows) {
		m->st_rows = 0;
		if (m->Xst.alloc((size_t)want * m->dims[0]) != cudaSuccess ||
		    m->Yst.alloc((size_t)want * m->members * m->dims[m->L]) != cudaSuccess) {
			cudaGetLastError();
			m->Xst.free();
			m->Yst.free();
			return m->rows;
		}
		m->st_rows = want;
	}
	return want;
}

// Makes the pages of host memory that is about to be copied into present by a write to each.
static void touch_pages(char* p, size_t bytes) {
	const size_t page = (size_t)sysconf(_SC_PAGESIZE);
	volatile char* c = p;
	for (size_t o = 0; o < bytes; o += page) c[o] = 0;
	if (bytes) c[bytes - 1] = 0;
}

// Rows r0 .. r0 + b of every member's result, src [members][b][out] on the device, into the
// host's y [members][n][out].  The pages are made present first, while the kernels run: a copy
// into new host memory otherwise takes a fault of the device a page (30,000 rows x 5 members
// x 66, 40 MB: 32.4 ms, 1.8 this way).  Not for a result over the input: a write could come
// before the copy that reads the input (those pages are present anyway).  Several chunks: a
// strided copy into pageable memory reaches a whole pitch behind its last row's start, from
// the second chunk on past the end of y, which may be nobody's memory; the last member's rows
// go in a copy of their own.
static cudaError_t result_to_host(mf_mlp* m, const float* x, int n, float* y, int r0, int b, const float* src) {
	const size_t row = (size_t)m->dims[m->L] * 4, part = b * row, pitch = n * row;
	char* dst = reinterpret_cast<char*>(y) + r0 * row;
	const uintptr_t xa = (uintptr_t)x, ya = (uintptr_t)y;
	if (xa + (size_t)n * m->dims[0] * 4 <= ya || ya + m->members * pitch <= xa)
		for (int z = 0; z < m->members; z++) touch_pages(dst + z * pitch, part);
	const char* from = reinterpret_cast<const char*>(src);
	if (b == n) return cudaMemcpyAsync(dst, from, m->members * part, cudaMemcpyDefault, m->stream);
	const int strided = m->members - 1;
	cudaError_t e = cudaSuccess;
	if (strided) e = cudaMemcpy2DAsync(dst, pitch, from, part, part, strided, cudaMemcpyDefault, m->stream);
	if (e != cudaSuccess) return e;
	return cudaMemcpyAsync(dst + strided * pitch, from + strided * part, part, cudaMemcpyDefault, m->stream);
}

MF_API mf_status mf_mlp_predict(mf_mlp* m, const float* x, int32_t n, float* y) {
	if (!m || n < 0 || (n > 0 && (!x || !y))) return MF_ERR_ARG;
	MCK(cudaSetDevice(m->device));
	cudaStream_t s = m->stream;
	const int in = m->dims[0], out = m->dims[m->L];
	if (n > 0 && fused_eligible(m)) {
		mf_status st = fused_prepare(m);
		if (st != MF_OK) return st;
		const bool xd = device_pointer(x), yd = device_pointer(y);
		if (xd && yd) {  // one launch over every row, straight from x into y
			MCK(fused_forward(m, x, 0, n, y, (long long)n * out, out));
		} else {
			const int chunk = stage_chunk(m, n);
			float *xst = chunk > m->rows ? m->Xst.p : m->Xin.p, *yst = chunk > m->rows ? m->Yst.p : m->Yin.p;
			for (int r0 = 0; r0 < n; r0 += chunk) {
				const int b = std::min(chunk, n - r0);
				const float* xs = x + (size_t)r0 * in;
				if (!xd) {
					MCK(cudaMemcpyAsync(xst, xs, (size_t)b * in * 4, cudaMemcpyDefault, s));
					xs = xst;
				}
				if (yd) {
					MCK(fused_forward(m, xs, 0, b, y + (size_t)r0 * out, (long long)n * out, out));
				} else {
					MCK(fused_forward(m, xs, 0, b, yst, (long long)b * out, out));
					MCK(result_to_host(m, x, n, y, r0, b, yst));
				}
			}
		}
		MCK(cudaStreamSynchronize(s));
		return tc_status(m);
	}
	// the layers' own path: passes of max_batch rows, each straight into y or into the staging
	const bool yd = n > 0 && device_pointer(y);
	const int chunk = yd || n == 0 ? n : stage_chunk(m, n);
	for (int r0 = 0; r0 < n; r0 += chunk) {
		const int b = std::min(chunk, n - r0);
		float* yo = yd ? y : chunk > m->rows ? m->Yst.p : m->Yin.p;
		for (int q0 = 0; q0 < b; q0 += m->rows) {
			const int c = std::min(m->rows, b - q0);
			MCK(cudaMemcpyAsync(m->Xin.p, x + (size_t)(r0 + q0) * in, (size_t)c * in * 4, cudaMemcpyDefault, s));
			const long long per = (long long)c * m->pd[0];
			k_input<<<nblk(per * m->members, 256), 256, 0, s>>>(m->members, c, in, m->pd[0], m->Xin.p, 0, m->H[0].p, sH(m, 0));
			m->launches++;
			MCK(cudaGetLastError());
			MCK(forward_layers(m, c, yo + (size_t)q0 * out, (long long)b * out));
		}
		if (!yd) MCK(result_to_host(m, x, n, y, r0, b, yo));
	}
	MCK(cudaStreamSynchronize(s));
	return tc_status(m);
}

MF_API mf_status mf_mlp_launch_count(const mf_mlp* m, uint64_t* launches) {
	if (!m || !launches) return MF_ERR_ARG;
	*launches = m->launches;
	return MF_OK;
}

MF_API mf_status mf_mlp_get_stream(const mf_mlp* m, void** stream) {
	if (!m || !stream) return MF_ERR_ARG;
	*stream = (void*)m->stream;
	return MF_OK;
}

MF_API mf_status mf_mlp_set_option(mf_mlp* m, const char* key, int64_t value) {
	if (!m || !key) return MF_ERR_ARG;
	if (!strcmp(key, "tcgen05")) {
		if (value != 0 && value != 1) return MF_ERR_ARG;
		int major = 0;
		MCK(cudaDeviceGetAttribute(&major, cudaDevAttrComputeCapabilityMajor, m->device));
		if (value && !(major == 10 && tensor_map_encoder())) {
			m->err = "tcgen05: needs a compute capability 10.x device and the driver's tensor-map encoder";
			return MF_ERR_STATE;
		}
		if (value && !m->tc) {
			MCK(cudaFuncSetAttribute(tc::k_gemm_tc, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)TC_SMEM_MAX));
			MCK(cudaFuncSetAttribute(fz::k_mlp_fused, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)TC_SMEM_MAX));
		}
		m->tc = value != 0;
		drop_graph(m);  // the captured training step holds the old launches
		return MF_OK;
	}
	if (!strcmp(key, "fused")) {
		if (value != 0 && value != 1) return MF_ERR_ARG;
		m->fused = value != 0;
		return MF_OK;
	}
	m->err = std::string("unknown option ") + key;
	return MF_ERR_ARG;
}

MF_API mf_status mf_mlp_get_option(const mf_mlp* m, const char* key, int64_t* value) {
	if (!m || !key || !value) return MF_ERR_ARG;
	if (!strcmp(key, "tcgen05")) {
		*value = m->tc ? 1 : 0;
		return MF_OK;
	}
	if (!strcmp(key, "fused")) {  // 1 when predict runs the fused kernel
		*value = fused_eligible(m) ? 1 : 0;
		return MF_OK;
	}
	return MF_ERR_ARG;
}

}  // extern "C"
