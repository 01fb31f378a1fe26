// Updated-Lagrangian (Gray-Monaghan) SPH time-step kernels.
//
// One derivative evaluation of the reference (body::compute_time_derivatives for
// particle_ul, body.h:125-148) rebuilds the cell grid, sorts the particles by cell
// hash, builds Verlet lists, evaluates the kernel per pair and runs the action list
// (rings.cpp:86-96).  Here that becomes, per RK4 stage, for all bodies at once:
//
//   ul_bbox      per-body bounding box and h_max        (grid.h:83-104)
//   ul_geom      per-body cell geometry, cell offsets   (grid.h:105-115)
//   ul_hash      global cell key per row                (grid.h:35-41)
//   CUB radix sort of (key, row)                        (body.h:137)
//   ul_gather    the cell start table, empty cells filled from the right (grid.h:48-81);
//                the rows' stage state in cell order, with the per-particle actions
//                EOS (material.h:37-64), artificial stress (correctors.h:37-81) and
//                integration weights (riemann_integration.h:28-33) fused in
//   ul_pair      the row's cells of the stencil (FP64: 3x3 cells of the reference grid,
//                grid.h:117-177, four lanes a row; mixed: up to 5x5 half-size cells, one
//                thread a row, or eight lanes where rows are few): tests the candidates,
//                evaluates W/gradW (kernel.cpp:20-55) and every pair
//                action at once -- derive_stress_monaghan (derivatives.h:378-443),
//                derive_velocity (:32-66), artificial viscosity (correctors.h:83-137),
//                XSPH (:139-169) -- then the per-particle actions Jaumann rate
//                (material.h:66-100), continuity, momentum and advection
//                (cont_mech.h:32-49,108-142) and the RK4 update (rk4.h:52-108).
//
// Neighbour lists are never stored: the pair kernel re-derives them from the cell
// table with the reference's predicate r^2 <= 4 h_i^2 + eps, evaluated without FMA
// contraction so the neighbour sets are the reference's, bit for bit.
#include <cub/device/device_radix_sort.cuh>

#include "mf_common.cuh"
#include "mf_launch.cuh"
#include "mf_kernels.h"

using namespace mfk;
using mfk_host::BodyParams;
using mfk_host::Geom;
using mfk_host::ULArgs;

namespace MF_NS {
namespace {

enum : uint32_t {
	A_RIEMANN = 1u << 1,
	A_EOS = 1u << 2,
	A_ART_STRESS = 1u << 3,
	A_STRESS_MGHN = 1u << 4,
	A_DERIVE_VEL = 1u << 5,
	A_ART_VISC = 1u << 6,
	A_XSPH = 1u << 7,
	A_JAUMANN = 1u << 8,
	A_CONTINUITY = 1u << 9,
	A_MOMENTUM_UL = 1u << 10,
	A_ADVECTION = 1u << 11,
	A_GOD_CONT = mfk_host::FLAG_GODUNOV_CONTINUITY,
	A_GOD_MOM = mfk_host::FLAG_GODUNOV_MOMENTUM,
	// the whole Gray-Monaghan list (rings.cpp:86-96): the mixed pair pass is compiled for it,
	// so that no pair tests a flag
	A_MONAGHAN = A_RIEMANN | A_EOS | A_ART_STRESS | A_STRESS_MGHN | A_DERIVE_VEL | A_ART_VISC | A_XSPH | A_JAUMANN |
	             A_CONTINUITY | A_MOMENTUM_UL | A_ADVECTION,
};

// Cell-ordered record of one particle's stage state plus per-particle derived
// quantities.  FP64 form: 16 doubles = 128 bytes, loaded as 8 x 16 B.  With the
// Godunov actions (which exclude the artificial stress) Rxx holds the pressure p and
// Rxy the stress Syy itself.
struct __align__(16) Rec64 {
	double x, y, vx, vy;
	double m, h, rho, sxx;   // sxx = Sxx - p
	double sxy, syy, Rxx, Rxy;
	double Ryy, c, qw, rho21;  // c = sqrt(K/rho), qw = m/rho (or the stored weight), rho21 = 1/rho^2
};
// Mixed form: positions and velocities as float-float, the rest FP32: five 16-byte parts.
struct __align__(16) Rec32 {
	FF x, y, vx, vy;
	float m, h, rho, sxx;
	float sxy, syy, Rxx, Rxy;
	float Ryy, c, qw, rho21;
};

__device__ __forceinline__ Rec64 load_rec(const Rec64* p) {
	Rec64 r;
	const double2* s = reinterpret_cast<const double2*>(p);
	double2* d = reinterpret_cast<double2*>(&r);
#pragma unroll
	for (int i = 0; i < 8; i++) d[i] = __ldg(s + i);
	return r;
}
// The mixed records are stored as five float4 arrays of n rows (16-byte part f of row k at
// rec[f * n + k]): the 32 lanes of a warp reach the same part of mostly consecutive rows,
// 4 cache lines an access where 80-byte records spread it over 20 (with them the L1 data
// pipe was 60 % busy in the pair pass).
__device__ __forceinline__ Rec32 load_rec(const float4* rec, size_t n, uint32_t k, float4 head) {
	Rec32 r;
	float4* d = reinterpret_cast<float4*>(&r);
	d[0] = head;  // (x, y: already loaded)
#pragma unroll
	for (int f = 1; f < 5; f++) d[f] = __ldg(rec + f * n + k);
	return r;
}
__device__ __forceinline__ void store_rec(float4* rec, size_t n, uint32_t k, const Rec32& r) {
	const float4* s = reinterpret_cast<const float4*>(&r);
#pragma unroll
	for (int f = 0; f < 5; f++) rec[f * n + k] = s[f];
}

// ------------------------------------------------------- per-body failures
// With per-body masking (failed != nullptr) an error found on a row fails the row's
// body alone; without it, it fails the step (the status word).
__device__ __forceinline__ void fail_body(uint32_t* failed, DevStatus* st, uint32_t bit, uint32_t row, uint32_t body) {
	if (failed) atomicOr(&failed[body], bit);
	else raise(st, bit, row);
}
__device__ __forceinline__ bool is_failed(const uint32_t* failed, uint32_t body) {
	return failed && *(volatile const uint32_t*)&failed[body];
}

// --------------------------------------------------------------- grid build
__global__ void k_bbox_init(uint32_t nb, unsigned long long* bb) {
	after_previous();
	uint32_t b = blockIdx.x * blockDim.x + threadIdx.x;
	if (b >= nb) return;
	bb[6 * b + 0] = ord_encode(1.7976931348623157e308);   // min x
	bb[6 * b + 1] = ord_encode(1.7976931348623157e308);   // min y
	bb[6 * b + 2] = ord_encode(-1.7976931348623157e308);  // max x
	bb[6 * b + 3] = ord_encode(-1.7976931348623157e308);  // max y
	bb[6 * b + 4] = ord_encode(-1.7976931348623157e308);  // h_max
	bb[6 * b + 5] = ord_encode(0.);                       // max |v|^2 (mixed form)
}

// Bounding box and h_max per body (grid.h:83-104).  Rows of a body are contiguous,
// so a warp whose rows share one body reduces in registers and issues one atomic
// per quantity.  The mixed form also takes the largest speed, which sizes cells that
// stay valid for all four stages of a step.
__global__ void k_bbox(uint32_t n, const double* __restrict__ x, const double* __restrict__ y,
                       const double* __restrict__ h, const double* __restrict__ vx, const double* __restrict__ vy,
                       const uint32_t* __restrict__ body_of, int mixed, unsigned long long* bb,
                       const uint32_t* failed) {
	after_previous();
	uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
	bool valid = i < n;
	uint32_t b = valid ? body_of[i] : 0xffffffffu;
	if (valid && is_failed(failed, b)) {  // a failed body's rows are left out
		valid = false;
		b = 0xffffffffu;
	}
	unsigned long long mnx = ~0ull, mny = ~0ull, mxx = 0ull, mxy = 0ull, mh = 0ull, mv = 0ull;
	if (valid) {
		mnx = mxx = ord_encode(x[i]);
		mny = mxy = ord_encode(y[i]);
		mh = ord_encode(h[i]);
		// the square of the speed (the square root once per body: a correctly rounded root
		// is monotonic, so the root of the largest square is the largest root)
		mv = mixed ? ord_encode(vx[i] * vx[i] + vy[i] * vy[i]) : ord_encode(0.);
	}
	uint32_t lane = threadIdx.x & 31;
	uint32_t b0 = __shfl_sync(0xffffffffu, b, 0);
	bool uniform = __all_sync(0xffffffffu, b == b0) && b0 != 0xffffffffu;
	if (uniform) {
#pragma unroll
		for (int o = 16; o > 0; o >>= 1) {
			mnx = min(mnx, __shfl_xor_sync(0xffffffffu, mnx, o));
			mny = min(mny, __shfl_xor_sync(0xffffffffu, mny, o));
			mxx = max(mxx, __shfl_xor_sync(0xffffffffu, mxx, o));
			mxy = max(mxy, __shfl_xor_sync(0xffffffffu, mxy, o));
			mh = max(mh, __shfl_xor_sync(0xffffffffu, mh, o));
			mv = max(mv, __shfl_xor_sync(0xffffffffu, mv, o));
		}
		if (lane == 0) {
			atomicMin(&bb[6 * b0 + 0], mnx);
			atomicMin(&bb[6 * b0 + 1], mny);
			atomicMax(&bb[6 * b0 + 2], mxx);
			atomicMax(&bb[6 * b0 + 3], mxy);
			atomicMax(&bb[6 * b0 + 4], mh);
			atomicMax(&bb[6 * b0 + 5], mv);
		}
	} else if (valid) {
		atomicMin(&bb[6 * b + 0], mnx);
		atomicMin(&bb[6 * b + 1], mny);
		atomicMax(&bb[6 * b + 2], mxx);
		atomicMax(&bb[6 * b + 3], mxy);
		atomicMax(&bb[6 * b + 4], mh);
		atomicMax(&bb[6 * b + 5], mv);
	}
}

// Cell geometry of one body (grid.h:105-115) from its bounding box, h_max and (mixed form)
// largest squared speed; bad: not a valid grid (one cell, or too many, is set).
__device__ Geom body_geometry(const BodyParams& pr, int mixed, double bminx, double bminy, double bmaxx, double bmaxy,
                              double hmax, double v2max, bool& bad) {
	Geom g{};
	bminx -= 1e-6; bminy -= 1e-6;
	bmaxx += 1e-6; bmaxy += 1e-6;
	double dx = hmax * 2.;
	double slack = 0.;
	uint32_t span = 1;
	double lx = bmaxx - bminx, ly = bmaxy - bminy;
	if (mixed) {
		// a particle moves at most ~ |v| dt per step; allow twice the fastest speed
		slack = 2. * sqrt(v2max) * pr.dt;
		dx = 2. * hmax + 2. * slack;
		// half-size cells with a 5x5 stencil cover the same reach with ~40 % fewer
		// candidates than 3x3 cells of the full reach; used while the body's cells
		// stay below twice its particles
		double hx = 0.5 * dx;
		if (ceil(lx / hx) * ceil(ly / hx) <= 2.0 * pr.n) {
			dx = hx;
			span = 2;
		}
	}
	double fnx = ceil(lx / dx), fny = ceil(ly / dx);
	uint32_t nx = (uint32_t)fnx, ny = (uint32_t)fny;
	uint32_t num_cell = nx * ny;
	bad = false;
	if (!(num_cell < pr.n) && !mixed) bad = true;
	if (!(fnx * fny < 4.0e9) || nx == 0 || ny == 0) {
		nx = ny = 1;
		num_cell = 1;
		bad = true;
	}
	g.bbmin_x = bminx; g.bbmin_y = bminy; g.dx = dx; g.slack = slack;
	g.nx = nx; g.ny = ny; g.num_cell = num_cell; g.span = span;
	return g;
}

// Cell geometry per body (grid.h:105-115) and the exclusive scan of cell counts.
// One block; bodies are processed serially in chunks for the scan.
__global__ void k_geom(uint32_t nb, const unsigned long long* bb, const BodyParams* P, int mixed, Geom* G,
                       uint32_t* total_cells, uint32_t cell_cap, DevStatus* st, uint32_t* failed) {
	after_previous();
	__shared__ uint32_t s_cnt[1024];
	__shared__ uint32_t s_base;
	if (threadIdx.x == 0) s_base = 0;
	__syncthreads();
	for (uint32_t c0 = 0; c0 < nb; c0 += blockDim.x) {
		uint32_t b = c0 + threadIdx.x;
		uint32_t cnt = 0;
		Geom g{};
		if (b < nb && is_failed(failed, b)) {  // a failed body gets no cells
			g.nx = g.ny = 1;
			g.dx = 1.;
			g.span = 1;
		} else if (b < nb) {
			bool bad;
			g = body_geometry(P[b], mixed, ord_decode(bb[6 * b + 0]), ord_decode(bb[6 * b + 1]), ord_decode(bb[6 * b + 2]),
			                  ord_decode(bb[6 * b + 3]), ord_decode(bb[6 * b + 4]), ord_decode(bb[6 * b + 5]), bad);
			if (bad) {
				fail_body(failed, st, ERR_GRID, P[b].off, b);
				if (failed) g.num_cell = 0;  // masked from this stage on
			}
			cnt = g.num_cell;
		}
		s_cnt[threadIdx.x] = cnt;
		__syncthreads();
		if (threadIdx.x == 0) {
			uint32_t run = s_base;
			uint32_t lim = min((uint32_t)blockDim.x, nb - c0);
			for (uint32_t t = 0; t < lim; t++) {
				uint32_t c = s_cnt[t];
				s_cnt[t] = run;
				run += c;
			}
			s_base = run;
		}
		__syncthreads();
		if (b < nb) {
			g.cell_off = s_cnt[threadIdx.x];
			G[b] = g;
		}
		__syncthreads();
	}
	if (threadIdx.x == 0) {
		uint32_t tot = s_base;
		if (tot > cell_cap) {
			raise(st, ERR_GRID, 0);
			tot = 0;  // downstream kernels see an empty grid
		}
		*total_cells = tot;
	}
}

// Global cell key of each row (grid.h:35-41): cell_off + ix*ny + iy.
__global__ void k_hash(uint32_t n, const double* __restrict__ x, const double* __restrict__ y,
                       const uint32_t* __restrict__ body_of, const Geom* __restrict__ G,
                       const uint32_t* __restrict__ total_cells, uint32_t* keys, uint32_t* vals, DevStatus* st,
                       uint32_t* failed) {
	after_previous();
	uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
	if (i >= n) return;
	const uint32_t b = body_of[i], tot = *total_cells;
	vals[i] = i;
	if (is_failed(failed, b) && tot != 0) {  // past every cell: no stencil reaches it
		keys[i] = tot;
		return;
	}
	Geom g = G[b];
	uint32_t ix = (uint32_t)((x[i] - g.bbmin_x) / g.dx);
	uint32_t iy = (uint32_t)((y[i] - g.bbmin_y) / g.dx);
	if (ix >= g.nx || iy >= g.ny || tot == 0) {
		if (tot != 0 && failed) {
			atomicOr(&failed[b], ERR_GRID);
			keys[i] = tot;
			return;
		}
		raise(st, ERR_GRID, i);
		ix = min(ix, g.nx - 1);
		iy = min(iy, g.ny - 1);
	}
	uint32_t key = g.cell_off + ix * g.ny + iy;
	keys[i] = (tot == 0) ? 0u : key;
}

// Cell start table over all bodies' cells (grid.h:48-81): cell_start[c] is the first
// sorted position with key >= c, so empty cells get the next start.  Position k (up to
// and including n) fills in the cells that start there; run by the gather kernels.
__device__ __forceinline__ void fill_cells(const ULArgs& a, uint32_t k) {
	const uint32_t n = a.n_total, tot = *a.total_cells;
	if (k == n) {
		const uint32_t last = a.keys_sorted[n - 1] + 1;
		for (uint32_t c = last; c <= tot; c++) a.cell_start[c] = n;
		return;
	}
	const uint32_t key = min(a.keys_sorted[k], tot);
	const uint32_t prev = (k == 0) ? 0u : min(a.keys_sorted[k - 1], tot) + 1;
	if (k == 0 || a.keys_sorted[k] != a.keys_sorted[k - 1])
		for (uint32_t c = prev; c <= key; c++) a.cell_start[c] = k;
}

// ---- The grid of small bodies (at most GRID_BODY_MAX rows each): a block per body does
// what the kernels above do in eight launches -- bounding box, geometry, keys, the sort
// and the cell table -- in two (k_body_box, k_body_sort), and one body in one.  The
// rows of a body stay in its own range of the cell order; a counting sort over its cells,
// each cell's rows then put in ascending order, gives the radix sort's stable order.
// 256 small impacts (512 bodies of some 600 rows): 90 us a step in 13 launches -> 30 us.
// Larger bodies (ul_small_grid), and contexts that mask failed bodies (whose rows leave
// the cell order), take the general kernels.
constexpr uint32_t GRID_BODY_MAX = 4608;    // rows: two cells each and a 16-bit index fit 48 KB
constexpr uint32_t GRID_MAX_BODIES = 4096;  // every block adds up the cells of the bodies before it

// Block-wide reduction in shared memory (blockDim.x a multiple of 32, at most 1024)
template <class T, class Op>
__device__ __forceinline__ T block_reduce(T v, T* s, T identity, Op op) {
#pragma unroll
	for (int o = 16; o > 0; o >>= 1) v = op(v, __shfl_xor_sync(0xffffffffu, v, o));
	__syncthreads();
	if ((threadIdx.x & 31u) == 0) s[threadIdx.x >> 5] = v;
	__syncthreads();
	v = (threadIdx.x & 31u) < (blockDim.x >> 5) ? s[threadIdx.x & 31u] : identity;
#pragma unroll
	for (int o = 16; o > 0; o >>= 1) v = op(v, __shfl_xor_sync(0xffffffffu, v, o));
	return v;
}

// Bounding box, h_max, largest squared speed and from them the geometry of body b
// (cell_off left 0); every thread returns it
__device__ __forceinline__ Geom body_box(const ULArgs& a, int mixed, uint32_t b) {
	typedef unsigned long long u64;
	__shared__ u64 s_red[32];
	__shared__ Geom s_geom;
	const BodyParams& pr = a.params[b];
	const mfk_host::StateSoA& sv = a.stage == 0 ? a.base : a.st;
	u64 mnx = ord_encode(1.7976931348623157e308), mny = mnx, mxx = ord_encode(-1.7976931348623157e308), mxy = mxx, mh = mxx;
	u64 mv = ord_encode(0.);
	for (uint32_t i = pr.off + threadIdx.x; i < pr.off + pr.n; i += blockDim.x) {
		const u64 ex = ord_encode(sv.x[i]), ey = ord_encode(sv.y[i]);
		mnx = min(mnx, ex);
		mxx = max(mxx, ex);
		mny = min(mny, ey);
		mxy = max(mxy, ey);
		mh = max(mh, ord_encode(a.h[i]));
		if (mixed) {
			const double vx = sv.vx[i], vy = sv.vy[i];
			mv = max(mv, ord_encode(vx * vx + vy * vy));
		}
	}
	auto lo = [](u64 p, u64 q) { return min(p, q); };
	auto hi = [](u64 p, u64 q) { return max(p, q); };
	mnx = block_reduce(mnx, s_red, ~0ull, lo);
	mny = block_reduce(mny, s_red, ~0ull, lo);
	mxx = block_reduce(mxx, s_red, 0ull, hi);
	mxy = block_reduce(mxy, s_red, 0ull, hi);
	mh = block_reduce(mh, s_red, 0ull, hi);
	if (mixed) mv = block_reduce(mv, s_red, 0ull, hi);
	if (threadIdx.x == 0) {
		bool bad;
		s_geom = body_geometry(pr, mixed, ord_decode(mnx), ord_decode(mny), ord_decode(mxx), ord_decode(mxy), ord_decode(mh),
		                       ord_decode(mv), bad);
		if (bad) raise(reinterpret_cast<DevStatus*>(a.status), ERR_GRID, pr.off);
	}
	__syncthreads();
	return s_geom;
}

__global__ void __launch_bounds__(1024) k_body_box(ULArgs a, int mixed, uint32_t* cells) {
	after_previous();
	const uint32_t b = blockIdx.x;
	const Geom g = body_box(a, mixed, b);
	if (threadIdx.x == 0) {
		a.geom[b] = g;
		cells[b] = g.num_cell;
	}
}

// The body's rows in cell order and its part of the cell table.  ONE: a single body, its
// geometry computed here; else `cells` holds every body's cell count.
template <bool ONE>
__global__ void __launch_bounds__(1024) k_body_sort(ULArgs a, int mixed, const uint32_t* cells, uint32_t hist_cap,
                                                    uint32_t cell_cap) {
	after_previous();
	extern __shared__ uint32_t s_dyn[];  // [hist_cap] cell counters, then 16-bit row indices
	__shared__ unsigned long long s_red[32];
	__shared__ uint32_t s_warp[32];
	uint16_t* slot = reinterpret_cast<uint16_t*>(s_dyn + hist_cap);
	const uint32_t b = blockIdx.x, T = blockDim.x, tid = threadIdx.x;
	const mfk_host::StateSoA& sv = a.stage == 0 ? a.base : a.st;
	const uint32_t off = a.params[b].off, n = a.params[b].n;
	Geom g;
	unsigned long long before = 0, total;
	if (ONE) {
		g = body_box(a, mixed, b);
		total = g.num_cell;
	} else {
		g = a.geom[b];
		total = 0;
		for (uint32_t q = tid; q < a.n_bodies; q += T) {
			const uint32_t c = cells[q];
			total += c;
			if (q < b) before += c;
		}
		auto add = [](unsigned long long p, unsigned long long q) { return p + q; };
		total = block_reduce(total, s_red, 0ull, add);
		before = block_reduce(before, s_red, 0ull, add);
	}
	const bool fits = total <= cell_cap;
	if (!fits) before = 0;
	g.cell_off = (uint32_t)before;
	if (tid == 0) {
		a.geom[b] = g;
		if (b == 0) {
			*a.total_cells = fits ? (uint32_t)total : 0u;
			if (!fits) raise(reinterpret_cast<DevStatus*>(a.status), ERR_GRID, 0);
		}
	}
	if (!fits) {  // downstream kernels see an empty grid
		for (uint32_t i = tid; i < n; i += T) {
			a.perm[off + i] = off + i;
			a.keys_sorted[off + i] = 0;
		}
		return;
	}
	// the cells' counters: shared memory, or (scattered particles: more cells than the
	// block's share) the body's part of the cell table itself
	const uint32_t nc = g.num_cell;
	volatile uint32_t* hist = nc <= hist_cap ? s_dyn : a.cell_start + g.cell_off;
	for (uint32_t c = tid; c < nc; c += T) hist[c] = 0;
	__syncthreads();
	for (uint32_t i = tid; i < n; i += T) {
		uint32_t ix = (uint32_t)((sv.x[off + i] - g.bbmin_x) / g.dx);
		uint32_t iy = (uint32_t)((sv.y[off + i] - g.bbmin_y) / g.dx);
		if (ix >= g.nx || iy >= g.ny) {
			raise(reinterpret_cast<DevStatus*>(a.status), ERR_GRID, off + i);
			ix = min(ix, g.nx - 1);
			iy = min(iy, g.ny - 1);
		}
		const uint32_t key = ix * g.ny + iy;
		a.keys[off + i] = key;
		atomicAdd(const_cast<uint32_t*>(&hist[key]), 1u);
	}
	__syncthreads();
	// exclusive scan: each thread a contiguous piece
	const uint32_t per = (nc + T - 1) / T, c0 = min(tid * per, nc), c1 = min(c0 + per, nc);
	uint32_t sum = 0;
	for (uint32_t c = c0; c < c1; c++) sum += hist[c];
	uint32_t run = sum;
#pragma unroll
	for (int o = 1; o < 32; o <<= 1) {
		const uint32_t up = __shfl_up_sync(0xffffffffu, run, o);
		if ((tid & 31u) >= (uint32_t)o) run += up;
	}
	if ((tid & 31u) == 31u) s_warp[tid >> 5] = run;
	__syncthreads();
	uint32_t start = run - sum;
	for (uint32_t w = 0; w < (tid >> 5); w++) start += s_warp[w];
	for (uint32_t c = c0; c < c1; c++) {
		const uint32_t k = hist[c];
		hist[c] = start;
		start += k;
	}
	__syncthreads();
	for (uint32_t i = tid; i < n; i += T) slot[atomicAdd(const_cast<uint32_t*>(&hist[a.keys[off + i]]), 1u)] = (uint16_t)i;
	__syncthreads();
	// every cell's rows ascending (hist[c] is now the end of cell c)
	for (uint32_t c = tid; c < nc; c += T) {
		const uint32_t s0 = c ? hist[c - 1] : 0u, s1 = hist[c];
		for (uint32_t p = s0 + 1; p < s1; p++) {
			const uint16_t v = slot[p];
			uint32_t q = p;
			for (; q > s0 && slot[q - 1] > v; q--) slot[q] = slot[q - 1];
			slot[q] = v;
		}
	}
	__syncthreads();
	for (uint32_t p = tid; p < n; p += T) {
		const uint32_t i = slot[p];
		a.perm[off + p] = off + i;
		a.keys_sorted[off + p] = g.cell_off + a.keys[off + i];
	}
	// the cell table: the first row of every cell, from the ends just used (in place where
	// they stand in the table: piece by piece from the top, the piece's lower end read first)
	uint32_t prev = c0 < c1 && c0 > 0 ? hist[c0 - 1] : 0u;
	__syncthreads();
	for (uint32_t c = c0; c < c1; c++) {
		const uint32_t end = hist[c];
		a.cell_start[g.cell_off + c] = off + prev;
		prev = end;
	}
	if (b == a.n_bodies - 1 && tid == 0) a.cell_start[(uint32_t)total] = a.n_total;
}

// ---------------------------------------------------------------- gather
template <bool MIXED>
struct StageView;

// Reads the stage state of row i: stage 0 reads the base state (k1 is a copy of
// the particles, rk4.h:76-78), later stages the RK stage arrays.
template <>
struct StageView<false> {
	const double *x, *y, *vx, *vy, *rho, *Sxx, *Sxy, *Syy;
	__device__ void load(uint32_t i, double& X, double& Y, double& VX, double& VY, double& R, double& A, double& B,
	                     double& C) const {
		X = x[i]; Y = y[i]; VX = vx[i]; VY = vy[i]; R = rho[i]; A = Sxx[i]; B = Sxy[i]; C = Syy[i];
	}
};
template <>
struct StageView<true> {
	const double *x, *y, *vx, *vy;
	const float *rho, *Sxx, *Sxy, *Syy;
	__device__ void load(uint32_t i, double& X, double& Y, double& VX, double& VY, float& R, float& A, float& B,
	                     float& C) const {
		X = x[i]; Y = y[i]; VX = vx[i]; VY = vy[i]; R = rho[i]; A = Sxx[i]; B = Sxy[i]; C = Syy[i];
	}
};

template <bool MIXED>
__device__ StageView<MIXED> stage_view(const ULArgs& a);
template <>
__device__ StageView<false> stage_view<false>(const ULArgs& a) {
	const mfk_host::StateSoA& s = a.stage == 0 ? a.base : a.st;
	return StageView<false>{s.x, s.y, s.vx, s.vy, s.rho, s.Sxx, s.Sxy, s.Syy};
}
template <>
__device__ StageView<true> stage_view<true>(const ULArgs& a) {
	const mfk_host::StateSoA& s = a.stage == 0 ? a.base : a.st;
	return StageView<true>{s.x, s.y, s.vx, s.vy, s.rho_f, s.Sxx_f, s.Sxy_f, s.Syy_f};
}

// Per-particle actions of one stage: EOS, artificial stress, integration weight.
template <class T>
__device__ __forceinline__ void per_particle(uint32_t flags, const BodyParams& pr, T m, T rho, T qw0, T Sxx, T Sxy,
                                             T Syy, T& sxx_o, T& syy_o, T& Rxx, T& Rxy, T& Ryy, T& c, T& qw,
                                             T& rho21) {
	T p = T(0);
	if (flags & A_EOS) p = T(pr.c0sq) * (rho - T(pr.rho0));  // c0*c0*(rho - rho0)
	T sxx = Sxx - p, syy = Syy - p, sxy = Sxy;
	Rxx = Rxy = Ryy = T(0);
	if (flags & A_ART_STRESS) {
		T eps = T(pr.mghn_eps);
		T theta = T(0.5) * atan2(T(2.) * sxy, sxx - syy + T(0.));
		T cs = cos(theta), sn = sin(theta);
		T cs2 = cs * cs, sn2 = sn * sn;
		T rot_sxx = cs2 * sxx + T(2.0) * cs * sn * sxy + sn2 * syy;
		T rot_syy = sn2 * sxx - T(2.0) * cs * sn * sxy + cs2 * syy;
		T rot_rxx = T(0), rot_ryy = T(0);
		if (rot_sxx > T(0)) rot_rxx = -eps * rot_sxx / (rho * rho);
		if (rot_syy > T(0)) rot_ryy = -eps * rot_syy / (rho * rho);
		Rxx = cs2 * rot_rxx + sn2 * rot_ryy;
		Rxy = cs * sn * (rot_rxx - rot_ryy);
		Ryy = sn2 * rot_rxx + cs2 * rot_ryy;
	}
	sxx_o = sxx;
	syy_o = syy;
	c = sqrt(T(pr.K) / rho);
	qw = (flags & A_RIEMANN) ? m / rho : qw0;
	rho21 = T(1.) / (rho * rho);
}

// The same in FP32 for the mixed gather, from the parameters' FP32 copies, the EOS from
// the stored rho - rho0 (no cancellation of rho - rho0 in FP32)
__device__ __forceinline__ void per_particle32(uint32_t flags, const BodyParams& pr, float m, float rho, float drho,
                                               float qw0, float Sxx, float Sxy, float Syy, float& sxx_o, float& syy_o,
                                               float& Rxx, float& Rxy, float& Ryy, float& c, float& qw,
                                               float& rho21) {
	float p = 0.f;
	if (flags & A_EOS) p = pr.fc0sq * drho;
	float sxx = Sxx - p, syy = Syy - p, sxy = Sxy;
	Rxx = Rxy = Ryy = 0.f;
	if (flags & A_ART_STRESS) {
		// principal stresses from the stress circle; cos 2 theta and sin 2 theta (halved) as
		// its components over its radius, in place of atan2f, cosf and sinf of the angle
		float dev = sxx - syy, twice = 2.f * sxy;
		const float mean = 0.5f * (sxx + syy);
		// (an exponent whose square could leave the range: scaled by a power of two)
		const uint32_t e = max(__float_as_uint(fabsf(dev)), __float_as_uint(fabsf(twice))) >> 23;
		const uint32_t k = min(max(e, 1u), 253u);
		const bool scaled = e - 80u > 94u;
		if (scaled) {
			dev *= __uint_as_float((254u - k) << 23);
			twice *= __uint_as_float((254u - k) << 23);
		}
		const float R2 = dev * dev + twice * twice;
		const float R1 = R2 > 1e-30f ? rsqrtf(R2) : 0.f;
		float radius = 0.5f * R2 * R1;
		if (scaled) radius *= __uint_as_float(k << 23);
		const float c2 = R2 > 1e-30f ? 0.5f * dev * R1 : 0.5f, s2 = 0.5f * twice * R1;
		const float eps = -pr.fmghn_eps / (rho * rho);
		const float ra = eps * fmaxf(mean + radius, 0.f), rb = eps * fmaxf(mean - radius, 0.f);
		Rxx = (0.5f + c2) * ra + (0.5f - c2) * rb;
		Ryy = (0.5f - c2) * ra + (0.5f + c2) * rb;
		Rxy = s2 * (ra - rb);
	}
	sxx_o = sxx;
	syy_o = syy;
	c = sqrtf(pr.fK / rho);
	qw = (flags & A_RIEMANN) ? m / rho : qw0;
	rho21 = 1.f / (rho * rho);
}

#if !MF_STRICT_FORM
// The same for the fast FP64 gather, which the narrow FP64 pipe bounds: the principal
// stresses from the stress circle, cos 2 theta and sin 2 theta as its components over its
// radius, in place of atan2, cos and sin of the angle (337k rows: 100 -> 41 us).
__device__ __forceinline__ void per_particle64(uint32_t flags, const BodyParams& pr, double m, double rho, double qw0,
                                               double Sxx, double Sxy, double Syy, Rec64& r) {
	const double p = (flags & A_EOS) ? pr.c0sq * (rho - pr.rho0) : 0.;
	const double rho1 = rcp64(rho);
	r.sxx = Sxx - p;
	r.syy = Syy - p;
	r.sxy = Sxy;
	r.rho21 = rho1 * rho1;
	r.qw = (flags & A_RIEMANN) ? m * rho1 : qw0;
	r.c = sqrt(pr.K * rho1);
	r.Rxx = r.Rxy = r.Ryy = 0.;
	if (flags & A_ART_STRESS) {
		double dev = r.sxx - r.syy, twice = 2. * Sxy;
		const double mean = 0.5 * (r.sxx + r.syy);
		// (an exponent whose square could leave the range: scaled by a power of two)
		const uint32_t e = (uint32_t)max(__double2hiint(fabs(dev)), __double2hiint(fabs(twice))) >> 20;
		const uint32_t k = min(max(e, 1u), 2045u);
		const bool scaled = e - 600u > 800u;
		if (scaled) {
			dev *= __hiloint2double((int)((2046u - k) << 20), 0);
			twice *= __hiloint2double((int)((2046u - k) << 20), 0);
		}
		const double R2 = fma(dev, dev, twice * twice);
		const double R1 = R2 > 0. ? rsqrt64(R2) : 0.;
		double radius = 0.5 * R2 * R1;
		if (scaled) radius *= __hiloint2double((int)(k << 20), 0);
		const double c2 = R2 > 0. ? 0.5 * dev * R1 : 0.5, s2 = 0.5 * twice * R1;  // halves of cos, sin 2 theta
		const double eps = -pr.mghn_eps * r.rho21;
		const double ra = eps * clamp0(mean + radius), rb = eps * clamp0(mean - radius);
		r.Rxx = (0.5 + c2) * ra + (0.5 - c2) * rb;
		r.Ryy = (0.5 - c2) * ra + (0.5 + c2) * rb;
		r.Rxy = s2 * (ra - rb);
	}
}
#endif

__global__ void k_gather64(ULArgs a, const BodyParams* __restrict__ P) {
	after_previous();
	uint32_t k = blockIdx.x * blockDim.x + threadIdx.x;
	if (a.fill_cells && k <= a.n_total) fill_cells(a, k);
	if (k >= a.n_total) return;
	uint32_t i = a.perm[k];
	StageView<false> v = stage_view<false>(a);
	double x, y, vx, vy, rho, Sxx, Sxy, Syy;
	v.load(i, x, y, vx, vy, rho, Sxx, Sxy, Syy);
	uint32_t b = a.body_of[i];
	Rec64 r;
	r.x = x; r.y = y; r.vx = vx; r.vy = vy;
	r.m = a.m[i]; r.h = a.h[i]; r.rho = rho;
#if MF_STRICT_FORM
	per_particle<double>(a.flags, P[b], r.m, rho, a.qw0[i], Sxx, Sxy, Syy, r.sxx, r.syy, r.Rxx, r.Rxy, r.Ryy, r.c, r.qw,
	                     r.rho21);
	r.sxy = Sxy;
#else
	per_particle64(a.flags, P[b], r.m, rho, a.qw0[i], Sxx, Sxy, Syy, r);
#endif
	if (a.flags & (A_GOD_CONT | A_GOD_MOM)) {
		r.Rxx = (a.flags & A_EOS) ? P[b].c0sq * (rho - P[b].rho0) : 0.;
		r.Rxy = Syy;
	}
#if !MF_STRICT_FORM
	else {  // pair64_fast takes the stresses times 1/rho^2 and c times alpha / 2
		r.c *= 0.5 * P[b].alpha;
		r.sxx *= r.rho21;
		r.sxy *= r.rho21;
		r.syy *= r.rho21;
	}
#endif
	// float-float positions for the candidate tests
	const FF fx = ff_split_bits(x), fy = ff_split_bits(y);
	reinterpret_cast<float4*>(a.pos)[k] = make_float4(fx.hi, fx.lo, fy.hi, fy.lo);
	Rec64* out = reinterpret_cast<Rec64*>(a.rec) + k;
	const double2* s = reinterpret_cast<const double2*>(&r);
	double2* d = reinterpret_cast<double2*>(out);
#pragma unroll
	for (int q = 0; q < 8; q++) d[q] = s[q];
	a.rec_body[k] = b;
}

// The record of particle i (body parameters pr) from its stage state, as row k of rec.
__device__ __forceinline__ void put_rec32(const ULArgs& a, const BodyParams& pr, uint32_t i, void* rec, uint32_t k,
                                          double x, double y, double vx, double vy, float rho_dev, float Sxx, float Sxy,
                                          float Syy) {
	const float rho = rho_dev + pr.frho0;  // the mixed state holds rho - rho0
	Rec32 r;
	r.x = ff_split_bits(x); r.y = ff_split_bits(y); r.vx = ff_split_bits(vx); r.vy = ff_split_bits(vy);
	r.m = (float)a.m[i]; r.h = (float)a.h[i]; r.rho = rho;
	per_particle32(a.flags, pr, r.m, rho, rho_dev, (float)a.qw0[i], Sxx, Sxy, Syy, r.sxx, r.syy, r.Rxx, r.Rxy, r.Ryy,
	               r.c, r.qw, r.rho21);
	r.sxy = Sxy;
	if (a.flags & (A_GOD_CONT | A_GOD_MOM)) {  // p from the stored deviation, the stress Syy itself
		r.Rxx = (a.flags & A_EOS) ? pr.fc0sq * rho_dev : 0.f;
		r.Rxy = Syy;
	} else {  // pair32_fast takes the stresses times 1/rho^2 and c times alpha / 2
		r.c *= 0.5f * pr.falpha;
		r.sxx *= r.rho21;
		r.sxy *= r.rho21;
		r.syy *= r.rho21;
	}
	store_rec(reinterpret_cast<float4*>(rec), a.n_total, k, r);
}

__global__ void k_gather32(ULArgs a, const BodyParams* __restrict__ P) {
	after_previous();
	uint32_t k = blockIdx.x * blockDim.x + threadIdx.x;
	if (a.fill_cells && k <= a.n_total) fill_cells(a, k);
	if (k >= a.n_total) return;
	uint32_t i = a.perm[k];
	StageView<true> v = stage_view<true>(a);
	double x, y, vx, vy;
	float rho, Sxx, Sxy, Syy;
	v.load(i, x, y, vx, vy, rho, Sxx, Sxy, Syy);
	uint32_t b = a.body_of[i];
	put_rec32(a, P[b], i, a.rec, k, x, y, vx, vy, rho, Sxx, Sxy, Syy);
	a.rec_body[k] = b;
}

__device__ __forceinline__ void stencil(const Geom& g, uint32_t key, int& lo_i, int& hi_i, int& lo_j, int& hi_j) {
	uint32_t b = key - g.cell_off;
	uint32_t gi = b / g.ny;
	uint32_t gj = b - gi * g.ny;
	const int sp = (int)g.span;
	lo_i = (int)gi - sp < 0 ? 0 : (int)gi - sp;
	lo_j = (int)gj - sp < 0 ? 0 : (int)gj - sp;
	hi_i = (int)gi + sp + 1 > (int)g.nx ? (int)g.nx : (int)gi + sp + 1;
	hi_j = (int)gj + sp + 1 > (int)g.ny ? (int)g.ny : (int)gj + sp + 1;
}

// ----------------------------------------------------------- pair kernel FP64
// GB300 issues FP64 at 2 lanes a clock and SM: a warp instruction holds the pipe for 16
// clocks however few of its lanes are active, so these kernels' time is their FP64 warp
// instructions.  Three things keep them low.
//
// 1. Four lanes share a row (P64_L).  They test the row's candidates in FP32, from the
//    float-float positions the gather writes, and list the ones within reach in shared
//    memory; then lane l takes the listed pairs l, l + 4, ...  A warp's eight rows finish
//    in ceil(most neighbours / 4) pair evaluations with nearly every lane at work, where
//    one thread a row ran the pair terms for every candidate that some lane accepted.
//    The split depends on the row's own candidates alone, never on the launch, so a body
//    gets the same bits in any batch.
// 2. The FP32 test decides only what it can: the offsets' error is at most
//    2^-23 |d| + 2^-46 |x| (the split keeps 48 bits), under 2e-6 of the squared distance
//    while |x| <= 2^26 h; a candidate within 2e-5 of the reference's limit, and every
//    candidate of a row outside those ranges, is decided by the reference's FP64
//    predicate, so the counts and the neighbour sets are the reference's.
// 3. The fast form rearranges the Gray-Monaghan pair terms (pair64_fast).
//
// Ensemble of 16 ring impacts (337k rows), per stage: 4.89 ms with one thread a row and
// the FP64 test, 1.27 ms now (503 FP64 instructions a warp of eight rows, the FP64 pipe
// 87 % busy); rings at dx = 1 mm (4,408 rows), parity form, per step: 1.76 ms -> 0.42 ms
// (there the 35 blocks of 128 rows had also left 117 of the 152 SMs empty).
constexpr uint32_t P64_L = 4;        // lanes per row
constexpr uint32_t P64_CAP = 96;    // listed pairs per row before they are worked off
constexpr uint32_t P64_THREADS = 128;
constexpr uint32_t P64_ROWS = P64_THREADS / P64_L;

// The pair sums of one row (a lane's share of them)
struct Acc64 {
	double Sxx_x = 0., Sxy_y = 0., Sxy_x = 0., Syy_y = 0.;
	double vx_x = 0., vx_y = 0., vy_x = 0., vy_y = 0.;
	double av_x = 0., av_y = 0., xs_x = 0., xs_y = 0.;
	double god_rho = 0., god_vx = 0., god_vy = 0.;
};

// All pair terms in the reference's expressions (the records hold the stress itself; 1/rho^2 is
// applied here).
template <bool GOD>
__device__ __forceinline__ void pair64_ref(uint32_t flags, const BodyParams& pr, const Rec64& ri, const Rec64& rj,
                                           Acc64& s) {
	const double hi = ri.h;
	double xij = __dsub_rn(ri.x, rj.x);
	double yij = __dsub_rn(ri.y, rj.y);
	double r2 = __dadd_rn(__dmul_rn(xij, xij), __dmul_rn(yij, yij));
	KR64 w = cubic_spline(xij, yij, hi);
	if (flags & A_STRESS_MGHN) {
		double Rxx = 0., Rxy = 0., Ryy = 0.;
		if (pr.wdeltap > 0) {
			double fab = w.w / pr.wdeltap;
			if (pr.corr_exp == 4.) {
				double f2 = fab * fab;
				fab = f2 * f2;
			} else {
				fab = pow(fab, pr.corr_exp);
			}
			Rxx = fab * (ri.Rxx + rj.Rxx);
			Rxy = fab * (ri.Rxy + rj.Rxy);
			Ryy = fab * (ri.Ryy + rj.Ryy);
		}
		const double rhoi21 = ri.rho21;
		s.Sxx_x += rj.m * (ri.sxx * rhoi21 + rj.sxx * rj.rho21 + Rxx) * w.w_x;
		s.Sxy_y += rj.m * (ri.sxy * rhoi21 + rj.sxy * rj.rho21 + Rxy) * w.w_y;
		s.Sxy_x += rj.m * (ri.sxy * rhoi21 + rj.sxy * rj.rho21 + Rxy) * w.w_x;
		s.Syy_y += rj.m * (ri.syy * rhoi21 + rj.syy * rj.rho21 + Ryy) * w.w_y;
	}
	if (flags & A_DERIVE_VEL) {
		s.vx_x += (rj.vx - ri.vx) * w.w_x * rj.qw;
		s.vx_y += (rj.vx - ri.vx) * w.w_y * rj.qw;
		s.vy_x += (rj.vy - ri.vy) * w.w_x * rj.qw;
		s.vy_y += (rj.vy - ri.vy) * w.w_y * rj.qw;
	}
	double vijx = ri.vx - rj.vx, vijy = ri.vy - rj.vy;
	if (flags & A_ART_VISC) {
		double vijposij = vijx * xij + vijy * yij;
		if (vijposij < 0.) {
			double cij = 0.5 * (ri.c + rj.c);
			double hij = 0.5 * (hi + rj.h);
			double rhoij = 0.5 * (ri.rho + rj.rho);
			double r2ij = xij * xij + yij * yij;
			double muij = (hij * vijposij) / (r2ij + pr.eta * pr.eta * hij * hij);
			double piij = (-pr.alpha * cij * muij + pr.beta * muij * muij) / rhoij;
			s.av_x += -rj.m * piij * w.w_x;
			s.av_y += -rj.m * piij * w.w_y;
		}
	}
	if (flags & A_XSPH) {
		double rhoij = 0.5 * (ri.rho + rj.rho);
		double fac = -pr.xsph_eps * w.w * ri.m / rhoij;
		s.xs_x += fac * vijx;
		s.xs_y += fac * vijy;
	}
	if (GOD) {
		// |x_j - x_i| from the predicate's own sum (the same value as the
		// reference's sqrt(dx*dx + dy*dy) and sqrt(dot(R, R)))
		const double mag_r = sqrt(r2);
		// the acoustic Riemann denominator, the same expression in both actions
		const double frac = 1. / (ri.rho * ri.c + rj.rho * rj.c);
#if !MF_STRICT_FORM
		const double inv_r = 1. / mag_r;
#endif
		if (flags & A_GOD_CONT) {  // godunov_continuity, godunov.h:144-187
#if MF_STRICT_FORM
			double nx = xij / mag_r, ny = yij / mag_r;
#else
			double nx = xij * inv_r, ny = yij * inv_r;
#endif
			double vir = ri.vx * nx + ri.vy * ny;
			double vjr = rj.vx * nx + rj.vy * ny;
			// riemann_solver_acoustic (godunov.h:41-54); Rxx = p
			double ustar = frac * (vir * ri.rho * ri.c + vjr * rj.rho * rj.c - ri.Rxx + rj.Rxx);
			s.god_rho += 2 * ri.rho * (vir - ustar) * (w.w_x * nx + w.w_y * ny) * rj.qw;
		}
		if (flags & A_GOD_MOM) {  // godunov_get_trafo + godunov_momentum, godunov.h:56-142
			const double two_rhoi = 2. / ri.rho;  // godunov.h:127-133's 2./rhoi, the same per pair
			double rx = rj.x - ri.x, ry = rj.y - ri.y;
#if MF_STRICT_FORM
			double inv = 1. / mag_r;  // glm::normalize: v * (1 / sqrt(dot(v, v)))
#else
			double inv = inv_r;
#endif
			double Rx = rx * inv, Ry = ry * inv, Sx = ry * inv, Sy = -rx * inv;
			// the frame matrix is single precision (a glm::mat2x2 of the unit vectors)
			double lRx = (double)__double2float_rn(Rx), lRy = (double)__double2float_rn(Ry);
			double lSx = (double)__double2float_rn(Sx), lSy = (double)__double2float_rn(Sy);
			// stress times R: (Sxx - p, Sxy; Sxy, Syy), Rxy = Syy
			double siR0 = ri.sxx * Rx + ri.sxy * Ry, siR1 = ri.sxy * Rx + ri.Rxy * Ry;
			double sjR0 = rj.sxx * Rx + rj.sxy * Ry, sjR1 = rj.sxy * Rx + rj.Rxy * Ry;
			double si0 = lRx * siR0 + lSx * siR1;
			double sj0 = lRx * sjR0 + lSx * sjR1, sj1 = lRy * sjR0 + lSy * sjR1;
			double vi0 = lRx * ri.vx + lSx * ri.vy, vi1 = lRy * ri.vx + lSy * ri.vy;
			double vj0 = lRx * rj.vx + lSx * rj.vy, vj1 = lRy * rj.vx + lSy * rj.vy;
			// the second component takes sigma_j twice (godunov.h:116), as the reference does
			double S0 = frac * (sj0 * ri.rho * ri.c + si0 * rj.rho * rj.c + ri.rho * ri.c * rj.rho * rj.c * (vj0 - vi0));
			double S1 = frac * (sj1 * ri.rho * ri.c + sj1 * rj.rho * rj.c + ri.rho * ri.c * rj.rho * rj.c * (vj1 - vi1));
			double SR0 = lRx * S0 + lRy * S1, SR1 = lSx * S0 + lSy * S1;
			if (fabs(rx) > 0.) s.god_vx += two_rhoi * w.w_x * mag_r / rx * SR0 * rj.qw;
			if (fabs(ry) > 0.) s.god_vy += two_rhoi * w.w_y * mag_r / ry * SR1 * rj.qw;
		}
	}
}

#if !MF_STRICT_FORM
// The Gray-Monaghan pair terms for the fast form: the same sums in ~70 FP64 instructions
// a pair against ~150 (square root and five divisions included).
//  * the spline through t = 2 - q and u = max(1 - q, 0): W = fac (t^3 / 4 - u^3) and
//    dW/dq = 3 fac (u^2 - t^2 / 4), one expression for both pieces (t clamped at 0 beyond
//    2h); the factor 3 fac is applied to the row's gradient sums at the end;
//  * 1/r, 1/(r^2 + eta^2 h^2) and 1/(rho_i + rho_j) by one third-order step from an FP32
//    seed (rsqrt64, rcp64);
//  * stress and viscosity share one gradient sum, (s_i + s_j + R - Pi) grad W, since the
//    momentum equation takes only the sums' totals and its rho_i / rho_i cancels; they
//    collect in av_x, av_y;
//  * mu and Pi with the factors 1/2 of the pair means folded into the constants, the
//    records' stresses already times 1/rho^2 and their c times alpha / 2 (k_gather64).
struct Row64 {
	double h1, w_wdp, eta2q, half_beta, xs_c;
	bool stress, art;
};
__device__ __forceinline__ void pair64_fast(uint32_t flags, const Row64& k, double corr_exp, const Rec64& ri,
                                            const Rec64& rj, Acc64& s) {
	const double xij = ri.x - rj.x, yij = ri.y - rj.y;
	const double r2 = fma(yij, yij, xij * xij);
	const bool apart = __double_as_longlong(r2) > __double_as_longlong(1e-24);  // kernel.cpp's r > 1e-12
	const double sr = apart ? rsqrt64(r2) * k.h1 : 0.;  // 1 / (r h)
	const double q = r2 * sr;
	const double t = clamp0(2. - q), u = clamp0(1. - q);
	const double u2 = u * u, t2q = 0.25 * t * t;
	const double w = fma(t2q, t, -u2 * u);  // W / fac
	const double g = (u2 - t2q) * sr;       // |grad W| / (3 fac r)
	const double gx = xij * g, gy = yij * g;
	const double dvx = rj.vx - ri.vx, dvy = rj.vy - ri.vy;
	const double inv_rs = rcp64(ri.rho + rj.rho);
	double piij = 0.;
	if (flags & A_ART_VISC) {
		const double dot = fma(dvy, yij, dvx * xij);  // -v_ij . x_ij
		const bool approach = above0(dot);
		const double hs = ri.h + rj.h;
		const double D = approach ? fma(k.eta2q * hs, hs, r2) : 1.;
		const double mu2 = hs * dot * rcp64(D);  // -2 mu_ij
		const double p = mu2 * fma(k.half_beta, mu2, ri.c + rj.c) * inv_rs;
		piij = approach ? p : 0.;
	}
	if (k.stress) {
		double txx = ri.sxx + rj.sxx, txy = ri.sxy + rj.sxy, tyy = ri.syy + rj.syy;
		if (k.art) {
			double fab = w * k.w_wdp;
			if (corr_exp == 4.) {
				fab *= fab;
				fab *= fab;
			} else {
				fab = pow(fab, corr_exp);
			}
			txx = fma(fab, ri.Rxx + rj.Rxx, txx);
			txy = fma(fab, ri.Rxy + rj.Rxy, txy);
			tyy = fma(fab, ri.Ryy + rj.Ryy, tyy);
		}
		const double mx = rj.m * gx, my = rj.m * gy;
		s.av_x = fma(txx - piij, mx, fma(txy, my, s.av_x));
		s.av_y = fma(txy, mx, fma(tyy - piij, my, s.av_y));
	} else if (flags & A_ART_VISC) {
		const double mp = rj.m * piij;
		s.av_x = fma(-mp, gx, s.av_x);
		s.av_y = fma(-mp, gy, s.av_y);
	}
	if (flags & A_DERIVE_VEL) {
		const double qx = rj.qw * gx, qy = rj.qw * gy;
		s.vx_x = fma(dvx, qx, s.vx_x);
		s.vx_y = fma(dvx, qy, s.vx_y);
		s.vy_x = fma(dvy, qx, s.vy_x);
		s.vy_y = fma(dvy, qy, s.vy_y);
	}
	if (flags & A_XSPH) {
		const double f = w * inv_rs;
		s.xs_x = fma(f, dvx, s.xs_x);
		s.xs_y = fma(f, dvy, s.xs_y);
	}
}
#endif

// The row's totals of N sums (N a multiple of its four lanes) into every lane: each lane
// adds up a quarter of them, N / 2 + N / 4 additions where a butterfly per sum takes 2 N,
// and reads the others' (the shuffles do not use the FP64 pipe).
template <int N>
__device__ __forceinline__ void row_sums64(double (&v)[N], uint32_t lane) {
	double h[N / 2], t[N / 4];
#pragma unroll
	for (int i = 0; i < N / 2; i++) {
		const double keep = (lane & 2u) ? v[N / 2 + i] : v[i], give = (lane & 2u) ? v[i] : v[N / 2 + i];
		h[i] = keep + __shfl_xor_sync(0xffffffffu, give, 2);
	}
#pragma unroll
	for (int i = 0; i < N / 4; i++) {
		const double keep = (lane & 1u) ? h[N / 4 + i] : h[i], give = (lane & 1u) ? h[i] : h[N / 4 + i];
		t[i] = keep + __shfl_xor_sync(0xffffffffu, give, 1);
	}
#pragma unroll
	for (int l = 0; l < 4; l++)
#pragma unroll
		for (int i = 0; i < N / 4; i++) v[(l >> 1) * (N / 2) + (l & 1) * (N / 4) + i] = __shfl_sync(0xffffffffu, t[i], l, P64_L);
}

// Every lane of a warp stays to the end (a row past the last, or of a failed body, lists
// no pairs and writes nothing), so the shuffles take the whole warp.
template <bool GOD>
__global__ void __launch_bounds__(P64_THREADS) k_pair64(ULArgs a, const BodyParams* __restrict__ P,
                                                        const Geom* __restrict__ G, DevStatus* st) {
	after_previous();
	__shared__ uint32_t s_list[P64_ROWS][P64_CAP + 1];  // (+ 1: rows start in different banks)
	constexpr unsigned FULL = 0xffffffffu;
	const uint32_t lane = threadIdx.x % P64_L;
	const uint32_t k = (blockIdx.x * P64_THREADS + threadIdx.x) / P64_L;
	const bool in_range = k < a.n_total;
	const uint32_t kk = in_range ? k : a.n_total - 1;
	uint32_t* list = s_list[threadIdx.x / P64_L];
	const uint32_t b = a.rec_body[kk];
	// the row's four lanes must agree on a word that other rows may set meanwhile
	bool live = in_range && !is_failed(a.failed, b);
	live = __shfl_sync(FULL, live, 0, P64_L);
	const Rec64* rec = reinterpret_cast<const Rec64*>(a.rec);
	const float4* pos = reinterpret_cast<const float4*>(a.pos);
	const Rec64 ri = load_rec(rec + kk);
	const float4 pi = __ldg(pos + kk);
	const BodyParams& pr = P[b];
	const Geom g = G[b];
	const uint32_t i = a.perm[kk];
	const uint32_t flags = a.flags;
	int lo_i, hi_i, lo_j, hi_j;
	stencil(g, a.keys_sorted[kk], lo_i, hi_i, lo_j, hi_j);
	if (!live) hi_i = lo_i;
	const uint32_t tot = *a.total_cells;

	// the FP32 test's bands: beyond `far` a pair cannot contribute (q >= 2 gives exactly
	// zero); below `sure_in` / above `sure_out` it is certainly within / beyond the
	// reference's limit 4 h^2 + eps.  In FP32 from h's leading bits, out of the FP64 pipe's way.
	const int he = __double2hiint(ri.h), eexp = ((__double2hiint(ri.h) >> 20) & 0x7ff) + 26;  // |x| < 2^26 h
	const float hf = seed_f32(ri.h), limf = 4.f * hf * hf + a.nbh_eps_f;
	const bool fp32 = he >= 0x3cd203af && he < 0x430c6bf5 /* 1e-15 <= h < 1e15 */ && limf < 1e30f && a.nbh_eps_f >= 0.f &&
	                  ((__double2hiint(ri.x) >> 20) & 0x7ff) < eexp && ((__double2hiint(ri.y) >> 20) & 0x7ff) < eexp;
	const float far = 4.f * hf * hf * 1.00002f, sure_in = limf * 0.99998f, sure_out = limf * 1.00002f;
	Acc64 s;
#if !MF_STRICT_FORM
	Row64 rk;
	rk.h1 = rcp64(ri.h);
	const double fac = 10 * (K_1_PI) / 7.0 * rk.h1 * rk.h1;
	rk.art = pr.wdeltap > 0;
	rk.w_wdp = rk.art ? fac * rcp64(pr.wdeltap) : 0.;
	rk.eta2q = 0.25 * pr.eta * pr.eta;
	rk.half_beta = 0.5 * pr.beta;
	rk.stress = (flags & A_MOMENTUM_UL) != 0;
#endif
	auto pairs = [&](uint32_t n) {
		for (uint32_t e = lane; e < n; e += P64_L) {
			const uint32_t kj = list[e];
			const Rec64 rj = load_rec(rec + kj);
#if MF_STRICT_FORM
			pair64_ref<GOD>(flags, pr, ri, rj, s);
#else
			if (GOD) pair64_ref<GOD>(flags, pr, ri, rj, s);
			else pair64_fast(flags, rk, pr.corr_exp, ri, rj, s);
#endif
		}
	};
	uint32_t cnt = 0, listed = 0;
	bool alone = true;
	const int cols = __reduce_max_sync(FULL, hi_i - lo_i);
	for (int c = 0; c < cols; c++) {
		uint32_t j0 = 0, j1 = 0;
		if (lo_i + c < hi_i) {
			const uint32_t row = g.cell_off + (uint32_t)(lo_i + c) * g.ny;
			j0 = a.cell_start[min(row + (uint32_t)lo_j, tot)];
			j1 = a.cell_start[min(row + (uint32_t)hi_j, tot)];
		}
		for (uint32_t base = j0; __any_sync(FULL, base < j1); base += 32) {
			uint32_t mask = 0u;  // of the 32 candidates from base on, those to list
#pragma unroll
			for (uint32_t t = 0; t < 32; t += P64_L) {
				const uint32_t kj = base + t + lane;
				if (base >= j1 || kj >= j1) break;
				const float4 pj = __ldg(pos + kj);
				const float dx = (pi.x - pj.x) + (pi.y - pj.y), dy = (pi.z - pj.z) + (pi.w - pj.w);
				const float r2 = dx * dx + dy * dy;
				bool list_it = !(r2 > far), in = r2 <= sure_in;
				if (!fp32 || !(in || r2 > sure_out)) {  // the reference's predicate decides
					const double2 xy = __ldg(reinterpret_cast<const double2*>(rec + kj));
					const double xij = __dsub_rn(ri.x, xy.x), yij = __dsub_rn(ri.y, xy.y);
					const double d2 = __dadd_rn(__dmul_rn(xij, xij), __dmul_rn(yij, yij));
					const double h2 = __dmul_rn(ri.h, ri.h);
					in = d2 <= __dadd_rn(__dmul_rn(__dmul_rn(h2, 2.), 2.), a.nbh_eps);
					if (!fp32) list_it = !(d2 > 4.0000001 * h2);
				}
				cnt += in ? 1u : 0u;
				// (the row itself counts, but adds nothing to any sum)
				if (list_it && kj != k) mask |= 1u << (t + lane);
			}
			uint32_t own = mask;
#pragma unroll
			for (uint32_t o = P64_L / 2; o > 0; o >>= 1) mask |= __shfl_xor_sync(FULL, mask, o);
			while (own) {
				const uint32_t bit = (uint32_t)__ffs(own) - 1u;
				own &= own - 1u;
				list[listed + __popc(mask & ((1u << bit) - 1u))] = base + bit;
			}
			listed += __popc(mask);
			const bool full = listed > P64_CAP - 32;
			if (__any_sync(FULL, full)) {  // a full row works its list off now (the others go on listing)
				__syncwarp();
				pairs(full ? listed : 0u);
				if (full) {
					listed = 0u;
					alone = false;
				}
				__syncwarp();
			}
		}
	}
	// a row without neighbours takes itself: zero terms, unless its stress is not finite or its
	// h zero, which then shows in the sums as it does through any neighbour
	if (!GOD && live && alone && listed == 0u) {
		if (lane == 0) list[0] = k;
		listed = 1u;
	}
	__syncwarp();
	pairs(listed);
	for (uint32_t o = P64_L / 2; o > 0; o >>= 1) cnt += __shfl_xor_sync(FULL, cnt, o);

	// per-particle actions, in the reference's list order; every lane of the row holds the
	// totals, and lane q then updates the state components q and q + 4
	double d[8] = {0., 0., 0., 0., 0., 0., 0., 0.};
	const double rhoi = ri.rho;
#if MF_STRICT_FORM
	constexpr bool SUMS = true;
#else
	constexpr bool SUMS = GOD;  // (pair64_fast adds the stress forces to av)
#endif
	constexpr int NS = GOD ? 16 : SUMS ? 12 : 8;
	double v[NS] = {s.av_x, s.av_y, s.vx_x, s.vx_y, s.vy_x, s.vy_y, s.xs_x, s.xs_y};
	if (SUMS) {
		v[8 % NS] = s.Sxx_x; v[9 % NS] = s.Sxy_y; v[10 % NS] = s.Sxy_x; v[11 % NS] = s.Syy_y;
	}
	if (GOD) {
		v[12 % NS] = s.god_rho; v[13 % NS] = s.god_vx; v[14 % NS] = s.god_vy; v[15 % NS] = 0.;
	}
	row_sums64<NS>(v, lane);
	double vx_x = v[2], vx_y = v[3], vy_x = v[4], vy_y = v[5];
#if !MF_STRICT_FORM
	if (!GOD) {  // the factors that pair64_fast left out
		const double gsc = 3. * fac, xsc = 2. * pr.xsph_eps * ri.m * fac;
		v[0] *= gsc; v[1] *= gsc; v[6] *= xsc; v[7] *= xsc;
		vx_x *= gsc; vx_y *= gsc; vy_x *= gsc; vy_y *= gsc;
	}
	const bool av = (flags & A_ART_VISC) || (!GOD && rk.stress);
#else
	const bool av = (flags & A_ART_VISC) != 0;
#endif
	if (av) { d[2] = v[0]; d[3] = v[1]; }
	if (flags & A_XSPH) { d[0] = v[6]; d[1] = v[7]; }
	if (flags & A_JAUMANN) {
		// the Jaumann rate uses the stage stress itself (not S - p)
		const mfk_host::StateSoA& sv = a.stage == 0 ? a.base : a.st;
#if MF_STRICT_FORM
		jaumann<double>(vx_x, vx_y, vy_x, vy_y, sv.Sxx[i], sv.Sxy[i], sv.Syy[i], pr.G, d[5], d[6], d[7]);
#else
		jaumann_plane(vx_x, vx_y, vy_x, vy_y, sv.Sxx[i], sv.Sxy[i], sv.Syy[i], pr.G, d[5], d[6], d[7]);
#endif
	}
	if (flags & A_CONTINUITY) d[4] = -(rhoi * (vx_x + vy_y));
	if (GOD) {
		if (flags & A_GOD_CONT) d[4] = v[12 % NS];
		if (flags & A_GOD_MOM) {
			d[2] += v[13 % NS] + a.fcx[i] / ri.m;
			d[3] += v[14 % NS] + a.fcy[i] / ri.m;
		}
	}
	if (flags & A_MOMENTUM_UL) {
#if MF_STRICT_FORM
		const double fmx = a.fcx[i] / ri.m, fmy = a.fcy[i] / ri.m;
#else
		const double m1 = rcp64(ri.m), fmx = a.fcx[i] * m1, fmy = a.fcy[i] * m1;
#endif
		if (SUMS) {
			d[2] += 1. / rhoi * (v[8 % NS] * rhoi + v[9 % NS] * rhoi) + fmx;
			d[3] += 1. / rhoi * (v[10 % NS] * rhoi + v[11 % NS] * rhoi) + fmy;
		} else {
			d[2] += fmx;
			d[3] += fmy;
		}
	}
	if (flags & A_ADVECTION) { d[0] += ri.vx; d[1] += ri.vy; }
	// (lanes 1 to 3 now replace the stage stress that every lane has read)
	__syncwarp();
	if (!live) return;
	if (lane == 0) {
		if (a.max_nbh && cnt >= a.max_nbh) fail_body(a.failed, st, ERR_NBH_OVERFLOW, i, b);
		if (cnt == 0) fail_body(a.failed, st, ERR_NO_NEIGHBOR, i, b);
	}
	// rk4.h:52-69 (stage state = particles + c*dt*derivative) and :94-103 (final combine
	// with weights 1,2,2,1 / 6); d[] = x_t, y_t, vx_t, vy_t, rho_t, Sxx_t, Sxy_t, Syy_t
	double* bp[8] = {a.base.x, a.base.y, a.base.vx, a.base.vy, a.base.rho, a.base.Sxx, a.base.Sxy, a.base.Syy};
	double* ap[8] = {a.acc.x, a.acc.y, a.acc.vx, a.acc.vy, a.acc.rho, a.acc.Sxx, a.acc.Sxy, a.acc.Syy};
	double* sp[8] = {a.st.x, a.st.y, a.st.vx, a.st.vy, a.st.rho, a.st.Sxx, a.st.Sxy, a.st.Syy};
	const double dt = pr.dt;
	bool ok = true;
#pragma unroll
	for (uint32_t half = 0; half < 2; half++) {
		double dq = d[4 * half];
		double *B = bp[4 * half], *A = ap[4 * half], *S = sp[4 * half];
#pragma unroll
		for (uint32_t q = 1; q < 4; q++)
			if (lane == q) { dq = d[4 * half + q]; B = bp[4 * half + q]; A = ap[4 * half + q]; S = sp[4 * half + q]; }
		if (a.stage < 3) {
			const double dts = (a.stage == 2 ? 1.0 : 0.5) * dt;
			A[i] = (a.stage == 0) ? dq : A[i] + 2 * dq;
			S[i] = B[i] + dq * dts;
		} else {
			const double w6 = dt * 1. / 6.;
			const double v = B[i] + w6 * (A[i] + dq);
			B[i] = v;
			if (half == 0 || lane == 0) ok = ok && isfinite(v);  // x, y, vx, vy, rho
		}
	}
	if (!ok) fail_body(a.failed, st, ERR_NONFINITE, i, b);
}

// ---------------------------------------------------------- pair kernel mixed
// Instruction issue (60 % of the slots), the L1 data pipe (60 %) and the L2 reads behind it
// bound these kernels together, so the Gray-Monaghan pair terms are written for few
// instructions, as in pair64_fast: ~75 FP32 operations a pair against ~120 in the
// reference's expressions, no flag tests in the whole list's instance, the records as
// arrays.  Ensemble of 64 ring impacts (1.35M rows), per stage: 373 -> 285 us.  Measured
// and not kept: a list over all stencil columns in shared memory (fewer evaluations, 21
// against 25 a row, but the lanes drift apart: 300 against 271 us alone), 8-byte relative
// positions for the candidate tests (303: the tests on the records' own positions bring
// the lines that the pair terms read next), cells in blocks of 8 x 16 (381), a warp's
// records of the next column prefetched into L1 (285).

// The pair sums of one row (or a lane's share of them)
struct Acc32 {
	float Sxx_x = 0.f, Sxy_y = 0.f, Sxy_x = 0.f, Syy_y = 0.f;
	float vx_x = 0.f, vx_y = 0.f, vy_x = 0.f, vy_y = 0.f;
	float av_x = 0.f, av_y = 0.f, xs_x = 0.f, xs_y = 0.f;
	float god_rho = 0.f, god_vx = 0.f, god_vy = 0.f;
};
// Per-row constants of the pair terms (the parameters' FP32 copies: a conversion, let
// alone a division, in FP64 would run on the narrow FP64 pipe for every row)
struct Row32 {
	float h1, fac;                          // 1 / h, 10 / (7 pi h^2)
	float w_wdp, eta2q, half_beta, corr_exp;
	bool stress, art;
};

// 1/x and 1/sqrt(x) by the special-function unit alone (2 ulp, no rescaling of
// subnormals: r^2, eta^2 h^2 and densities are far above them)
__device__ __forceinline__ float rcp_approx(float x) {
	float y;
	asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
	return y;
}
__device__ __forceinline__ float rsqrt_approx(float x) {
	float y;
	asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
	return y;
}

// The Gray-Monaghan pair terms at the offset (xij, yij) = x_i - x_j, r2 its square.
struct Terms32 {
	float ax = 0.f, ay = 0.f;                // of av
	float dvx, dvy, qx = 0.f, qy = 0.f;      // of vx_x .. vy_y: dv times q
	float f = 0.f;                           // of xs: dv times f
};
__device__ __forceinline__ Terms32 pair32_terms(uint32_t flags, const Row32& k, const Rec32& ri, const Rec32& rj, float xij,
                                                float yij, float r2) {
	Terms32 o;
	// W = fac (t^3 / 4 - u^3), |grad W| = 3 fac (t^2 / 4 - u^2) / h with t = 2 - q,
	// u = max(1 - q, 0) (t clamped at 0 beyond 2h); 3 fac is applied to the row's sums
	const float sr = r2 > 1e-24f ? rsqrt_approx(r2) * k.h1 : 0.f;  // 1 / (r h); kernel.cpp's r > 1e-12
	const float q = r2 * sr;
	const float t = fmaxf(2.f - q, 0.f), u = fmaxf(1.f - q, 0.f);
	const float u2 = u * u, t2q = 0.25f * t * t;
	const float w = t2q * t - u2 * u;
	const float g = (u2 - t2q) * sr;
	const float gx = xij * g, gy = yij * g;
	const float dvx = ff_diff(rj.vx, ri.vx), dvy = ff_diff(rj.vy, ri.vy);
	o.dvx = dvx;
	o.dvy = dvy;
	const float inv_rs = rcp_approx(ri.rho + rj.rho);
	float piij = 0.f;
	if (flags & A_ART_VISC) {
		const float dot = dvx * xij + dvy * yij;  // -v_ij . x_ij
		const float hs = ri.h + rj.h;
		const float mu2 = hs * dot * rcp_approx(r2 + k.eta2q * hs * hs);  // -2 mu_ij
		const float p = mu2 * (k.half_beta * mu2 + (ri.c + rj.c)) * inv_rs;
		piij = dot > 0.f ? p : 0.f;  // approaching
	}
	if (k.stress) {  // the records' stresses are already times 1/rho^2
		float txx = ri.sxx + rj.sxx, txy = ri.sxy + rj.sxy, tyy = ri.syy + rj.syy;
		if (k.art) {
			float fab = w * k.w_wdp;
			if (k.corr_exp == 4.f) {
				fab *= fab;
				fab *= fab;
			} else {
				fab = powf(fab, k.corr_exp);
			}
			txx += fab * (ri.Rxx + rj.Rxx);
			txy += fab * (ri.Rxy + rj.Rxy);
			tyy += fab * (ri.Ryy + rj.Ryy);
		}
		const float mx = rj.m * gx, my = rj.m * gy;
		o.ax = __fmaf_rn(txx - piij, mx, __fmul_rn(txy, my));
		o.ay = __fmaf_rn(txy, mx, __fmul_rn(tyy - piij, my));
	} else if (flags & A_ART_VISC) {
		const float mp = rj.m * piij;
		o.ax = -mp * gx;
		o.ay = -mp * gy;
	}
	if (flags & A_DERIVE_VEL) {
		o.qx = rj.qw * gx;
		o.qy = rj.qw * gy;
	}
	if (flags & A_XSPH) o.f = w * inv_rs;
	return o;
}
// ... and their sums, every rounding spelled out: the walks of a row by one thread and by
// eight lanes (row_by_lanes) agree to the bit.
__device__ __forceinline__ void pair32_fast(uint32_t flags, const Row32& k, const Rec32& ri, const Rec32& rj, float xij,
                                            float yij, float r2, Acc32& s) {
	const Terms32 o = pair32_terms(flags, k, ri, rj, xij, yij, r2);
	s.av_x = __fadd_rn(s.av_x, o.ax);
	s.av_y = __fadd_rn(s.av_y, o.ay);
	if (flags & A_DERIVE_VEL) {
		s.vx_x = __fmaf_rn(o.dvx, o.qx, s.vx_x);
		s.vx_y = __fmaf_rn(o.dvx, o.qy, s.vx_y);
		s.vy_x = __fmaf_rn(o.dvy, o.qx, s.vy_x);
		s.vy_y = __fmaf_rn(o.dvy, o.qy, s.vy_y);
	}
	if (flags & A_XSPH) {
		s.xs_x = __fmaf_rn(o.f, o.dvx, s.xs_x);
		s.xs_y = __fmaf_rn(o.f, o.dvy, s.xs_y);
	}
}

// The pair terms of a pipeline with Godunov actions, in the reference's expressions.
__device__ __forceinline__ void pair32_godunov(uint32_t flags, const BodyParams& pr, const Row32& k, const Rec32& ri,
                                               const Rec32& rj, float xij, float yij, float r2, Acc32& s) {
	KR32 w = cubic_spline_f(xij, yij, k.h1, k.fac);
	if (flags & A_STRESS_MGHN) {
		float Rxx = 0.f, Rxy = 0.f, Ryy = 0.f;
		if (pr.fwdp1 > 0.f) {
			float fab = w.w * pr.fwdp1;
			if (pr.fcorr_exp == 4.f) {
				float f2 = fab * fab;
				fab = f2 * f2;
			} else {
				fab = powf(fab, pr.fcorr_exp);
			}
			Rxx = fab * (ri.Rxx + rj.Rxx);
			Rxy = fab * (ri.Rxy + rj.Rxy);
			Ryy = fab * (ri.Ryy + rj.Ryy);
		}
		float tsx = rj.m * (ri.sxy * ri.rho21 + rj.sxy * rj.rho21 + Rxy);
		s.Sxx_x += rj.m * (ri.sxx * ri.rho21 + rj.sxx * rj.rho21 + Rxx) * w.w_x;
		s.Sxy_y += tsx * w.w_y;
		s.Sxy_x += tsx * w.w_x;
		s.Syy_y += rj.m * (ri.syy * ri.rho21 + rj.syy * rj.rho21 + Ryy) * w.w_y;
	}
	float dvx = ff_diff(rj.vx, ri.vx), dvy = ff_diff(rj.vy, ri.vy);
	if (flags & A_DERIVE_VEL) {
		float qx = w.w_x * rj.qw, qy = w.w_y * rj.qw;
		s.vx_x += dvx * qx;
		s.vx_y += dvx * qy;
		s.vy_x += dvy * qx;
		s.vy_y += dvy * qy;
	}
	if (flags & A_ART_VISC) {
		float vijposij = -(dvx * xij + dvy * yij);
		if (vijposij < 0.f) {
			float cij = 0.5f * (ri.c + rj.c);
			float hij = 0.5f * (ri.h + rj.h);
			float rhoij = 0.5f * (ri.rho + rj.rho);
			float muij = __fdividef(hij * vijposij, r2 + pr.feta2 * hij * hij);
			float piij = __fdividef(-pr.falpha * cij * muij + pr.fbeta * muij * muij, rhoij);
			s.av_x += -rj.m * piij * w.w_x;
			s.av_y += -rj.m * piij * w.w_y;
		}
	}
	if (flags & A_XSPH) {
		float rhoij = 0.5f * (ri.rho + rj.rho);
		float f = __fdividef(-pr.fxsph_eps * w.w * ri.m, rhoij);
		s.xs_x -= f * dvx;
		s.xs_y -= f * dvy;
	}
	{
		// godunov_continuity / godunov_momentum (godunov.h:86-187) in FP32: velocity
		// differences from the float-float records, the Riemann state in the form
		// v_i - u* = (Z_j (v_i - v_j).n + p_i - p_j) / (Z_i + Z_j), Z = rho c;
		// Rxx holds p, Rxy the stress Syy itself
		const float mag_r = sqrtf(r2), inv = 1.f / mag_r;
		const float Zi = ri.rho * ri.c, Zj = rj.rho * rj.c;
		const float frac = 1.f / (Zi + Zj);
		if (flags & A_GOD_CONT) {
			float nx = xij * inv, ny = yij * inv;
			float dvn = -(dvx * nx + dvy * ny);  // (v_i - v_j).n
			float vi_us = frac * (Zj * dvn + (ri.Rxx - rj.Rxx));
			s.god_rho += 2.f * ri.rho * vi_us * (w.w_x * nx + w.w_y * ny) * rj.qw;
		}
		if (flags & A_GOD_MOM) {
			float rx = -xij, ry = -yij;
			float Rx = rx * inv, Ry = ry * inv, Sx = ry * inv, Sy = -rx * inv;  // the float frame
			float siR0 = ri.sxx * Rx + ri.sxy * Ry;
			float sjR0 = rj.sxx * Rx + rj.sxy * Ry, sjR1 = rj.sxy * Rx + rj.Rxy * Ry;
			float si0 = Rx * siR0 + Sx * (ri.sxy * Rx + ri.Rxy * Ry);
			float sj0 = Rx * sjR0 + Sx * sjR1, sj1 = Ry * sjR0 + Sy * sjR1;
			float dv0 = Rx * dvx + Sx * dvy, dv1 = Ry * dvx + Sy * dvy;  // frame (v_j - v_i)
			// the second component takes sigma_j twice (godunov.h:116), as the reference does
			float S0 = frac * (sj0 * Zi + si0 * Zj + Zi * Zj * dv0);
			float S1 = frac * (sj1 * Zi + sj1 * Zj + Zi * Zj * dv1);
			float SR0 = Rx * S0 + Ry * S1, SR1 = Sx * S0 + Sy * S1;
			if (fabsf(rx) > 0.f) s.god_vx += (2.f / ri.rho) * __fdividef(w.w_x * mag_r, rx) * SR0 * rj.qw;
			if (fabsf(ry) > 0.f) s.god_vy += (2.f / ri.rho) * __fdividef(w.w_y * mag_r, ry) * SR1 * rj.qw;
		}
	}
}

// L threads per row (L = 1: one thread walks the row's whole stencil): lane takes every
// L-th candidate of each stencil row, the partial sums are added across the L lanes,
// and lane 0 finishes the row.  L > 1 puts more rows' work in flight when the rows are
// few (the launch would otherwise cover a handful of SMs); it changes the order of the
// pair sums, not their terms.
// ORDERED (L = 8, no Godunov actions): the lanes split the tests and the pair terms, and
// each sums one of the eight sums over the row's pairs in their order: a thread's result,
// to the bit.
constexpr uint32_t ORD_CAP = 64;  // neighbours listed before they are evaluated
struct OrdRow {
	float term[8][8];
	uint32_t list[ORD_CAP];
	float pad[8];  // (the four rows of a warp 8 banks apart)
};
template <bool GOD, bool FULL, int L = 1, bool ORDERED = false>
__device__ __forceinline__ void pair32_row(const ULArgs& a, const BodyParams* __restrict__ P,
                                           const Geom* __restrict__ G, DevStatus* st, uint32_t k,
                                           uint32_t lane = 0, OrdRow* sh = nullptr) {
	uint32_t b = a.rec_body[k];
	// a failed body stays as it was (all L lanes of the row, on the first one's reading: another
	// row may be failing the body just now)
	bool failed = is_failed(a.failed, b);
	if (L > 1) failed = __shfl_sync(((1u << L) - 1u) << (threadIdx.x & 31u & ~(unsigned)(L - 1)), failed, 0, L);
	if (failed) return;
	const float4* rec = reinterpret_cast<const float4*>(a.rec);
	const size_t n = a.n_total;
	const Rec32 ri = load_rec(rec, n, k, __ldg(rec + k));
	const BodyParams& pr = P[b];
	Geom g = G[b];
	uint32_t i = a.perm[k];
	const uint32_t flags = FULL ? A_MONAGHAN : a.flags;
	int lo_i, hi_i, lo_j, hi_j;
	stencil(g, a.keys_sorted[k], lo_i, hi_i, lo_j, hi_j);
	const uint32_t tot = *a.total_cells;

	Row32 rk;
	rk.h1 = 1.f / ri.h;
	rk.fac = (float)(10 * (K_1_PI) / 7.0) * rk.h1 * rk.h1;
	rk.art = pr.fwdp1 > 0.f;
	rk.w_wdp = rk.fac * pr.fwdp1;
	rk.eta2q = 0.25f * pr.feta2;
	rk.half_beta = 0.5f * pr.fbeta;
	rk.corr_exp = pr.fcorr_exp;
	rk.stress = (flags & A_MOMENTUM_UL) != 0;
	const float reach2 = 4.0001f * ri.h * ri.h;
	Acc32 s;
	// the pair terms of candidate kj within reach (xij, yij: x_i - x_j; r2 = |x_i - x_j|^2)
	auto pair = [&](uint32_t kj, float4 head, float xij, float yij, float r2) {
		const Rec32 rj = load_rec(rec, n, kj, head);
		if (GOD) pair32_godunov(flags, pr, rk, ri, rj, xij, yij, r2, s);
		else pair32_fast(flags, rk, ri, rj, xij, yij, r2, s);
	};
	// candidate offsets and squared distance, one rounding each (the same values in both
	// walks below)
	auto offs = [&](float4 head, float& xij, float& yij) {
		xij = __fadd_rn(__fsub_rn(ri.x.hi, head.x), __fsub_rn(ri.x.lo, head.y));
		yij = __fadd_rn(__fsub_rn(ri.y.hi, head.z), __fsub_rn(ri.y.lo, head.w));
		return __fmaf_rn(yij, yij, __fmul_rn(xij, xij));
	};
	if (ORDERED) {
		const uint32_t shift = threadIdx.x & 24u, gmask = 0xffu << shift;
		// this lane's sum, and which factors of a pair it adds: {ax, ay, dvx, dvy, qx, qy, f, 1}
		const uint32_t fa = 0x66332210u >> (4 * lane) & 15u, fb = 0x32545477u >> (4 * lane) & 15u;
		float acc = 0.f;
		uint32_t cnt = 0;
		auto evaluate = [&] {
			__syncwarp(gmask);
			for (uint32_t p0 = 0; p0 < cnt; p0 += 8) {
				if (p0 + lane < cnt) {
					const uint32_t kj = sh->list[p0 + lane];
					const float4 head = __ldg(rec + kj);
					float xij, yij;
					const float r2 = offs(head, xij, yij);
					const Terms32 o = pair32_terms(flags, rk, ri, load_rec(rec, n, kj, head), xij, yij, r2);
					float4* t = reinterpret_cast<float4*>(sh->term[lane]);
					t[0] = make_float4(o.ax, o.ay, o.dvx, o.dvy);
					t[1] = make_float4(o.qx, o.qy, o.f, 1.f);
				}
				__syncwarp(gmask);
				const uint32_t m = min(cnt - p0, 8u);
#pragma unroll
				for (uint32_t u = 0; u < 8; u++)
					if (u < m) acc = __fmaf_rn(sh->term[u][fa], sh->term[u][fb], acc);
				__syncwarp(gmask);
			}
			cnt = 0;
		};
		for (int n0 = lo_i; n0 < hi_i; n0 += 8) {
			// a lane per stencil column, then the columns' candidates as one range
			uint32_t j0 = 0, len = 0;
			if (n0 + (int)lane < hi_i) {
				const uint32_t cell = g.cell_off + (uint32_t)(n0 + (int)lane) * g.ny;
				j0 = a.cell_start[min(cell + (uint32_t)lo_j, tot)];
				len = a.cell_start[min(cell + (uint32_t)hi_j, tot)] - j0;
			}
			uint32_t end = len;
#pragma unroll
			for (int o = 1; o < 8; o <<= 1) {
				const uint32_t v = __shfl_up_sync(gmask, end, o, 8);
				if ((int)lane >= o) end += v;
			}
			const uint32_t base = j0 - (end - len), total = __shfl_sync(gmask, end, 7, 8);
			uint32_t ends[7];
#pragma unroll
			for (int q = 0; q < 7; q++) ends[q] = __shfl_sync(gmask, end, q, 8);
			for (uint32_t c0 = 0; c0 < total; c0 += 32) {
				if (cnt + 32u > ORD_CAP) evaluate();
				uint32_t kj[4];
				bool in[4];
#pragma unroll
				for (int r = 0; r < 4; r++) {
					const uint32_t cand = c0 + 8 * r + lane;
					uint32_t col = 0;
#pragma unroll
					for (int q = 0; q < 7; q++) col += cand >= ends[q];
					kj[r] = __shfl_sync(gmask, base, col, 8) + cand;
					in[r] = cand < total && kj[r] != k;
				}
				float4 head[4];
#pragma unroll
				for (int r = 0; r < 4; r++)
					if (in[r]) head[r] = __ldg(rec + kj[r]);
#pragma unroll
				for (int r = 0; r < 4; r++) {
					float xij, yij;
					in[r] = in[r] && !(offs(head[r], xij, yij) > reach2);
					const uint32_t hit = __ballot_sync(gmask, in[r]) >> shift & 255u;
					if (in[r]) sh->list[cnt + __popc(hit & ((1u << lane) - 1u))] = kj[r];
					cnt += __popc(hit);
				}
			}
		}
		evaluate();
		float* sums[8] = {&s.av_x, &s.av_y, &s.vx_x, &s.vx_y, &s.vy_x, &s.vy_y, &s.xs_x, &s.xs_y};
#pragma unroll
		for (int q = 0; q < 8; q++) *sums[q] = __shfl_sync(gmask, acc, q, 8);
		if (lane != 0) return;
	}
	for (int ni = lo_i; !ORDERED && ni < hi_i; ni++) {
		uint32_t c0 = min(g.cell_off + (uint32_t)ni * g.ny + (uint32_t)lo_j, tot);
		uint32_t c1 = min(g.cell_off + (uint32_t)ni * g.ny + (uint32_t)hi_j, tot);
		uint32_t j0 = a.cell_start[c0], j1 = a.cell_start[c1];
		if (L == 1 && j1 - j0 <= 32u) {
			// this stencil column's candidates tested first, into one mask, then the pair
			// terms of those within reach in ascending order: a warp runs as many pair
			// evaluations as its lane with the most neighbours in the column, instead of one
			// for every candidate that some lane accepts (the same pairs in the same order)
			uint32_t mask = 0u;
			for (uint32_t kj = j0; kj < j1; kj++) {
				float xij, yij;
				const float r2 = offs(__ldg(rec + kj), xij, yij);
				if (!(r2 > reach2)) mask |= 1u << (kj - j0);
			}
			if (k - j0 < 32u) mask &= ~(1u << (k - j0));  // (the row itself adds nothing to any sum)
			while (mask) {
				const uint32_t kj = j0 + (uint32_t)(__ffs(mask) - 1);
				mask &= mask - 1u;
				const float4 head = __ldg(rec + kj);
				float xij, yij;
				const float r2 = offs(head, xij, yij);
				pair(kj, head, xij, yij, r2);
			}
		} else {
			for (uint32_t kj = j0 + lane; kj < j1; kj += L) {
				// positions first: most candidates of the stencil lie beyond the reach
				const float4 head = __ldg(rec + kj);
				float xij, yij;
				const float r2 = offs(head, xij, yij);
				if (r2 > reach2 || kj == k) continue;
				pair(kj, head, xij, yij, r2);
			}
		}
	}
	if (L > 1 && !ORDERED) {
		const unsigned gmask = ((1u << L) - 1u) << ((threadIdx.x & 31u) & ~(unsigned)(L - 1));
		constexpr int NS = GOD ? 15 : 8;
		float* acc[15] = {&s.vx_x, &s.vx_y, &s.vy_x, &s.vy_y, &s.av_x, &s.av_y, &s.xs_x, &s.xs_y,
		                  &s.Sxx_x, &s.Sxy_y, &s.Sxy_x, &s.Syy_y, &s.god_rho, &s.god_vx, &s.god_vy};
#pragma unroll
		for (int q = 0; q < NS; q++)
#pragma unroll
			for (int o = L / 2; o > 0; o >>= 1) *acc[q] += __shfl_xor_sync(gmask, *acc[q], o, L);
		if (lane != 0) return;
	}
	float d[8] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
	const float rhoi = ri.rho;
	if (!GOD && rk.stress) {  // (a stress that is not finite shows in a row without neighbours too)
		s.av_x = __fmaf_rn(ri.sxx, 0.f, __fmaf_rn(ri.sxy, 0.f, s.av_x));
		s.av_y = __fmaf_rn(ri.syy, 0.f, s.av_y);
	}
	if (!GOD) {  // the factors that pair32_fast left out
		const float gsc = 3.f * rk.fac, xsc = 2.f * pr.fxsph_eps * ri.m * rk.fac;
		s.av_x *= gsc; s.av_y *= gsc;
		s.vx_x *= gsc; s.vx_y *= gsc; s.vy_x *= gsc; s.vy_y *= gsc;
		s.xs_x *= xsc; s.xs_y *= xsc;
	}
	if ((flags & A_ART_VISC) || (!GOD && rk.stress)) { d[2] = s.av_x; d[3] = s.av_y; }
	if (flags & A_XSPH) { d[0] = s.xs_x; d[1] = s.xs_y; }
	if (flags & A_JAUMANN) {
		const mfk_host::StateSoA& sv = a.stage == 0 ? a.base : a.st;
		jaumann<float>(s.vx_x, s.vx_y, s.vy_x, s.vy_y, sv.Sxx_f[i], sv.Sxy_f[i], sv.Syy_f[i], pr.fG, d[5], d[6], d[7]);
	}
	if (flags & A_CONTINUITY) d[4] = -(rhoi * (s.vx_x + s.vy_y));
	if (GOD && (flags & A_GOD_CONT)) d[4] = s.god_rho;
	if (GOD && (flags & A_GOD_MOM)) {
		d[2] += s.god_vx + (float)a.fcx[i] / ri.m;
		d[3] += s.god_vy + (float)a.fcy[i] / ri.m;
	}
	if (flags & A_MOMENTUM_UL) {
		if (GOD) {  // (pair32_fast added the stress forces to av, without rho / rho)
			d[2] += 1.f / rhoi * (s.Sxx_x * rhoi + s.Sxy_y * rhoi);
			d[3] += 1.f / rhoi * (s.Sxy_x * rhoi + s.Syy_y * rhoi);
		}
		d[2] += (float)a.fcx[i] / ri.m;
		d[3] += (float)a.fcy[i] / ri.m;
	}
	if (a.stage > 0) {
		// the cells were sized at stage 0 for moves up to g.slack; check that held
		double mx = a.st.x[i] - a.base.x[i], my = a.st.y[i] - a.base.y[i];
		if (mx * mx + my * my > g.slack * g.slack) fail_body(a.failed, st, ERR_GRID, i, b);
	}
	// advection: the FP64 velocity enters the FP64 position update below
	double dd0 = (double)d[0], dd1 = (double)d[1];
	if (flags & A_ADVECTION) {
		const mfk_host::StateSoA& sv = a.stage == 0 ? a.base : a.st;
		dd0 += sv.vx[i];
		dd1 += sv.vy[i];
	}
	// position/velocity in FP64, rho/S in FP32
	const uint32_t stg = a.stage;
	double dt = pr.dt;
	double dq[4] = {dd0, dd1, (double)d[2], (double)d[3]};
	double* bp[4] = {a.base.x, a.base.y, a.base.vx, a.base.vy};
	double* ap[4] = {a.acc.x, a.acc.y, a.acc.vx, a.acc.vy};
	double* sp[4] = {a.st.x, a.st.y, a.st.vx, a.st.vy};
	float* bq[4] = {a.base.rho_f, a.base.Sxx_f, a.base.Sxy_f, a.base.Syy_f};
	float* aq[4] = {a.acc.rho_f, a.acc.Sxx_f, a.acc.Sxy_f, a.acc.Syy_f};
	float* sq[4] = {a.st.rho_f, a.st.Sxx_f, a.st.Sxy_f, a.st.Syy_f};
	if (stg < 3) {
		double dts = (stg == 2 ? 1.0 : 0.5) * dt;
		double nv[4];  // the next stage's x, y, vx, vy
		float nf[4];   // and its rho - rho0, Sxx, Sxy, Syy
#pragma unroll
		for (int q = 0; q < 4; q++) {
			ap[q][i] = (stg == 0) ? dq[q] : ap[q][i] + 2 * dq[q];
			nv[q] = bp[q][i] + dq[q] * dts;
			sp[q][i] = nv[q];
			float dr = d[4 + q];
			aq[q][i] = (stg == 0) ? dr : aq[q][i] + 2.f * dr;
			nf[q] = bq[q][i] + dr * (float)dts;
			sq[q][i] = nf[q];
		}
		if (a.write_recs)
			put_rec32(a, pr, i, a.rec_next, k, nv[0], nv[1], nv[2], nv[3], nf[0], nf[1], nf[2], nf[3]);
	} else {
		double w6 = dt * 1. / 6.;
#pragma unroll
		for (int q = 0; q < 4; q++) {
			bp[q][i] = bp[q][i] + w6 * (ap[q][i] + dq[q]);
			bq[q][i] = bq[q][i] + (float)w6 * (aq[q][i] + d[4 + q]);
		}
		if (!(isfinite(bp[0][i]) && isfinite(bp[1][i]) && isfinite(bp[2][i]) && isfinite(bp[3][i]) &&
		      isfinite(bq[0][i])))
			fail_body(a.failed, st, ERR_NONFINITE, i, b);
	}
}

// The mixed pair pass with L threads per row (plain grid)
template <bool GOD, bool FULL, int L>
__global__ void __launch_bounds__(256, 3) k_pair_split(ULArgs a, const BodyParams* __restrict__ P,
                                                       const Geom* __restrict__ G, DevStatus* st) {
	after_previous();
	const uint32_t t = blockIdx.x * blockDim.x + threadIdx.x;
	const uint32_t k = t / L;
	if (k >= a.n_total) return;  // a row's L lanes leave together (L divides the warp)
	pair32_row<GOD, FULL, L>(a, P, G, st, k, t % L);
}

// The same walk by eight lanes a row, for few rows: a row's tests and pairs are a chain of
// gathers, 18 us a stage with a thread a row whether there are 4,400 rows or 17,600.  As
// long as the blocks fit the SMs at once (4 of 16 rows by their registers, 9,728 rows on 152
// SMs) the lanes make it shorter: 4,408 rows 17.9 -> 12.0 us, 9,176 rows 18.0 -> 14.1; 9,860
// rows would take 20.6.
constexpr unsigned ORD_THREADS = 128;
template <bool FULL>
__global__ void __launch_bounds__(ORD_THREADS, 4) k_pair_ordered(ULArgs a, const BodyParams* __restrict__ P,
                                                                 const Geom* __restrict__ G, DevStatus* st) {
	after_previous();
	__shared__ __align__(16) OrdRow rows[ORD_THREADS / 8];
	const uint32_t t = blockIdx.x * ORD_THREADS + threadIdx.x, k = t / 8;
	if (k >= a.n_total) return;  // a row's 8 lanes leave together
	pair32_row<false, FULL, 8, true>(a, P, G, st, k, t % 8, rows + threadIdx.x / 8);
}

// Rows an SM from which the mixed pair pass runs with four blocks of 256 an SM at 64
// registers (some constants of a row spilled) instead of three at 80: the deeper occupancy
// pays once every SM has several rounds of blocks, 27 of 128 rows here.  Per step, three / four
// blocks, ring impacts of 4k to 110k rows: 223,600 rows 355 / 380 us, 316,600 462 / 487,
// 445,512 598 / 588, 518,680 671 / 681, 600,448 759 / 733, 1,053,456 1182 / 1155, 1,349,144
// 1461 / 1430; of 4.4k rows: 331,944 452 / 476, 671,232 745 / 727, 3,348,184 3245 / 3090.
constexpr uint32_t PAIR_ROWS_MB4 = 3450;

// The mixed pair kernel.  Plain form: one thread per cell-ordered row.  Persistent form
// (one launch per stage over all bodies): a fixed grid whose blocks take chunks of
// rows -- consecutive cell-ordered rows, so a chunk is a run of cells of one body --
// from an atomic counter until the rows run out; no block ever waits on another.
// MB: blocks of 256 per SM the register budget is cut for (3: 80 registers; 4: 64, with
// some constants of a row spilled) -- the same arithmetic, so the same results.
template <bool GOD, bool FULL, int MB>
__global__ void __launch_bounds__(256, MB) k_pair(ULArgs a, const BodyParams* __restrict__ P, const Geom* __restrict__ G,
                                                 DevStatus* st) {
	after_previous();
	if (!a.persistent) {
		uint32_t k = blockIdx.x * blockDim.x + threadIdx.x;
		if (k >= a.n_total) return;
		pair32_row<GOD, FULL>(a, P, G, st, k);
		return;
	}
	__shared__ uint32_t s_chunk;
	const uint32_t rows = blockDim.x * a.chunk;
	for (;;) {
		if (threadIdx.x == 0) s_chunk = atomicAdd(a.work, 1u);
		__syncthreads();
		uint64_t base = (uint64_t)s_chunk * rows;
		__syncthreads();
		if (base >= a.n_total) break;
		for (uint32_t r = threadIdx.x; r < rows; r += blockDim.x) {
			uint64_t k = base + r;
			if (k < a.n_total) pair32_row<GOD, FULL>(a, P, G, st, (uint32_t)k);
		}
	}
}

// Neighbour lists of the current grid (test/debug): pass 0 counts, pass 1 writes
// the rows of each list (as global rows) at offs[row].
__global__ void k_neighbors(ULArgs a, const Geom* __restrict__ G, uint32_t* counts, uint32_t* idx,
                            const uint64_t* offs, int pass) {
	uint32_t k = blockIdx.x * blockDim.x + threadIdx.x;
	if (k >= a.n_total) return;
	const Rec64* rec = reinterpret_cast<const Rec64*>(a.rec);
	const Rec64 ri = load_rec(rec + k);
	Geom g = G[a.rec_body[k]];
	uint32_t i = a.perm[k];
	int lo_i, hi_i, lo_j, hi_j;
	stencil(g, a.keys_sorted[k], lo_i, hi_i, lo_j, hi_j);
	const uint32_t tot = *a.total_cells;
	double hi = ri.h;
	double radius2 = __dmul_rn(__dmul_rn(__dmul_rn(hi, hi), 2.), 2.);
	double lim = __dadd_rn(radius2, a.nbh_eps);
	uint32_t cnt = 0;
	for (int ni = lo_i; ni < hi_i; ni++) {
		uint32_t c0 = min(g.cell_off + (uint32_t)ni * g.ny + (uint32_t)lo_j, tot);
		uint32_t c1 = min(g.cell_off + (uint32_t)ni * g.ny + (uint32_t)hi_j, tot);
		for (uint32_t kj = a.cell_start[c0]; kj < a.cell_start[c1]; kj++) {
			const Rec64 rj = load_rec(rec + kj);
			double xij = __dsub_rn(ri.x, rj.x);
			double yij = __dsub_rn(ri.y, rj.y);
			double r2 = __dadd_rn(__dmul_rn(xij, xij), __dmul_rn(yij, yij));
			if (r2 <= lim) {
				if (pass == 1) idx[offs[i] + cnt] = a.perm[kj];
				cnt++;
			}
		}
	}
	if (pass == 0) counts[i] = cnt;
}

inline unsigned grid1(uint64_t n, unsigned bs) { return (unsigned)((n + bs - 1) / bs); }

// Threads a block of the kernels with a thread a row: fewer where 256 would leave SMs without
// a block, since an SM's rows share its narrow FP64 pipe
// (4,408 rows, strict gather: 15.0 us on 18 SMs, 9.5 on 138).
unsigned row_block(const ULArgs& a) {
	unsigned bs = 256;
	while (bs > 32 && grid1(a.n_total, bs) < a.sm_count) bs >>= 1;
	return bs;
}

// One block's FP64 divisions for the cell keys hold its SM's narrow pipe for 7.5 ns a row.
// Up to 1024 rows that is a fraction of the launches saved (one body of 856 rows, mixed step:
// 63 us with the general kernels, 61 this way); from there on a lone body's block is the
// longer one (1,684 rows 68 / 70 us, 2,608 72 / 80, 4,408 76 / 96).  With a body for every SM
// the blocks share the work: 152 bodies of 1,096 rows 281 / 215 us, of 4,408 771 / 696 (FP64
// 3044 / 2796 and 11,338 / 11,037).  The line between lies where every SM is known to have
// one; it could lie lower (19 bodies of 1,096 rows 134 / 104 us, of 4,408 198 / 163).
bool ul_small_grid(const ULArgs& a) {
	const uint32_t limit = a.n_bodies >= a.sm_count && a.sm_count ? GRID_BODY_MAX : 1024u;
	return a.max_body && a.max_body <= limit && a.n_bodies <= GRID_MAX_BODIES && !a.failed;
}

// The grid of the stage's positions; the caller's gather comes next.
cudaError_t build_grid(ULArgs& a, bool mixed, cudaStream_t s) {
	DevStatus* st = reinterpret_cast<DevStatus*>(a.status);
	const uint32_t cell_cap = a.cell_cap ? a.cell_cap : a.n_total + 1;
	if (ul_small_grid(a)) {
		const uint32_t hist_cap = (mixed ? 2u : 1u) * a.max_body + 16u;
		const size_t smem = hist_cap * sizeof(uint32_t) + a.max_body * sizeof(uint16_t);
		const unsigned T = a.max_body > 1024u ? 1024u : 256u;
		uint32_t* cells = reinterpret_cast<uint32_t*>(a.bbox);  // (the general kernels' bounding boxes)
		if (a.n_bodies == 1) {
			launch_after(k_body_sort<true>, 1, T, smem, s, a, mixed ? 1 : 0, cells, hist_cap, cell_cap);
		} else {
			launch_after(k_body_box, a.n_bodies, T, 0, s, a, mixed ? 1 : 0, cells);
			launch_after(k_body_sort<false>, a.n_bodies, T, smem, s, a, mixed ? 1 : 0, cells, hist_cap, cell_cap);
		}
		return cudaGetLastError();
	}
	launch_after(k_bbox_init, grid1(a.n_bodies, 128), 128, 0, s, a.n_bodies, a.bbox);
	const mfk_host::StateSoA& sv = a.stage == 0 ? a.base : a.st;
	launch_after(k_bbox, grid1(a.n_total, 256), 256, 0, s, a.n_total, sv.x, sv.y, a.h, sv.vx, sv.vy, a.body_of, mixed ? 1 : 0, a.bbox, a.failed);
	launch_after(k_geom, 1, 1024, 0, s, a.n_bodies, a.bbox, a.params, mixed ? 1 : 0, a.geom, a.total_cells, cell_cap, st, a.failed);
	launch_after(k_hash, grid1(a.n_total, row_block(a)), row_block(a), 0, s, a.n_total, sv.x, sv.y, a.body_of, a.geom, a.total_cells,
	             a.keys, a.perm_in, st, a.failed);
	size_t tmp = a.sort_tmp_bytes;
	cudaError_t e = cub::DeviceRadixSort::SortPairs(a.sort_tmp, tmp, a.keys, a.keys_sorted, a.perm_in, a.perm,
	                                                (int)a.n_total, 0, a.sort_bits, s);
	if (e != cudaSuccess) return e;
	a.fill_cells = 1;  // (the gather that follows also fills the cell table)
	return cudaGetLastError();
}

}  // namespace

size_t ul_sort_tmp_bytes(uint32_t n, int bits) {
	size_t bytes = 0;
	cub::DeviceRadixSort::SortPairs(nullptr, bytes, (uint32_t*)nullptr, (uint32_t*)nullptr, (uint32_t*)nullptr,
	                                (uint32_t*)nullptr, (int)n, 0, bits);
	return bytes;
}

// Kernels of this file that ul_stage launches: the grid's (CUB's sort not counted), the
// gather, the pair pass.
uint32_t ul_stage_launches(const ULArgs& a) {
	if (a.n_total == 0) return 0;
	const bool grid = a.strict_grid || a.stage == 0;
	return (!grid ? 0u : !ul_small_grid(a) ? 4u : a.n_bodies == 1 ? 1u : 2u) + (a.skip_gather ? 1u : 2u);
}

size_t ul_rec_bytes(bool mixed) { return mixed ? sizeof(Rec32) : sizeof(Rec64); }

cudaError_t ul_stage(const ULArgs& args, bool mixed, cudaStream_t s) {
	if (args.n_total == 0) return cudaSuccess;
	ULArgs a = args;
	DevStatus* st = reinterpret_cast<DevStatus*>(a.status);
	if (a.strict_grid || a.stage == 0) {
		cudaError_t e = build_grid(a, mixed, s);
		if (e != cudaSuccess) return e;
	}
	const unsigned rb = row_block(a);
	if (mixed) {
		if (!a.skip_gather) launch_after(k_gather32, grid1((uint64_t)a.n_total + 1, rb), rb, 0, s, a, a.params);
	} else {
		launch_after(k_gather64, grid1((uint64_t)a.n_total + 1, rb), rb, 0, s, a, a.params);
	}
	unsigned bs = a.block ? a.block : 128;
	unsigned grid = a.persistent ? a.grid : grid1(a.n_total, bs);
	if (mixed && a.persistent) {
		cudaError_t e = cudaMemsetAsync(a.work, 0, sizeof(uint32_t), s);
		if (e != cudaSuccess) return e;
	}
	if (a.ev_pair0) cudaEventRecord(a.ev_pair0, s);
	const bool god = a.flags & (A_GOD_CONT | A_GOD_MOM);
	if (mixed) {
		const bool full = !god && (a.flags & A_MONAGHAN) == A_MONAGHAN;
		const uint32_t split = !a.persistent && (a.split == 4 || a.split == 8) ? a.split : 1u;
		auto launch = [&](auto kernel) {
			launch_after(kernel, split > 1 ? grid1((uint64_t)a.n_total * split, bs) : grid, bs, 0, s, a, a.params, a.geom, st);
		};
		if (split == 1 && !god && !a.persistent && a.n_total <= a.sm_count * (4u * ORD_THREADS / 8u))
			launch_after(full ? k_pair_ordered<true> : k_pair_ordered<false>, grid1(8ull * a.n_total, ORD_THREADS), ORD_THREADS, 0, s, a, a.params, a.geom, st);
		else if (split == 4) launch(god ? k_pair_split<true, false, 4> : full ? k_pair_split<false, true, 4> : k_pair_split<false, false, 4>);
		else if (split == 8) launch(god ? k_pair_split<true, false, 8> : full ? k_pair_split<false, true, 8> : k_pair_split<false, false, 8>);
		else if (god || !full) launch(god ? k_pair<true, false, 3> : k_pair<false, false, 3>);
		else launch(a.n_total / PAIR_ROWS_MB4 >= a.sm_count ? k_pair<false, true, 4> : k_pair<false, true, 3>);
	} else {
		const unsigned g64 = grid1(a.n_total, P64_ROWS);
		if (god) launch_after(k_pair64<true>, g64, P64_THREADS, 0, s, a, a.params, a.geom, st);
		else launch_after(k_pair64<false>, g64, P64_THREADS, 0, s, a, a.params, a.geom, st);
	}
	if (a.ev_pair1) cudaEventRecord(a.ev_pair1, s);
	return cudaGetLastError();
}

// left/right_bndry_fun_ul (tensile.cpp:44-66) on the particles after the RK4 combine
// (rk4.h:105): of what they set only the velocity outlives the step, since every
// derivative evaluation starts from zeroed rates
__global__ void k_ul_bc(uint32_t n_bc, const uint32_t* __restrict__ rows, const double* __restrict__ v, double* vx,
                        double* vy) {
	uint32_t k = blockIdx.x * blockDim.x + threadIdx.x;
	if (k >= n_bc) return;
	uint32_t i = rows[k];
	vx[i] = v[k];
	vy[i] = 0.;
}

cudaError_t ul_bc(uint32_t n_bc, const uint32_t* rows, const double* v, double* vx, double* vy, cudaStream_t s) {
	k_ul_bc<<<grid1(n_bc, 128), 128, 0, s>>>(n_bc, rows, v, vx, vy);
	return cudaGetLastError();
}

cudaError_t ul_neighbors(const ULArgs& args, uint32_t* counts, uint32_t* idx, const uint64_t* offs, int pass,
                         cudaStream_t s) {
	if (args.n_total == 0) return cudaSuccess;
	ULArgs a = args;
	if (pass == 0) {
		cudaError_t e = build_grid(a, false, s);
		if (e != cudaSuccess) return e;
		launch_after(k_gather64, grid1((uint64_t)a.n_total + 1, 256), 256, 0, s, a, a.params);
	}
	k_neighbors<<<grid1(a.n_total, 128), 128, 0, s>>>(a, a.geom, counts, idx, offs, pass);
	return cudaGetLastError();
}

}  // namespace MF_NS
