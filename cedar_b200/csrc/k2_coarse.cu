// k2_coarse.cu -- the coarse end of a 2D V-cycle in one kernel launch.
//
// Below ~64x64 points a level's kernels are latency bound: each launch of the
// point, line and transfer kernels costs several microseconds however little
// work it has.  This kernel runs the whole sub-cycle from a coarse level down to
// the coarsest and back (cycle::vcycle::ncycle_helper,
// include/cedar/cycle/vcycle.h:57-115: pre-smoothing, residual, restriction,
// zero coarse iterate, ..., banded Cholesky, ..., interpolate-add,
// post-smoothing) with one CTA per problem and a barrier between steps.  Every
// point formula is the shared helper the separate kernels use (k2_point.cuh),
// and in FP64 the line solves run DPTTS2's sequential substitutions, so the
// result is the one the separate kernels give in CDR_LINES_EXACT mode.
//
// All levels of the sub-cycle live in shared memory for the whole launch (with
// compact rows): the operators, smoother factors and interpolation weights are
// staged once at entry, b of the first level is read and its x written back at
// exit, and nothing else touches global memory.  Loops map rows to warps and
// positions to lanes (no per-element division).  By default a cycle of a single
// problem or a plane fuses the levels of at most 32^2 in FP64 and 64^2 in FP32, as
// far as shared memory holds them (the callers' rules: pick_fused_level,
// Batch2::pick_fused); batches fuse from 32^2 in both.
#include <algorithm>

#include "k2_point.cuh"
#include "kernels2d.cuh"

namespace cdrgpu {

// 512 threads: a colour of 32-point lines needs 16 warps, a barrier of 32 warps costs
// more than the second round of the point steps, and two CTAs share an SM in a batch
constexpr int CC_THREADS = 512;
constexpr int CC_WARPS = CC_THREADS / 32;

// f(i, j) for i in [i0, i1], j in [j0, j1]: rows over the warps, positions over the lanes
template <typename F>
__device__ __forceinline__ void cc_rows(int i0, int i1, int j0, int j1, F f)
{
	const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
	for (int j = j0 + warp; j <= j1; j += CC_WARPS)
		for (int i = i0 + lane; i <= i1; i += 32) f(i, j);
}

// Planes of smoother factors kept for a relaxation type
__host__ __device__ inline int cc_sor_planes(int relax)
{
	return relax == CDR_RELAX_POINT ? 1 : relax == CDR_RELAX_LINE_Y ? 0 : 2;
}
__host__ __device__ inline int cc_sory_planes(int relax)
{
	return relax == CDR_RELAX_LINE_Y || relax == CDR_RELAX_LINE_XY ? 2 : 0;
}

// Shared-memory offsets (elements) of a level's arrays, -1 where it has none;
// rows of nx+2 elements, y-line factors transposed with rows of ny+2.
struct CcOffsets {
	int so, sor, sory, ci, x, b, r;
};
// One plane to stage: global source of problem 0, elements between problems,
// source pitch, rows of rowlen elements (back to back in shared memory at dst);
// pairs: rows move as 8-byte FP32 pairs.
struct CcPlane {
	const void *src;
	int pstride, spitch, dst;
	unsigned short rowlen, rows : 15, pairs : 1;
};
static_assert(sizeof(CcPlane) == 24, "one plane of the kernel parameter");
// a level stages at most its operator (5), both directions' factors (2 + 2) and
// its weights (8); the first one b and x in place of the weights
constexpr int kMaxCcPlanes = (5 + 2 + 2 + 8) * kMaxCoarseLevels;
// What a launch needs beside the levels, laid out on the host: the levels' x, r
// and restricted b first (zeroed as one range), then the staged planes, the line
// right-hand sides, and the coarsest solve's vector and factor in FP64.
template <typename T>
struct CcPlan {
	CoarseCycle<T> cc;
	CcOffsets off[kMaxCoarseLevels];
	int nzero = 0, lines = 0, dbl_byte = 0, nplanes = 0;
	size_t bytes = 0;
	CcPlane plane[kMaxCcPlanes];
};

// Byte counts stay in size_t until a level is known to fit: the plan is also the
// fit test for levels of any size, and its table holds ints.  bytes = SIZE_MAX:
// beyond the shared-memory limit or the plane table.
template <typename T>
static CcPlan<T> cc_plan(const CoarseCycle<T> &cc)
{
	// a kernel parameter: within the classic 4 KB (a plane smoother's graph holds
	// about a hundred of these launches, whose parameters every launch copies)
	static_assert(sizeof(CcPlan<T>) <= 4096, "plan within 4 KB");
	CcPlan<T> P;
	P.cc = cc;
	P.bytes = SIZE_MAX;
	size_t at = 0, ln = 0;
	int nplanes = 0;  // wanted, in the table or not
	auto fits = [&]() { return at * sizeof(T) <= kCoarseSmemMax && nplanes <= kMaxCcPlanes; };
	auto take = [&](size_t n) {
		const size_t o = at;
		at += n;
		return (int)o;
	};
	for (int l = 0; l < cc.nl; ++l) {
		const CoarseLevel<T> &L = cc.lv[l];
		const size_t pl = (size_t)(L.nx + 2) * (L.ny + 2);
		const bool last = l == cc.nl - 1;
		P.off[l] = CcOffsets{-1, -1, -1, -1, -1, -1, -1};
		if (l > 0 || !cc.x0) P.off[l].x = take(pl);
		if (!last) P.off[l].r = take(pl);
		if (l > 0) P.off[l].b = take(pl);
	}
	if (!fits()) return P;
	P.nzero = (int)at;
	for (int l = 0; l < cc.nl; ++l) {
		const CoarseLevel<T> &L = cc.lv[l];
		const int ii = L.nx + 2, jj = L.ny + 2;
		const size_t gpl = (size_t)L.pitch * jj;
		const bool last = l == cc.nl - 1;
		// planes of one array: rowlen x rows elements each, back to back in shared memory
		auto stage = [&](const T *src, int spitch, size_t splane, int rowlen, int rows, int planes) {
			const int o = take((size_t)rowlen * rows * planes);
			nplanes += planes;
			if (!fits()) return o;
			for (int q = 0; q < planes; ++q) {
				CcPlane &c = P.plane[P.nplanes++];
				c.src = src + q * splane;
				c.pstride = (int)(splane * planes);
				c.spitch = spitch;
				c.dst = o + q * rowlen * rows;
				c.rowlen = (unsigned short)rowlen;
				c.rows = (unsigned short)rows;
				c.pairs = sizeof(T) == 4 && rowlen % 2 == 0 && spitch % 2 == 0 && c.dst % 2 == 0 &&
				          c.pstride % 2 == 0 && (uintptr_t)c.src % 8 == 0;
			}
			return o;
		};
		if (!last) {
			P.off[l].so = stage(L.so, L.pitch, gpl, ii, jj, L.ns);
			// point relaxation keeps one plane of the two allocated
			const int np = cc_sor_planes(cc.relax);
			if (np) {
				P.off[l].sor = stage(L.sor, L.pitch, gpl, ii, jj, np);
				for (int q = 0; q < np && fits(); ++q) P.plane[P.nplanes - 1 - q].pstride = 2 * (int)gpl;
			}
			if (cc_sory_planes(cc.relax)) P.off[l].sory = stage(L.sory, L.tpitch, (size_t)L.tpitch * ii, jj, ii, 2);
			const size_t a = (size_t)((L.ny + 1) / 2) * L.nx, b = (size_t)((L.nx + 1) / 2) * L.ny;
			// FP32 lines of up to 64 points stay in registers
			if (sizeof(T) == 8 || L.nx > 64 || L.ny > 64) ln = std::max(ln, std::max(a, b));
		}
		if (l > 0) P.off[l].ci = stage(L.ci, L.pitch, gpl, ii, jj, 8);
		if (l == 0) P.off[l].b = stage(L.b, L.pitch, gpl, ii, jj, 1);
		if (l == 0 && cc.x0) P.off[l].x = stage(L.x, L.pitch, gpl, ii, jj, 1);
		if (!fits()) return P;
	}
	P.lines = take(ln);
	if (!fits()) return P;
	P.dbl_byte = (int)((at * sizeof(T) + 7) / 8 * 8);
	const CoarseLevel<T> &Cg = cc.lv[cc.nl - 1];
	const size_t n = (size_t)Cg.nx * Cg.ny;
	P.bytes = P.dbl_byte + (n + (size_t)(Cg.nx + 2) * n) * sizeof(double);
	return P;
}

// Shared copy of level l
template <typename T>
__device__ CoarseLevel<T> cc_view(const CcPlan<T> &P, int l, T *base)
{
	const CcOffsets &o = P.off[l];
	CoarseLevel<T> S;
	S.nx = P.cc.lv[l].nx;
	S.ny = P.cc.lv[l].ny;
	S.ns = P.cc.lv[l].ns;
	S.pitch = S.nx + 2;
	S.tpitch = S.ny + 2;
	S.so = base + o.so;
	S.sor = base + o.sor;
	S.sory = base + o.sory;
	S.ci = base + o.ci;
	S.x = base + o.x;
	S.b = base + o.b;
	S.r = base + o.r;
	return S;
}

// Staging by asynchronous copies (cp.async), every one in flight at once: a warp
// takes a plane and walks its rows, lanes along the row.  One loop over the
// host's plane table, so that its code is fetched once (a separate copy per
// array cost a microsecond of instruction fetch each).
template <int N>
__device__ __forceinline__ void cp_async(unsigned dst, const void *src)
{
	asm volatile("cp.async.ca.shared.global [%0], [%1], %2;\n" ::"r"(dst), "l"(src), "n"(N) : "memory");
}

template <typename T>
__device__ __forceinline__ void cc_stage(const CcPlan<T> &P, T *base)
{
	const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
	const long long prob = (long long)blockIdx.x * P.cc.bstep;
	const unsigned sbase = (unsigned)__cvta_generic_to_shared(base);
	for (int q = warp; q < P.nplanes; q += CC_WARPS) {
		const CcPlane &c = P.plane[q];
		const T *src = static_cast<const T *>(c.src) + prob * c.pstride;
		unsigned dst = sbase + (unsigned)c.dst * (unsigned)sizeof(T);
		const int rowlen = c.rowlen, rows = c.rows, spitch = c.spitch;
		const unsigned drow = (unsigned)(rowlen * (int)sizeof(T));
		if (sizeof(T) == 4 && c.pairs) {
			for (int j = 0; j < rows; ++j, src += spitch, dst += drow)
				for (int i = lane; i < rowlen / 2; i += 32) cp_async<8>(dst + 8 * i, src + 2 * i);
		} else {
			for (int j = 0; j < rows; ++j, src += spitch, dst += drow)
				for (int i = lane; i < rowlen; i += 32) cp_async<sizeof(T)>(dst + (unsigned)sizeof(T) * i, src + i);
		}
	}
}

// r = b - A x on the level (all interior points)
template <typename T, int NS>
__device__ void cc_residual(const CoarseLevel<T> &L)
{
	const size_t ps = (size_t)L.pitch * (L.ny + 2);
	cc_rows(1, L.nx, 1, L.ny, [&](int i, int j) {
		const size_t k = (size_t)j * L.pitch + i;
		L.r[k] = resid_at<T, NS>(L.so, ps, L.x, L.b, k, L.pitch);
	});
}

// coarse b = P^T r_fine
template <typename T>
__device__ void cc_restrict(const CoarseLevel<T> &F, const CoarseLevel<T> &C)
{
	const Dims2 f{F.nx, F.ny, F.pitch}, c{C.nx, C.ny, C.pitch};
	cc_rows(1, C.nx, 1, C.ny, [&](int ic, int jc) { restrict_at<T>(C.ci, F.r, C.b, f, c, ic, jc); });
}

// x_fine += P x_coarse + r/c on the fine-only points
template <typename T>
__device__ void cc_interp(const CoarseLevel<T> &F, const CoarseLevel<T> &C)
{
	const Dims2 f{F.nx, F.ny, F.pitch}, c{C.nx, C.ny, C.pitch};
	cc_rows(1, F.nx / 2 + 1, 1, F.ny / 2 + 1, [&](int ic, int jc) { interp_at<T>(C.ci, C.x, F.r, F.so, F.x, f, c, ic, jc); });
}

template <typename T, int NS>
__device__ void cc_gs(const CoarseLevel<T> &L, int updown)
{
	const size_t ps = (size_t)L.pitch * (L.ny + 2);
	if (NS == 5) {
		// DOWN: rows of odd j (0-based), in a row odd then even i, then the rows of even
		// j; UP: the reverse.  A row's second colour depends on its first only inside
		// the row, so the row's warp does both: two barriers per sweep instead of four.
		const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, first = updown == CDR_DOWN ? 1 : 2;
		for (int h = 0; h < 2; ++h) {
			for (int j = (h == 0 ? first : 3 - first) + 2 * warp; j <= L.ny; j += 2 * CC_WARPS)
				for (int c = 0; c < 2; ++c) {
					for (int i = (c == 0 ? first : 3 - first) + 2 * lane; i <= L.nx; i += 64)
						gs_at<T, 5>(L.so, ps, L.x, L.b, L.sor, (size_t)j * L.pitch + i, L.pitch);
					__syncwarp();
				}
			__syncthreads();
		}
	} else {
		for (int c = 0; c < 2; ++c) {
			const int par = updown == CDR_DOWN ? c : 1 - c;
			const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
			for (int j = 1 + warp; j <= L.ny; j += CC_WARPS) {
				const int i0 = ((1 + j) & 1) == par ? 1 : 2;
				for (int i = i0 + 2 * lane; i <= L.nx; i += 64)
					gs_at<T, 3>(L.so, ps, L.x, L.b, L.sor, (size_t)j * L.pitch + i, L.pitch);
			}
			__syncthreads();
		}
	}
}

// FP32 solve of a line of n <= 32 CS points by one warp, CS consecutive positions
// per lane in registers from their right-hand sides to their solution: the
// chunk form of cc_lines (affine maps of the chunks scanned over the lanes) with
// its operations and bits.  dd / ee: factors of position p (from 1) at dd[p], ee[p].
template <typename T, int CS, typename RHS, typename PUT>
__device__ __forceinline__ void cc_line(const T *dd, const T *ee, int n, RHS rhs, PUT put)
{
	const int lane = threadIdx.x & 31, lo = lane * CS;
	T r[CS], e[CS + 1], dv[CS];  // e[c]: multiplier of position lo + c, e[CS] of the one after the chunk
#pragma unroll
	for (int c = 0; c <= CS; ++c) e[c] = lo + c > 0 && lo + c < n ? ee[lo + c + 1] : T(0);
#pragma unroll
	for (int c = 0; c < CS; ++c) {
		dv[c] = lo + c < n ? dd[lo + c + 1] : T(0);
		r[c] = lo + c < n ? rhs(lo + c) : T(0);
	}
	T A = T(1), B = T(0);
#pragma unroll
	for (int c = 0; c < CS; ++c)
		if (lo + c < n) {
			B = madd(-e[c], B, r[c]);
			A = -e[c] * A;
		}
#pragma unroll
	for (int off = 1; off < 32; off <<= 1) {
		const T a2 = __shfl_up_sync(0xffffffffu, A, off), b2 = __shfl_up_sync(0xffffffffu, B, off);
		if (lane >= off) { B = madd(A, b2, B); A = A * a2; }
	}
	T v = __shfl_up_sync(0xffffffffu, B, 1);
	if (lane == 0) v = T(0);
#pragma unroll
	for (int c = 0; c < CS; ++c)
		if (lo + c < n) {
			v = lo + c == 0 ? r[c] : madd(-v, e[c], r[c]);
			r[c] = pivot_div(v, dv[c]);
		}
	A = T(1);
	B = T(0);
#pragma unroll
	for (int c = CS - 1; c >= 0; --c)
		if (lo + c < n) {
			B = madd(-e[c + 1], B, r[c]);
			A = -e[c + 1] * A;
		}
#pragma unroll
	for (int off = 1; off < 32; off <<= 1) {
		const T a2 = __shfl_down_sync(0xffffffffu, A, off), b2 = __shfl_down_sync(0xffffffffu, B, off);
		if (lane + off < 32) { B = madd(A, b2, B); A = A * a2; }
	}
	v = __shfl_down_sync(0xffffffffu, B, 1);
	if (lane == 31) v = T(0);
#pragma unroll
	for (int c = CS - 1; c >= 0; --c)
		if (lo + c < n) {
			v = lo + c == n - 1 ? r[c] : madd(-v, e[c + 1], r[c]);
			put(lo + c, v);
		}
}

// One zebra line sweep (both colours, relax_lines_2d's order).  Each colour:
// each line's warp forms its right-hand sides into sm (the other warps solve
// lines of the same colour, which this line does not read), then the
// substitutions run with the level's (shared-memory) pivots and multipliers:
// DPTTS2's sequential order in FP64 (one warp per line), affine-map scans over
// the lanes of one warp per line in FP32 (the preconditioner has no bitwise
// target; the separate FP32 kernels scan too).
template <typename T, int NS, int DIR>
__device__ void cc_lines(const CoarseLevel<T> &L, int updown, T *sm)
{
	const Dims2 d{L.nx, L.ny, L.pitch};
	const size_t ps = d.plane();
	const int n = DIR == CDR_DIR_X ? L.nx : L.ny;    // line length
	const int nl = DIR == CDR_DIR_X ? L.ny : L.nx;   // lines
	const T *fac = DIR == CDR_DIR_X ? L.sor : L.sory;
	const size_t eplane = DIR == CDR_DIR_X ? ps : (size_t)L.tpitch * (L.nx + 2);
	const int firsts[2] = {updown == CDR_DOWN ? 2 : 1, updown == CDR_DOWN ? 1 : 2};
	// x of position m (0-based) of line lc: the solves write their lines' x
	// directly (lines of one colour read only lines of the other)
	auto xat = [&](int lc, int m) -> size_t { return DIR == CDR_DIR_X ? d.at(m + 1, lc) : d.at(lc, m + 1); };
	for (int c = 0; c < 2; ++c) {
		const int first = firsts[c];
		const int ml = first > nl ? 0 : (nl - first) / 2 + 1;  // lines of this colour
		T *R = sm;
		if constexpr (sizeof(T) == 8) {
			// FP64: DPTTS2's sequential substitutions, one warp per line: the
			// line's right-hand sides and the quotients of the backward
			// substitution (which do not depend on its recurrence) by all lanes,
			// the two recurrences by lane 0, four positions per step with their
			// operands loaded ahead of the arithmetic
			const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
			for (int g = warp; g < ml; g += CC_THREADS / 32) {
				const int lc = first + 2 * g;
				// factors of position p at dd[p], ee[p] (position 1 is r[0])
				const T *dd = fac + (DIR == CDR_DIR_X ? (size_t)lc * L.pitch : (size_t)lc * L.tpitch);
				const T *ee = dd + eplane;
				T *r = R + g * n;
				for (int m = lane; m < n; m += 32) r[m] = line_rhs<T, NS, DIR>(L.so, ps, L.x, L.b, xat(lc, m), L.pitch);
				__syncwarp();
				if (lane == 0) {  // y(m) = r(m) - y(m-1) e(m+1), y(0) = r(0)
					T y = r[0];
					int m = 1;
					for (; m + 3 < n; m += 4) {
						const T e0 = ee[m + 1], e1 = ee[m + 2], e2 = ee[m + 3], e3 = ee[m + 4];
						const T a0 = r[m], a1 = r[m + 1], a2 = r[m + 2], a3 = r[m + 3];
						y = a0 - y * e0;
						r[m] = y;
						y = a1 - y * e1;
						r[m + 1] = y;
						y = a2 - y * e2;
						r[m + 2] = y;
						y = a3 - y * e3;
						r[m + 3] = y;
					}
					for (; m < n; ++m) {
						y = r[m] - y * ee[m + 1];
						r[m] = y;
					}
				}
				__syncwarp();
				for (int m = lane; m < n; m += 32) r[m] = pivot_div(r[m], dd[m + 1]);
				__syncwarp();
				if (lane == 0) {  // x(m) = y(m)/d(m+1) - x(m+1) e(m+2), x(n-1) = y(n-1)/d(n)
					T xv = r[n - 1];
					L.x[xat(lc, n - 1)] = xv;
					int m = n - 2;
					for (; m >= 3; m -= 4) {
						const T e0 = ee[m + 2], e1 = ee[m + 1], e2 = ee[m], e3 = ee[m - 1];
						const T q0 = r[m], q1 = r[m - 1], q2 = r[m - 2], q3 = r[m - 3];
						xv = q0 - xv * e0;
						L.x[xat(lc, m)] = xv;
						xv = q1 - xv * e1;
						L.x[xat(lc, m - 1)] = xv;
						xv = q2 - xv * e2;
						L.x[xat(lc, m - 2)] = xv;
						xv = q3 - xv * e3;
						L.x[xat(lc, m - 3)] = xv;
					}
					for (; m >= 0; --m) {
						xv = r[m] - xv * ee[m + 2];
						L.x[xat(lc, m)] = xv;
					}
				}
				__syncwarp();
			}
		} else {
			const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
			if (n <= 64) {
				for (int g = warp; g < ml; g += CC_WARPS) {
					const int lc = first + 2 * g;
					const T *dd = fac + (DIR == CDR_DIR_X ? (size_t)lc * L.pitch : (size_t)lc * L.tpitch);
					auto rhs = [&](int m) { return line_rhs<T, NS, DIR>(L.so, ps, L.x, L.b, xat(lc, m), L.pitch); };
					auto put = [&](int m, T v) { L.x[xat(lc, m)] = v; };
					if (n <= 32) cc_line<T, 1>(dd, dd + eplane, n, rhs, put);
					else cc_line<T, 2>(dd, dd + eplane, n, rhs, put);
				}
				__syncthreads();
				continue;
			}
			// FP32: one warp per line, each lane a chunk of consecutive positions;
			// both substitutions as affine-map scans over the lanes (shuffles)
			const int cs = (n + 31) / 32;  // chunk length
			for (int g = warp; g < ml; g += CC_THREADS / 32) {
				const int lc = first + 2 * g;
				const T *dd = fac + (DIR == CDR_DIR_X ? (size_t)lc * L.pitch : (size_t)lc * L.tpitch);
				const T *ee = dd + eplane;
				T *r = R + g * n;
				// the line's right-hand sides by its own warp (the other warps solve
				// lines of the same colour, which this line does not read)
				for (int m = lane; m < n; m += 32) r[m] = line_rhs<T, NS, DIR>(L.so, ps, L.x, L.b, xat(lc, m), L.pitch);
				__syncwarp();
				const int lo = lane * cs < n ? lane * cs : n, hi = lo + cs < n ? lo + cs : n;
				// forward y(m) = r(m) - y(m-1) E(m+1), y(0) = r(0)
				T A = T(1), B = T(0);
				for (int m = lo; m < hi; ++m) {
					const T a = m == 0 ? T(0) : -ee[m + 1];
					B = madd(a, B, r[m]);
					A = a * A;
				}
				for (int off = 1; off < 32; off <<= 1) {
					const T a2 = __shfl_up_sync(0xffffffffu, A, off), b2 = __shfl_up_sync(0xffffffffu, B, off);
					if (lane >= off) { B = madd(A, b2, B); A = A * a2; }
				}
				T y = __shfl_up_sync(0xffffffffu, B, 1);
				if (lane == 0) y = T(0);
				for (int m = lo; m < hi; ++m) {
					y = m == 0 ? r[0] : madd(-y, ee[m + 1], r[m]);
					r[m] = pivot_div(y, dd[m + 1]);
				}
				__syncwarp();
				// backward x(m) = y(m)/D(m+1) - x(m+1) E(m+2), x(n-1) = y(n-1)/D(n)
				A = T(1);
				B = T(0);
				for (int m = hi - 1; m >= lo; --m) {
					const T a = m == n - 1 ? T(0) : -ee[m + 2];
					B = madd(a, B, r[m]);
					A = a * A;
				}
				for (int off = 1; off < 32; off <<= 1) {
					const T a2 = __shfl_down_sync(0xffffffffu, A, off), b2 = __shfl_down_sync(0xffffffffu, B, off);
					if (lane + off < 32) { B = madd(A, b2, B); A = A * a2; }
				}
				T xv = __shfl_down_sync(0xffffffffu, B, 1);
				if (lane == 31) xv = T(0);
				for (int m = hi - 1; m >= lo; --m) {
					xv = m == n - 1 ? r[m] : madd(-xv, ee[m + 2], r[m]);
					L.x[xat(lc, m)] = xv;
				}
				__syncwarp();
			}
		}
		__syncthreads();  // this colour's lines are written into x
	}
}

template <typename T, int NS>
__device__ void cc_smooth(const CoarseCycle<T> &cc, const CoarseLevel<T> &L, int updown, T *sm)
{
	const int nrel = updown == CDR_DOWN ? cc.npre : cc.npost;
	for (int it = 0; it < nrel; ++it) {
		switch (cc.relax) {
		case CDR_RELAX_POINT: cc_gs<T, NS>(L, updown); break;
		case CDR_RELAX_LINE_X: cc_lines<T, NS, CDR_DIR_X>(L, updown, sm); break;
		case CDR_RELAX_LINE_Y: cc_lines<T, NS, CDR_DIR_Y>(L, updown, sm); break;
		default:  // x then y down, y then x up: one copy of each direction's code
			for (int h = 0; h < 2; ++h) {
				if ((h == 0) == (updown == CDR_DOWN)) cc_lines<T, NS, CDR_DIR_X>(L, updown, sm);
				else cc_lines<T, NS, CDR_DIR_Y>(L, updown, sm);
			}
		}
	}
}

// BMG2_SymStd_SOLVE_cg with DPBTRS('U') on the coarsest level by one warp
// (band_solve_warp): the right-hand side in shared memory (xs), the factor after
// it (staged with the levels).
template <typename T>
__device__ void cc_cg(const CoarseLevel<T> &L, double *xs)
{
	const int ldab = L.nx + 2, n = L.nx * L.ny;
	const double *abs = xs + n;
	cc_rows(1, L.nx, 1, L.ny, [&](int i, int j) { xs[(j - 1) * L.nx + i - 1] = (double)L.b[(size_t)j * L.pitch + i]; });
	__syncthreads();
	if (threadIdx.x < 32) band_solve_warp(abs, ldab, n, xs);
	__syncthreads();
	cc_rows(1, L.nx, 1, L.ny, [&](int i, int j) { L.x[(size_t)j * L.pitch + i] = (T)xs[(j - 1) * L.nx + i - 1]; });
}

template <typename T>
__global__ void __launch_bounds__(CC_THREADS, sizeof(T) == 4 ? 2 : 1) k_coarse_cycle(const __grid_constant__ CcPlan<T> P)
{
	await_previous();
	extern __shared__ __align__(16) unsigned char cc_smem[];
	const CoarseCycle<T> &cc = P.cc;
	T *base = reinterpret_cast<T *>(cc_smem);
	T *sm = base + P.lines;  // line right-hand sides
	double *xs = reinterpret_cast<double *>(cc_smem + P.dbl_byte);
	const int nl = cc.nl;
	// stage: operators, factors and weights of every level, b (and, with x0, x) of
	// the first level, and after the coarsest right-hand side xs its band factor; the
	// other x, r and b zero (ghost rings included)
	cc_stage<T>(P, base);
	{
		const CoarseLevel<T> &Cg = cc.lv[nl - 1];
		const int n = Cg.nx * Cg.ny, nab = (Cg.nx + 2) * n;
		const double *src = cc.abd + (size_t)blockIdx.x * cc.bstep * nab;
		const unsigned dst = (unsigned)__cvta_generic_to_shared(xs + n);
		for (int e = threadIdx.x; e < nab; e += CC_THREADS) cp_async<8>(dst + 8u * e, src + e);
	}
	for (int e = threadIdx.x; e < P.nzero; e += CC_THREADS) base[e] = T(0);
	asm volatile("cp.async.wait_all;\n" ::: "memory");
	__syncthreads();
	// The cycle as one sequence of steps (down: smooth, residual, restriction,
	// and the coarsest solve after the last; up: interpolation, smooth), so that
	// the code of each kind of step exists once: the first fetch of a code
	// region from instruction memory costs several microseconds, and separate
	// copies for the two legs paid it twice.
	if (nl == 1) {
		cc_cg<T>(cc_view(P, 0, base), xs);
		__syncthreads();
	}
	for (int step = 0; step < 2 * (nl - 1); ++step) {
		const bool down = step < nl - 1;
		const int l = down ? step : 2 * (nl - 1) - 1 - step;
		const CoarseLevel<T> F = cc_view(P, l, base), C = cc_view(P, l + 1, base);
		if (!down) {
			cc_interp<T>(F, C);
			__syncthreads();
		}
		const int updown = down ? CDR_DOWN : CDR_UP;
		if (F.ns == 5) cc_smooth<T, 5>(cc, F, updown, sm);
		else cc_smooth<T, 3>(cc, F, updown, sm);
		if (down) {
			if (F.ns == 5) cc_residual<T, 5>(F);
			else cc_residual<T, 3>(F);
			__syncthreads();
			cc_restrict<T>(F, C);  // the coarse iterate is still zero
			__syncthreads();
			if (l == nl - 2) {
				cc_cg<T>(cc_view(P, nl - 1, base), xs);
				__syncthreads();
			}
		} else {
			__syncthreads();
		}
	}
	{
		const CoarseLevel<T> S = cc_view(P, 0, base);
		const int gp = cc.lv[0].pitch;
		T *x = cc.lv[0].x + (size_t)blockIdx.x * cc.bstep * gp * (S.ny + 2);
		cc_rows(0, S.nx + 1, 0, S.ny + 1, [&](int i, int j) { x[(size_t)j * gp + i] = S.x[(size_t)j * S.pitch + i]; });
	}
}

// Shared memory a fused coarse cycle from level descriptor lv[0..nl) needs
template <typename T>
size_t coarse_cycle_bytes(const CoarseCycle<T> &cc)
{
	return cc_plan(cc).bytes;
}
template size_t coarse_cycle_bytes<double>(const CoarseCycle<double> &);
template size_t coarse_cycle_bytes<float>(const CoarseCycle<float> &);

template <typename T>
int coarse_cycle(const CoarseCycle<T> &cc, int nproblems, cudaStream_t st)
{
	if (cc.nl < 1 || cc.nl > kMaxCoarseLevels) {
		set_error(CDR_ERR_DIM, "fused coarse cycle over %d levels", cc.nl);
		return CDR_ERR_DIM;
	}
	const CcPlan<T> plan = cc_plan(cc);
	const size_t smem = plan.bytes;
	if (smem > kCoarseSmemMax) {
		set_error(CDR_ERR_DIM, "fused coarse cycle needs %zu bytes of shared memory", smem);
		return CDR_ERR_DIM;
	}
	launch(k_coarse_cycle<T>, nproblems, CC_THREADS, smem, st, plan);
	CDR_LAUNCH_CHECK();
	return CDR_OK;
}
template int coarse_cycle<double>(const CoarseCycle<double> &, int, cudaStream_t);

// Opt the fused kernels into the large shared-memory carve-out (once per
// process, before any graph capture: called from lines_prepare).
int coarse_prepare()
{
	CDR_CUDA_TRY(cudaFuncSetAttribute(k_coarse_cycle<double>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kCoarseSmemMax));
	CDR_CUDA_TRY(cudaFuncSetAttribute(k_coarse_cycle<float>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kCoarseSmemMax));
	return CDR_OK;
}
template int coarse_cycle<float>(const CoarseCycle<float> &, int, cudaStream_t);

}  // namespace cdrgpu
