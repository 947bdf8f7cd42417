// k2_stencil.cu -- 2D BoxMG point kernels for sm_100a.
//
// All kernels are HBM-bandwidth bound stencil sweeps: one thread per output
// point, coalesced along i, no tensor cores.  Arithmetic is written in the
// reference's operand order and the library is compiled without FMA
// contraction, so residual, point Gauss-Seidel, restriction, interpolation and
// the interpolation setup give the same bits as Cedar's serial kernels.
#include <cstdint>
#include <type_traits>

#include "k2_point.cuh"
#include "kernels2d.cuh"

namespace cdrgpu {

constexpr int NORM_MAX_BLOCKS = 2048;

// Blocks per problem of a residual with norm: all 2048 partial-sum slots for a
// single problem, an equal share of them for each problem of a batch (the
// tile -> block map, hence the summation order, is fixed for a given batch).
int norm_blocks(Dims2 d)
{
	const int ntiles = ceil_div(d.nx, TX) * ceil_div(d.ny, TY);
	int per = NORM_MAX_BLOCKS / (d.nb > 0 ? d.nb : 1);
	if (per < 1) per = 1;
	return ntiles < per ? ntiles : per;
}

// ------------------------------------------------------------------ residual
// Grid-stride over 32x8 tiles; with NORM each block leaves the sum of r^2 over
// its tiles in partial[blockIdx.x] (fixed tile->block map: deterministic).
template <typename T, int NS, bool NORM>
__global__ void __launch_bounds__(TX *TY) k_residual(const T *__restrict__ so, const T *__restrict__ q,
                                                     const T *__restrict__ qf, T *__restrict__ res, Dims2 d,
                                                     double *__restrict__ partial)
{
	await_previous();
	__shared__ double sh[TX * TY / 32];
	const int tiles_x = (d.nx + TX - 1) / TX;
	const int ntiles = tiles_x * ((d.ny + TY - 1) / TY);
	const size_t ps = d.plane();
	so += d.bofs(NS * ps);
	q += d.bofs(ps);
	qf += d.bofs(ps);
	res += d.bofs(ps);
	double acc = 0.0;
	for (int t = blockIdx.x; t < ntiles; t += gridDim.x) {
		int i = (t % tiles_x) * TX + threadIdx.x + 1;
		int j = (t / tiles_x) * TY + threadIdx.y + 1;
		if (i <= d.nx && j <= d.ny) {
			size_t k = d.at(i, j);
			T r = resid_at<T, NS>(so, ps, q, qf, k, d.pitch);
			res[k] = r;
			if (NORM) acc += (double)r * (double)r;
		}
	}
	if (NORM) {
		double s = block_sum<TX * TY / 32>(acc, sh);
		if (threadIdx.x == 0 && threadIdx.y == 0) partial[(size_t)blockIdx.z * gridDim.x + blockIdx.x] = s;
	}
}

// The same residual with V = 16 / sizeof(T) consecutive points of a row per
// thread (16-byte loads; rows 16-byte aligned): a tile is 32 V x 8 points.
// The left and right neighbours of the vector are separate loads (L1 hits).
// Per point the operand order of resid_at, so the bits are the same.
template <typename T, int NS, bool NORM>
__global__ void __launch_bounds__(TX *TY) k_residual_v(const T *__restrict__ so, const T *__restrict__ q,
                                                       const T *__restrict__ qf, T *__restrict__ res, Dims2 d,
                                                       double *__restrict__ partial)
{
	await_previous();
	constexpr int V = 16 / sizeof(T);
	using VT = typename std::conditional<sizeof(T) == 4, float4, double2>::type;
	__shared__ double sh[TX * TY / 32];
	const int tiles_x = (d.nx + TX * V) / (TX * V);  // columns 0 .. nx
	const int ntiles = tiles_x * ((d.ny + TY - 1) / TY);
	const size_t ps = d.plane();
	const int P = d.pitch;
	so += d.bofs(NS * ps);
	q += d.bofs(ps);
	qf += d.bofs(ps);
	res += d.bofs(ps);
	const T *c = so, *w = so + ps, *s = so + 2 * ps, *sw = so + (NS == 5 ? 3 : 0) * ps,
	        *nw = so + (NS == 5 ? 4 : 0) * ps;
	auto vld = [](const T *p, T *out) {
		const VT t = *reinterpret_cast<const VT *>(p);
		const T *e = reinterpret_cast<const T *>(&t);
#pragma unroll
		for (int m = 0; m < V; ++m) out[m] = e[m];
	};
	double acc = 0.0;
	for (int t = NORM ? blockIdx.x : 0; t < (NORM ? ntiles : 1); t += NORM ? gridDim.x : 1) {
		const int tx = NORM ? t % tiles_x : blockIdx.x, ty = NORM ? t / tiles_x : blockIdx.y;
		const int i0 = (tx * TX + threadIdx.x) * V;
		const int j = ty * TY + threadIdx.y + 1;
		if (i0 > d.nx || j > d.ny) continue;
		const size_t k = (size_t)j * P + i0;
		const bool lft = i0 >= 1, rgt = i0 + V <= d.nx + 1;
		// rows j - 1 (m), j (c), j + 1 (p) of q with the left and right neighbours
		T qm[V + 2], qc[V + 2], qp[V + 2];
		vld(q + k - P, qm + 1);
		vld(q + k, qc + 1);
		vld(q + k + P, qp + 1);
		qm[0] = lft ? q[k - P - 1] : T(0);
		qc[0] = lft ? q[k - 1] : T(0);
		qp[0] = lft ? q[k + P - 1] : T(0);
		qm[V + 1] = rgt ? q[k - P + V] : T(0);
		qc[V + 1] = rgt ? q[k + V] : T(0);
		qp[V + 1] = rgt ? q[k + P + V] : T(0);
		T cc[V], ww[V + 1], s0[V], s1[V], bb[V];
		vld(c + k, cc);
		vld(w + k, ww);
		ww[V] = rgt ? w[k + V] : T(0);
		vld(s + k, s0);
		vld(s + k + P, s1);
		vld(qf + k, bb);
		T sw0[V], sw1[V + 1], nw0[V + 1], nw1[V];
		if (NS == 5) {
			vld(sw + k, sw0);
			vld(sw + k + P, sw1);
			sw1[V] = rgt ? sw[k + P + V] : T(0);
			vld(nw + k, nw0);
			nw0[V] = rgt ? nw[k + V] : T(0);
			vld(nw + k + P, nw1);
		}
		T r[V];
#pragma unroll
		for (int m = 0; m < V; ++m) {
			// column i0 + m: index m + 1 of the q rows
			T a = madd(ww[m], qc[m], bb[m]);
			a = madd(ww[m + 1], qc[m + 2], a);
			a = madd(s0[m], qm[m + 1], a);
			a = madd(s1[m], qp[m + 1], a);
			if (NS == 5) {
				a = madd(sw0[m], qm[m], a);
				a = madd(nw0[m + 1], qm[m + 2], a);
				a = madd(nw1[m], qp[m], a);
				a = madd(sw1[m + 1], qp[m + 2], a);
			}
			r[m] = madd(-cc[m], qc[m + 1], a);
		}
		if (lft && i0 + V - 1 <= d.nx) {
			VT o;
			T *e = reinterpret_cast<T *>(&o);
#pragma unroll
			for (int m = 0; m < V; ++m) e[m] = r[m];
			*reinterpret_cast<VT *>(res + k) = o;
		} else {
#pragma unroll
			for (int m = 0; m < V; ++m)
				if (i0 + m >= 1 && i0 + m <= d.nx) res[k + m] = r[m];
		}
		if (NORM) {
#pragma unroll
			for (int m = 0; m < V; ++m)
				if (i0 + m >= 1 && i0 + m <= d.nx) acc += (double)r[m] * (double)r[m];
		}
	}
	if (NORM) {
		double sum = block_sum<TX * TY / 32>(acc, sh);
		if (threadIdx.x == 0 && threadIdx.y == 0) partial[(size_t)blockIdx.z * gridDim.x + blockIdx.x] = sum;
	}
}

// one block per problem: out[b] = sqrt(sum of partial[b*n .. b*n+n))
__global__ void __launch_bounds__(1024) k_norm_finish(const double *__restrict__ partial, int n, double *out)
{
	await_previous();
	__shared__ double sh[32];
	partial += (size_t)blockIdx.x * n;
	out += blockIdx.x;
	double v = 0;
	for (int i = threadIdx.x; i < n; i += blockDim.x) v += partial[i];
	for (int o = 16; o > 0; o >>= 1) v += __shfl_down_sync(0xffffffffu, v, o);
	if ((threadIdx.x & 31) == 0) sh[threadIdx.x >> 5] = v;
	__syncthreads();
	if (threadIdx.x < 32) {
		v = sh[threadIdx.x];
		for (int o = 16; o > 0; o >>= 1) v += __shfl_down_sync(0xffffffffu, v, o);
		if (threadIdx.x == 0) *out = sqrt(v);
	}
}

template <typename T>
int residual_2d(const T *so, int nstencil, const T *x, const T *b, T *r, Dims2 d, double *norm_out,
                double *partial, cudaStream_t st)
{
	const int ntiles = ceil_div(d.nx, TX) * ceil_div(d.ny, TY);
	dim3 blk(TX, TY);
	// 16-byte rows: the vector kernel (its tiles are V times wider, so fewer partials)
	constexpr int V = 16 / sizeof(T);
	if (((uintptr_t)so | (uintptr_t)x | (uintptr_t)b | (uintptr_t)r) % 16 == 0 && d.pitch % V == 0) {
		const int tx = ceil_div(d.nx + 1, TX * V), ty = ceil_div(d.ny, TY);
		if (norm_out) {
			int nb = norm_blocks(d);
			nb = nb < tx * ty ? nb : tx * ty;
			if (nstencil == 5) launch(k_residual_v<T, 5, true>, dim3(nb, 1, d.nb), blk, 0, st, so, x, b, r, d, partial);
			else launch(k_residual_v<T, 3, true>, dim3(nb, 1, d.nb), blk, 0, st, so, x, b, r, d, partial);
			CDR_LAUNCH_CHECK();
			launch(k_norm_finish, d.nb, 1024, 0, st, partial, nb, norm_out);
		} else {
			if (nstencil == 5) launch(k_residual_v<T, 5, false>, dim3(tx, ty, d.nb), blk, 0, st, so, x, b, r, d, nullptr);
			else launch(k_residual_v<T, 3, false>, dim3(tx, ty, d.nb), blk, 0, st, so, x, b, r, d, nullptr);
		}
		CDR_LAUNCH_CHECK();
		return CDR_OK;
	}
	if (norm_out) {
		int nb = norm_blocks(d);
		if (nstencil == 5) launch(k_residual<T, 5, true>, dim3(nb, 1, d.nb), blk, 0, st, so, x, b, r, d, partial);
		else launch(k_residual<T, 3, true>, dim3(nb, 1, d.nb), blk, 0, st, so, x, b, r, d, partial);
		CDR_LAUNCH_CHECK();
		launch(k_norm_finish, d.nb, 1024, 0, st, partial, nb, norm_out);
	} else {
		if (nstencil == 5) launch(k_residual<T, 5, false>, dim3(ntiles, 1, d.nb), blk, 0, st, so, x, b, r, d, nullptr);
		else launch(k_residual<T, 3, false>, dim3(ntiles, 1, d.nb), blk, 0, st, so, x, b, r, d, nullptr);
	}
	CDR_LAUNCH_CHECK();
	return CDR_OK;
}
template int residual_2d<double>(const double *, int, const double *, const double *, double *, Dims2, double *,
                                 double *, cudaStream_t);

template int residual_2d<float>(const float *, int, const float *, const float *, float *, Dims2, double *,
                                double *, cudaStream_t);

// ------------------------------------------------------------ point smoother
// BMG2_SymStd_SETUP_recip (src/2d/ftn/BMG2_SymStd_SETUP_recip.f90:63-67).
template <typename T>
__global__ void k_recip(const T *__restrict__ so, int ns, T *__restrict__ sor, Dims2 d)
{
	await_previous();
	so += d.bofs(ns * d.plane());
	sor += d.bofs(2 * d.plane());
	int i = blockIdx.x * TX + threadIdx.x + 1, j = blockIdx.y * TY + threadIdx.y + 1;
	if (i <= d.nx && j <= d.ny) sor[d.at(i, j)] = T(1) / so[d.at(i, j)];
}

template <typename T>
int setup_recip_2d(const T *so, T *sor, Dims2 d, cudaStream_t st, int ns)
{
	launch(k_recip<T>, dim3(ceil_div(d.nx, TX), ceil_div(d.ny, TY), d.nb), dim3(TX, TY), 0, st, so, ns, sor, d);
	CDR_LAUNCH_CHECK();
	return CDR_OK;
}
template int setup_recip_2d<double>(const double *, double *, Dims2, cudaStream_t, int);
template int setup_recip_2d<float>(const float *, float *, Dims2, cudaStream_t, int);

// One colour of BMG2_SymStd_relax_GS (src/2d/ftn/BMG2_SymStd_relax_GS.f90:93-133).
// 5-point: points with (i + j) % 2 == par (red-black); 9-point: points with
// i % 2 == pi and j % 2 == pj (four colours).  Points of one colour are
// independent, so one launch per colour reproduces the sequential sweep.  LEAD: the
// next kernel is let in (await_previous).
template <typename T, int NS, bool LEAD = true>
__global__ void __launch_bounds__(TX *TY) k_gs_colour(const T *__restrict__ so, T *__restrict__ q,
                                                      const T *__restrict__ qf, const T *__restrict__ sor,
                                                      Dims2 d, int pi, int pj)
{
	if (LEAD) await_previous();
	else await_previous_only();
	const size_t ps = d.plane();
	const int pitch = d.pitch;
	so += d.bofs(NS * ps);
	q += d.bofs(ps);
	qf += d.bofs(ps);
	sor += d.bofs(2 * ps);
	int j, i;
	if (NS == 3) {
		j = blockIdx.y * TY + threadIdx.y + 1;
		int i0 = ((1 + j) & 1) == pi ? 1 : 2;  // pi carries the (i+j) parity here
		i = i0 + 2 * (blockIdx.x * TX + threadIdx.x);
	} else {
		j = (pj ? 1 : 2) + 2 * (blockIdx.y * TY + threadIdx.y);
		i = (pi ? 1 : 2) + 2 * (blockIdx.x * TX + threadIdx.x);
	}
	if (i > d.nx || j > d.ny) return;
	gs_at<T, NS>(so, ps, q, qf, sor, d.at(i, j), pitch);
}

// Two colours of the nine-point sweep (BMG2_SymStd_relax_GS.f90:93-133) in one
// pass: the rows of one parity, first the points of one x-parity, then the
// others.  A row's second colour depends on the first only inside the row, so a
// block that owns whole rows needs no other block, and a sweep is two launches.
// A thread takes the points a = 2t, b = 2t + 1 (0-based) and loads every operand
// of both at once: a row's operator lines are read once with all of their bytes
// used (one colour per launch uses every second element, and reads each line
// twice).  A visit of a 1000 x 701 FP64 level (two sweeps, residual, transfers)
// 65 -> 54 us; in segments of 512 pairs 70 us.  Rows longer than
// 2 W points run in segments from the side whose first colour the second one
// reads.  SECOND_A: b first, then a (DOWN); else a, then b (UP).
template <typename T, bool VEC, bool SECOND_A>
__global__ void __launch_bounds__(256) k_gs_rows(const T *__restrict__ so, T *__restrict__ q, const T *__restrict__ qf,
                                                 const T *__restrict__ sor, Dims2 d, int j0, int W)
{
	await_previous();
	using V2 = typename Vec2<T>::type;
	__shared__ T sh[256];    // first-colour values of the segment
	__shared__ T edge[256];  // per row: the first-colour value the next segment reads
	const size_t ps = d.plane();
	so += d.bofs(5 * ps);
	q += d.bofs(ps);
	qf += d.bofs(ps);
	sor += d.bofs(2 * ps);
	const int r = threadIdx.x / W, t0 = threadIdx.x - r * W;
	const int j = j0 + 2 * (int)(blockIdx.x * (blockDim.x / W) + r);
	const int nT = d.nx / 2 + 1, nseg = (nT + W - 1) / W, p = d.pitch;
	auto pair = [&](const T *x, T(&v)[2]) {
		if constexpr (VEC) {
			const V2 u = *reinterpret_cast<const V2 *>(x);
			v[0] = u.x;
			v[1] = u.y;
		} else {
			v[0] = x[0];
			v[1] = x[1];
		}
	};
	for (int s = 0; s < nseg; ++s) {
		const int t = (SECOND_A ? s : nseg - 1 - s) * W + t0;
		const bool live = j <= d.ny && t < nT, va = live && t >= 1, vb = live && 2 * t + 1 <= d.nx;
		const size_t k = (size_t)j * p + 2 * t;
		T f[2], ds[2], w[3], s0[2], s1[2], sw0[2], nw0[2], nw1[2], sw1[2], Y[4], M[4], P[4];
		T first = T(0);
		// point e (0: a, 1: b) from its row neighbours, in gs_at's operand order
		auto point = [&](int e, T left, T right) -> T {
			T acc = madd(w[e], left, f[e]);
			acc = madd(w[e + 1], right, acc);
			acc = madd(s0[e], M[1 + e], acc);
			acc = madd(s1[e], P[1 + e], acc);
			acc = madd(sw0[e], M[e], acc);
			acc = madd(nw0[e], M[2 + e], acc);
			acc = madd(nw1[e], P[e], acc);
			acc = madd(sw1[e], P[2 + e], acc);
			return acc * ds[e];
		};
		if (live) {
			auto row4 = [&](const T *x, T(&v)[4]) {  // left neighbour of a, a, b, right neighbour of b
				T c[2];
				pair(x, c);
				v[0] = t >= 1 ? x[-1] : T(0);
				v[1] = c[0];
				v[2] = c[1];
				v[3] = vb ? x[2] : T(0);
			};
			auto right = [&](const T *x, T(&v)[2]) {  // a plane at the right neighbours
				v[0] = x[1];
				v[1] = vb ? x[2] : T(0);
			};
			const T *cw = so + ps + k, *cs = so + 2 * ps + k, *csw = so + 3 * ps + k, *cnw = so + 4 * ps + k;
			T c[2];
			pair(cw, c);
			w[0] = c[0];
			w[1] = c[1];
			w[2] = vb ? cw[2] : T(0);
			pair(cs, s0);
			pair(cs + p, s1);
			pair(csw, sw0);
			right(cnw, nw0);
			pair(cnw + p, nw1);
			right(csw + p, sw1);
			pair(qf + k, f);
			pair(sor + k, ds);
			row4(q + k, Y);
			row4(q + k - p, M);
			row4(q + k + p, P);
			// a point outside the interior keeps its value
			if (SECOND_A) first = vb ? point(1, Y[1], Y[3]) : Y[2];
			else first = va ? point(0, Y[0], Y[2]) : Y[1];
		}
		sh[threadIdx.x] = first;
		__syncthreads();  // the segment's row is read, its first colour formed
		if (live) {
			T second;
			if (SECOND_A) second = va ? point(0, t0 > 0 ? sh[threadIdx.x - 1] : edge[r], first) : T(0);
			else second = vb ? point(1, first, t + 1 >= nT ? Y[3] : t0 + 1 < W ? sh[threadIdx.x + 1] : edge[r]) : T(0);
			const T na = SECOND_A ? second : first, nb = SECOND_A ? first : second;
			T *qo = q + k;
			if (VEC && va && vb) {
				V2 v;
				v.x = na;
				v.y = nb;
				*reinterpret_cast<V2 *>(qo) = v;
			} else {
				if (va) qo[0] = na;
				if (vb) qo[1] = nb;
			}
		}
		if (nseg > 1) {
			__syncthreads();  // edge and sh are read
			if (t0 == (SECOND_A ? W - 1 : 0)) edge[r] = first;
		}
	}
}


// Periodic branch (BMG2_SymStd_relax_GS.f90:139-226): the reference copies a
// row's x ghosts after the row's points of a colour and the y ghost rows after
// the whole sweep.  Points of a colour never read another row's x ghosts that
// the same colour changes (five-point: no diagonal couplings; nine-point: the
// rows of one colour are two apart), so one copy launch after each colour
// launch gives the same values.
template <typename T>
int relax_point_2d(const T *so, int nstencil, T *x, const T *b, const T *sor, Dims2 d, int updown,
                   cudaStream_t st, int per)
{
	dim3 blk(TX, TY);
	const bool perx = per & 1, pery = (per >> 1) & 1;
	// Nine-point rows, two colours per launch: W pairs of points per row and segment
	// (equal segments of at most 256), rows to a block of 128 threads or one longer
	// row.  A row of three segments or more is a chain of them in one block, so few
	// such rows leave the chip idle: they go by colours, which tile x as well.  The
	// line: 32 rows of a parity per segment, two to an SM at most.  Both sides, FP64
	// us a sweep, colours | rows: 1024 x 128 7.5 | 9.4, x 320 11.0 | 9.6; 2048 x 256
	// 11.2 | 13.5, x 384 15.4 | 15.1; 4096 x 512 37 | 47, x 640 74 | 58; 16384 x 16
	// 8.4 | 78, x 256 122 | 164, x 768 348 | 233; FP32 4096 x 256 11.8 | 16.5, 8192 x
	// 512 45 | 57, x 640 78 | 67.  Within a fifth of the line it costs some levels:
	// FP64 3000 x 600 29.5 | 32.7, 8192 x 512 124 | 99.  Rows of one or two segments
	// are the faster ones at any height (700 x 16 8.4 | 6.7).
	const int nT = d.nx / 2 + 1, nseg = ceil_div(nT, 256), W = ceil_div(nT, nseg), R = W < 128 ? 128 / W : 1;
	const long row_blocks = (long)(d.ny / 2) / R * d.nb;
	const bool rows = !per && (nseg <= 2 || row_blocks >= (32 * nseg < 296 ? 32 * nseg : 296));
	if (nstencil == 5 && rows) {
		const bool vec = d.pitch % 2 == 0 &&
		                 ((uintptr_t)so | (uintptr_t)x | (uintptr_t)b | (uintptr_t)sor) % (2 * sizeof(T)) == 0;
		for (int c = 0; c < 2; ++c) {
			// DOWN: rows of odd 0-based j first, i odd then even; UP: the reverse
			const int j0 = (updown == CDR_DOWN) == (c == 0) ? 1 : 2;
			if (j0 > d.ny) continue;
			const dim3 grd(ceil_div((d.ny - j0) / 2 + 1, R), 1, d.nb);
			// not early where the blocks crowd on the SMs that the launch before leaves free
			// (early | not, us a sweep): FP64 1200 x 1080 16.2 | 14.5, unaligned 1400 x 1260
			// 34.7 | 30.8; FP32 1000 x 900 9.6 | 8.5, 2048 x 1024 17.2 | 14.1; but 850 x 765
			// (40 SMs' worth) 6.7 | 7.5, FP64 2048 x 2048 (103) 74.1 | 75.4
			const double sms = launch_size(grd, R * W, 0).sms;
			const bool early = sms < 45.0 || (sizeof(T) == 8 && sms > 90.0);
			if (updown == CDR_DOWN) {
				if (vec) launch_as(early, k_gs_rows<T, true, true>, grd, R * W, 0, st, so, x, b, sor, d, j0, W);
				else launch_as(early, k_gs_rows<T, false, true>, grd, R * W, 0, st, so, x, b, sor, d, j0, W);
			} else {
				if (vec) launch_as(early, k_gs_rows<T, true, false>, grd, R * W, 0, st, so, x, b, sor, d, j0, W);
				else launch_as(early, k_gs_rows<T, false, false>, grd, R * W, 0, st, so, x, b, sor, d, j0, W);
			}
			CDR_LAUNCH_CHECK();
		}
	} else if (nstencil == 5) {
		// DOWN: (JBEG, IBEG) = (2,2),(2,3),(3,2),(3,3) with JBEG outer; UP reversed.
		// Fortran index 2 is 0-based 1 (odd), 3 is 0-based 2 (even).
		const int order[4][2] = {{1, 1}, {1, 0}, {0, 1}, {0, 0}};  // (j odd?, i odd?)
		dim3 grd(ceil_div((d.nx + 1) / 2, TX), ceil_div((d.ny + 1) / 2, TY), d.nb);
		// FP64 beyond 90 SMs' worth not early, as the rows above (3000 x 300 18.6 | 16.6,
		// 4096 x 256 18.4 | 17.4; FP32 11.6 | 12.5)
		const bool early = sizeof(T) == 4 || launch_size(grd, blk, 0).sms <= 90.0;
		for (int c = 0; c < 4; ++c) {
			int o = updown == CDR_DOWN ? c : 3 - c;
			launch_as(early, k_gs_colour<T, 5>, grd, blk, 0, st, so, x, b, sor, d, order[o][1], order[o][0]);
			CDR_LAUNCH_CHECK();
			if (perx) CDR_TRY(ghost_copy_2d<T>(x, d, 1, 1, 0, order[o][0], st));
		}
	} else {
		// DOWN: JO = 2 then 3; a point is swept in pass JO when (I + J + JO) is even,
		// i.e. 0-based (i + j) even first, odd second.  UP reversed.
		dim3 grd(ceil_div((d.nx + 1) / 2, TX), ceil_div(d.ny, TY), d.nb);
		for (int c = 0; c < 2; ++c) {
			int par = updown == CDR_DOWN ? c : 1 - c;
			// FP32 blocks are so short that beyond two waves the next kernel is not let in:
			// 2000 x 1800 19.0 -> 17.3 us a sweep, 1400 x 1260 10.2 -> 9.6
			if (sizeof(T) == 4 && (long)grd.x * grd.y * grd.z > 2 * 8 * 148)
				launch(k_gs_colour<T, 3, sizeof(T) != 4>, grd, blk, 0, st, so, x, b, sor, d, par, 0);
			else
				launch(k_gs_colour<T, 3>, grd, blk, 0, st, so, x, b, sor, d, par, 0);
			CDR_LAUNCH_CHECK();
			if (perx) CDR_TRY(ghost_copy_2d<T>(x, d, 1, 1, 0, -1, st));
		}
	}
	if (pery) CDR_TRY(ghost_copy_2d<T>(x, d, 1, 0, 1, -1, st));
	return CDR_OK;
}
template int relax_point_2d<double>(const double *, int, double *, const double *, const double *, Dims2, int,
                                    cudaStream_t, int);
template int relax_point_2d<float>(const float *, int, float *, const float *, const float *, Dims2, int,
                                   cudaStream_t, int);

// ---------------------------------------------------------------- restriction
// BMG2_SymStd_restrict (src/2d/ftn/BMG2_SymStd_restrict.f90:72-92): coarse
// (ic, jc) sits on fine (2ic-1, 2jc-1) (0-based, ghosts at 0).
template <typename T, typename TC = T>
__global__ void __launch_bounds__(TX *TY) k_restrict(const TC *__restrict__ ci, const T *__restrict__ q,
                                                     TC *__restrict__ qc, Dims2 f, Dims2 c)
{
	await_previous();
	int ic = blockIdx.x * TX + threadIdx.x + 1, jc = blockIdx.y * TY + threadIdx.y + 1;
	if (ic > c.nx || jc > c.ny) return;
	const size_t cps = c.plane();
	ci += c.bofs(8 * cps);
	q += f.bofs(f.plane());
	qc += c.bofs(cps);
	restrict_at<T, TC>(ci, q, qc, f, c, ic, jc);
}

template <typename T>
int restrict_2d(const T *ci, const T *rf, T *bc, Dims2 f, Dims2 c, cudaStream_t st)
{
	launch(k_restrict<T>, dim3(ceil_div(c.nx, TX), ceil_div(c.ny, TY), c.nb), dim3(TX, TY), 0, st, ci, rf, bc, f, c);
	CDR_LAUNCH_CHECK();
	return CDR_OK;
}
template int restrict_2d<double>(const double *, const double *, double *, Dims2, Dims2, cudaStream_t);
template int restrict_2d<float>(const float *, const float *, float *, Dims2, Dims2, cudaStream_t);

int restrict_2d_mixed(const double *ci, const float *rf, double *bc, Dims2 f, Dims2 c, cudaStream_t st)
{
	launch(k_restrict<float, double>, dim3(ceil_div(c.nx, TX), ceil_div(c.ny, TY), c.nb), dim3(TX, TY), 0, st, ci, rf, bc,
	                                                                                                     f, c);
	CDR_LAUNCH_CHECK();
	return CDR_OK;
}

// ------------------------------------------------------------ interpolate-add
// BMG2_SymStd_interp_add (src/2d/ftn/BMG2_SymStd_interp_add.f90:101-137).  One
// thread per coarse cell (IC, JC) of the reference loop (0-based ic in
// [1, nxf/2+1]); it owns fine points (i, j), (i-1, j), (i, j-1), (i-1, j-1) with
// i = 2ic-1.  r/c is formed on the fly instead of dividing r in place.
template <typename T, typename TC = T>
__global__ void __launch_bounds__(TX *TY) k_interp_add(const TC *__restrict__ ci, const TC *__restrict__ qc,
                                                       const T *__restrict__ res, const T *__restrict__ soc,
                                                       T *__restrict__ q, Dims2 f, Dims2 c, int nsf)
{
	await_previous();
	int ic = blockIdx.x * TX + threadIdx.x + 1, jc = blockIdx.y * TY + threadIdx.y + 1;
	if (ic > f.nx / 2 + 1 || jc > f.ny / 2 + 1) return;
	const size_t cps = c.plane();
	ci += c.bofs(8 * cps);
	qc += c.bofs(cps);
	res += f.bofs(f.plane());
	soc += f.bofs(nsf * f.plane());
	q += f.bofs(f.plane());
	interp_at<T, TC>(ci, qc, res, soc, q, f, c, ic, jc);
}

template <typename T>
int interp_add_2d(const T *ci, const T *xc, const T *rf, const T *sof, T *xf, Dims2 f, Dims2 c, cudaStream_t st,
                  int nsf)
{
	launch(k_interp_add<T>, dim3(ceil_div(f.nx / 2 + 1, TX), ceil_div(f.ny / 2 + 1, TY), f.nb), dim3(TX, TY), 0, st, ci, xc, rf, sof, xf, f, c, nsf);
	CDR_LAUNCH_CHECK();
	return CDR_OK;
}
template int interp_add_2d<double>(const double *, const double *, const double *, const double *, double *,
                                   Dims2, Dims2, cudaStream_t, int);
template int interp_add_2d<float>(const float *, const float *, const float *, const float *, float *, Dims2,
                                  Dims2, cudaStream_t, int);

int interp_add_2d_mixed(const double *ci, const double *xc, const float *rf, const float *sof, float *xf, Dims2 f,
                        Dims2 c, cudaStream_t st, int nsf)
{
	launch(k_interp_add<float, double>, dim3(ceil_div(f.nx / 2 + 1, TX), ceil_div(f.ny / 2 + 1, TY), f.nb), dim3(TX, TY), 0,
	                              st, ci, xc, rf, sof, xf, f, c, nsf);
	CDR_LAUNCH_CHECK();
	return CDR_OK;
}

// The same interpolate-add on the FP32 cycle's fine level when its iterate is
// widened: xout (FP64) = xin (FP32) + P xc + r/c, formed in FP64 from the FP32
// weights, coarse iterate and residual (the points and ghost positions
// interp_at writes).
__global__ void __launch_bounds__(TX *TY) k_interp_add_wide(const float *__restrict__ ci, const float *__restrict__ qc,
                                                            const float *__restrict__ res,
                                                            const float *__restrict__ soc,
                                                            const float *__restrict__ qin, double *__restrict__ qout,
                                                            Dims2 f, Dims2 c, int nsf)
{
	await_previous();
	const int ic = blockIdx.x * TX + threadIdx.x + 1, jc = blockIdx.y * TY + threadIdx.y + 1;
	if (ic > f.nx / 2 + 1 || jc > f.ny / 2 + 1) return;
	const size_t cps = c.plane();
	ci += c.bofs(8 * cps);
	qc += c.bofs(cps);
	res += f.bofs(f.plane());
	soc += f.bofs(nsf * f.plane());
	qin += f.bofs(f.plane());
	qout += f.bofs(f.plane());
	const int cp = c.pitch, fp = f.pitch;
	const int i = 2 * ic - 1, j = 2 * jc - 1;
	const size_t kc = c.at(ic, jc), kf = f.at(i, j);
	auto rc = [&](size_t k, int ii, int jj) -> double {
		return (ii <= f.nx && jj <= f.ny) ? (double)res[k] / (double)soc[k] : (double)res[k];
	};
	auto W = [&](int plane, size_t k) -> double { return (double)ci[plane * cps + k]; };
	auto QC = [&](size_t k) -> double { return (double)qc[k]; };
	const double qcc = QC(kc);
	qout[kf] = (double)qin[kf] + qcc;
	if (ic >= 2) {
		const double a = W(IL, kc) * QC(kc - 1) + W(IR, kc) * qcc;
		const size_t k = kf - 1;
		qout[k] = (double)qin[k] + a + rc(k, i - 1, j);
	}
	if (jc >= 2) {
		const double a = W(IB, kc) * QC(kc - cp) + W(IA, kc) * qcc;
		const size_t k = kf - fp;
		qout[k] = (double)qin[k] + a + rc(k, i, j - 1);
	}
	if (ic >= 2 && jc >= 2) {
		double a = W(INW, kc) * QC(kc - 1) + W(ISW, kc) * QC(kc - cp - 1);
		a += W(INE, kc) * qcc;
		a += W(ISE, kc) * QC(kc - cp);
		const size_t k = kf - fp - 1;
		qout[k] = (double)qin[k] + a + rc(k, i - 1, j - 1);
	}
}

// The same interpolate-add by fine rows: thread (ic, jf) forms the fine points
// (2ic - 2, jf) and (2ic - 1, jf) of row jf (a coarse row: the x-edge point and
// the coarse point; otherwise the interior point and the y-edge point), with
// k_interp_add_wide's arithmetic for each, so that a warp reads and writes 64
// consecutive fine points of one row (8- and 16-byte accesses).  It covers the
// points of k_interp_add_wide: ic = 1 .. nxf/2 + 1, jf = 1 .. 2 (nyf/2) + 1.
__global__ void __launch_bounds__(256) k_interp_add_wide_rows(const float *__restrict__ ci,
                                                             const float *__restrict__ qc,
                                                             const float *__restrict__ res,
                                                             const float *__restrict__ soc,
                                                             const float *__restrict__ qin,
                                                             double *__restrict__ qout, Dims2 f, Dims2 c)
{
	await_previous();
	const int ic = blockIdx.x * blockDim.x + threadIdx.x + 1, jf = blockIdx.y + 1;
	if (ic > f.nx / 2 + 1) return;
	const size_t cps = c.plane();
	const int cp = c.pitch;
	const int i = 2 * ic - 1;
	auto rc = [&](size_t k, int ii, int jj) -> double {
		return (ii <= f.nx && jj <= f.ny) ? (double)res[k] / (double)soc[k] : (double)res[k];
	};
	auto W = [&](int plane, size_t k) -> double { return (double)ci[plane * cps + k]; };
	auto QC = [&](size_t k) -> double { return (double)qc[k]; };
	const size_t k = f.at(i, jf);  // i odd, rows 16-byte aligned: k - 1 is even
	double v0 = 0.0, v1;           // points (i - 1, jf) and (i, jf)
	float2 x01 = make_float2(0.f, 0.f);
	if (ic >= 2) x01 = *reinterpret_cast<const float2 *>(qin + k - 1);
	else x01.y = qin[k];
	if (jf & 1) {  // coarse row jc: the x-edge point, then the coarse point
		const size_t kc = c.at(ic, (jf + 1) / 2);
		const double qcc = QC(kc);
		v1 = (double)x01.y + qcc;
		if (ic >= 2) {
			const double a = W(IL, kc) * QC(kc - 1) + W(IR, kc) * qcc;
			v0 = (double)x01.x + a + rc(k - 1, i - 1, jf);
		}
	} else {  // between coarse rows jc - 1 and jc: the interior point, then the y-edge point
		const size_t kc = c.at(ic, jf / 2 + 1);
		const double qcc = QC(kc);
		const double a = W(IB, kc) * QC(kc - cp) + W(IA, kc) * qcc;
		v1 = (double)x01.y + a + rc(k, i, jf);
		if (ic >= 2) {
			double b = W(INW, kc) * QC(kc - 1) + W(ISW, kc) * QC(kc - cp - 1);
			b += W(INE, kc) * qcc;
			b += W(ISE, kc) * QC(kc - cp);
			v0 = (double)x01.x + b + rc(k - 1, i - 1, jf);
		}
	}
	if (ic >= 2) *reinterpret_cast<double2 *>(qout + k - 1) = make_double2(v0, v1);
	else qout[k] = v1;
}

// Row-sum excess of a level's operator, dg = c - (w(i,j) + w(i+1,j) + s(i,j) +
// s(i,j+1) [+ sw(i,j) + sw(i+1,j+1) + nw(i+1,j) + nw(i,j+1)]), in FP64 and
// rounded once.
__global__ void k_rowsum_excess(const double *__restrict__ so, int ns, float *__restrict__ dg, Dims2 d)
{
	await_previous();
	const size_t ps = d.plane();
	const int P = d.pitch;
	const int i = blockIdx.x * TX + threadIdx.x + 1, j = blockIdx.y * TY + threadIdx.y + 1;
	if (i > d.nx || j > d.ny) return;
	const size_t k = d.at(i, j);
	const double *w = so + ps, *s = so + 2 * ps;
	double a = w[k] + w[k + 1] + s[k] + s[k + P];
	if (ns == 5) {
		const double *sw = so + 3 * ps, *nw = so + 4 * ps;
		a = a + sw[k] + sw[k + P + 1] + nw[k + 1] + nw[k + P];
	}
	dg[k] = (float)(so[k] - a);
}

int rowsum_excess_2d(const double *so, int ns, float *dg, Dims2 d, cudaStream_t st)
{
	launch(k_rowsum_excess, dim3(ceil_div(d.nx, TX), ceil_div(d.ny, TY)), dim3(TX, TY), 0, st, so, ns, dg, d);
	CDR_LAUNCH_CHECK();
	return CDR_OK;
}

// Residual of the FP32 cycle's widened fine-level iterate (FP64 x) over the
// FP32 operator in difference form, in FP64 arithmetic:
//   r = b - dg x - sum over the couplings a of a (x - x_nb),
// rounded to FP32, with dg the row-sum excess (k_rowsum_excess).  The sum is
// the residual of the operator whose couplings and row-sum excess are the FP32
// values: a zero row sum stays zero, and its rounding error scales with the
// differences x - x_nb, not with x.  The post-smoothing that follows starts
// from zero on r, so the kernel also zeroes that iterate (zero).  Four points
// of a row per thread (rows 16-byte aligned, pitch a multiple of 4).
template <int NS>
__global__ void __launch_bounds__(TX *TY) k_residual_wide(const float *__restrict__ so, const float *__restrict__ dg,
                                                          const double *__restrict__ q, const float *__restrict__ qf,
                                                          float *__restrict__ res, float *__restrict__ zero, Dims2 d)
{
	await_previous();
	constexpr int V = 4;
	const size_t ps = d.plane();
	const int P = d.pitch;
	const int i0 = (blockIdx.x * TX + threadIdx.x) * V;
	const int j = blockIdx.y * TY + threadIdx.y + 1;
	if (i0 > d.nx || j > d.ny) return;
	const size_t k = (size_t)j * P + i0;
	const bool lft = i0 >= 1, rgt = i0 + V <= d.nx + 1;
	auto ld4 = [](const float *p, float *o) {
		const float4 t = *reinterpret_cast<const float4 *>(p);
		o[0] = t.x; o[1] = t.y; o[2] = t.z; o[3] = t.w;
	};
	auto ldq = [&](size_t kk, double *o) {  // o[0] = q[kk-1], o[1..4] = q[kk..kk+3], o[5] = q[kk+4]
		const double2 a = *reinterpret_cast<const double2 *>(q + kk), b = *reinterpret_cast<const double2 *>(q + kk + 2);
		o[1] = a.x; o[2] = a.y; o[3] = b.x; o[4] = b.y;
		o[0] = lft ? q[kk - 1] : 0.0;
		o[V + 1] = rgt ? q[kk + V] : 0.0;
	};
	double qm[V + 2], qc[V + 2], qp[V + 2];
	ldq(k - P, qm);
	ldq(k, qc);
	ldq(k + P, qp);
	const float *w = so + ps, *s = so + 2 * ps, *sw = so + (NS == 5 ? 3 : 0) * ps, *nw = so + (NS == 5 ? 4 : 0) * ps;
	float dd[V], bb[V], ww[V + 1], s0[V], s1[V];
	ld4(dg + k, dd);
	ld4(qf + k, bb);
	ld4(w + k, ww);
	ww[V] = rgt ? w[k + V] : 0.f;
	ld4(s + k, s0);
	ld4(s + k + P, s1);
	float sw0[V], sw1[V + 1], nw0[V + 1], nw1[V];
	if (NS == 5) {
		ld4(sw + k, sw0);
		ld4(sw + k + P, sw1);
		sw1[V] = rgt ? sw[k + P + V] : 0.f;
		ld4(nw + k, nw0);
		nw0[V] = rgt ? nw[k + V] : 0.f;
		ld4(nw + k + P, nw1);
	}
	float r[V];
#pragma unroll
	for (int m = 0; m < V; ++m) {
		const double qk = qc[m + 1];
		double a = (double)bb[m] - (double)dd[m] * qk;
		a -= (double)ww[m] * (qk - qc[m]);
		a -= (double)ww[m + 1] * (qk - qc[m + 2]);
		a -= (double)s0[m] * (qk - qm[m + 1]);
		a -= (double)s1[m] * (qk - qp[m + 1]);
		if (NS == 5) {
			a -= (double)sw0[m] * (qk - qm[m]);
			a -= (double)nw0[m + 1] * (qk - qm[m + 2]);
			a -= (double)nw1[m] * (qk - qp[m]);
			a -= (double)sw1[m + 1] * (qk - qp[m + 2]);
		}
		r[m] = (float)a;
	}
	if (lft && i0 + V - 1 <= d.nx) {
		*reinterpret_cast<float4 *>(res + k) = make_float4(r[0], r[1], r[2], r[3]);
		if (zero) *reinterpret_cast<float4 *>(zero + k) = make_float4(0.f, 0.f, 0.f, 0.f);
	} else {
#pragma unroll
		for (int m = 0; m < V; ++m)
			if (i0 + m >= 1 && i0 + m <= d.nx) {
				res[k + m] = r[m];
				if (zero) zero[k + m] = 0.f;
			}
	}
}

int residual_2d_wide(const float *so, const float *dg, int ns, const double *x, const float *b, float *r, float *zero,
                     Dims2 d, cudaStream_t st)
{
	if (((uintptr_t)so | (uintptr_t)dg | (uintptr_t)x | (uintptr_t)b | (uintptr_t)r | (uintptr_t)zero) % 16 != 0 ||
	    d.pitch % 4 != 0 || d.nb != 1) {
		set_error(CDR_ERR_ARG, "wide residual: rows must be 16-byte aligned with a pitch that is a multiple of 4");
		return CDR_ERR_ARG;
	}
	const dim3 g(ceil_div(d.nx + 1, TX * 4), ceil_div(d.ny, TY)), blk(TX, TY);
	if (ns == 5) launch(k_residual_wide<5>, g, blk, 0, st, so, dg, x, b, r, zero, d);
	else launch(k_residual_wide<3>, g, blk, 0, st, so, dg, x, b, r, zero, d);
	CDR_LAUNCH_CHECK();
	return CDR_OK;
}

int interp_add_2d_wide(const float *ci, const float *xc, const float *rf, const float *sof, const float *xin,
                       double *xout, Dims2 f, Dims2 c, cudaStream_t st, int nsf)
{
	// rows of 16-byte alignment, a single problem: the row kernel; otherwise by
	// 2 x 2 blocks of fine points
	if (f.nb == 1 && f.pitch % 4 == 0 && ((uintptr_t)xin | (uintptr_t)xout) % 16 == 0) {
		launch(k_interp_add_wide_rows, dim3(ceil_div(f.nx / 2 + 1, 256), 2 * (f.ny / 2) + 1), 256, 0, st, ci, xc, rf, sof, xin, xout, f, c);
	} else {
		launch(k_interp_add_wide, dim3(ceil_div(f.nx / 2 + 1, TX), ceil_div(f.ny / 2 + 1, TY), f.nb), dim3(TX, TY), 0,
		                    st, ci, xc, rf, sof, xin, xout, f, c, nsf);
	}
	CDR_LAUNCH_CHECK();
	return CDR_OK;
}

// ------------------------------------------------ operator-induced interpolation
// BMG2_SymStd_SETUP_interp_OI (src/2d/ftn/BMG2_SymStd_SETUP_interp_OI.f90:109-253).
// Phase 1 computes the edge weights, phase 2 the corner weights that read
// neighbouring edge weights.  emach = D1MACH(3) = 2^-53.

template <int NS>
__global__ void k_oi_edges(const double *__restrict__ so, double *__restrict__ ci, Dims2 f, Dims2 c)
{
	await_previous();
	int ic = blockIdx.x * TX + threadIdx.x + 1, jc = blockIdx.y * TY + threadIdx.y + 1;
	const size_t ps = f.plane(), cps = c.plane();
	const int fp = f.pitch;
	so += f.bofs(NS * ps);
	ci += c.bofs(8 * cps);
	const double *C = so, *W = so + ps, *S = so + 2 * ps, *SW = so + 3 * ps, *NW = so + 4 * ps;
	size_t kc = c.at(ic, jc);
	// x-edge weights at coarse (ic, jc), ic in [2, nxf/2+1], jc in [1, nyc]
	if (ic >= 2 && ic <= f.nx / 2 + 1 && jc <= c.ny) {
		size_t k = f.at(2 * ic - 1, 2 * jc - 1);  // fine point right of the x-edge point k-1
		double A, B;
		if (NS == 5) {
			A = W[k] + NW[k] + SW[k + fp];
			B = W[k - 1] + SW[k - 1] + NW[k - 1 + fp];
		} else {
			A = W[k];
			B = W[k - 1];
		}
		double o = C[k - 1];
		double ep = fmin(fabs(A / o), fabs(B / o));
		double sum = A + B + S[k - 1] + S[k - 1 + fp];
		sum = A + B + (o - sum) * fmax(o - (1.0 + ep) * sum, 0.0) / (fabs(o - (1.0 + ep) * sum) + 1.1102230246251565e-16);
		sum = 1.0 / sum;
		ci[IR * cps + kc] = A * sum;
		ci[IL * cps + kc] = B * sum;
	}
	// y-edge weights at coarse (ic, jc), ic in [1, nxc], jc in [2, nyf/2+1]
	if (ic <= c.nx && jc >= 2 && jc <= f.ny / 2 + 1) {
		size_t k = f.at(2 * ic - 1, 2 * jc - 1);  // fine point above the y-edge point k-fp
		double A, B;
		if (NS == 5) {
			A = S[k] + NW[k] + SW[k + 1];
			B = S[k - fp] + SW[k - fp] + NW[k + 1 - fp];
		} else {
			A = S[k];
			B = S[k - fp];
		}
		double o = C[k - fp];
		double ep = fmin(fabs(A / o), fabs(B / o));
		double sum = A + B + W[k - fp] + W[k + 1 - fp];
		sum = A + B + (o - sum) * fmax(o - (1.0 + ep) * sum, 0.0) / (fabs(o - (1.0 + ep) * sum) + 1.1102230246251565e-16);
		sum = 1.0 / sum;
		ci[IA * cps + kc] = A * sum;
		ci[IB * cps + kc] = B * sum;
	}
}

template <int NS>
__global__ void k_oi_corners(const double *__restrict__ so, double *__restrict__ ci, Dims2 f, Dims2 c)
{
	await_previous();
	int ic = blockIdx.x * TX + threadIdx.x + 2, jc = blockIdx.y * TY + threadIdx.y + 2;
	if (ic > f.nx / 2 + 1 || jc > f.ny / 2 + 1) return;
	const size_t ps = f.plane(), cps = c.plane();
	const int fp = f.pitch, cp = c.pitch;
	so += f.bofs(NS * ps);
	ci += c.bofs(8 * cps);
	const double *C = so, *W = so + ps, *S = so + 2 * ps, *SW = so + 3 * ps, *NW = so + 4 * ps;
	size_t kc = c.at(ic, jc);
	size_t k = f.at(2 * ic - 1, 2 * jc - 1);  // (I, J); the centre point is (I-1, J-1)
	size_t kw = k - 1, ks = k - fp, ksw = k - fp - 1;
	double o = C[ksw];
	double ciLL_s = ci[IL * cps + kc - cp], ciLR_s = ci[IR * cps + kc - cp];
	double ciLB_w = ci[IB * cps + kc - 1], ciLA_w = ci[IA * cps + kc - 1];
	double ciLL = ci[IL * cps + kc], ciLR = ci[IR * cps + kc], ciLB = ci[IB * cps + kc], ciLA = ci[IA * cps + kc];
	double sum, ep;
	if (NS == 5) {
		sum = W[ksw] + NW[kw] + S[kw] + SW[k] + W[ks] + NW[ks] + S[ksw] + SW[ksw];
		ep = fmin(fmin(fabs((SW[ksw] + W[ksw] + NW[kw]) / o), fabs((NW[kw] + S[kw] + SW[k]) / o)),
		          fmin(fabs((SW[k] + W[ks] + NW[ks]) / o), fabs((NW[ks] + S[ksw] + SW[ksw]) / o)));
	} else {
		sum = W[ksw] + S[kw] + W[ks] + S[ksw];
		ep = fmin(fmin(fabs(W[ksw] / o), fabs(S[kw] / o)), fmin(fabs(W[ks] / o), fabs(S[ksw] / o)));
	}
	sum = sum + (o - sum) * fmax(o - (1.0 + ep) * sum, 0.0) / (fabs(o - (1.0 + ep) * sum) + 1.1102230246251565e-16);
	double s = 1.0 / sum;
	if (NS == 5) {
		ci[ISW * cps + kc] = (S[ksw] * ciLL_s + W[ksw] * ciLB_w + SW[ksw]) * s;
		ci[ISE * cps + kc] = (S[ksw] * ciLR_s + W[ks] * ciLB + NW[ks]) * s;
		ci[INW * cps + kc] = (W[ksw] * ciLA_w + S[kw] * ciLL + NW[kw]) * s;
		ci[INE * cps + kc] = (S[kw] * ciLR + W[ks] * ciLA + SW[k]) * s;
	} else {
		ci[ISW * cps + kc] = (S[ksw] * ciLL_s + W[ksw] * ciLB_w) * s;
		ci[ISE * cps + kc] = (S[ksw] * ciLR_s + W[ks] * ciLB) * s;
		ci[INW * cps + kc] = (W[ksw] * ciLA_w + S[kw] * ciLL) * s;
		ci[INE * cps + kc] = (S[kw] * ciLR + W[ks] * ciLA) * s;
	}
}

int setup_interp_2d(const double *so, int nstencil, double *ci, Dims2 f, Dims2 c, cudaStream_t st)
{
	CDR_CUDA_TRY(cudaMemsetAsync(ci, 0, sizeof(double) * c.plane() * 8 * c.nb, st));
	dim3 blk(TX, TY);
	dim3 g1(ceil_div(c.nx + 1, TX), ceil_div(c.ny + 1, TY), c.nb);
	dim3 g2(ceil_div(f.nx / 2, TX), ceil_div(f.ny / 2, TY), c.nb);
	if (nstencil == 5) {
		launch(k_oi_edges<5>, g1, blk, 0, st, so, ci, f, c);
		CDR_LAUNCH_CHECK();
		launch(k_oi_corners<5>, g2, blk, 0, st, so, ci, f, c);
	} else {
		launch(k_oi_edges<3>, g1, blk, 0, st, so, ci, f, c);
		CDR_LAUNCH_CHECK();
		launch(k_oi_corners<3>, g2, blk, 0, st, so, ci, f, c);
	}
	CDR_LAUNCH_CHECK();
	return CDR_OK;
}

// ------------------------------------------------------------ Galerkin coarse op
// Coarse operator P^T A P for the operator-induced P, BMG2_SymStd_SETUP_ITLI_ex
// (src/2d/ftn/BMG2_SymStd_SETUP_ITLI_ex.f90:94-214 nine-point fine operator,
// :252-331 five-point), one thread per coarse point.  The partial products
// (C*) and their order are the reference's, so the result is bit-identical.
// (A generic local P^T A P over the 3x3 supports gives the same operator up to
// summation order; the OI weights of the next level amplify such differences,
// so the reference's order is kept.)
template <int NS>
__global__ void k_galerkin(const double *__restrict__ so, const double *__restrict__ ci, double *__restrict__ soc,
                           Dims2 f, Dims2 c)
{
	await_previous();
	const int ic = blockIdx.x * TX + threadIdx.x + 1, jc = blockIdx.y * TY + threadIdx.y + 1;
	if (ic > c.nx || jc > c.ny) return;
	const size_t ps = f.plane(), cps = c.plane();
	const int fp = f.pitch, cp = c.pitch;
	so += f.bofs(NS * ps);
	ci += c.bofs(8 * cps);
	soc += c.bofs(5 * cps);
	const size_t k0 = f.at(2 * ic - 1, 2 * jc - 1), kc0 = c.at(ic, jc);
	// fine stencil relative to (I, J) and weights relative to (IC, JC)
	auto O = [&](int di, int dj) { return so[k0 + (long)dj * fp + di]; };
	auto W = [&](int di, int dj) { return so[ps + k0 + (long)dj * fp + di]; };
	auto S = [&](int di, int dj) { return so[2 * ps + k0 + (long)dj * fp + di]; };
	auto SW = [&](int di, int dj) { return NS == 5 ? so[3 * ps + k0 + (long)dj * fp + di] : 0.0; };
	auto NW = [&](int di, int dj) { return NS == 5 ? so[4 * ps + k0 + (long)dj * fp + di] : 0.0; };
	auto P = [&](int di, int dj, int pl) { return ci[pl * cps + kc0 + (long)dj * cp + di]; };
	double CO, CS, CSW, CW, CNW, CN, CNE, CE, CSE;
	if (NS == 5) {
		CO = NW(0, 1) * P(0, 1, ISW) + W(0, 0) * P(0, 0, IL) + SW(0, 0) * P(0, 0, INW);
		CS = W(0, -1) * P(0, 0, INW) + NW(0, 0) * P(0, 0, IL);
		CSW = -O(-1, -1) * P(0, 0, INW) + W(-1, -1) * P(-1, 0, IA) + NW(-1, 0) + S(-1, 0) * P(0, 0, IL);
		CW = -O(-1, 0) * P(0, 0, IL) + S(-1, 0) * P(0, 0, INW) + SW(-1, 0) * P(-1, 0, IA) + W(-1, 0)
		     + NW(-1, 1) * P(-1, 1, IB) + S(-1, 1) * P(0, 1, ISW);
		CNW = -O(-1, 1) * P(0, 1, ISW) + S(-1, 1) * P(0, 0, IL) + SW(-1, 1) + W(-1, 1) * P(-1, 1, IB);
		CN = SW(0, 1) * P(0, 0, IL) + W(0, 1) * P(0, 1, ISW);
		soc[PW * cps + kc0] = CO + P(0, 0, IA) * CS + P(0, 0, INE) * CSW + P(0, 0, IR) * CW + P(0, 1, ISE) * CNW
		                      + P(0, 1, IB) * CN;
		double COSW = SW(0, 0) * P(0, 0, ISW);
		double CSSW = SW(0, -1) * P(0, -1, IL) + W(0, -1) * P(0, 0, ISW);
		double CSWSW = -O(-1, -1) * P(0, 0, ISW) + S(-1, -1) * P(0, -1, IL) + SW(-1, -1) + W(-1, -1) * P(-1, 0, IB);
		double CWSW = S(-1, 0) * P(0, 0, ISW) + SW(-1, 0) * P(-1, 0, IB);
		soc[PSW * cps + kc0] = COSW + P(0, 0, IA) * CSSW + P(0, 0, INE) * CSWSW + P(0, 0, IR) * CWSW;
		double COA = SW(0, 0) * P(0, 0, ISE) + S(0, 0) * P(0, 0, IB) + NW(1, 0) * P(1, 0, ISW);
		double CEA = S(1, 0) * P(1, 0, ISW) + SW(1, 0) * P(0, 0, IB);
		double CSEA = -O(1, -1) * P(1, 0, ISW) + S(1, -1) * P(1, -1, IL) + SW(1, -1) + W(1, -1) * P(0, 0, IB);
		double CSA = -O(0, -1) * P(0, 0, IB) + W(1, -1) * P(1, 0, ISW) + NW(1, -1) * P(1, -1, IL) + S(0, -1)
		             + SW(0, -1) * P(0, -1, IR) + W(0, -1) * P(0, 0, ISE);
		double CSWA = -O(-1, -1) * P(0, 0, ISE) + W(0, -1) * P(0, 0, IB) + NW(0, -1) + S(-1, -1) * P(0, -1, IR);
		double CWA = NW(0, 0) * P(0, 0, IB) + S(-1, 0) * P(0, 0, ISE);
		soc[PS * cps + kc0] = COA + P(1, 0, IL) * CEA + P(1, 0, INW) * CSEA + P(0, 0, IA) * CSA + P(0, 0, INE) * CSWA
		                      + P(0, 0, IR) * CWA;
		double CONW = NW(-1, 0) * P(0, 0, ISE);
		double CENW = NW(0, 0) * P(0, 0, IB) + S(-1, 0) * P(0, 0, ISE);
		double CSENW = -O(-1, -1) * P(0, 0, ISE) + W(0, -1) * P(0, 0, IB) + NW(0, -1) + S(-1, -1) * P(0, -1, IR);
		double CFNW = W(-1, -1) * P(0, 0, ISE) + NW(-1, -1) * P(0, -1, IR);
		soc[PNW * cps + kc0] = CONW + P(0, 0, IL) * CENW + P(0, 0, INW) * CSENW + P(-1, 0, IA) * CFNW;
		CO = W(0, 0) * P(0, 0, IR) + NW(0, 1) * P(0, 1, ISE) + S(0, 1) * P(0, 1, IB) + SW(1, 1) * P(1, 1, ISW)
		     + W(1, 0) * P(1, 0, IL) + NW(1, 0) * P(1, 0, INW) + S(0, 0) * P(0, 0, IA) + SW(0, 0) * P(0, 0, INE)
		     - O(0, 0);
		CW = -O(-1, 0) * P(0, 0, IR) + S(-1, 1) * P(0, 1, ISE) + SW(0, 1) * P(0, 1, IB) + W(0, 0)
		     + NW(0, 0) * P(0, 0, IA) + S(-1, 0) * P(0, 0, INE);
		CNW = -O(-1, 1) * P(0, 1, ISE) + W(0, 1) * P(0, 1, IB) + NW(0, 1) + S(-1, 1) * P(0, 0, IR);
		CN = -O(0, 1) * P(0, 1, IB) + NW(1, 1) * P(1, 0, IL) + S(0, 1) + SW(0, 1) * P(0, 0, IR)
		     + W(0, 1) * P(0, 1, ISE) + W(1, 1) * P(1, 1, ISW);
		CNE = -O(1, 1) * P(1, 1, ISW) + S(1, 1) * P(1, 0, IL) + SW(1, 1) + W(1, 1) * P(0, 1, IB);
		CE = -O(1, 0) * P(1, 0, IL) + S(1, 0) * P(1, 0, INW) + SW(1, 0) * P(0, 0, IA) + W(1, 0)
		     + NW(1, 1) * P(0, 1, IB) + S(1, 1) * P(1, 1, ISW);
		CSE = -O(1, -1) * P(1, 0, INW) + W(1, -1) * P(0, 0, IA) + NW(1, 0) + S(1, 0) * P(1, 0, IL);
		CS = -O(0, -1) * P(0, 0, IA) + W(0, -1) * P(0, 0, INE) + NW(0, 0) * P(0, 0, IR) + S(0, 0)
		     + SW(1, 0) * P(1, 0, IL) + W(1, -1) * P(1, 0, INW);
		CSW = -O(-1, -1) * P(0, 0, INE) + S(-1, 0) * P(0, 0, IR) + SW(0, 0) + W(0, -1) * P(0, 0, IA);
	} else {
		CO = W(0, 0) * P(0, 0, IL);
		CS = W(0, -1) * P(0, 0, INW);
		CSW = -O(-1, -1) * P(0, 0, INW) + W(-1, -1) * P(-1, 0, IA) + S(-1, 0) * P(0, 0, IL);
		CW = -O(-1, 0) * P(0, 0, IL) + S(-1, 0) * P(0, 0, INW) + W(-1, 0) + S(-1, 1) * P(0, 1, ISW);
		CNW = -O(-1, 1) * P(0, 1, ISW) + S(-1, 1) * P(0, 0, IL) + W(-1, 1) * P(-1, 1, IB);
		CN = W(0, 1) * P(0, 1, ISW);
		soc[PW * cps + kc0] = CO + P(0, 0, IA) * CS + P(0, 0, INE) * CSW + P(0, 0, IR) * CW + P(0, 1, ISE) * CNW
		                      + P(0, 1, IB) * CN;
		double CSSW = W(0, -1) * P(0, 0, ISW);
		double CSWSW = -O(-1, -1) * P(0, 0, ISW) + S(-1, -1) * P(0, -1, IL) + W(-1, -1) * P(-1, 0, IB);
		double CWSW = S(-1, 0) * P(0, 0, ISW);
		soc[PSW * cps + kc0] = P(0, 0, IA) * CSSW + P(0, 0, INE) * CSWSW + P(0, 0, IR) * CWSW;
		double COA = S(0, 0) * P(0, 0, IB);
		double CEA = S(1, 0) * P(1, 0, ISW);
		double CSEA = -O(1, -1) * P(1, 0, ISW) + S(1, -1) * P(1, -1, IL) + W(1, -1) * P(0, 0, IB);
		double CSA = -O(0, -1) * P(0, 0, IB) + W(1, -1) * P(1, 0, ISW) + S(0, -1) + W(0, -1) * P(0, 0, ISE);
		double CSWA = -O(-1, -1) * P(0, 0, ISE) + W(0, -1) * P(0, 0, IB) + S(-1, -1) * P(0, -1, IR);
		double CWA = S(-1, 0) * P(0, 0, ISE);
		soc[PS * cps + kc0] = COA + P(1, 0, IL) * CEA + P(1, 0, INW) * CSEA + P(0, 0, IA) * CSA + P(0, 0, INE) * CSWA
		                      + P(0, 0, IR) * CWA;
		double CENW = S(-1, 0) * P(0, 0, ISE);
		double CSENW = -O(-1, -1) * P(0, 0, ISE) + W(0, -1) * P(0, 0, IB) + S(-1, -1) * P(0, -1, IR);
		double CSNW = W(-1, -1) * P(0, 0, ISE);
		soc[PNW * cps + kc0] = P(0, 0, IL) * CENW + P(0, 0, INW) * CSENW + P(-1, 0, IA) * CSNW;
		CO = W(0, 0) * P(0, 0, IR) + S(0, 1) * P(0, 1, IB) + W(1, 0) * P(1, 0, IL) + S(0, 0) * P(0, 0, IA) - O(0, 0);
		CW = -O(-1, 0) * P(0, 0, IR) + S(-1, 1) * P(0, 1, ISE) + W(0, 0) + S(-1, 0) * P(0, 0, INE);
		CNW = -O(-1, 1) * P(0, 1, ISE) + W(0, 1) * P(0, 1, IB) + S(-1, 1) * P(0, 0, IR);
		CN = -O(0, 1) * P(0, 1, IB) + S(0, 1) + W(0, 1) * P(0, 1, ISE) + W(1, 1) * P(1, 1, ISW);
		CNE = -O(1, 1) * P(1, 1, ISW) + S(1, 1) * P(1, 0, IL) + W(1, 1) * P(0, 1, IB);
		CE = -O(1, 0) * P(1, 0, IL) + S(1, 0) * P(1, 0, INW) + W(1, 0) + S(1, 1) * P(1, 1, ISW);
		CSE = -O(1, -1) * P(1, 0, INW) + W(1, -1) * P(0, 0, IA) + S(1, 0) * P(1, 0, IL);
		CS = -O(0, -1) * P(0, 0, IA) + W(0, -1) * P(0, 0, INE) + S(0, 0) + W(1, -1) * P(1, 0, INW);
		CSW = -O(-1, -1) * P(0, 0, INE) + S(-1, 0) * P(0, 0, IR) + W(0, -1) * P(0, 0, IA);
	}
	soc[PC * cps + kc0] = -P(0, 1, ISE) * CNW - P(0, 1, IB) * CN - P(1, 1, ISW) * CNE - P(0, 0, IR) * CW - CO
	                      - P(1, 0, IL) * CE - P(0, 0, INE) * CSW - P(0, 0, IA) * CS - P(1, 0, INW) * CSE;
}

int galerkin_2d(const double *so, int nstencil, const double *ci, double *soc, Dims2 f, Dims2 c, cudaStream_t st)
{
	CDR_CUDA_TRY(cudaMemsetAsync(soc, 0, sizeof(double) * c.plane() * 5 * c.nb, st));
	dim3 g(ceil_div(c.nx, TX), ceil_div(c.ny, TY), c.nb);
	if (nstencil == 5) launch(k_galerkin<5>, g, dim3(TX, TY), 0, st, so, ci, soc, f, c);
	else launch(k_galerkin<3>, g, dim3(TX, TY), 0, st, so, ci, soc, f, c);
	CDR_LAUNCH_CHECK();
	return CDR_OK;
}

// --------------------------------------------------- coarsest banded Cholesky
// ABD fill of BMG2_SymStd_SETUP_cg_LU (src/2d/ftn/BMG2_SymStd_SETUP_cg_LU.f90:92-104,
// 229-241) and LAPACK DPBTF2('U') (unblocked upper band Cholesky; DPBTRF takes it
// for KD < 32).  The grid is at most a few dozen points: one thread.
__global__ void __launch_bounds__(1024) k_cg_factor(const double *__restrict__ so, int ns, Dims2 d,
                                                    double *__restrict__ ab, int *info)
{
	await_previous();
	__shared__ double rcp_s;
	__shared__ int stop_s;
	const int tid = threadIdx.x, nt = blockDim.x;
	const int ldab = d.nx + 2, kd = d.nx + 1, n = d.nx * d.ny;
	const size_t ps = d.plane();
	so += d.bofs(ns * ps);
	ab += d.bofs((size_t)ldab * n);
	for (size_t e = tid; e < (size_t)ldab * n; e += nt) ab[e] = 0.0;
	__syncthreads();
	for (int kk = tid; kk < n; kk += nt) {
		const size_t k = d.at(kk % d.nx + 1, kk / d.nx + 1);
		double *col = ab + (size_t)kk * ldab;  // column kk, rows 0..ldab-1
		col[ldab - 1] = so[k];
		col[ldab - 2] = -so[ps + k];
		col[2] = ns == 5 ? -so[4 * ps + k + 1] : 0.0;
		col[1] = -so[2 * ps + k];
		col[0] = ns == 5 ? -so[3 * ps + k] : 0.0;
	}
	// DPBTF2('U'): column jj's pivot by one thread, then its scaling and the
	// rank-1 update of the trailing band triangle by all threads.  Every
	// element receives the sequential routine's updates in the same order.
	const int kld = ldab - 1;
	int st = 0;
	for (int jj = 0; jj < n; ++jj) {
		__syncthreads();
		if (tid == 0) {
			double ajj = ab[(size_t)jj * ldab + kd];
			stop_s = ajj <= 0.0;
			if (!stop_s) {
				ajj = sqrt(ajj);
				ab[(size_t)jj * ldab + kd] = ajj;
				rcp_s = 1.0 / ajj;
			}
		}
		__syncthreads();
		if (stop_s) { st = jj + 1; break; }
		const int kn = kd < n - jj - 1 ? kd : n - jj - 1;
		if (kn <= 0) continue;
		double *x = ab + (size_t)(jj + 1) * ldab + (kd - 1);
		for (int p = tid; p < kn; p += nt) x[(size_t)p * kld] = rcp_s * x[(size_t)p * kld];
		__syncthreads();
		double *a = ab + (size_t)(jj + 1) * ldab + kd;
		for (int e = tid; e < kn * kn; e += nt) {
			const int q = e / kn, p = e - q * kn;
			if (p > q) continue;
			const double xq = x[(size_t)q * kld];
			if (xq != 0.0) {
				const double temp = -1.0 * xq;
				a[(size_t)p + (size_t)q * kld] = a[(size_t)p + (size_t)q * kld] + x[(size_t)p * kld] * temp;
			}
		}
	}
	// a batch records the first failure it meets (the caller zeroes info)
	if (info && tid == 0) {
		if (gridDim.z == 1) *info = st;
		else if (st) atomicCAS(info, 0, st);
	}
}

// BMG2_SymStd_SOLVE_cg (src/2d/ftn/BMG2_SymStd_SOLVE_cg.f90:93-123) with DPBTRS('U'):
// U^T y = b then U x = y, in FP64 whatever the grid-function type.
template <typename T>
__global__ void k_cg_solve(const double *__restrict__ ab, T *__restrict__ q, const T *__restrict__ qf, Dims2 d)
{
	await_previous();
	extern __shared__ double xs[];
	const int ldab = d.nx + 2, n = d.nx * d.ny, lane = threadIdx.x;
	ab += d.bofs((size_t)ldab * n);
	q += d.bofs(d.plane());
	qf += d.bofs(d.plane());
	for (int m = lane; m < n; m += 32) xs[m] = (double)qf[d.at(m % d.nx + 1, m / d.nx + 1)];
	__syncwarp();
	band_solve_warp(ab, ldab, n, xs);
	for (int m = lane; m < n; m += 32) q[d.at(m % d.nx + 1, m / d.nx + 1)] = (T)xs[m];
}

int setup_cg_2d(const double *so, int nstencil, Dims2 d, double *abd, int *info, cudaStream_t st)
{
	launch(k_cg_factor, dim3(1, 1, d.nb), 1024, 0, st, so, nstencil, d, abd, info);
	CDR_LAUNCH_CHECK();
	return CDR_OK;
}

template <typename T>
int solve_cg_2d(const double *abd, T *x, const T *b, Dims2 d, cudaStream_t st)
{
	size_t sm = sizeof(double) * (size_t)d.nx * d.ny;
	if (sm > 48 * 1024) {
		set_error(CDR_ERR_DIM, "coarsest grid %dx%d too large for the direct solve", d.nx, d.ny);
		return CDR_ERR_DIM;
	}
	launch(k_cg_solve<T>, dim3(1, 1, d.nb), 32, sm, st, abd, x, b, d);
	CDR_LAUNCH_CHECK();
	return CDR_OK;
}
template int solve_cg_2d<double>(const double *, double *, const double *, Dims2, cudaStream_t);
template int solve_cg_2d<float>(const double *, float *, const float *, Dims2, cudaStream_t);

// ------------------------------------------------------------ precision helpers
template <typename TO, typename TI>
__global__ void k_convert(const TI *__restrict__ in, TO *__restrict__ out, size_t n)
{
	await_previous();
	for (size_t e = blockIdx.x * (size_t)blockDim.x + threadIdx.x; e < n; e += (size_t)gridDim.x * blockDim.x)
		out[e] = (TO)in[e];
}

int convert_f64_f32(const double *in, float *out, size_t n, cudaStream_t st)
{
	int nb = (int)((n + 255) / 256);
	if (nb > 148 * 16) nb = 148 * 16;
	if (nb < 1) nb = 1;
	launch(k_convert<float, double>, nb, 256, 0, st, in, out, n);
	CDR_LAUNCH_CHECK();
	return CDR_OK;
}

// One launch for the two buffers of a refinement or Krylov solve: a second copy
// command cost a small solve 17 us (400^2, six cycles of 125 us).
__global__ void __launch_bounds__(256) k_copy_to_both(const double *__restrict__ x, double *__restrict__ a,
                                                      double *__restrict__ b, size_t n)
{
	await_previous();
	const size_t step = (size_t)gridDim.x * blockDim.x, t = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
	for (size_t e = t; e < n / 2; e += step) {
		const double2 v = reinterpret_cast<const double2 *>(x)[e];
		reinterpret_cast<double2 *>(a)[e] = v;
		reinterpret_cast<double2 *>(b)[e] = v;
	}
	if (t == 0 && n % 2) a[n - 1] = b[n - 1] = x[n - 1];
}

int copy_to_both(const double *x, double *a, double *b, size_t n, cudaStream_t st)
{
	const size_t nb = (n / 2 + 255) / 256;
	launch(k_copy_to_both, (unsigned)(nb < 1 ? 1 : nb > 148 * 8 ? 148 * 8 : nb), 256, 0, st, x, a, b, n);
	CDR_LAUNCH_CHECK();
	return CDR_OK;
}

__global__ void __launch_bounds__(256) k_copy_rings(const double *__restrict__ x, double *__restrict__ y, Dims2 d)
{
	await_previous();
	const int w = d.nx + 2, t = blockIdx.x * 256 + threadIdx.x;
	if (t >= 2 * w + 2 * d.ny) return;
	const int s = t - 2 * w;  // rows 0 and ny + 1, then columns 0 and nx + 1
	const int i = s < 0 ? t % w : s % 2 * (d.nx + 1), j = s < 0 ? t / w * (d.ny + 1) : s / 2 + 1;
	const size_t k = d.bofs(d.plane()) + d.at(i, j);
	y[k] = x[k];
}

int copy_rings(const double *x, double *y, Dims2 d, cudaStream_t st)
{
	launch(k_copy_rings, dim3(ceil_div(2 * (d.nx + 2) + 2 * d.ny, 256), 1, d.nb), 256, 0, st, x, y, d);
	CDR_LAUNCH_CHECK();
	return CDR_OK;
}

// Outer refinement step of the mixed-precision solve:
//   x_out = x_in + e32 on the interior, r64 = b64 - A64 x_out, r32 = (float) r64
//   and ||r64||^2 per block.  The residual at a point needs the corrected x at
//   its neighbours, so each thread forms x_in + e32 for its 3x3 neighbourhood on
//   the fly; x_in and x_out are different buffers (ping-pong), so no thread
//   reads a value another thread has already corrected.  apply = 0 skips e; in a
//   batch, a problem whose active[z] is 0 (converged) skips e as well.
template <int NS>
__global__ void __launch_bounds__(TX *TY) k_ir_residual(const double *__restrict__ so, const double *__restrict__ x,
                                                        const float *__restrict__ e, const double *__restrict__ b,
                                                        double *__restrict__ xo, float *__restrict__ r32, Dims2 d,
                                                        Dims2 d32, double *__restrict__ partial, int apply,
                                                        const int *__restrict__ active)
{
	await_previous();
	__shared__ double sh[TX * TY / 32];
	const int tiles_x = (d.nx + TX - 1) / TX;
	const int ntiles = tiles_x * ((d.ny + TY - 1) / TY);
	const size_t ps = d.plane();
	const int p = d.pitch, p32 = d32.pitch;
	so += d.bofs(NS * ps);
	x += d.bofs(ps);
	b += d.bofs(ps);
	xo += d.bofs(ps);
	e += d32.bofs(d32.plane());
	r32 += d32.bofs(d32.plane());
	if (active && !active[blockIdx.z * d.bstep]) apply = 0;
	double acc = 0.0;
	for (int t = blockIdx.x; t < ntiles; t += gridDim.x) {
		int i = (t % tiles_x) * TX + threadIdx.x + 1;
		int j = (t / tiles_x) * TY + threadIdx.y + 1;
		if (i <= d.nx && j <= d.ny) {
			const size_t k = d.at(i, j), k32 = d32.at(i, j);
			double xn[3][3];
#pragma unroll
			for (int dj = -1; dj <= 1; ++dj)
#pragma unroll
				for (int di = -1; di <= 1; ++di) {
					double v = x[k + (long)dj * p + di];
					xn[dj + 1][di + 1] = apply ? v + (double)e[k32 + (long)dj * p32 + di] : v;
				}
			const double *c = so, *w = so + ps, *s = so + 2 * ps;
			double rr;
			if (NS == 5) {
				const double *sw = so + 3 * ps, *nw = so + 4 * ps;
				rr = b[k] + w[k] * xn[1][0] + w[k + 1] * xn[1][2] + s[k] * xn[0][1] + s[k + p] * xn[2][1]
				     + sw[k] * xn[0][0] + nw[k + 1] * xn[0][2] + nw[k + p] * xn[2][0] + sw[k + p + 1] * xn[2][2]
				     - c[k] * xn[1][1];
			} else {
				rr = b[k] + w[k] * xn[1][0] + w[k + 1] * xn[1][2] + s[k] * xn[0][1] + s[k + p] * xn[2][1]
				     - c[k] * xn[1][1];
			}
			acc += rr * rr;
			r32[k32] = (float)rr;
			xo[k] = xn[1][1];
		}
	}
	double s = block_sum<TX * TY / 32>(acc, sh);
	if (threadIdx.x == 0 && threadIdx.y == 0) partial[(size_t)blockIdx.z * gridDim.x + blockIdx.x] = s;
}

// The same step with two points per thread, i0 and i0 + 1 (i0 even, 16-byte
// loads and stores along the rows; the neighbours beyond the pair as single
// loads): k_ir_residual's operations on each point in its order, so xo and r32
// are the same bits; the norm's partial sums run in another order.
template <int NS>
__global__ void __launch_bounds__(TX *TY) k_ir_residual_v(const double *__restrict__ so, const double *__restrict__ x,
                                                          const float *__restrict__ e, const double *__restrict__ b,
                                                          double *__restrict__ xo, float *__restrict__ r32, Dims2 d,
                                                          Dims2 d32, double *__restrict__ partial, int apply,
                                                          const int *__restrict__ active)
{
	await_previous();
	__shared__ double sh[TX * TY / 32];
	const int tiles_x = (d.nx + 2 * TX) / (2 * TX);  // pairs (0,1), (2,3), ... up to nx
	const int ntiles = tiles_x * ((d.ny + TY - 1) / TY);
	const size_t ps = d.plane();
	const int p = d.pitch, p32 = d32.pitch;
	so += d.bofs(NS * ps);
	x += d.bofs(ps);
	b += d.bofs(ps);
	xo += d.bofs(ps);
	e += d32.bofs(d32.plane());
	r32 += d32.bofs(d32.plane());
	if (active && !active[blockIdx.z * d.bstep]) apply = 0;
	const double *c = so, *w = so + ps, *s = so + 2 * ps, *sw = so + (NS == 5 ? 3 : 0) * ps,
	             *nw = so + (NS == 5 ? 4 : 0) * ps;
	auto ld2 = [](const double *q) { return *reinterpret_cast<const double2 *>(q); };
	double acc = 0.0;
	for (int t = blockIdx.x; t < ntiles; t += gridDim.x) {
		const int i0 = (t % tiles_x) * 2 * TX + 2 * threadIdx.x;
		const int j = (t / tiles_x) * TY + threadIdx.y + 1;
		if (i0 > d.nx || j > d.ny) continue;
		const bool v0 = i0 >= 1, v1 = i0 + 1 <= d.nx;  // the pair's points inside the grid
		const size_t k = d.at(i0, j), k32 = d32.at(i0, j);
		// x (+ e) at columns i0 - 1 .. i0 + 2 of rows j - 1, j, j + 1
		double xn[3][4];
#pragma unroll
		for (int dj = -1; dj <= 1; ++dj) {
			const size_t kr = k + (long)dj * p, kr32 = k32 + (long)dj * p32;
			const double2 m = ld2(x + kr);
			double v[4] = {v0 ? x[kr - 1] : 0.0, m.x, m.y, v1 ? x[kr + 2] : 0.0};
			if (apply) {
				const float2 em = *reinterpret_cast<const float2 *>(e + kr32);
				v[0] = v0 ? v[0] + (double)e[kr32 - 1] : 0.0;
				v[1] = v[1] + (double)em.x;
				v[2] = v[2] + (double)em.y;
				v[3] = v1 ? v[3] + (double)e[kr32 + 2] : 0.0;
			}
#pragma unroll
			for (int q = 0; q < 4; ++q) xn[dj + 1][q] = v[q];
		}
		const double2 cc = ld2(c + k), bb = ld2(b + k), ww = ld2(w + k), s0 = ld2(s + k), s1 = ld2(s + k + p);
		const double w2 = v1 ? w[k + 2] : 0.0;
		double rr[2];
		if (NS == 5) {
			const double2 sw0 = ld2(sw + k), sw1 = ld2(sw + k + p), nw0 = ld2(nw + k), nw1 = ld2(nw + k + p);
			const double sw12 = v1 ? sw[k + p + 2] : 0.0, nw02 = v1 ? nw[k + 2] : 0.0;
			// point i0 (column index 1 of xn), then i0 + 1 (index 2)
			rr[0] = bb.x + ww.x * xn[1][0] + ww.y * xn[1][2] + s0.x * xn[0][1] + s1.x * xn[2][1] + sw0.x * xn[0][0] +
			        nw0.y * xn[0][2] + nw1.x * xn[2][0] + sw1.y * xn[2][2] - cc.x * xn[1][1];
			rr[1] = bb.y + ww.y * xn[1][1] + w2 * xn[1][3] + s0.y * xn[0][2] + s1.y * xn[2][2] + sw0.y * xn[0][1] +
			        nw02 * xn[0][3] + nw1.y * xn[2][1] + sw12 * xn[2][3] - cc.y * xn[1][2];
		} else {
			rr[0] = bb.x + ww.x * xn[1][0] + ww.y * xn[1][2] + s0.x * xn[0][1] + s1.x * xn[2][1] - cc.x * xn[1][1];
			rr[1] = bb.y + ww.y * xn[1][1] + w2 * xn[1][3] + s0.y * xn[0][2] + s1.y * xn[2][2] - cc.y * xn[1][2];
		}
		if (v0 && v1) {
			acc += rr[0] * rr[0];
			acc += rr[1] * rr[1];
			*reinterpret_cast<float2 *>(r32 + k32) = make_float2((float)rr[0], (float)rr[1]);
			*reinterpret_cast<double2 *>(xo + k) = make_double2(xn[1][1], xn[1][2]);
		} else if (v0) {
			acc += rr[0] * rr[0];
			r32[k32] = (float)rr[0];
			xo[k] = xn[1][1];
		} else if (v1) {
			acc += rr[1] * rr[1];
			r32[k32 + 1] = (float)rr[1];
			xo[k + 1] = xn[1][2];
		}
	}
	double sum = block_sum<TX * TY / 32>(acc, sh);
	if (threadIdx.x == 0 && threadIdx.y == 0) partial[(size_t)blockIdx.z * gridDim.x + blockIdx.x] = sum;
}

int ir_residual_2d(const double *so, int nstencil, const double *x, const float *e, const double *b, double *xo,
                   float *r32, Dims2 d, Dims2 d32, double *norm_out, double *partial, int apply, cudaStream_t st,
                   const int *active)
{
	const int nb = norm_blocks(d);
	const dim3 grd(nb, 1, d.nb);
	// pairs of points along 16-byte rows where the pitches allow it
	const bool vec = d.pitch % 2 == 0 && d32.pitch % 2 == 0 && (d.bstep * d.plane()) % 2 == 0 &&
	                 (d32.bstep * d32.plane()) % 2 == 0 &&
	                 ((uintptr_t)so | (uintptr_t)x | (uintptr_t)b | (uintptr_t)xo) % 16 == 0 &&
	                 ((uintptr_t)e | (uintptr_t)r32) % 8 == 0;
	if (vec && nstencil == 5)
		launch(k_ir_residual_v<5>, grd, dim3(TX, TY), 0, st, so, x, e, b, xo, r32, d, d32, partial, apply, active);
	else if (vec)
		launch(k_ir_residual_v<3>, grd, dim3(TX, TY), 0, st, so, x, e, b, xo, r32, d, d32, partial, apply, active);
	else if (nstencil == 5)
		launch(k_ir_residual<5>, grd, dim3(TX, TY), 0, st, so, x, e, b, xo, r32, d, d32, partial, apply, active);
	else
		launch(k_ir_residual<3>, grd, dim3(TX, TY), 0, st, so, x, e, b, xo, r32, d, d32, partial, apply, active);
	CDR_LAUNCH_CHECK();
	launch(k_norm_finish, d.nb, 1024, 0, st, partial, nb, norm_out);
	CDR_LAUNCH_CHECK();
	return CDR_OK;
}

}  // namespace cdrgpu
