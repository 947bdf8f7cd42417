// k3.cu -- 3D BoxMG kernels (27- and 7-point fine operators) for sm_100a.
//
// Layout: Cedar's 3D arrays with one ghost layer, i fastest, rows padded to a
// pitch; a k-slice is pitch*(ny+2) elements, a stencil plane
// pitch*(ny+2)*(nz+2).  Stencil planes (include/cedar/3d/base_types.h:4-20,
// 1-based as in src/3d/ftn/BMG_stencils_f90.h): kp kpw kps kb kpsw kpnw kbw kbnw
// kbn kbne kbe kbse kbs kbsw; interpolation weights: 26 planes lxyl .. ltse.
// A seven-point operator (include/cedar/3d/base_types.h seven_pt) keeps the
// first four planes only: p, pw, ps, b.
// Kernel bodies address arrays with the reference's 1-based (I, J, K) through
// the macros below and keep its operand order, so they reproduce its bits
// (the library is built without FMA contraction).

#include "k2_bulk.cuh"
#include "k2_point.cuh"
#include "kernels3d.cuh"

namespace cdrgpu {

#define SO(i, j, k, p) so[(size_t)((p)-1) * F.plane() + F.at1(i, j, k)]
#define Q(i, j, k) q[F.at1(i, j, k)]
#define QF(i, j, k) qf[F.at1(i, j, k)]
#define CI(i, j, k, l) ci[(size_t)((l)-1) * C.plane() + C.at1(i, j, k)]
#define QC(i, j, k) qc[C.at1(i, j, k)]

// qf plus the 26 neighbour terms of BMG3_SymStd_residual.f90:76-101, in its
// order; xq(i, j, k) supplies the iterate (a plain load, or x + e in the
// refinement step)
template <typename T, typename XQ>
__device__ __forceinline__ T nb27(const T *__restrict__ so, XQ xq, T qf, Dims3 F, int i, int j, int k)
{
	T nb = qf + SO(i, j, k, KPW) * xq(i - 1, j, k);
	nb = nb + SO(i, j + 1, k, KPNW) * xq(i - 1, j + 1, k) + SO(i, j + 1, k, KPS) * xq(i, j + 1, k)
	     + SO(i + 1, j + 1, k, KPSW) * xq(i + 1, j + 1, k) + SO(i + 1, j, k, KPW) * xq(i + 1, j, k)
	     + SO(i + 1, j, k, KPNW) * xq(i + 1, j - 1, k) + SO(i, j, k, KPS) * xq(i, j - 1, k)
	     + SO(i, j, k, KPSW) * xq(i - 1, j - 1, k) + SO(i, j, k, KB) * xq(i, j, k - 1)
	     + SO(i, j, k, KBW) * xq(i - 1, j, k - 1) + SO(i, j + 1, k, KBNW) * xq(i - 1, j + 1, k - 1)
	     + SO(i, j + 1, k, KBN) * xq(i, j + 1, k - 1) + SO(i + 1, j + 1, k, KBNE) * xq(i + 1, j + 1, k - 1)
	     + SO(i + 1, j, k, KBE) * xq(i + 1, j, k - 1) + SO(i + 1, j, k, KBSE) * xq(i + 1, j - 1, k - 1)
	     + SO(i, j, k, KBS) * xq(i, j - 1, k - 1) + SO(i, j, k, KBSW) * xq(i - 1, j - 1, k - 1)
	     + SO(i, j, k + 1, KB) * xq(i, j, k + 1) + SO(i, j, k + 1, KBE) * xq(i - 1, j, k + 1)
	     + SO(i, j + 1, k + 1, KBSE) * xq(i - 1, j + 1, k + 1) + SO(i, j + 1, k + 1, KBS) * xq(i, j + 1, k + 1)
	     + SO(i + 1, j + 1, k + 1, KBSW) * xq(i + 1, j + 1, k + 1) + SO(i + 1, j, k + 1, KBW) * xq(i + 1, j, k + 1)
	     + SO(i + 1, j, k + 1, KBNW) * xq(i + 1, j - 1, k + 1) + SO(i, j, k + 1, KBN) * xq(i, j - 1, k + 1)
	     + SO(i, j, k + 1, KBNE) * xq(i - 1, j - 1, k + 1);
	return nb;
}

// qf plus the 6 neighbour terms of the seven-point branch
// (BMG3_SymStd_residual.f90:104-119), in its order.
template <typename T, typename XQ>
__device__ __forceinline__ T nb7(const T *__restrict__ so, XQ xq, T qf, Dims3 F, int i, int j, int k)
{
	return qf + SO(i, j, k, KPW) * xq(i - 1, j, k) + SO(i, j + 1, k, KPS) * xq(i, j + 1, k)
	       + SO(i + 1, j, k, KPW) * xq(i + 1, j, k) + SO(i, j, k, KPS) * xq(i, j - 1, k)
	       + SO(i, j, k, KB) * xq(i, j, k - 1) + SO(i, j, k + 1, KB) * xq(i, j, k + 1);
}

// Neighbour sum of an NS-plane operator: 14 (27-point) or 4 (seven-point).
template <int NS, typename T, typename XQ>
__device__ __forceinline__ T nbs(const T *__restrict__ so, XQ xq, T qf, Dims3 F, int i, int j, int k)
{
	if constexpr (NS == 4) return nb7<T>(so, xq, qf, F, i, j, k);
	else return nb27<T>(so, xq, qf, F, i, j, k);
}

// every pointer a multiple of n bytes
template <typename... P>
static bool aligned_to(size_t n, const P *...p)
{
	return ((reinterpret_cast<uintptr_t>(p) % n == 0) && ...);
}

template <typename T>
struct Load3 {
	const T *__restrict__ q;
	Dims3 F;
	__device__ __forceinline__ T operator()(int i, int j, int k) const { return q[F.at1(i, j, k)]; }
};

// --------------------------------------------------------------- residual
// BMG3_SymStd_residual (src/3d/ftn/BMG3_SymStd_residual.f90:67-121); grid-stride
// over 32x8 tiles of every k-slice, FP64 partial sums of r^2 per block.
// TO: type of the stored residual.
template <typename T, bool NORM, int NS, typename TO = T>
__global__ void __launch_bounds__(TX *TY) k3_residual(const T *__restrict__ so, const T *__restrict__ q,
                                                      const T *__restrict__ qf, TO *__restrict__ res, Dims3 F,
                                                      double *__restrict__ partial)
{
	await_previous();
	__shared__ double sh[TX * TY / 32];
	const int tx = (F.nx + TX - 1) / TX, ty = (F.ny + TY - 1) / TY;
	const long ntiles = (long)tx * ty * F.nz;
	double acc = 0.0;
	for (long t = blockIdx.x; t < ntiles; t += gridDim.x) {
		const int kk = (int)(t / ((long)tx * ty));
		const int rem = (int)(t - (long)kk * tx * ty);
		const int i = (rem % tx) * TX + threadIdx.x + 2, j = (rem / tx) * TY + threadIdx.y + 2, k = kk + 2;
		if (i <= F.nx + 1 && j <= F.ny + 1) {
			const T r = nbs<NS, T>(so, Load3<T>{q, F}, QF(i, j, k), F, i, j, k) - SO(i, j, k, KP) * Q(i, j, k);
			res[F.at1(i, j, k)] = (TO)r;
			if (NORM) acc += (double)r * (double)r;
		}
	}
	if (NORM) {
		const double s = block_sum<TX * TY / 32>(acc, sh);
		if (threadIdx.x == 0 && threadIdx.y == 0) partial[blockIdx.x] = s;
	}
}

__global__ void __launch_bounds__(1024) k3_norm_finish(const double *__restrict__ partial, int n, double *out)
{
	await_previous();
	__shared__ double sh[32];
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

// ----------------------------------------------------------------- smoother
// BMG3_SymStd_SETUP_recip (src/3d/ftn/BMG3_SymStd_SETUP_recip.f90:63-69)
template <typename T>
__global__ void k3_recip(const T *__restrict__ so, T *__restrict__ sor, Dims3 F)
{
	await_previous();
	const int i = blockIdx.x * TX + threadIdx.x + 2, j = blockIdx.y * TY + threadIdx.y + 2, k = blockIdx.z + 2;
	if (i > F.nx + 1 || j > F.ny + 1) return;
	sor[F.at1(i, j, k)] = T(1) / SO(i, j, k, KP);
}

// The points a = 2t, b = 2t + 1 (0-based) of a row: the sum of the colour swept
// first, and the second point's terms, held as products (in nb27's order) until
// its row neighbours (terms 0 and 4, coefficients c0 and c4) have their new values.
template <typename T>
struct GsPair {
	T pr[26], c0, c4, first, rhs, ds;
};

// crow(plane, dj, dk) and qrow(dj, dk) point at element a of an operator row and
// of the iterate's rows around (j, k); qf and sor at element a of b and 1/c.
// SECOND_A: b first, then a (the sweep UP, colours 1..8); else a, then b (DOWN).
// t >= 1: a has a left neighbour; vb: b is an interior point.
template <typename T, bool VEC, bool SECOND_A, typename CR, typename QR>
__device__ __forceinline__ void gs_pair_terms(CR crow, QR qrow, const T *qf, const T *sor, int t, bool va, bool vb,
                                              GsPair<T> &g, T &far)
{
	using V2 = typename Vec2<T>::type;
	auto pair = [&](const T *x, T &a, T &b) {
		if constexpr (VEC) {
			const V2 v = *reinterpret_cast<const V2 *>(x);
			a = v.x;
			b = v.y;
		} else {
			a = x[0];
			b = x[1];
		}
	};
	auto row4 = [&](const T *x, T(&v)[4]) {  // left neighbour of a, a, b, right neighbour of b
		v[0] = t >= 1 ? x[-1] : T(0);
		pair(x, v[1], v[2]);
		v[3] = vb ? x[2] : T(0);
	};
	T X[4] = {}, Y[4], Z[4], ca, cb, fa, fb, wa, wb, wr, sa, sb;
	pair(qf, fa, fb);
	T acc = SECOND_A ? fb : fa;
	// one term: coefficients of a and of b, iterates of a and of b
	auto term = [&](int m, T ka, T xa, T kb, T xb) {
		if (SECOND_A) {
			acc = acc + kb * xb;
			g.pr[m] = ka * xa;
		} else {
			acc = acc + ka * xa;
			g.pr[m] = kb * xb;
		}
	};
	// coefficient planes at the point, and at its right neighbour; x: the
	// neighbour's offset along the row
	auto own = [&](int m, const T *c, int x) {
		pair(c, ca, cb);
		term(m, ca, X[1 + x], cb, X[2 + x]);
	};
	auto right = [&](int m, const T *c, int x) {
		ca = c[1];
		cb = vb ? c[2] : T(0);
		term(m, ca, X[1 + x], cb, X[2 + x]);
	};
	auto use = [&](const T(&v)[4]) {
#pragma unroll
		for (int m = 0; m < 4; ++m) X[m] = v[m];
	};
	row4(qrow(0, 0), Y);
	const T *pw = crow(KPW, 0, 0);
	pair(pw, wa, wb);
	wr = vb ? pw[2] : T(0);
	if (SECOND_A) {  // b: left a (old), right a' (old); a waits for both new b
		acc = acc + wb * Y[1];
		g.c0 = wa;
		g.c4 = wb;
	} else {  // a: left b (old), right b (old); b waits for both new a
		acc = acc + wa * Y[0];
		g.c0 = wb;
		g.c4 = wr;
	}
	row4(qrow(1, 0), X);
	own(1, crow(KPNW, 1, 0), -1);
	own(2, crow(KPS, 1, 0), 0);
	right(3, crow(KPSW, 1, 0), 1);
	if (SECOND_A) acc = acc + wr * Y[3];
	else acc = acc + wb * Y[2];
	row4(qrow(-1, 0), X);
	right(5, crow(KPNW, 0, 0), 1);
	own(6, crow(KPS, 0, 0), 0);
	own(7, crow(KPSW, 0, 0), -1);
	row4(qrow(0, -1), Z);
	use(Z);
	own(8, crow(KB, 0, 0), 0);
	own(9, crow(KBW, 0, 0), -1);
	row4(qrow(1, -1), X);
	own(10, crow(KBNW, 1, 0), -1);
	own(11, crow(KBN, 1, 0), 0);
	right(12, crow(KBNE, 1, 0), 1);
	use(Z);
	right(13, crow(KBE, 0, 0), 1);
	row4(qrow(-1, -1), X);
	right(14, crow(KBSE, 0, 0), 1);
	own(15, crow(KBS, 0, 0), 0);
	own(16, crow(KBSW, 0, 0), -1);
	row4(qrow(0, 1), Z);
	use(Z);
	own(17, crow(KB, 0, 1), 0);
	own(18, crow(KBE, 0, 1), -1);
	row4(qrow(1, 1), X);
	own(19, crow(KBSE, 1, 1), -1);
	own(20, crow(KBS, 1, 1), 0);
	right(21, crow(KBSW, 1, 1), 1);
	use(Z);
	right(22, crow(KBW, 0, 1), 1);
	row4(qrow(-1, 1), X);
	right(23, crow(KBNW, 0, 1), 1);
	own(24, crow(KBN, 0, 1), 0);
	own(25, crow(KBNE, 0, 1), -1);
	pair(sor, sa, sb);
	// a point outside the interior keeps its value
	if (SECOND_A) g.first = vb ? acc * sb : Y[2];
	else g.first = va ? acc * sa : Y[1];
	g.rhs = SECOND_A ? fa : fb;
	g.ds = SECOND_A ? sa : sb;
	far = Y[3];
}

// the second point, given the new values of its row neighbours
template <typename T>
__device__ __forceinline__ T gs_pair_second(const GsPair<T> &g, T left, T right)
{
	T v = g.rhs + g.c0 * left;
	v = v + g.pr[1] + g.pr[2] + g.pr[3] + g.c4 * right;
#pragma unroll
	for (int m = 5; m < 26; ++m) v = v + g.pr[m];
	return v * g.ds;
}

template <typename T, bool VEC>
__device__ __forceinline__ void gs_pair_store(T *qo, T a, T b, bool va, bool vb)
{
	if (VEC && va && vb) {
		typename Vec2<T>::type v;
		v.x = a;
		v.y = b;
		*reinterpret_cast<typename Vec2<T>::type *>(qo) = v;
	} else {
		if (va) qo[0] = a;
		if (vb) qo[1] = b;
	}
}

// Two colours of BMG3_SymStd_relax_GS (src/3d/ftn/BMG3_SymStd_relax_GS.f90:94-136)
// in one pass: the rows (j, k) of one parity pair, first the points of one
// x-parity, then the others.  A row's second colour depends on the first only
// inside the row, and rows of one parity pair do not touch each other, so a
// block that owns whole rows needs no other block: four launches per sweep.
// Bound by latency and DRAM: a thread takes a pair of points and loads every
// coefficient of both at once, so a row's operator lines are read once with all
// of their bytes used (one colour per launch reads every second point of a row,
// and each line twice), and the second point's terms wait as products, so that
// its sum keeps the reference's order and bits.  Rows longer than 2 W points run
// in segments from the side whose first colour the second one reads.
template <typename T, bool VEC, bool SECOND_A>
__global__ void __launch_bounds__(256) k3_gs_rows(const T *__restrict__ so, T *__restrict__ q,
                                                  const T *__restrict__ qf, const T *__restrict__ sor, Dims3 F, int pj,
                                                  int pk, int nrj, int nrows, int W)
{
	await_previous();
	__shared__ T sh[256];    // first-colour values of the segment
	__shared__ T edge[256];  // per row: the first-colour value the next segment reads
	const int r = threadIdx.x / W, t0 = threadIdx.x - r * W;
	const int row = blockIdx.x * (blockDim.x / W) + r;
	const int nT = F.nx / 2 + 1, nseg = (nT + W - 1) / W;
	const int rk = row / nrj, j = 1 + pj + 2 * (row - rk * nrj), k = 1 + pk + 2 * rk;
	const size_t ps = F.plane(), sl = F.slice();
	const int p = F.pitch;
	const size_t base = ((size_t)k * (F.ny + 2) + j) * p;
	for (int s = 0; s < nseg; ++s) {
		const int t = (SECOND_A ? s : nseg - 1 - s) * W + t0;
		const bool live = row < nrows && t < nT;
		const bool va = live && t >= 1, vb = live && 2 * t + 1 <= F.nx;
		const size_t o = base + 2 * t;
		GsPair<T> g;
		T far = T(0);
		g.first = T(0);
		if (live)
			gs_pair_terms<T, VEC, SECOND_A>(
			    [&](int plane, int dj, int dk) { return so + (size_t)(plane - 1) * ps + o + dj * p + dk * sl; },
			    [&](int dj, int dk) { return q + o + (ptrdiff_t)dj * p + (ptrdiff_t)dk * (ptrdiff_t)sl; }, qf + o, sor + o, t,
			    va, vb, g, far);
		sh[threadIdx.x] = g.first;
		__syncthreads();  // the segment's row is read, its first colour formed
		if (live) {
			T left, right;  // new row neighbours of the second point
			if (SECOND_A) {
				left = t0 > 0 ? sh[threadIdx.x - 1] : edge[r];
				right = g.first;
			} else {
				left = g.first;
				right = t + 1 >= nT ? far : t0 + 1 < W ? sh[threadIdx.x + 1] : edge[r];
			}
			const T second = gs_pair_second<T>(g, left, right);
			gs_pair_store<T, VEC>(q + o, SECOND_A ? second : g.first, SECOND_A ? g.first : second, va, vb);
		}
		if (nseg > 1) {
			__syncthreads();  // edge and sh are read
			if (t0 == (SECOND_A ? W - 1 : 0)) edge[r] = g.first;
		}
	}
}

// --------------------------------------------------------------- staged rows
// The sweep and the residual of a row read 36 rows: with loads into registers
// they are bound by latency (159^3 FP32: 22 warps per SM, DRAM at 55 % of peak).
// Where rows start on 16 bytes, a block takes one row and its 36 input rows arrive
// in shared memory by 16-byte asynchronous copies, all in flight at once and
// without registers; several blocks to an SM overlap copies and arithmetic.
// the 25 operator rows of a row's terms, in shared-memory order
struct Row27 {
	int plane, dj, dk;
};
constexpr int GS_OPS = 25, GS_ROWS = GS_OPS + 2 + 9;  // then b, 1/c and the iterate's nine rows
__host__ __device__ constexpr Row27 gs_op(int m)
{
	constexpr Row27 t[GS_OPS] = {
	    {KPW, 0, 0},  {KPNW, 0, 0}, {KPS, 0, 0},  {KPSW, 0, 0}, {KB, 0, 0},   {KBW, 0, 0},  {KBE, 0, 0},
	    {KBSE, 0, 0}, {KBS, 0, 0},  {KBSW, 0, 0}, {KPNW, 1, 0}, {KPS, 1, 0},  {KPSW, 1, 0}, {KBNW, 1, 0},
	    {KBN, 1, 0},  {KBNE, 1, 0}, {KB, 0, 1},   {KBE, 0, 1},  {KBW, 0, 1},  {KBNW, 0, 1}, {KBN, 0, 1},
	    {KBNE, 0, 1}, {KBSE, 1, 1}, {KBS, 1, 1},  {KBSW, 1, 1}};
	return t[m];
}
__host__ __device__ constexpr int gs_op_index(int plane, int dj, int dk)
{
	for (int m = 0; m < GS_OPS; ++m)
		if (gs_op(m).plane == plane && gs_op(m).dj == dj && gs_op(m).dk == dk) return m;
	return -1;
}


__device__ __forceinline__ void cp_async16(void *dst, const void *src)
{
	asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"(smem_u32(dst)), "l"(src) : "memory");
}

// 16-byte chunks of a staged row
template <typename T>
__host__ __device__ __forceinline__ int staged_chunks(Dims3 F)
{
	constexpr int VPC = 16 / sizeof(T);
	return (F.nx + 2 + VPC - 1) / VPC;
}

// Copies of the row at `base` (element offset of (j, k)): rl elements apart in
// shared memory; slot GS_OPS holds qf's row, slot GS_OPS + 1 the row of `extra`.
template <typename T>
__device__ __forceinline__ void stage_rows(T *rows, int nch, const T *__restrict__ so, const T *q,
                                           const T *__restrict__ qf, const T *__restrict__ extra, size_t base, Dims3 F)
{
	constexpr int VPC = 16 / sizeof(T);
	const size_t ps = F.plane(), sl = F.slice();
	const int p = F.pitch, rl = nch * VPC;
	for (int c = threadIdx.x; c < nch; c += blockDim.x) {
		const T *src = so + base + c * VPC, *qs = q + base + c * VPC;
		T *dst = rows + c * VPC;
#pragma unroll
		for (int m = 0; m < GS_OPS; ++m) {
			const Row27 r = gs_op(m);
			cp_async16(dst + m * rl, src + (size_t)(r.plane - 1) * ps + r.dj * p + r.dk * sl);
		}
		cp_async16(dst + GS_OPS * rl, qf + base + c * VPC);
		cp_async16(dst + (GS_OPS + 1) * rl, extra + base + c * VPC);
#pragma unroll
		for (int m = 0; m < 9; ++m)
			cp_async16(dst + (GS_OPS + 2 + m) * rl,
			           qs + (ptrdiff_t)(m % 3 - 1) * p + (ptrdiff_t)(m / 3 - 1) * (ptrdiff_t)sl);
	}
	asm volatile("cp.async.wait_all;\n" ::: "memory");
	__syncthreads();
}

constexpr size_t kStageSmemMax = 104 * 1024;  // two blocks to an SM
// threads of a block at that limit (a pair of points each, whole warps): 384 in FP32
// (rows of 734 points), 192 in FP64 (366).  The kernels' launch bounds ask for more,
// which caps their registers at 64 and 128: with bounds of 384 and 192 threads they
// take 80 and 168, fewer blocks share an SM, and most sizes lose (FP32 sweep 95^3 20.7
// -> 22.5 us, 159^3 103.5 -> 105.7, 255^3 365 -> 372, norm 200^3 131 -> 148; FP64 sweep
// 95^3 40.5 -> 42.9, 255^3 820 -> 750).
template <typename T>
constexpr int kStagedThreads =
    ((int)(kStageSmemMax / (GS_ROWS * 16)) * (16 / (int)sizeof(T)) - 2) / 2 / 32 * 32 + 32;
static_assert(kStagedThreads<float> == 384 && kStagedThreads<double> == 192, "within the launch bounds");

// k3_gs_rows with the row staged; block = row.
template <typename T, bool SECOND_A>
__global__ void __launch_bounds__(512, sizeof(T) == 4 ? 2 : 1)
    k3_gs_staged(const T *__restrict__ so, T *__restrict__ q, const T *__restrict__ qf, const T *__restrict__ sor,
                 Dims3 F, int pj, int pk, int nrj)
{
	await_previous();
	extern __shared__ __align__(16) unsigned char k3_raw[];
	T *rows = reinterpret_cast<T *>(k3_raw);
	const int nch = staged_chunks<T>(F), rl = nch * (16 / (int)sizeof(T)), t = threadIdx.x;
	const int rk = blockIdx.x / nrj, j = 1 + pj + 2 * (blockIdx.x - rk * nrj), k = 1 + pk + 2 * rk;
	const size_t base = ((size_t)k * (F.ny + 2) + j) * F.pitch;
	stage_rows<T>(rows, nch, so, q, qf, sor, base, F);
	const bool live = t < F.nx / 2 + 1, va = live && t >= 1, vb = live && 2 * t + 1 <= F.nx;
	T *center = rows + (GS_OPS + 2 + 4) * rl;
	GsPair<T> g;
	if (live) {
		T far;
		gs_pair_terms<T, true, SECOND_A>(
		    [&](int plane, int dj, int dk) { return rows + gs_op_index(plane, dj, dk) * rl + 2 * t; },
		    [&](int dj, int dk) { return rows + (GS_OPS + 2 + 3 * (dk + 1) + dj + 1) * rl + 2 * t; },
		    rows + GS_OPS * rl + 2 * t, rows + (GS_OPS + 1) * rl + 2 * t, t, va, vb, g, far);
		// the first colour goes into the staged row: no thread's first sum reads these points
		if (SECOND_A ? vb : va) center[2 * t + (SECOND_A ? 1 : 0)] = g.first;
	}
	__syncthreads();
	if (va || vb) {
		T second = T(0);
		if (SECOND_A && va) second = gs_pair_second<T>(g, center[2 * t - 1], center[2 * t + 1]);
		if (!SECOND_A && vb) second = gs_pair_second<T>(g, center[2 * t], center[2 * t + 2]);
		gs_pair_store<T, true>(q + base + 2 * t, SECOND_A ? second : g.first, SECOND_A ? g.first : second, va, vb);
	}
}

// r = b - A x (27-point) of the points a = 2t, b = 2t + 1 of a staged row, in
// the order of nb27
template <typename T>
__device__ __forceinline__ void residual_pair(const T *rows, int rl, int t, bool vb, T &ra, T &rb)
{
	using V2 = typename Vec2<T>::type;
	const T *r0 = rows + 2 * t;
	auto pair = [&](const T *x, T &a, T &b) {
		const V2 v = *reinterpret_cast<const V2 *>(x);
		a = v.x;
		b = v.y;
	};
	T X[4] = {}, Y[4], Z[4], ca, cb;
	auto row4 = [&](int dj, int dk, T(&v)[4]) {
		const T *x = r0 + (GS_OPS + 2 + 3 * (dk + 1) + dj + 1) * rl;
		v[0] = t >= 1 ? x[-1] : T(0);
		pair(x, v[1], v[2]);
		v[3] = vb ? x[2] : T(0);
	};
	auto own = [&](int plane, int dj, int dk, int x) {
		pair(r0 + gs_op_index(plane, dj, dk) * rl, ca, cb);
		ra = ra + ca * X[1 + x];
		rb = rb + cb * X[2 + x];
	};
	auto right = [&](int plane, int dj, int dk, int x) {
		const T *c = r0 + gs_op_index(plane, dj, dk) * rl;
		ra = ra + c[1] * X[1 + x];
		rb = rb + (vb ? c[2] : T(0)) * X[2 + x];
	};
	auto use = [&](const T(&v)[4]) {
#pragma unroll
		for (int m = 0; m < 4; ++m) X[m] = v[m];
	};
	pair(r0 + GS_OPS * rl, ra, rb);
	row4(0, 0, Y);
	use(Y);
	own(KPW, 0, 0, -1);
	row4(1, 0, X);
	own(KPNW, 1, 0, -1);
	own(KPS, 1, 0, 0);
	right(KPSW, 1, 0, 1);
	use(Y);
	right(KPW, 0, 0, 1);
	row4(-1, 0, X);
	right(KPNW, 0, 0, 1);
	own(KPS, 0, 0, 0);
	own(KPSW, 0, 0, -1);
	row4(0, -1, Z);
	use(Z);
	own(KB, 0, 0, 0);
	own(KBW, 0, 0, -1);
	row4(1, -1, X);
	own(KBNW, 1, 0, -1);
	own(KBN, 1, 0, 0);
	right(KBNE, 1, 0, 1);
	use(Z);
	right(KBE, 0, 0, 1);
	row4(-1, -1, X);
	right(KBSE, 0, 0, 1);
	own(KBS, 0, 0, 0);
	own(KBSW, 0, 0, -1);
	row4(0, 1, Z);
	use(Z);
	own(KB, 0, 1, 0);
	own(KBE, 0, 1, -1);
	row4(1, 1, X);
	own(KBSE, 1, 1, -1);
	own(KBS, 1, 1, 0);
	right(KBSW, 1, 1, 1);
	use(Z);
	right(KBW, 0, 1, 1);
	row4(-1, 1, X);
	right(KBNW, 0, 1, 1);
	own(KBN, 0, 1, 0);
	own(KBNE, 0, 1, -1);
	pair(r0 + (GS_OPS + 1) * rl, ca, cb);
	ra = ra - ca * Y[1];
	rb = rb - cb * Y[2];
}

// k3_residual with the rows staged: a block walks rows (NORM: at most 2048
// blocks, one partial sum each).
template <typename T, bool NORM>
__global__ void __launch_bounds__(512, 2)
    k3_residual_staged(const T *__restrict__ so, const T *__restrict__ q, const T *__restrict__ qf, T *__restrict__ res,
                       Dims3 F, double *__restrict__ partial)
{
	await_previous();
	extern __shared__ __align__(16) unsigned char k3_raw[];
	__shared__ double sh[kStagedThreads<T> / 32];
	T *rows = reinterpret_cast<T *>(k3_raw);
	const int nch = staged_chunks<T>(F), rl = nch * (16 / (int)sizeof(T)), t = threadIdx.x;
	const bool live = t < F.nx / 2 + 1, va = live && t >= 1, vb = live && 2 * t + 1 <= F.nx;
	const int nrows = F.ny * F.nz;
	double acc = 0.0;
	for (int row = blockIdx.x; row < nrows; row += gridDim.x) {
		const int k = row / F.ny + 1, j = row - (k - 1) * F.ny + 1;
		const size_t base = ((size_t)k * (F.ny + 2) + j) * F.pitch;
		stage_rows<T>(rows, nch, so, q, qf, so, base, F);
		if (live) {
			T ra, rb;
			residual_pair<T>(rows, rl, t, vb, ra, rb);
			gs_pair_store<T, true>(res + base + 2 * t, ra, rb, va, vb);
			if (NORM) {
				if (va) acc += (double)ra * (double)ra;
				if (vb) acc += (double)rb * (double)rb;
			}
		}
		__syncthreads();  // the staged rows are read
	}
	if (NORM) {
		for (int o = 16; o > 0; o >>= 1) acc += __shfl_down_sync(0xffffffffu, acc, o);
		if ((t & 31) == 0) sh[t >> 5] = acc;
		__syncthreads();
		if (t == 0) {
			double v = 0.0;
			for (int w = 0; w < (int)blockDim.x / 32; ++w) v += sh[w];
			partial[blockIdx.x] = v;
		}
	}
}

// Shared memory of a staged row, and whether a level's rows can be staged: one
// row to a block, two blocks to an SM at the least, rows on 16 bytes.  Against the
// rows with loads into registers, us a sweep: FP32 31^3 16.2 -> 8.2, 63^3 16.6 ->
// 14.4, 95^3 21.7 -> 20.6, 127^3 65 -> 45, 191^3 244 -> 166; FP64 31^3 17.8 -> 9.3,
// 79^3 27.6 -> 26.4, 95^3 65 -> 40, 127^3 151 -> 116, 191^3 543 -> 323.  At 63^3 FP64
// alone it was slower (19.1 -> 21.5; single colours 27): not worth a rule.
template <typename T>
static size_t staged_smem(Dims3 F)
{
	return (size_t)GS_ROWS * staged_chunks<T>(F) * 16;
}
template <typename T, typename... P>
static bool staged_ok(Dims3 F, const P *...p)
{
	return F.pitch % (16 / (int)sizeof(T)) == 0 && staged_smem<T>(F) <= kStageSmemMax && aligned_to(16, p...);
}
static int staged_block(Dims3 F) { return (F.nx / 2 + 1 + 31) / 32 * 32; }
// opts a staged kernel into its dynamic shared memory
static int staged_opt_in(const void *fn, size_t smem)
{
	if (smem > 40 * 1024)
		CDR_CUDA_TRY(cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kStageSmemMax));
	return CDR_OK;
}

template <typename T>
int residual_3d(const T *so, const T *x, const T *b, T *r, Dims3 F, double *norm_out, double *partial, cudaStream_t st,
                int ns)
{
	// FP32 27-point rows staged (255^3: 390 -> 239 us); in FP64 a staged row takes
	// 74 KB there and the point kernel is the faster one (863 against about 530 us)
	if constexpr (sizeof(T) == 4)
		if (ns == 14 && staged_ok<T>(F, so, x, b, r)) {
			const size_t smem = staged_smem<T>(F);
			const int nrows = F.ny * F.nz, blk = staged_block(F), nb = norm_out && nrows > 2048 ? 2048 : nrows;
			CDR_TRY(staged_opt_in(norm_out ? (const void *)k3_residual_staged<T, true>
			                               : (const void *)k3_residual_staged<T, false>, smem));
			if (norm_out) launch(k3_residual_staged<T, true>, nb, blk, smem, st, so, x, b, r, F, partial);
			else launch(k3_residual_staged<T, false>, nb, blk, smem, st, so, x, b, r, F, nullptr);
			CDR_LAUNCH_CHECK();
			if (norm_out) {
				launch(k3_norm_finish, 1, 1024, 0, st, partial, nb, norm_out);
				CDR_LAUNCH_CHECK();
			}
			return CDR_OK;
		}
	const long ntiles = (long)ceil_div(F.nx, TX) * ceil_div(F.ny, TY) * F.nz;
	const int nb = ntiles < 2048 ? (int)ntiles : 2048;
	if (norm_out) {
		if (ns == 4) launch(k3_residual<T, true, 4>, nb, dim3(TX, TY), 0, st, so, x, b, r, F, partial);
		else launch(k3_residual<T, true, 14>, nb, dim3(TX, TY), 0, st, so, x, b, r, F, partial);
		CDR_LAUNCH_CHECK();
		launch(k3_norm_finish, 1, 1024, 0, st, partial, nb, norm_out);
	} else {
		const int nb2 = ntiles < 148 * 64 ? (int)ntiles : 148 * 64;
		if (ns == 4) launch(k3_residual<T, false, 4>, nb2, dim3(TX, TY), 0, st, so, x, b, r, F, nullptr);
		else launch(k3_residual<T, false, 14>, nb2, dim3(TX, TY), 0, st, so, x, b, r, F, nullptr);
	}
	CDR_LAUNCH_CHECK();
	return CDR_OK;
}
template int residual_3d<double>(const double *, const double *, const double *, double *, Dims3, double *, double *,
                                 cudaStream_t, int);
template int residual_3d<float>(const float *, const float *, const float *, float *, Dims3, double *, double *,
                                cudaStream_t, int);

// One colour of the 27-point branch (BMG3_SymStd_relax_GS.f90:94-136): points of
// parities (pi, pj, pk).
template <typename T>
__global__ void __launch_bounds__(TX *TY) k3_gs_colour(const T *__restrict__ so, T *__restrict__ q,
                                                       const T *__restrict__ qf, const T *__restrict__ sor, Dims3 F,
                                                       int pi, int pj, int pk)
{
	await_previous();
	const int i = 2 + pi + 2 * (blockIdx.x * TX + threadIdx.x);
	const int j = 2 + pj + 2 * (blockIdx.y * TY + threadIdx.y);
	const int k = 2 + pk + 2 * blockIdx.z;
	if (i > F.nx + 1 || j > F.ny + 1 || k > F.nz + 1) return;
	const T acc = nb27<T>(so, Load3<T>{q, F}, QF(i, j, k), F, i, j, k);
	Q(i, j, k) = acc * sor[F.at1(i, j, k)];
}

// One colour of the seven-point branch of BMG3_SymStd_relax_GS
// (BMG3_SymStd_relax_GS.f90:141-180): colour pts (0 or 1) holds the points
// with I + J + K + pts even.
template <typename T>
__global__ void __launch_bounds__(TX *TY) k3_gs7_colour(const T *__restrict__ so, T *__restrict__ q,
                                                        const T *__restrict__ qf, const T *__restrict__ sor, Dims3 F,
                                                        int pts)
{
	await_previous();
	const int j = 2 + blockIdx.y * TY + threadIdx.y, k = 2 + blockIdx.z;
	const int i = 2 + ((j + k + pts) & 1) + 2 * (blockIdx.x * TX + threadIdx.x);
	if (i > F.nx + 1 || j > F.ny + 1) return;
	Q(i, j, k) = nb7<T>(so, Load3<T>{q, F}, QF(i, j, k), F, i, j, k) * sor[F.at1(i, j, k)];
}

// Whether a level whose rows cannot be staged goes by single colours, not by rows
// in nseg segments.  A row of several segments is a chain of them in one block, so
// rows need many blocks (two to an SM) and a level beyond L2 (126 MB), where each
// operator line read once instead of twice pays; and about the size of L2 the
// rows' order keeps less of the level there.  Level sizes count the operator, x, b
// and 1/c.  Both sides, us a sweep, colours | rows.  One segment: FP64 79^3 (67 MB)
// 38 | 24, 95^3 54 | 58, 103^3 69 | 84, 111^3 (186 MB) 87 | 95, 119^3 155 | 111; FP32
// 103^3 (74 MB) 38 | 37, 111^3 43 | 48, 119^3 (115 MB) 53 | 57, 127^3 63 | 62.
// Several: FP64 8192 x 8 x 8 33 | 319, 700 x 32 x 32 43 | 52, 1024 x 32 x 32 64 | 82,
// 600 x 64 x 64 210 | 179, 4096 x 24 x 24 202 | 281, 1024 x 64 x 64 346 | 381 (a row
// pitch of 1026), 1100 x 64 x 64 367 | 337; FP32 1500 x 32 x 32 49 | 75, 600 x 64 x 64
// 96 | 102, 1500 x 48 x 48 142 | 104.
template <typename T>
static bool gs3_by_colours(Dims3 F, int nseg)
{
	const double mb = 17e-6 * sizeof(T) * F.nx * F.ny * F.nz, hi = sizeof(T) == 8 ? 190.0 : 126.0;
	if (nseg == 1) return mb > 84.0 && mb < hi;
	return mb < hi || (long)(F.ny / 2) * (F.nz / 2) < 296;
}

template <typename T>
int relax_point_3d(const T *so, T *x, const T *b, const T *sor, Dims3 F, int updown, cudaStream_t st, int ns)
{
	if (ns == 4) {  // UP (and the non-symmetric sweep): colour 0 then 1; DOWN: 1 then 0
		const dim3 blk(TX, TY), grd(ceil_div((F.nx + 1) / 2, TX), ceil_div(F.ny, TY), F.nz);
		for (int c = 0; c < 2; ++c) {
			launch(k3_gs7_colour<T>, grd, blk, 0, st, so, x, b, sor, F, updown == CDR_DOWN ? 1 - c : c);
			CDR_LAUNCH_CHECK();
		}
		return CDR_OK;
	}
	// colours 1..8 (UP) or 8..1 (DOWN) are the parities (i, j, k), i fastest: pairs
	// of colours share the rows of one (j, k) parity.  Staged rows where they fit
	// (see staged_ok); else single colours (see gs3_by_colours) or W pairs of points
	// per row and segment (equal segments), as many rows to a block of 256 threads as
	// fit; two-element accesses where rows start aligned.
	const bool staged = staged_ok<T>(F, so, x, b, sor);
	const size_t smem = staged_smem<T>(F);
	if (staged)
		CDR_TRY(staged_opt_in(updown == CDR_UP ? (const void *)k3_gs_staged<T, true>
		                                       : (const void *)k3_gs_staged<T, false>, smem));
	const bool vec = F.pitch % 2 == 0 && aligned_to(2 * sizeof(T), so, x, b, sor);
	const int nT = F.nx / 2 + 1, nseg = ceil_div(nT, 256), W = ceil_div(nT, nseg), R = 256 / W;
	if (!staged && gs3_by_colours<T>(F, nseg)) {
		const dim3 blk(TX, TY), grd(ceil_div((F.nx + 1) / 2, TX), ceil_div((F.ny + 1) / 2, TY), (F.nz + 1) / 2);
		for (int c = 0; c < 8; ++c) {  // not early: 300 x 64 x 64 FP64 74 us a sweep, 100 with early launches
			const int bits = updown == CDR_UP ? c : 7 - c;
			launch_as(false, k3_gs_colour<T>, grd, blk, 0, st, so, x, b, sor, F, bits & 1, (bits >> 1) & 1, bits >> 2);
			CDR_LAUNCH_CHECK();
		}
		return CDR_OK;
	}
	for (int c = 0; c < 4; ++c) {
		const int bits = updown == CDR_UP ? c : 3 - c, pj = bits & 1, pk = bits >> 1;
		const int nrj = (F.ny - pj + 1) / 2, nrows = nrj * ((F.nz - pk + 1) / 2);
		if (nrows == 0) continue;
		if (staged) {
			if (updown == CDR_UP) launch(k3_gs_staged<T, true>, nrows, staged_block(F), smem, st, so, x, b, sor, F, pj, pk, nrj);
			else launch(k3_gs_staged<T, false>, nrows, staged_block(F), smem, st, so, x, b, sor, F, pj, pk, nrj);
			CDR_LAUNCH_CHECK();
			continue;
		}
		const int grd = ceil_div(nrows, R), blk = R * W;
		// not early where the blocks crowd on the SMs that the launch before leaves free
		// (unaligned, early | not, us a sweep): FP64 79^3 26.1 | 23.1; FP32 79^3 21.3 | 19.3,
		// 300 x 64 x 64 41.3 | 34.8; but 71^3 (22 SMs' worth) 23.9 | 24.2, FP64 119^3 (102)
		// 111.1 | 113.1
		const double sms = launch_size(grd, blk, 0).sms;
		const bool early = sms < 28.0 || sms > 90.0;
		if (updown == CDR_UP) {
			if (vec) launch_as(early, k3_gs_rows<T, true, true>, grd, blk, 0, st, so, x, b, sor, F, pj, pk, nrj, nrows, W);
			else launch_as(early, k3_gs_rows<T, false, true>, grd, blk, 0, st, so, x, b, sor, F, pj, pk, nrj, nrows, W);
		} else {
			if (vec) launch_as(early, k3_gs_rows<T, true, false>, grd, blk, 0, st, so, x, b, sor, F, pj, pk, nrj, nrows, W);
			else launch_as(early, k3_gs_rows<T, false, false>, grd, blk, 0, st, so, x, b, sor, F, pj, pk, nrj, nrows, W);
		}
		CDR_LAUNCH_CHECK();
	}
	return CDR_OK;
}
template int relax_point_3d<double>(const double *, double *, const double *, const double *, Dims3, int, cudaStream_t,
                                    int);
template int relax_point_3d<float>(const float *, float *, const float *, const float *, Dims3, int, cudaStream_t, int);

template <typename T>
int setup_recip_3d(const T *so, T *sor, Dims3 F, cudaStream_t st)
{
	launch(k3_recip<T>, dim3(ceil_div(F.nx, TX), ceil_div(F.ny, TY), F.nz), dim3(TX, TY), 0, st, so, sor, F);
	CDR_LAUNCH_CHECK();
	return CDR_OK;
}
template int setup_recip_3d<double>(const double *, double *, Dims3, cudaStream_t);

// ----------------------------------------------------------------- transfers
// BMG3_SymStd_restrict (src/3d/ftn/BMG3_SymStd_restrict.f90:114-154)
template <typename T>
__global__ void __launch_bounds__(TX *TY) k3_restrict(const T *__restrict__ ci, const T *__restrict__ q,
                                                      T *__restrict__ qc, Dims3 F, Dims3 C)
{
	await_previous();
	const int ic = blockIdx.x * TX + threadIdx.x + 2, jc = blockIdx.y * TY + threadIdx.y + 2, kc = blockIdx.z + 2;
	if (ic > C.nx + 1 || jc > C.ny + 1) return;
	const int i = 2 * ic - 2, j = 2 * jc - 2, k = 2 * kc - 2;
	QC(ic, jc, kc) = CI(ic, jc, kc, LXYNE) * Q(i - 1, j - 1, k) + CI(ic, jc, kc, LXYA) * Q(i, j - 1, k)
	                 + CI(ic + 1, jc, kc, LXYNW) * Q(i + 1, j - 1, k) + CI(ic, jc, kc, LXYR) * Q(i - 1, j, k) + Q(i, j, k)
	                 + CI(ic + 1, jc, kc, LXYL) * Q(i + 1, j, k) + CI(ic, jc + 1, kc, LXYSE) * Q(i - 1, j + 1, k)
	                 + CI(ic, jc + 1, kc, LXYB) * Q(i, j + 1, k) + CI(ic + 1, jc + 1, kc, LXYSW) * Q(i + 1, j + 1, k)
	                 + CI(ic, jc, kc, LTNE) * Q(i - 1, j - 1, k - 1) + CI(ic, jc, kc, LYZNW) * Q(i, j - 1, k - 1)
	                 + CI(ic + 1, jc, kc, LTNW) * Q(i + 1, j - 1, k - 1) + CI(ic, jc, kc, LXZNE) * Q(i - 1, j, k - 1)
	                 + CI(ic, jc, kc, LXZA) * Q(i, j, k - 1) + CI(ic + 1, jc, kc, LXZNW) * Q(i + 1, j, k - 1)
	                 + CI(ic, jc + 1, kc, LTSE) * Q(i - 1, j + 1, k - 1) + CI(ic, jc + 1, kc, LYZNE) * Q(i, j + 1, k - 1)
	                 + CI(ic + 1, jc + 1, kc, LTSW) * Q(i + 1, j + 1, k - 1) + CI(ic, jc, kc + 1, LBNE) * Q(i - 1, j - 1, k + 1)
	                 + CI(ic, jc, kc + 1, LYZSW) * Q(i, j - 1, k + 1) + CI(ic + 1, jc, kc + 1, LBNW) * Q(i + 1, j - 1, k + 1)
	                 + CI(ic, jc, kc + 1, LXZSE) * Q(i - 1, j, k + 1) + CI(ic, jc, kc + 1, LXZB) * Q(i, j, k + 1)
	                 + CI(ic + 1, jc, kc + 1, LXZSW) * Q(i + 1, j, k + 1) + CI(ic, jc + 1, kc + 1, LBSE) * Q(i - 1, j + 1, k + 1)
	                 + CI(ic, jc + 1, kc + 1, LYZSE) * Q(i, j + 1, k + 1) + CI(ic + 1, jc + 1, kc + 1, LBSW) * Q(i + 1, j + 1, k + 1);
}

// BMG3_SymStd_interp_add (src/3d/ftn/BMG3_SymStd_interp_add.f90:108-239).  The
// reference's three loop nests write disjoint sets of fine points and each
// update reads only its own target in q, so one thread per (IC, JC, KC) does the
// writes of all three nests.  r/c is formed on the fly (the reference divides
// r in place on interior points; a ghost-layer point, reached for even sizes,
// adds r undivided).
template <typename T>
__global__ void __launch_bounds__(TX *TY) k3_interp_add(const T *__restrict__ ci, const T *__restrict__ qc,
                                                        const T *__restrict__ res, const T *__restrict__ so,
                                                        T *__restrict__ q, Dims3 F, Dims3 C)
{
	await_previous();
	const int ic = blockIdx.x * TX + threadIdx.x + 2, jc = blockIdx.y * TY + threadIdx.y + 2, kc = blockIdx.z + 2;
	const int iic1 = C.nx + 1, kkc1 = C.nz + 1;
	const int iicf1 = F.nx / 2 + 2, jjcf1 = F.ny / 2 + 2, kkcf1 = F.nz / 2 + 2;
	if (ic > iicf1 || jc > jjcf1) return;
	auto RES = [&](int i, int j, int k) -> T {
		const size_t o = F.at1(i, j, k);
		const bool in = i >= 2 && i <= F.nx + 1 && j >= 2 && j <= F.ny + 1 && k >= 2 && k <= F.nz + 1;
		return in ? res[o] / so[o] : res[o];
	};
	if (kc <= kkc1) {  // coarse-aligned k-planes, k = 2KC-2: the 2D pattern
		const int k = 2 * kc - 2, i = 2 * ic - 2, j = 2 * jc - 2;
		Q(i, j, k) = Q(i, j, k) + QC(ic, jc, kc);
		if (ic >= 3) {
			const T a = CI(ic, jc, kc, LXYR) * QC(ic, jc, kc) + CI(ic, jc, kc, LXYL) * QC(ic - 1, jc, kc);
			Q(i - 1, j, k) = Q(i - 1, j, k) + a + RES(i - 1, j, k);
		}
		if (jc >= 3) {
			const T aq = CI(ic, jc, kc, LXYA) * QC(ic, jc, kc) + CI(ic, jc, kc, LXYB) * QC(ic, jc - 1, kc);
			Q(i, j - 1, k) = Q(i, j - 1, k) + aq + RES(i, j - 1, k);
		}
		if (ic >= 3 && jc >= 3) {
			const T a = CI(ic, jc, kc, LXYSW) * QC(ic - 1, jc - 1, kc) + CI(ic, jc, kc, LXYNW) * QC(ic - 1, jc, kc)
			            + CI(ic, jc, kc, LXYNE) * QC(ic, jc, kc) + CI(ic, jc, kc, LXYSE) * QC(ic, jc - 1, kc);
			Q(i - 1, j - 1, k) = Q(i - 1, j - 1, k) + a + RES(i - 1, j - 1, k);
		}
	}
	if (kc < 3 || kc > kkcf1) return;
	const int k = 2 * kc - 3, j = 2 * jc - 2;
	if (ic <= iic1) {  // fine-only k-planes, coarse-aligned x: i = 2IC-2
		const int i = 2 * ic - 2;
		Q(i, j, k) = Q(i, j, k) + CI(ic, jc, kc, LXZA) * QC(ic, jc, kc) + CI(ic, jc, kc, LXZB) * QC(ic, jc, kc - 1)
		             + RES(i, j, k);
		if (jc >= 3)
			Q(i, j - 1, k) = Q(i, j - 1, k) + CI(ic, jc, kc, LYZNW) * QC(ic, jc, kc) + CI(ic, jc, kc, LYZNE) * QC(ic, jc - 1, kc)
			                 + CI(ic, jc, kc, LYZSW) * QC(ic, jc, kc - 1) + CI(ic, jc, kc, LYZSE) * QC(ic, jc - 1, kc - 1)
			                 + RES(i, j - 1, k);
	}
	if (ic >= 3) {  // fine-only k-planes, fine-only x: i = 2IC-3
		const int i = 2 * ic - 3;
		Q(i, j, k) = Q(i, j, k) + CI(ic, jc, kc, LXZNW) * QC(ic - 1, jc, kc) + CI(ic, jc, kc, LXZNE) * QC(ic, jc, kc)
		             + CI(ic, jc, kc, LXZSW) * QC(ic - 1, jc, kc - 1) + CI(ic, jc, kc, LXZSE) * QC(ic, jc, kc - 1)
		             + RES(i, j, k);
		if (jc >= 3)
			Q(i, j - 1, k) = Q(i, j - 1, k) + CI(ic, jc, kc, LTNW) * QC(ic - 1, jc, kc) + CI(ic, jc, kc, LTNE) * QC(ic, jc, kc)
			                 + CI(ic, jc, kc, LTSW) * QC(ic - 1, jc - 1, kc) + CI(ic, jc, kc, LTSE) * QC(ic, jc - 1, kc)
			                 + CI(ic, jc, kc, LBNW) * QC(ic - 1, jc, kc - 1) + CI(ic, jc, kc, LBNE) * QC(ic, jc, kc - 1)
			                 + CI(ic, jc, kc, LBSW) * QC(ic - 1, jc - 1, kc - 1) + CI(ic, jc, kc, LBSE) * QC(ic, jc - 1, kc - 1)
			                 + RES(i, j - 1, k);
	}
}

template <typename T>
int restrict_3d(const T *ci, const T *rf, T *bc, Dims3 F, Dims3 C, cudaStream_t st)
{
	launch(k3_restrict<T>, dim3(ceil_div(C.nx, TX), ceil_div(C.ny, TY), C.nz), dim3(TX, TY), 0, st, ci, rf, bc, F, C);
	CDR_LAUNCH_CHECK();
	return CDR_OK;
}
template int restrict_3d<double>(const double *, const double *, double *, Dims3, Dims3, cudaStream_t);
template int restrict_3d<float>(const float *, const float *, float *, Dims3, Dims3, cudaStream_t);

template <typename T>
int interp_add_3d(const T *ci, const T *xc, const T *rf, const T *sof, T *xf, Dims3 F, Dims3 C, cudaStream_t st)
{
	const dim3 grd(ceil_div(F.nx / 2 + 1, TX), ceil_div(F.ny / 2 + 1, TY), F.nz / 2 + 1);
	launch(k3_interp_add<T>, grd, dim3(TX, TY), 0, st, ci, xc, rf, sof, xf, F, C);
	CDR_LAUNCH_CHECK();
	return CDR_OK;
}
template int interp_add_3d<double>(const double *, const double *, const double *, const double *, double *, Dims3,
                                   Dims3, cudaStream_t);
template int interp_add_3d<float>(const float *, const float *, const float *, const float *, float *, Dims3, Dims3,
                                  cudaStream_t);

// ------------------------------------------------ operator-induced interpolation
// BMG3_SymStd_SETUP_interp_OI (src/3d/ftn/BMG3_SymStd_SETUP_interp_OI.f90:121-537),
// non-periodic, 27-point fine operator.  Launch 0: edge weights (x-, y-, z-edges);
// launch 1: face weights (xy, xz, yz), which read edge weights; launch 2:
// interior weights, which read face and edge weights.  Every thread handles one
// (IC, JC, KC) and the fine point (2IC-2, 2JC-2, 2KC-2) the formulas are centred on.
__device__ __forceinline__ double dmin2(double a, double b) { return a < b ? a : b; }

__global__ void __launch_bounds__(TX *TY) k3_oi(const double *__restrict__ so, double *__restrict__ ci, Dims3 F,
                                                Dims3 C, int phase)
{
	await_previous();
	const int ic = blockIdx.x * TX + threadIdx.x + 2, jc = blockIdx.y * TY + threadIdx.y + 2, kc = blockIdx.z + 2;
	const int iic1 = C.nx + 1, jjc1 = C.ny + 1, kkc1 = C.nz + 1;
	const int iicf1 = F.nx / 2 + 2, jjcf1 = F.ny / 2 + 2, kkcf1 = F.nz / 2 + 2;
	const double emach = 1.1102230246251565e-16;
	const int i = 2 * ic - 2, j = 2 * jc - 2, k = 2 * kc - 2;
	double a, b, c, ep, dnw, dn, dne, dw, de, dsw, ds, dse, dp, sum;
	if (phase == 0) {
		if (kc <= kkc1 && jc <= jjc1 && ic >= 3 && ic <= iicf1) {  // x-edges: lxyl, lxyr
			a = SO(i - 1, j + 1, k, KPNW) + SO(i - 1, j, k, KPW) + SO(i - 1, j, k, KPSW) + SO(i - 1, j + 1, k, KBNW)
			    + SO(i - 1, j, k, KBW) + SO(i - 1, j, k, KBSW) + SO(i - 1, j + 1, k + 1, KBSE) + SO(i - 1, j, k + 1, KBE)
			    + SO(i - 1, j, k + 1, KBNE);
			b = SO(i, j + 1, k, KPSW) + SO(i, j, k, KPW) + SO(i, j, k, KPNW) + SO(i, j + 1, k, KBNE) + SO(i, j, k, KBE)
			    + SO(i, j, k, KBSE) + SO(i, j + 1, k + 1, KBSW) + SO(i, j, k + 1, KBW) + SO(i, j, k + 1, KBNW);
			c = a + b + SO(i - 1, j, k, KPS) + SO(i - 1, j + 1, k, KPS) + SO(i - 1, j + 1, k, KBN) + SO(i - 1, j, k, KB)
			    + SO(i - 1, j, k, KBS) + SO(i - 1, j + 1, k + 1, KBS) + SO(i - 1, j, k + 1, KB) + SO(i - 1, j, k + 1, KBN);
			ep = dmin2(fabs(a / SO(i - 1, j, k, KP)), fabs(b / SO(i - 1, j, k, KP)));
			c = a + b + (SO(i - 1, j, k, KP) - c) * fmax(SO(i - 1, j, k, KP) - (1.0 + ep) * c, 0.0)
			            / (fabs(SO(i - 1, j, k, KP) - (1.0 + ep) * c) + emach);
			CI(ic, jc, kc, LXYL) = a / c;
			CI(ic, jc, kc, LXYR) = b / c;
		}
		if (kc <= kkc1 && jc >= 3 && jc <= jjcf1 && ic <= iic1) {  // y-edges: lxya, lxyb
			a = SO(i, j, k, KPNW) + SO(i, j, k, KPS) + SO(i + 1, j, k, KPSW) + SO(i, j, k, KBNW) + SO(i, j, k, KBN)
			    + SO(i + 1, j, k, KBNE) + SO(i, j, k + 1, KBSE) + SO(i, j, k + 1, KBS) + SO(i + 1, j, k + 1, KBSW);
			b = SO(i, j - 1, k, KPSW) + SO(i, j - 1, k, KPS) + SO(i + 1, j - 1, k, KPNW) + SO(i, j - 1, k, KBSW)
			    + SO(i, j - 1, k, KBS) + SO(i + 1, j - 1, k, KBSE) + SO(i, j - 1, k + 1, KBNE) + SO(i, j - 1, k + 1, KBN)
			    + SO(i + 1, j - 1, k + 1, KBNW);
			ep = dmin2(fabs(a / SO(i, j - 1, k, KP)), fabs(b / SO(i, j - 1, k, KP)));
			c = a + b + SO(i, j - 1, k, KPW) + SO(i + 1, j - 1, k, KPW) + SO(i, j - 1, k, KBW) + SO(i, j - 1, k, KB)
			    + SO(i + 1, j - 1, k, KBE) + SO(i, j - 1, k + 1, KBE) + SO(i, j - 1, k + 1, KB) + SO(i + 1, j - 1, k + 1, KBW);
			c = a + b + (SO(i, j - 1, k, KP) - c) * fmax(SO(i, j - 1, k, KP) - (1.0 + ep) * c, 0.0)
			            / (fabs(SO(i, j - 1, k, KP) - (1.0 + ep) * c) + emach);
			CI(ic, jc, kc, LXYA) = a / c;
			CI(ic, jc, kc, LXYB) = b / c;
		}
		if (kc >= 3 && kc <= kkcf1 && jc <= jjc1 && ic <= iic1) {  // z-edges: lxza, lxzb
			a = SO(i, j + 1, k, KBSE) + SO(i, j + 1, k, KBS) + SO(i + 1, j + 1, k, KBSW) + SO(i, j, k, KBE) + SO(i, j, k, KB)
			    + SO(i + 1, j, k, KBW) + SO(i, j, k, KBNE) + SO(i, j, k, KBN) + SO(i + 1, j, k, KBNW);
			b = SO(i, j + 1, k - 1, KBNW) + SO(i, j + 1, k - 1, KBN) + SO(i + 1, j + 1, k - 1, KBNE) + SO(i, j, k - 1, KBW)
			    + SO(i, j, k - 1, KB) + SO(i + 1, j, k - 1, KBE) + SO(i, j, k - 1, KBSW) + SO(i, j, k - 1, KBS)
			    + SO(i + 1, j, k - 1, KBSE);
			c = a + b + SO(i, j, k - 1, KPW) + SO(i + 1, j, k - 1, KPW) + SO(i, j + 1, k - 1, KPNW) + SO(i, j + 1, k - 1, KPS)
			    + SO(i + 1, j + 1, k - 1, KPSW) + SO(i, j, k - 1, KPSW) + SO(i, j, k - 1, KPS) + SO(i + 1, j, k - 1, KPNW);
			ep = dmin2(fabs(a / SO(i, j, k - 1, KP)), fabs(b / SO(i, j, k - 1, KP)));
			c = a + b + (SO(i, j, k - 1, KP) - c) * fmax(SO(i, j, k - 1, KP) - (1.0 + ep) * c, 0.0)
			            / (fabs(SO(i, j, k - 1, KP) - (1.0 + ep) * c) + emach);
			CI(ic, jc, kc, LXZA) = a / c;
			CI(ic, jc, kc, LXZB) = b / c;
		}
	} else if (phase == 1) {
		if (kc <= kkc1 && jc >= 3 && jc <= jjcf1 && ic >= 3 && ic <= iicf1) {  // xy faces
			dnw = SO(i - 1, j, k, KPNW) + SO(i - 1, j, k, KBNW) + SO(i - 1, j, k + 1, KBSE);
			dn = SO(i - 1, j, k, KPS) + SO(i - 1, j, k, KBN) + SO(i - 1, j, k + 1, KBS);
			dne = SO(i, j, k, KPSW) + SO(i, j, k, KBNE) + SO(i, j, k + 1, KBSW);
			dw = SO(i - 1, j - 1, k, KPW) + SO(i - 1, j - 1, k, KBW) + SO(i - 1, j - 1, k + 1, KBE);
			de = SO(i, j - 1, k, KPW) + SO(i, j - 1, k, KBE) + SO(i, j - 1, k + 1, KBW);
			dsw = SO(i - 1, j - 1, k, KPSW) + SO(i - 1, j - 1, k, KBSW) + SO(i - 1, j - 1, k + 1, KBNE);
			ds = SO(i - 1, j - 1, k, KPS) + SO(i - 1, j - 1, k, KBS) + SO(i - 1, j - 1, k + 1, KBN);
			dse = SO(i, j - 1, k, KPNW) + SO(i, j - 1, k, KBSE) + SO(i, j - 1, k + 1, KBNW);
			const double o = SO(i - 1, j - 1, k, KP);
			ep = dmin2(dmin2(dmin2(fabs((dsw + dw + dnw) / o), fabs((dnw + dn + dne) / o)), fabs((dne + de + dse) / o)),
			           fabs((dse + ds + dsw) / o));
			dp = dw + dnw + dn + dne + de + dse + ds + dsw;
			sum = o - SO(i - 1, j - 1, k, KB) - SO(i - 1, j - 1, k + 1, KB);
			dp = dp + (sum - dp) * fmax(sum - (1.0 + ep) * dp, 0.0) / (fabs(sum - (1.0 + ep) * dp) + emach);
			dp = 1.0 / dp;
			CI(ic, jc, kc, LXYNW) = dp * (dnw + CI(ic - 1, jc, kc, LXYA) * dw + CI(ic, jc, kc, LXYL) * dn);
			CI(ic, jc, kc, LXYNE) = dp * (dne + CI(ic, jc, kc, LXYR) * dn + CI(ic, jc, kc, LXYA) * de);
			CI(ic, jc, kc, LXYSE) = dp * (dse + CI(ic, jc, kc, LXYB) * de + CI(ic, jc - 1, kc, LXYR) * ds);
			CI(ic, jc, kc, LXYSW) = dp * (dsw + CI(ic, jc - 1, kc, LXYL) * ds + CI(ic - 1, jc, kc, LXYB) * dw);
		}
		if (kc >= 3 && kc <= kkcf1 && jc <= jjc1 && ic >= 3 && ic <= iicf1) {  // xz faces
			dnw = SO(i - 1, j + 1, k, KBSE) + SO(i - 1, j, k, KBE) + SO(i - 1, j, k, KBNE);
			dn = SO(i - 1, j + 1, k, KBS) + SO(i - 1, j, k, KB) + SO(i - 1, j, k, KBN);
			dne = SO(i, j + 1, k, KBSW) + SO(i, j, k, KBW) + SO(i, j, k, KBNW);
			dw = SO(i - 1, j + 1, k - 1, KPNW) + SO(i - 1, j, k - 1, KPW) + SO(i - 1, j, k - 1, KPSW);
			de = SO(i, j + 1, k - 1, KPSW) + SO(i, j, k - 1, KPW) + SO(i, j, k - 1, KPNW);
			dsw = SO(i - 1, j + 1, k - 1, KBNW) + SO(i - 1, j, k - 1, KBW) + SO(i - 1, j, k - 1, KBSW);
			ds = SO(i - 1, j + 1, k - 1, KBN) + SO(i - 1, j, k - 1, KB) + SO(i - 1, j, k - 1, KBS);
			dse = SO(i, j + 1, k - 1, KBNE) + SO(i, j, k - 1, KBE) + SO(i, j, k - 1, KBSE);
			const double o = SO(i - 1, j, k - 1, KP);
			ep = dmin2(dmin2(dmin2(fabs((dsw + dw + dnw) / o), fabs((dnw + dn + dne) / o)), fabs((dne + de + dse) / o)),
			           fabs((dse + ds + dsw) / o));
			dp = dw + dnw + dn + dne + de + dse + ds + dsw;
			sum = o - SO(i - 1, j + 1, k - 1, KPS) - SO(i - 1, j, k - 1, KPS);
			dp = dp + (sum - dp) * fmax(sum - (1.0 + ep) * dp, 0.0) / (fabs(sum - (1.0 + ep) * dp) + emach);
			dp = 1.0 / dp;
			CI(ic, jc, kc, LXZNW) = dp * (dnw + CI(ic - 1, jc, kc, LXZA) * dw + CI(ic, jc, kc, LXYL) * dn);
			CI(ic, jc, kc, LXZNE) = dp * (dne + CI(ic, jc, kc, LXYR) * dn + CI(ic, jc, kc, LXZA) * de);
			CI(ic, jc, kc, LXZSE) = dp * (dse + CI(ic, jc, kc, LXZB) * de + CI(ic, jc, kc - 1, LXYR) * ds);
			CI(ic, jc, kc, LXZSW) = dp * (dsw + CI(ic, jc, kc - 1, LXYL) * ds + CI(ic - 1, jc, kc, LXZB) * dw);
		}
		if (kc >= 3 && kc <= kkcf1 && jc >= 3 && jc <= jjcf1 && ic <= iic1) {  // yz faces
			dnw = SO(i, j, k, KBSE) + SO(i, j, k, KBS) + SO(i + 1, j, k, KBSW);
			dn = SO(i, j - 1, k, KBE) + SO(i, j - 1, k, KB) + SO(i + 1, j - 1, k, KBW);
			dne = SO(i, j - 1, k, KBNE) + SO(i, j - 1, k, KBN) + SO(i + 1, j - 1, k, KBNW);
			dw = SO(i, j, k - 1, KPNW) + SO(i, j, k - 1, KPS) + SO(i + 1, j, k - 1, KPSW);
			de = SO(i, j - 1, k - 1, KPSW) + SO(i, j - 1, k - 1, KPS) + SO(i + 1, j - 1, k - 1, KPNW);
			dsw = SO(i, j, k - 1, KBNW) + SO(i, j, k - 1, KBN) + SO(i + 1, j, k - 1, KBNE);
			ds = SO(i, j - 1, k - 1, KBW) + SO(i, j - 1, k - 1, KB) + SO(i + 1, j - 1, k - 1, KBE);
			dse = SO(i, j - 1, k - 1, KBSW) + SO(i, j - 1, k - 1, KBS) + SO(i + 1, j - 1, k - 1, KBSE);
			const double o = SO(i, j - 1, k - 1, KP);
			ep = dmin2(dmin2(dmin2(fabs((dsw + dw + dnw) / o), fabs((dnw + dn + dne) / o)), fabs((dne + de + dse) / o)),
			           fabs((dse + ds + dsw) / o));
			dp = dw + dnw + dn + dne + de + dse + ds + dsw;
			sum = o - SO(i, j - 1, k - 1, KPW) - SO(i + 1, j - 1, k - 1, KPW);
			dp = dp + (sum - dp) * fmax(sum - (1.0 + ep) * dp, 0.0) / (fabs(sum - (1.0 + ep) * dp) + emach);
			dp = 1.0 / dp;
			CI(ic, jc, kc, LYZNW) = dp * (dnw + CI(ic, jc, kc, LXZA) * dw + CI(ic, jc, kc, LXYA) * dn);
			CI(ic, jc, kc, LYZNE) = dp * (dne + CI(ic, jc, kc, LXYB) * dn + CI(ic, jc - 1, kc, LXZA) * de);
			CI(ic, jc, kc, LYZSE) = dp * (dse + CI(ic, jc - 1, kc, LXZB) * de + CI(ic, jc, kc - 1, LXYB) * ds);
			CI(ic, jc, kc, LYZSW) = dp * (dsw + CI(ic, jc, kc - 1, LXYA) * ds + CI(ic, jc, kc, LXZB) * dw);
		}
	} else {
		if (!(kc >= 3 && kc <= kkcf1 && jc >= 3 && jc <= jjcf1 && ic >= 3 && ic <= iicf1)) return;
		double yp = SO(i - 1, j - 1, k - 1, KPW) + SO(i - 1, j, k - 1, KPNW) + SO(i - 1, j, k - 1, KPS)
		            + SO(i, j, k - 1, KPSW) + SO(i, j - 1, k - 1, KPW) + SO(i, j - 1, k - 1, KPNW)
		            + SO(i - 1, j - 1, k - 1, KPS) + SO(i - 1, j - 1, k - 1, KPSW) + SO(i - 1, j - 1, k - 1, KB)
		            + SO(i - 1, j - 1, k - 1, KBW) + SO(i - 1, j, k - 1, KBNW) + SO(i - 1, j, k - 1, KBN)
		            + SO(i, j, k - 1, KBNE) + SO(i, j - 1, k - 1, KBE) + SO(i, j - 1, k - 1, KBSE)
		            + SO(i - 1, j - 1, k - 1, KBS) + SO(i - 1, j - 1, k - 1, KBSW) + SO(i - 1, j - 1, k, KB)
		            + SO(i - 1, j - 1, k, KBE) + SO(i - 1, j, k, KBSE) + SO(i - 1, j, k, KBS) + SO(i, j, k, KBSW)
		            + SO(i, j - 1, k, KBW) + SO(i, j - 1, k, KBNW) + SO(i - 1, j - 1, k, KBN) + SO(i - 1, j - 1, k, KBNE);
		const double o = SO(i - 1, j - 1, k - 1, KP);
		const double m1 = fabs(SO(i - 1, j - 1, k - 1, KPW) + SO(i - 1, j, k - 1, KPNW) + SO(i - 1, j, k, KBSE)
		                       + SO(i - 1, j - 1, k, KBE) + SO(i - 1, j - 1, k, KBNE) + SO(i - 1, j - 1, k - 1, KPSW)
		                       + SO(i - 1, j - 1, k - 1, KBSW) + SO(i - 1, j - 1, k - 1, KBW) + SO(i - 1, j, k - 1, KBNW))
		                  / o;
		const double m2 = fabs(SO(i, j - 1, k - 1, KPW) + SO(i, j, k - 1, KPSW) + SO(i, j, k, KBSW) + SO(i, j - 1, k, KBW)
		                       + SO(i, j - 1, k, KBNW) + SO(i, j - 1, k - 1, KPNW) + SO(i, j - 1, k - 1, KBSE)
		                       + SO(i, j - 1, k - 1, KBE) + SO(i, j, k - 1, KBNE))
		                  / o;
		const double m3 = fabs(SO(i - 1, j, k - 1, KPS) + SO(i - 1, j, k - 1, KPNW) + SO(i - 1, j, k, KBSE) + SO(i - 1, j, k, KBS)
		                       + SO(i, j, k, KBSW) + SO(i, j, k - 1, KPSW) + SO(i, j, k - 1, KBNE) + SO(i - 1, j, k - 1, KBN)
		                       + SO(i - 1, j, k - 1, KBNW));
		const double m4 = fabs(SO(i - 1, j - 1, k - 1, KPS) + SO(i - 1, j - 1, k - 1, KPSW) + SO(i - 1, j - 1, k, KBNE)
		                       + SO(i - 1, j - 1, k, KBN) + SO(i, j - 1, k, KBNW) + SO(i, j - 1, k - 1, KPNW)
		                       + SO(i, j - 1, k - 1, KBSE) + SO(i - 1, j - 1, k - 1, KBS) + SO(i, j - 1, k - 1, KBSE))
		                  / o;
		double ypw = dmin2(dmin2(dmin2(m1, m2), m3), m4);  // third argument undivided, as the reference
		const double m5 = fabs(SO(i - 1, j - 1, k - 1, KB) + SO(i - 1, j - 1, k - 1, KBW) + SO(i - 1, j, k - 1, KBNW)
		                       + SO(i - 1, j, k - 1, KBN) + SO(i, j, k - 1, KBNE) + SO(i, j - 1, k - 1, KBE)
		                       + SO(i, j - 1, k - 1, KBSE) + SO(i - 1, j - 1, k - 1, KBS) + SO(i - 1, j - 1, k - 1, KBSW));
		const double m6 = fabs(SO(i - 1, j - 1, k, KB) + SO(i - 1, j - 1, k, KBE) + SO(i - 1, j, k, KBSE) + SO(i - 1, j, k, KBS)
		                       + SO(i, j, k, KBSW) + SO(i, j - 1, k, KBW) + SO(i, j - 1, k, KBNW) + SO(i - 1, j - 1, k, KBN)
		                       + SO(i - 1, j - 1, k, KBNE))
		                  / o;
		ypw = dmin2(dmin2(ypw, m5), m6);  // fifth argument undivided, as the reference
		yp = yp + (o - yp) * fmax(o - (1.0 + ypw) * yp, 0.0) / (fabs(o - (1.0 + ypw) * yp) + emach);
		yp = 1.0 / yp;
		CI(ic, jc, kc, LTNW) = yp * (SO(i - 1, j, k, KBSE) + CI(ic - 1, jc, kc, LYZNW) * SO(i - 1, j - 1, k - 1, KPW)
		                             + CI(ic - 1, jc, kc, LXZA) * SO(i - 1, j, k - 1, KPNW) + CI(ic, jc, kc, LXZNW) * SO(i - 1, j, k - 1, KPS)
		                             + CI(ic - 1, jc, kc, LXYA) * SO(i - 1, j - 1, k, KBE) + CI(ic, jc, kc, LXYL) * SO(i - 1, j, k, KBS)
		                             + CI(ic, jc, kc, LXYNW) * SO(i - 1, j - 1, k, KB));
		CI(ic, jc, kc, LTNE) = yp * (SO(i, j, k, KBSW) + CI(ic, jc, kc, LXZNE) * SO(i - 1, j, k - 1, KPS)
		                             + CI(ic, jc, kc, LXZA) * SO(i, j, k - 1, KPSW) + CI(ic, jc, kc, LYZNW) * SO(i, j - 1, k - 1, KPW)
		                             + CI(ic, jc, kc, LXYR) * SO(i - 1, j, k, KBS) + CI(ic, jc, kc, LXYA) * SO(i, j - 1, k, KBW)
		                             + CI(ic, jc, kc, LXYNE) * SO(i - 1, j - 1, k, KB));
		CI(ic, jc, kc, LBNW) = yp * (SO(i - 1, j, k - 1, KBNW) + CI(ic - 1, jc, kc - 1, LXYA) * SO(i - 1, j - 1, k - 1, KBW)
		                             + CI(ic, jc, kc - 1, LXYL) * SO(i - 1, j, k - 1, KBN) + CI(ic, jc, kc - 1, LXYNW) * SO(i - 1, j - 1, k - 1, KB)
		                             + CI(ic - 1, jc, kc, LYZSW) * SO(i - 1, j - 1, k - 1, KPW) + CI(ic - 1, jc, kc, LXZB) * SO(i - 1, j, k - 1, KPNW)
		                             + CI(ic, jc, kc, LXZSW) * SO(i - 1, j, k - 1, KPS));
		CI(ic, jc, kc, LBNE) = yp * (SO(i, j, k - 1, KBNE) + CI(ic, jc, kc - 1, LXYNE) * SO(i - 1, j - 1, k - 1, KB)
		                             + CI(ic, jc, kc - 1, LXYR) * SO(i - 1, j, k - 1, KBN) + CI(ic, jc, kc - 1, LXYA) * SO(i, j - 1, k - 1, KBE)
		                             + CI(ic, jc, kc, LXZSE) * SO(i - 1, j, k - 1, KPS) + CI(ic, jc, kc, LXZB) * SO(i, j, k - 1, KPSW)
		                             + CI(ic, jc, kc, LYZSW) * SO(i, j - 1, k - 1, KPW));
		CI(ic, jc, kc, LBSW) = yp * (SO(i - 1, j - 1, k - 1, KBSW) + CI(ic - 1, jc, kc - 1, LXYB) * SO(i - 1, j - 1, k - 1, KBW)
		                             + CI(ic, jc, kc - 1, LXYSW) * SO(i - 1, j - 1, k - 1, KB) + CI(ic, jc - 1, kc - 1, LXYL) * SO(i - 1, j - 1, k - 1, KBS)
		                             + CI(ic - 1, jc, kc, LYZSE) * SO(i - 1, j - 1, k - 1, KPW) + CI(ic, jc - 1, kc, LXZSW) * SO(i - 1, j - 1, k - 1, KPS)
		                             + CI(ic - 1, jc - 1, kc, LXZB) * SO(i - 1, j - 1, k - 1, KPSW));
		CI(ic, jc, kc, LTSW) = yp * (SO(i - 1, j - 1, k, KBNE) + CI(ic - 1, jc, kc, LXYB) * SO(i - 1, j - 1, k, KBE)
		                             + CI(ic, jc, kc, LXYSW) * SO(i - 1, j - 1, k, KB) + CI(ic, jc - 1, kc, LXYL) * SO(i - 1, j - 1, k, KBN)
		                             + CI(ic - 1, jc, kc, LYZNE) * SO(i - 1, j - 1, k - 1, KPW) + CI(ic, jc - 1, kc, LXZNW) * SO(i - 1, j - 1, k - 1, KPS)
		                             + CI(ic - 1, jc - 1, kc, LXZA) * SO(i - 1, j - 1, k - 1, KPSW));
		CI(ic, jc, kc, LTSE) = yp * (SO(i, j - 1, k, KBNW) + CI(ic, jc - 1, kc, LXYR) * SO(i - 1, j - 1, k, KBN)
		                             + CI(ic, jc, kc, LXYSE) * SO(i - 1, j - 1, k, KB) + CI(ic, jc, kc, LXYB) * SO(i, j - 1, k, KBW)
		                             + CI(ic, jc - 1, kc, LXZNE) * SO(i - 1, j - 1, k - 1, KPS) + CI(ic, jc, kc, LYZNE) * SO(i, j - 1, k - 1, KPW)
		                             + CI(ic, jc - 1, kc, LXZA) * SO(i, j - 1, k - 1, KPNW));
		CI(ic, jc, kc, LBSE) = yp * (SO(i, j - 1, k - 1, KBSE) + CI(ic, jc - 1, kc - 1, LXYR) * SO(i - 1, j - 1, k - 1, KBS)
		                             + CI(ic, jc, kc - 1, LXYSE) * SO(i - 1, j - 1, k - 1, KB) + CI(ic, jc, kc - 1, LXYB) * SO(i, j - 1, k - 1, KBE)
		                             + CI(ic, jc - 1, kc, LXZSE) * SO(i - 1, j - 1, k - 1, KPS) + CI(ic, jc, kc, LYZSE) * SO(i, j - 1, k - 1, KPW)
		                             + CI(ic, jc - 1, kc, LXZB) * SO(i, j - 1, k - 1, KPNW));
	}
}

// The seven-point branch of BMG3_SymStd_SETUP_interp_OI
// (BMG3_SymStd_SETUP_interp_OI.f90:543-807), same three phases.  Kept from the
// reference: the x-edge ep divides |b| (not b) by so(kp), and the interior
// correction is added after the product ((o - dp) * ... + dp).
__global__ void __launch_bounds__(TX *TY) k3_oi7(const double *__restrict__ so, double *__restrict__ ci, Dims3 F,
                                                 Dims3 C, int phase)
{
	await_previous();
	const int ic = blockIdx.x * TX + threadIdx.x + 2, jc = blockIdx.y * TY + threadIdx.y + 2, kc = blockIdx.z + 2;
	const int iic1 = C.nx + 1, jjc1 = C.ny + 1, kkc1 = C.nz + 1;
	const int iicf1 = F.nx / 2 + 2, jjcf1 = F.ny / 2 + 2, kkcf1 = F.nz / 2 + 2;
	const double emach = 1.1102230246251565e-16;
	const int i = 2 * ic - 2, j = 2 * jc - 2, k = 2 * kc - 2;
	double a, b, c, ep, dn, dw, de, ds, dp, sum, o;
	if (phase == 0) {
		if (kc <= kkc1 && jc <= jjc1 && ic >= 3 && ic <= iicf1) {  // x-edges: lxyl, lxyr
			a = SO(i - 1, j, k, KPW);
			b = SO(i, j, k, KPW);
			ep = dmin2(fabs(a / SO(i - 1, j, k, KP)), fabs(b) / SO(i - 1, j, k, KP));
			c = a + b + SO(i - 1, j, k, KPS) + SO(i - 1, j + 1, k, KPS) + SO(i - 1, j, k, KB) + SO(i - 1, j, k + 1, KB);
			c = a + b + (SO(i - 1, j, k, KP) - c) * fmax(SO(i - 1, j, k, KP) - (1.0 + ep) * c, 0.0)
			            / (fabs(SO(i - 1, j, k, KP) - (1.0 + ep) * c) + emach);
			CI(ic, jc, kc, LXYL) = a / c;
			CI(ic, jc, kc, LXYR) = b / c;
		}
		if (kc <= kkc1 && jc >= 3 && jc <= jjcf1 && ic <= iic1) {  // y-edges: lxya, lxyb
			a = SO(i, j, k, KPS);
			b = SO(i, j - 1, k, KPS);
			c = a + b + SO(i, j - 1, k, KPW) + SO(i + 1, j - 1, k, KPW) + SO(i, j - 1, k, KB) + SO(i, j - 1, k + 1, KB);
			ep = dmin2(fabs(a / SO(i, j - 1, k, KP)), fabs(b / SO(i, j - 1, k, KP)));
			c = a + b + (SO(i, j - 1, k, KP) - c) * fmax(SO(i, j - 1, k, KP) - (1.0 + ep) * c, 0.0)
			            / (fabs(SO(i, j - 1, k, KP) - (1.0 + ep) * c) + emach);
			CI(ic, jc, kc, LXYA) = a / c;
			CI(ic, jc, kc, LXYB) = b / c;
		}
		if (kc >= 3 && kc <= kkcf1 && jc <= jjc1 && ic <= iic1) {  // z-edges: lxza, lxzb
			a = SO(i, j, k, KB);
			b = SO(i, j, k - 1, KB);
			c = a + b + SO(i, j, k - 1, KPW) + SO(i + 1, j, k - 1, KPW) + SO(i, j + 1, k - 1, KPS) + SO(i, j, k - 1, KPS);
			ep = dmin2(fabs(a / SO(i, j, k - 1, KP)), fabs(b / SO(i, j, k - 1, KP)));
			c = a + b + (SO(i, j, k - 1, KP) - c) * fmax(SO(i, j, k - 1, KP) - (1.0 + ep) * c, 0.0)
			            / (fabs(SO(i, j, k - 1, KP) - (1.0 + ep) * c) + emach);
			CI(ic, jc, kc, LXZA) = a / c;
			CI(ic, jc, kc, LXZB) = b / c;
		}
	} else if (phase == 1) {
		if (ic >= 3 && ic <= iicf1 && jc >= 3 && jc <= jjcf1 && kc <= kkc1) {  // xy faces
			o = SO(i - 1, j - 1, k, KP);
			dn = SO(i - 1, j, k, KPS);
			dw = SO(i - 1, j - 1, k, KPW);
			de = SO(i, j - 1, k, KPW);
			ds = SO(i - 1, j - 1, k, KPS);
			dp = dw + dn + de + ds;
			sum = o - SO(i - 1, j - 1, k, KB) - SO(i - 1, j - 1, k + 1, KB);
			ep = dmin2(dmin2(dmin2(fabs(dw / o), fabs(dn / o)), fabs(de / o)), fabs(ds / o));
			dp = dp + (sum - dp) * fmax(sum - (1.0 + ep) * dp, 0.0) / (fabs(sum - (1.0 + ep) * dp) + emach);
			dp = 1.0 / dp;
			CI(ic, jc, kc, LXYNW) = dp * (CI(ic - 1, jc, kc, LXYA) * dw + CI(ic, jc, kc, LXYL) * dn);
			CI(ic, jc, kc, LXYNE) = dp * (CI(ic, jc, kc, LXYR) * dn + CI(ic, jc, kc, LXYA) * de);
			CI(ic, jc, kc, LXYSE) = dp * (CI(ic, jc, kc, LXYB) * de + CI(ic, jc - 1, kc, LXYR) * ds);
			CI(ic, jc, kc, LXYSW) = dp * (CI(ic, jc - 1, kc, LXYL) * ds + CI(ic - 1, jc, kc, LXYB) * dw);
		}
		if (kc >= 3 && kc <= kkcf1 && jc <= jjc1 && ic >= 3 && ic <= iicf1) {  // xz faces
			o = SO(i - 1, j, k - 1, KP);
			dn = SO(i - 1, j, k, KB);
			dw = SO(i - 1, j, k - 1, KPW);
			de = SO(i, j, k - 1, KPW);
			ds = SO(i - 1, j, k - 1, KB);
			dp = dw + dn + de + ds;
			sum = o - SO(i - 1, j + 1, k - 1, KPS) - SO(i - 1, j, k - 1, KPS);
			ep = dmin2(dmin2(dmin2(fabs(dw / o), fabs(dn / o)), fabs(de / o)), fabs(ds / o));
			dp = dp + (sum - dp) * fmax(sum - (1.0 + ep) * dp, 0.0) / (fabs(sum - (1.0 + ep) * dp) + emach);
			dp = 1.0 / dp;
			CI(ic, jc, kc, LXZNW) = dp * (CI(ic - 1, jc, kc, LXZA) * dw + CI(ic, jc, kc, LXYL) * dn);
			CI(ic, jc, kc, LXZNE) = dp * (CI(ic, jc, kc, LXYR) * dn + CI(ic, jc, kc, LXZA) * de);
			CI(ic, jc, kc, LXZSE) = dp * (CI(ic, jc, kc, LXZB) * de + CI(ic, jc, kc - 1, LXYR) * ds);
			CI(ic, jc, kc, LXZSW) = dp * (CI(ic, jc, kc - 1, LXYL) * ds + CI(ic - 1, jc, kc, LXZB) * dw);
		}
		if (kc >= 3 && kc <= kkcf1 && jc >= 3 && jc <= jjcf1 && ic <= iic1) {  // yz faces
			o = SO(i, j - 1, k - 1, KP);
			dn = SO(i, j - 1, k, KB);
			dw = SO(i, j, k - 1, KPS);
			de = SO(i, j - 1, k - 1, KPS);
			ds = SO(i, j - 1, k - 1, KB);
			dp = dw + dn + de + ds;
			sum = o - SO(i, j - 1, k - 1, KPW) - SO(i + 1, j - 1, k - 1, KPW);
			ep = dmin2(dmin2(dmin2(fabs(dw / o), fabs(dn / o)), fabs(de / o)), fabs(ds / o));
			dp = dp + (sum - dp) * fmax(sum - (1.0 + ep) * dp, 0.0) / (fabs(sum - (1.0 + ep) * dp) + emach);
			dp = 1.0 / dp;
			CI(ic, jc, kc, LYZNW) = dp * (CI(ic, jc, kc, LXZA) * dw + CI(ic, jc, kc, LXYA) * dn);
			CI(ic, jc, kc, LYZNE) = dp * (CI(ic, jc, kc, LXYB) * dn + CI(ic, jc - 1, kc, LXZA) * de);
			CI(ic, jc, kc, LYZSE) = dp * (CI(ic, jc - 1, kc, LXZB) * de + CI(ic, jc, kc - 1, LXYB) * ds);
			CI(ic, jc, kc, LYZSW) = dp * (CI(ic, jc, kc - 1, LXYA) * ds + CI(ic, jc, kc, LXZB) * dw);
		}
	} else if (kc >= 3 && kc <= kkcf1 && jc >= 3 && jc <= jjcf1 && ic >= 3 && ic <= iicf1) {  // interior points
		o = SO(i - 1, j - 1, k - 1, KP);
		const double sw = SO(i - 1, j - 1, k - 1, KPW), sn = SO(i - 1, j, k - 1, KPS), se = SO(i, j - 1, k - 1, KPW);
		const double ss = SO(i - 1, j - 1, k - 1, KPS), sb = SO(i - 1, j - 1, k - 1, KB), st = SO(i - 1, j - 1, k, KB);
		dp = sw + sn + se + ss + sb + st;
		ep = dmin2(dmin2(dmin2(dmin2(dmin2(fabs(sw / o), fabs(sn / o)), fabs(se / o)), fabs(ss / o)), fabs(sb / o)),
		           fabs(st / o));
		dp = (o - dp) * fmax(o - (1.0 + ep) * dp, 0.0) / (fabs(o - (1.0 + ep) * dp) + emach) + dp;
		dp = 1.0 / dp;
		CI(ic, jc, kc, LTNW) = dp * (CI(ic - 1, jc, kc, LYZNW) * sw + CI(ic, jc, kc, LXZNW) * sn + CI(ic, jc, kc, LXYNW) * st);
		CI(ic, jc, kc, LTNE) = dp * (CI(ic, jc, kc, LXZNE) * sn + CI(ic, jc, kc, LYZNW) * se + CI(ic, jc, kc, LXYNE) * st);
		CI(ic, jc, kc, LBNW) =
		    dp * (CI(ic, jc, kc - 1, LXYNW) * sb + CI(ic - 1, jc, kc, LYZSW) * sw + CI(ic, jc, kc, LXZSW) * sn);
		CI(ic, jc, kc, LBNE) = dp * (CI(ic, jc, kc - 1, LXYNE) * sb + CI(ic, jc, kc, LXZSE) * sn + CI(ic, jc, kc, LYZSW) * se);
		CI(ic, jc, kc, LBSW) =
		    dp * (CI(ic, jc, kc - 1, LXYSW) * sb + CI(ic - 1, jc, kc, LYZSE) * sw + CI(ic, jc - 1, kc, LXZSW) * ss);
		CI(ic, jc, kc, LTSW) =
		    dp * (CI(ic, jc, kc, LXYSW) * st + CI(ic - 1, jc, kc, LYZNE) * sw + CI(ic, jc - 1, kc, LXZNW) * ss);
		CI(ic, jc, kc, LTSE) = dp * (CI(ic, jc, kc, LXYSE) * st + CI(ic, jc - 1, kc, LXZNE) * ss + CI(ic, jc, kc, LYZNE) * se);
		CI(ic, jc, kc, LBSE) =
		    dp * (CI(ic, jc, kc - 1, LXYSE) * sb + CI(ic, jc - 1, kc, LXZSE) * ss + CI(ic, jc, kc, LYZSE) * se);
	}
}

int setup_interp_3d(const double *so, double *ci, Dims3 F, Dims3 C, cudaStream_t st, int ns)
{
	CDR_CUDA_TRY(cudaMemsetAsync(ci, 0, sizeof(double) * C.plane() * 26, st));
	const dim3 grd(ceil_div(F.nx / 2 + 1, TX), ceil_div(F.ny / 2 + 1, TY), F.nz / 2 + 1);
	for (int ph = 0; ph < 3; ++ph) {
		if (ns == 4) launch(k3_oi7, grd, dim3(TX, TY), 0, st, so, ci, F, C, ph);
		else launch(k3_oi, grd, dim3(TX, TY), 0, st, so, ci, F, C, ph);
		CDR_LAUNCH_CHECK();
	}
	return CDR_OK;
}

// ------------------------------------------------------------- Galerkin (P^T A P)
// Same loops, order and skips as the CPU restatement of the product that
// BMG3_SymStd_SETUP_ITLI27_ex expands (cdr3 oracle).
// A seven-point operator (NS == 4) has no planes beyond kb: those couplings
// read as 0, as the zero-filled planes of a 14-plane copy would.
template <int NS>
__device__ __forceinline__ double a3(const double *__restrict__ so, Dims3 F, int i, int j, int k, int di, int dj, int dk)
{
	auto S = [&](int ii, int jj, int kk, int p) -> double { return (NS == 4 && p > KB) ? 0.0 : SO(ii, jj, kk, p); };
	if (di == 0 && dj == 0 && dk == 0) return SO(i, j, k, KP);
	double c = 0.0;
	switch ((dk + 1) * 9 + (dj + 1) * 3 + (di + 1)) {
	case 9 + 3 + 0: c = S(i, j, k, KPW); break;
	case 9 + 6 + 0: c = S(i, j + 1, k, KPNW); break;
	case 9 + 6 + 1: c = S(i, j + 1, k, KPS); break;
	case 9 + 6 + 2: c = S(i + 1, j + 1, k, KPSW); break;
	case 9 + 3 + 2: c = S(i + 1, j, k, KPW); break;
	case 9 + 0 + 2: c = S(i + 1, j, k, KPNW); break;
	case 9 + 0 + 1: c = S(i, j, k, KPS); break;
	case 9 + 0 + 0: c = S(i, j, k, KPSW); break;
	case 0 + 3 + 1: c = S(i, j, k, KB); break;
	case 0 + 3 + 0: c = S(i, j, k, KBW); break;
	case 0 + 6 + 0: c = S(i, j + 1, k, KBNW); break;
	case 0 + 6 + 1: c = S(i, j + 1, k, KBN); break;
	case 0 + 6 + 2: c = S(i + 1, j + 1, k, KBNE); break;
	case 0 + 3 + 2: c = S(i + 1, j, k, KBE); break;
	case 0 + 0 + 2: c = S(i + 1, j, k, KBSE); break;
	case 0 + 0 + 1: c = S(i, j, k, KBS); break;
	case 0 + 0 + 0: c = S(i, j, k, KBSW); break;
	case 18 + 3 + 1: c = S(i, j, k + 1, KB); break;
	case 18 + 3 + 0: c = S(i, j, k + 1, KBE); break;
	case 18 + 6 + 0: c = S(i, j + 1, k + 1, KBSE); break;
	case 18 + 6 + 1: c = S(i, j + 1, k + 1, KBS); break;
	case 18 + 6 + 2: c = S(i + 1, j + 1, k + 1, KBSW); break;
	case 18 + 3 + 2: c = S(i + 1, j, k + 1, KBW); break;
	case 18 + 0 + 2: c = S(i + 1, j, k + 1, KBNW); break;
	case 18 + 0 + 1: c = S(i, j, k + 1, KBN); break;
	case 18 + 0 + 0: c = S(i, j, k + 1, KBNE); break;
	}
	return -c;
}

__device__ __forceinline__ double p3(const double *__restrict__ ci, Dims3 C, int ic, int jc, int kc, int dx, int dy, int dz)
{
	if (dz == 0) {
		if (dx == 0 && dy == 0) return 1.0;
		if (dy == 0) return dx < 0 ? CI(ic, jc, kc, LXYR) : CI(ic + 1, jc, kc, LXYL);
		if (dx == 0) return dy < 0 ? CI(ic, jc, kc, LXYA) : CI(ic, jc + 1, kc, LXYB);
		if (dy < 0) return dx < 0 ? CI(ic, jc, kc, LXYNE) : CI(ic + 1, jc, kc, LXYNW);
		return dx < 0 ? CI(ic, jc + 1, kc, LXYSE) : CI(ic + 1, jc + 1, kc, LXYSW);
	}
	const int ko = dz < 0 ? 0 : 1;
	if (dx == 0 && dy == 0) return dz < 0 ? CI(ic, jc, kc, LXZA) : CI(ic, jc, kc + 1, LXZB);
	if (dx == 0) {
		if (dy < 0) return dz < 0 ? CI(ic, jc, kc, LYZNW) : CI(ic, jc, kc + 1, LYZSW);
		return dz < 0 ? CI(ic, jc + 1, kc, LYZNE) : CI(ic, jc + 1, kc + 1, LYZSE);
	}
	if (dy == 0) {
		if (dx < 0) return dz < 0 ? CI(ic, jc, kc, LXZNE) : CI(ic, jc, kc + 1, LXZSE);
		return dz < 0 ? CI(ic + 1, jc, kc, LXZNW) : CI(ic + 1, jc, kc + 1, LXZSW);
	}
	const int io = dx < 0 ? 0 : 1, jo = dy < 0 ? 0 : 1;
	int l;
	if (dz < 0) l = dy < 0 ? (dx < 0 ? LTNE : LTNW) : (dx < 0 ? LTSE : LTSW);
	else l = dy < 0 ? (dx < 0 ? LBNE : LBNW) : (dx < 0 ? LBSE : LBSW);
	return CI(ic + io, jc + jo, kc + ko, l);
}

template <int NS>
__device__ double rap3(const double *__restrict__ so, const double *__restrict__ ci, Dims3 F, Dims3 C, int i1, int j1,
                       int k1, int i2, int j2, int k2)
{
	const int F1x = 2 * i1 - 2, F1y = 2 * j1 - 2, F1z = 2 * k1 - 2;
	double tot = 0.0;
#pragma unroll 1
	for (int dz1 = -1; dz1 <= 1; ++dz1)
#pragma unroll 1
		for (int dy1 = -1; dy1 <= 1; ++dy1)
			for (int dx1 = -1; dx1 <= 1; ++dx1) {
				const int fx = F1x + dx1, fy = F1y + dy1, fz = F1z + dz1;
				if (fx < 2 || fx > F.nx + 1 || fy < 2 || fy > F.ny + 1 || fz < 2 || fz > F.nz + 1) continue;
				double inner = 0.0;
				for (int ddz = -1; ddz <= 1; ++ddz)
					for (int ddy = -1; ddy <= 1; ++ddy)
						for (int ddx = -1; ddx <= 1; ++ddx) {
							const int ex = dx1 + ddx - 2 * (i2 - i1), ey = dy1 + ddy - 2 * (j2 - j1), ez = dz1 + ddz - 2 * (k2 - k1);
							if (ex < -1 || ex > 1 || ey < -1 || ey > 1 || ez < -1 || ez > 1) continue;
							inner += a3<NS>(so, F, fx, fy, fz, ddx, ddy, ddz) * p3(ci, C, i2, j2, k2, ex, ey, ez);
						}
				tot += p3(ci, C, i1, j1, k1, dx1, dy1, dz1) * inner;
			}
	return tot;
}

// One thread per (coarse point, stencil plane): the 14 entries are independent.
template <int NS>
__global__ void __launch_bounds__(TX *TY) k3_galerkin(const double *__restrict__ so, const double *__restrict__ ci,
                                                      double *__restrict__ soc, Dims3 F, Dims3 C)
{
	await_previous();
	const int ic = blockIdx.x * TX + threadIdx.x + 2, jc = blockIdx.y * TY + threadIdx.y + 2;
	const int kc = blockIdx.z / 14 + 2, pl = blockIdx.z % 14 + 1;
	if (ic > C.nx + 1 || jc > C.ny + 1) return;
	// (fine-side coarse point, partner coarse point) offsets of each plane, and
	// the sign: KP = R(c,c); the others -R(c1, c2) (BMG3_SymStd_SETUP_ITLI27_ex)
	int a1 = 0, b1 = 0, c1 = 0, a2 = 0, b2 = 0, c2 = 0;
	switch (pl) {
	case KP: break;
	case KPW: a2 = -1; break;
	case KPS: b2 = -1; break;
	case KB: c2 = -1; break;
	case KPSW: a2 = -1; b2 = -1; break;
	case KPNW: b1 = -1; a2 = -1; break;
	case KBW: a2 = -1; c2 = -1; break;
	case KBNW: b1 = -1; a2 = -1; c2 = -1; break;
	case KBN: b1 = -1; c2 = -1; break;
	case KBNE: a1 = -1; b1 = -1; c2 = -1; break;
	case KBE: a1 = -1; c2 = -1; break;
	case KBSE: a1 = -1; b2 = -1; c2 = -1; break;
	case KBS: b2 = -1; c2 = -1; break;
	case KBSW: a2 = -1; b2 = -1; c2 = -1; break;
	}
	const double v = rap3<NS>(so, ci, F, C, ic + a1, jc + b1, kc + c1, ic + a2, jc + b2, kc + c2);
	soc[(size_t)(pl - 1) * C.plane() + C.at1(ic, jc, kc)] = pl == KP ? v : -v;
}

int galerkin_3d(const double *so, const double *ci, double *soc, Dims3 F, Dims3 C, cudaStream_t st, int ns)
{
	CDR_CUDA_TRY(cudaMemsetAsync(soc, 0, sizeof(double) * C.plane() * 14, st));
	const dim3 grd(ceil_div(C.nx, TX), ceil_div(C.ny, TY), C.nz * 14);
	if (ns == 4) launch(k3_galerkin<4>, grd, dim3(TX, TY), 0, st, so, ci, soc, F, C);
	else launch(k3_galerkin<14>, grd, dim3(TX, TY), 0, st, so, ci, soc, F, C);
	CDR_LAUNCH_CHECK();
	return CDR_OK;
}

// ---------------------------------------------------------- coarsest Cholesky
// ABD fill of BMG3_SymStd_SETUP_cg_LU (src/3d/ftn/BMG3_SymStd_SETUP_cg_LU.f90:106-130),
// KD = IBW = (II-2)*(JJ-1)+1, then DPBTF2('U') as in 2D.
// NS == 4: a seven-point operator (a one-level hierarchy); the couplings it
// lacks enter the band as -0.0, as from zero-filled planes.
template <int NS>
__global__ void k3_cg_factor(const double *__restrict__ so, Dims3 F, double *__restrict__ abd, int nabd1, int *info)
{
	await_previous();
	auto S = [&](int ii, int jj, int kk, int p) -> double { return (NS == 4 && p > KB) ? 0.0 : SO(ii, jj, kk, p); };
	if (threadIdx.x != 0 || blockIdx.x != 0) return;
	const int II = F.nx + 2, JJ = F.ny + 2, KK = F.nz + 2;
	const int i1 = II - 1, j1 = JJ - 1, k1 = KK - 1, i2 = i1 - 1;
	const int ibw = i2 * j1 + 1;
	const int n = F.nx * F.ny * F.nz;
	for (size_t e = 0; e < (size_t)nabd1 * n; ++e) abd[e] = 0.0;
#define ABD(r, c) abd[(size_t)((c)-1) * nabd1 + ((r)-1)]
	int kl = 0;
	for (int k = 2; k <= k1; ++k)
		for (int j = 2; j <= j1; ++j)
			for (int i = 2; i <= i1; ++i) {
				kl++;
				ABD(ibw + 1, kl) = S(i, j, k, KP);
				ABD(ibw, kl) = -S(i, j, k, KPW);
				ABD(ibw - i1 + 3, kl) = -S(i + 1, j, k, KPNW);
				ABD(ibw - i1 + 2, kl) = -S(i, j, k, KPS);
				ABD(ibw - i1 + 1, kl) = -S(i, j, k, KPSW);
				ABD(ibw - (j1 - 2) * i2 + 2, kl) = -S(i + 1, j + 1, k, KBNE);
				ABD(ibw - (j1 - 2) * i2 + 1, kl) = -S(i, j + 1, k, KBN);
				ABD(ibw - (j1 - 2) * i2, kl) = -S(i, j + 1, k, KBNW);
				ABD(ibw - (j1 - 1) * i2 + 2, kl) = -S(i + 1, j, k, KBE);
				ABD(ibw - (j1 - 1) * i2 + 1, kl) = -S(i, j, k, KB);
				ABD(ibw - (j1 - 1) * i2, kl) = -S(i, j, k, KBW);
				ABD(3, kl) = -S(i + 1, j, k, KBSE);
				ABD(2, kl) = -S(i, j, k, KBS);
				ABD(1, kl) = -S(i, j, k, KBSW);
			}
#undef ABD
	// DPBTF2('U', n, kd = ibw)
	const int kd = ibw, ldab = nabd1, kld = ldab - 1;
	int stt = 0;
	for (int jj = 0; jj < n; ++jj) {
		double ajj = abd[(size_t)jj * ldab + kd];
		if (ajj <= 0.0) { stt = jj + 1; break; }
		ajj = sqrt(ajj);
		abd[(size_t)jj * ldab + kd] = ajj;
		const int kn = kd < n - jj - 1 ? kd : n - jj - 1;
		if (kn > 0) {
			const double rcp = 1.0 / ajj;
			double *xv = abd + (size_t)(jj + 1) * ldab + (kd - 1);
			for (int p = 0; p < kn; ++p) xv[(size_t)p * kld] = rcp * xv[(size_t)p * kld];
			double *a = abd + (size_t)(jj + 1) * ldab + kd;
			for (int qq = 0; qq < kn; ++qq) {
				const double xq = xv[(size_t)qq * kld];
				if (xq != 0.0) {
					const double temp = -1.0 * xq;
					for (int p = 0; p <= qq; ++p)
						a[(size_t)p + (size_t)qq * kld] = a[(size_t)p + (size_t)qq * kld] + xv[(size_t)p * kld] * temp;
				}
			}
		}
	}
	if (info) *info = stt;
}

// BMG3_SymStd_SOLVE_cg (src/3d/ftn/BMG3_SymStd_SOLVE_cg.f90:105-131) with DPBTRS('U').
// Bound by the chain of 2n quotients, one per unknown and sweep.  The forward
// sweep runs by columns like the backward one: once unknown i is final, thread m
// subtracts its term from unknown i + 1 + m, so every unknown still receives its
// terms in DTBSV's ascending order (the same bits) while a step costs one
// quotient and one update.  Every thread forms the quotient itself.  WARP: the
// band has at most 32 entries, one warp runs the steps.  STAGED: the factor fits
// in shared memory beside the right-hand side.
template <typename T, bool WARP, bool STAGED>
__global__ void __launch_bounds__(WARP ? 128 : 1024) k3_cg_solve(const double *__restrict__ ab, int ldab, T *__restrict__ q,
                                                    const T *__restrict__ qf, Dims3 F)
{
	await_previous();
	extern __shared__ double xs[];
	const int kd = ldab - 1, n = F.nx * F.ny * F.nz, tid = threadIdx.x;
	auto at = [&](int m) -> size_t {  // unknown m, x fastest
		const int r = m / F.nx;
		return F.at1(m - r * F.nx + 2, r % F.ny + 2, r / F.ny + 2);
	};
	for (int m = tid; m < n; m += blockDim.x) xs[m] = (double)qf[at(m)];
	const double *A = ab;
	if (STAGED) {
		double *sa = xs + n;
		for (int m = tid; m < n * ldab; m += blockDim.x) sa[m] = ab[m];
		A = sa;
	}
	__syncthreads();
	if (!WARP || tid < 32) {
		const int nt = WARP ? 32 : blockDim.x;
		auto sync = [&]() {
			if (WARP) __syncwarp();
			else __syncthreads();
		};
		auto coef = [&](int r, int c) { return A[(size_t)c * ldab + kd + r - c]; };  // U(r, c), r <= c
		// the thread's first coefficient and the pivot of the next step load a step ahead
		double prev = 0.0, d = coef(0, 0), a = tid < kd && 1 + tid < n ? coef(0, 1 + tid) : 0.0;
		for (int i = 0; i < n; ++i) {
			const double dn = i + 1 < n ? coef(i + 1, i + 1) : 1.0;
			const double an = tid < kd && i + 2 + tid < n ? coef(i + 1, i + 2 + tid) : 0.0;
			const double xi = xs[i] / d;
			if (tid == 0 && i > 0) xs[i - 1] = prev;
			if (tid < kd && i + 1 + tid < n) xs[i + 1 + tid] = xs[i + 1 + tid] - a * xi;
			for (int m = tid + nt; m < kd && i + 1 + m < n; m += nt)
				xs[i + 1 + m] = xs[i + 1 + m] - coef(i, i + 1 + m) * xi;
			prev = xi;
			d = dn;
			a = an;
			sync();
		}
		if (tid == 0) xs[n - 1] = prev;
		sync();
		d = coef(n - 1, n - 1);
		a = tid < kd && n - 2 - tid >= 0 ? coef(n - 2 - tid, n - 1) : 0.0;
		for (int j = n - 1; j >= 0; --j) {
			const double dn = j > 0 ? coef(j - 1, j - 1) : 1.0;
			const double an = tid < kd && j - 2 - tid >= 0 ? coef(j - 2 - tid, j - 1) : 0.0;
			const double xj = xs[j];
			if (tid == 0 && j + 1 < n) xs[j + 1] = prev;
			prev = xj;
			if (xj != 0.0) {
				const double t = xj / d;
				if (tid < kd && j - 1 - tid >= 0) xs[j - 1 - tid] = xs[j - 1 - tid] - t * a;
				for (int m = tid + nt; m < kd && j - 1 - m >= 0; m += nt)
					xs[j - 1 - m] = xs[j - 1 - m] - t * coef(j - 1 - m, j);
				prev = t;
			}
			d = dn;
			a = an;
			sync();
		}
		if (tid == 0) xs[0] = prev;
	}
	__syncthreads();
	for (int m = tid; m < n; m += blockDim.x) q[at(m)] = (T)xs[m];
}

int setup_cg_3d(const double *so, Dims3 F, double *abd, int *info, cudaStream_t st, int ns)
{
	if (ns == 4) launch(k3_cg_factor<4>, 1, 32, 0, st, so, F, abd, F.nx * (F.ny + 1) + 2, info);
	else launch(k3_cg_factor<14>, 1, 32, 0, st, so, F, abd, F.nx * (F.ny + 1) + 2, info);
	CDR_LAUNCH_CHECK();
	return CDR_OK;
}

template <typename T>
int solve_cg_3d(const double *abd, T *x, const T *b, Dims3 F, cudaStream_t st)
{
	const int n = F.nx * F.ny * F.nz, ldab = cg3_ldab(F), kd = ldab - 1;
	const size_t sm = sizeof(double) * (size_t)n, staged = sm * (ldab + 1);
	if (sm > 48 * 1024) {
		set_error(CDR_ERR_DIM, "coarsest grid %dx%dx%d too large for the direct solve", F.nx, F.ny, F.nz);
		return CDR_ERR_DIM;
	}
	const int blk = kd <= 128 ? 128 : kd < 1024 ? (kd + 31) / 32 * 32 : 1024;
	if (staged <= 48 * 1024) {
		if (kd <= 32) launch(k3_cg_solve<T, true, true>, 1, blk, staged, st, abd, ldab, x, b, F);
		else launch(k3_cg_solve<T, false, true>, 1, blk, staged, st, abd, ldab, x, b, F);
	} else {
		if (kd <= 32) launch(k3_cg_solve<T, true, false>, 1, blk, sm, st, abd, ldab, x, b, F);
		else launch(k3_cg_solve<T, false, false>, 1, blk, sm, st, abd, ldab, x, b, F);
	}
	CDR_LAUNCH_CHECK();
	return CDR_OK;
}
template int solve_cg_3d<double>(const double *, double *, const double *, Dims3, cudaStream_t);
template int solve_cg_3d<float>(const double *, float *, const float *, Dims3, cudaStream_t);

// Outer refinement step of the mixed-precision 3D solve (as the 2D one):
//   x_out = x_in + e32, r64 = b - A x_out, r32 = (float) r64, ||r64||^2 per
//   block; x_in and x_out are different buffers.  apply = 0 skips e (x_out is
//   then not needed and may be left unwritten).
// Seven-point levels: each thread forms x_in + e32 over its neighbours on the fly.
struct LoadIR3 {
	const double *__restrict__ x;
	const float *__restrict__ e;
	Dims3 F;
	int apply;
	__device__ __forceinline__ double operator()(int i, int j, int k) const
	{
		const size_t o = F.at1(i, j, k);
		return apply ? x[o] + (double)e[o] : x[o];
	}
};

__global__ void __launch_bounds__(TX *TY) k3_ir_residual7(const double *__restrict__ so, const double *__restrict__ x,
                                                          const float *__restrict__ e, const double *__restrict__ b,
                                                          double *__restrict__ xo, float *__restrict__ r32, Dims3 F,
                                                          double *__restrict__ partial, int apply)
{
	await_previous();
	__shared__ double sh[TX * TY / 32];
	const int tx = (F.nx + TX - 1) / TX, ty = (F.ny + TY - 1) / TY;
	const long ntiles = (long)tx * ty * F.nz;
	const LoadIR3 xq{x, e, F, apply};
	double acc = 0.0;
	for (long t = blockIdx.x; t < ntiles; t += gridDim.x) {
		const int kk = (int)(t / ((long)tx * ty));
		const int rem = (int)(t - (long)kk * tx * ty);
		const int i = (rem % tx) * TX + threadIdx.x + 2, j = (rem / tx) * TY + threadIdx.y + 2, k = kk + 2;
		if (i <= F.nx + 1 && j <= F.ny + 1) {
			const double xc = xq(i, j, k);
			const double r = nb7<double>(so, xq, b[F.at1(i, j, k)], F, i, j, k) - SO(i, j, k, KP) * xc;
			acc += r * r;
			r32[F.at1(i, j, k)] = (float)r;
			xo[F.at1(i, j, k)] = xc;
		}
	}
	const double s = block_sum<TX * TY / 32>(acc, sh);
	if (threadIdx.x == 0 && threadIdx.y == 0) partial[blockIdx.x] = s;
}

// x_out = x_in + e32 on the interior
__global__ void __launch_bounds__(256) k3_ir_add(const double *__restrict__ x, const float *__restrict__ e,
                                                 double *__restrict__ xo, Dims3 F)
{
	await_previous();
	const int i = blockIdx.x * 64 + threadIdx.x + 1, j = blockIdx.y * 4 + threadIdx.y + 1, k = blockIdx.z + 1;
	if (i > F.nx || j > F.ny) return;
	const size_t o = ((size_t)k * (F.ny + 2) + j) * F.pitch + i;
	xo[o] = x[o] + (double)e[o];
}

// 27-point levels form x_out first and then its residual: forming x_in + e for
// each of the 27 neighbours cost 81 loads and 27 conversions a point (255^3:
// 1058 us at 32 % of the DRAM rate, now 65 us and about 530); the extra read of
// x_out is 8 of about 156 bytes.
int ir_residual_3d(const double *so, const double *x, const float *e, const double *b, double *xo, float *r32,
                   Dims3 d, double *norm_out, double *partial, int apply, cudaStream_t st, int ns)
{
	const long ntiles = (long)ceil_div(d.nx, TX) * ceil_div(d.ny, TY) * d.nz;
	const int nb = ntiles < 2048 ? (int)ntiles : 2048;
	if (ns == 4) {
		launch(k3_ir_residual7, nb, dim3(TX, TY), 0, st, so, x, e, b, xo, r32, d, partial, apply);
	} else {
		if (apply) {
			launch(k3_ir_add, dim3(ceil_div(d.nx, 64), ceil_div(d.ny, 4), d.nz), dim3(64, 4), 0, st, x, e, xo, d);
			CDR_LAUNCH_CHECK();
		}
		launch(k3_residual<double, true, 14, float>, nb, dim3(TX, TY), 0, st, so, apply ? xo : x, b, r32, d, partial);
	}
	CDR_LAUNCH_CHECK();
	launch(k3_norm_finish, 1, 1024, 0, st, partial, nb, norm_out);
	CDR_LAUNCH_CHECK();
	return CDR_OK;
}

#undef SO
#undef Q
#undef QF
#undef CI
#undef QC

}  // namespace cdrgpu
