// Hessians of particle-conserving fits in number sectors (k_ws_grad, k_ws_hess).  Included by
// mgcu_engine.cu inside its anonymous namespace, after mgcu_fit.cuh, whose factored blocks, moves
// and finishing kernels it shares.
//
// When every gate of the target and of the fitted circuit conserves the particle number (corner
// blocks diagonal, as in the fits of particle-conserving models: their gradients keep them so),
// every state, derivative and tangent state of a column of n ones lives on the C(L, n) indices
// of n ones (of n -+ 2 for the tangents of the two off-diagonal corner entries): a third of the
// parity sector at L = 12.  A block keeps 2^ln columns of one sector in shared memory, rows
// with the columns adjacent.  The rows of a wire pair come from one table per pair: for every
// value of the other wires, ordered by its number of ones m, the rows of its completions |00>
// (in sector m), |01>, |10> (m + 1) and |11> (m + 2).  So sector n's center pairs are the
// entries with m = n - 1, its |00> rows those with m = n and its |11> rows those with m = n - 2,
// and an entry also links the |00> and |11> rows of sectors two apart.
//
// Gates are applied in levels (runs of gates on disjoint wires, a brickwall layer); states and
// derivatives are cached once per level, after its last gate, where all of the level's
// contractions are made without a barrier.
//
// Measured against the parity sectors (k_fit with derivative cache, k_fit_hess; the whole items of
// an evaluation): L=12, 5 layers, complex128 6.8 + 128 -> 1.8 + 25.6 ms; L=12, 9 layers,
// translation-invariant, float-float 4.1 + 101 -> 1.6 + 33.4 ms; L=10, 5 layers, float-float
// 0.22 + 1.81 -> 0.12 + 0.80 ms.  Bound: the FP64 pipe in complex128, issue and the L2 reads of
// the cached derivatives in float-float.

struct WsLevel { int gbeg, gend; };
template <class T> struct WsGate { T p, q; int sw, pair, blk, pad; };
struct WsSec { int first, n, rlo, rhi; };    // columns: rows [rlo, rhi) of sector n, in groups from `first`

template <class P>
struct WsArgs
{
	typedef typename P::T T;
	int L, nlev, ngates, ln, dmax, nsec, ngroups, nblocks;
	int rstart[17], pstart[17];     // first row position per n; first entry of a pair table per m
	const WsLevel* levels;
	const WsGate<T>* gates;
	const ushort4* pairs;           // [pair][2^(L-2)]
	const T* tables;                // [level, then final][2^L], by row position
	const unsigned* rows;           // full index by row position
	const WsSec* sec;
	const T* dense;
	long dense_b0, S;
	T* ycache;                      // [group][level][dmax][2^ln]
	T* ecache;
	double* part;                   // [group blocks][nblocks][16]
	// Hessian items
	const int *place, *place_level, *block;
	const double* place_w;
	int nplace, mdim, hgroup;
	long placewise;                 // as in FitHessArgs
	double* part_h;
};

constexpr int WS_NT = 256;
constexpr int WS_MAXG = 128;   // fitted gates kept in shared memory

// the center blocks' M of one gate on the pairs of sector n in the tile
template <class P, bool QC, bool TR>
__device__ __forceinline__ void ws_rotate(const WsArgs<P>& a, const WsGate<typename P::T>& g, int n, unsigned tb)
{
	typedef typename P::T T;
	if (n < 1 || n >= a.L) return;
	const ushort4* e = a.pairs + ((size_t)g.pair << (a.L - 2)) + a.pstart[n - 1];
	const unsigned cnt = (unsigned)(a.pstart[n] - a.pstart[n - 1]) << a.ln, cm = (1u << a.ln) - 1u;
	const T p = g.p, q = g.q;
	for (unsigned t = threadIdx.x; t < cnt; t += WS_NT)
	{
		const ushort4 r = e[t >> a.ln];
		const unsigned ay = tb + ((((unsigned)r.y) << a.ln) | (t & cm)) * (unsigned)sizeof(T), az = tb + ((((unsigned)r.z) << a.ln) | (t & cm)) * (unsigned)sizeof(T);
		T y = lds<T>(ay), z = lds<T>(az);
		fit_pair<P, QC, TR>(y, z, p, q, g.sw);
		sts<T>(ay, y); sts<T>(az, z);
	}
}

template <class P>
__device__ __forceinline__ void ws_flush(const WsArgs<P>& a, int l, int n, unsigned tb)
{
	typedef typename P::T T;
	const unsigned cnt = (unsigned)(a.rstart[n + 1] - a.rstart[n]) << a.ln;
	const T* tab = a.tables + ((size_t)l << a.L) + a.rstart[n];
	for (unsigned t = threadIdx.x; t < cnt; t += WS_NT)
	{
		const unsigned ad = tb + t * (unsigned)sizeof(T);
		sts<T>(ad, P::mul(tab[t >> a.ln], lds<T>(ad)));
	}
}

// R sums of a gate: derivative (sector n) and state (sector n, or n - 2 / n + 2 with shift
// -1 / 1); DT: the derivative is in the tile and the state in memory, else the other way round
template <class P, bool DT>
__device__ __forceinline__ void ws_contract(const WsArgs<P>& a, int pair, int n, int shift, unsigned tb, const typename P::T* __restrict__ mem,
	typename P::Acc (&acc)[8])
{
	typedef typename P::T T;
	const ushort4* e = a.pairs + ((size_t)pair << (a.L - 2));
	const unsigned cm = (1u << a.ln) - 1u, c = threadIdx.x & cm;
	auto M = [&](unsigned row) { return mem[(row << a.ln) | c]; };
	auto S = [&](unsigned row) { return lds<T>(tb + ((row << a.ln) | c) * (unsigned)sizeof(T)); };
	const unsigned st = WS_NT >> a.ln, t0 = threadIdx.x >> a.ln;
	// two entries at a time, the reads from memory first: their latency is the bound
	auto rows = [&](int m, bool w, int k) {
		unsigned t = a.pstart[m] + t0;
		const unsigned end = a.pstart[m + 1];
		for (; t + st < end; t += 2 * st)
		{
			const ushort4 e0 = e[t], e1 = e[t + st];
			const unsigned r0 = w ? e0.w : e0.x, r1 = w ? e1.w : e1.x;
			const T m0 = M(r0), m1 = M(r1), s0 = S(r0), s1 = S(r1);
			P::acc_mul_add_short(acc[k], DT ? s0 : m0, DT ? m0 : s0);
			P::acc_mul_add_short(acc[k], DT ? s1 : m1, DT ? m1 : s1);
		}
		if (t < end)
		{
			const unsigned r0 = w ? e[t].w : e[t].x;
			const T m0 = M(r0), s0 = S(r0);
			P::acc_mul_add_short(acc[k], DT ? s0 : m0, DT ? m0 : s0);
		}
	};
	auto pair4 = [&](const T& my, const T& mz, const T& sy, const T& sz) {
		const T &dy = DT ? sy : my, &dz = DT ? sz : mz, &y = DT ? my : sy, &z = DT ? mz : sz;
		P::acc_mul_add_short(acc[0], dy, y); P::acc_mul_add_short(acc[1], dy, z);
		P::acc_mul_add_short(acc[2], dz, y); P::acc_mul_add_short(acc[3], dz, z);
	};
	if (shift == 0)
	{
		if (n >= 1 && n < a.L)
		{
			unsigned t = a.pstart[n - 1] + t0;
			const unsigned end = a.pstart[n];
			for (; t + st < end; t += 2 * st)
			{
				const ushort4 e0 = e[t], e1 = e[t + st];
				const T y0 = M(e0.y), z0 = M(e0.z), y1 = M(e1.y), z1 = M(e1.z);
				pair4(y0, z0, S(e0.y), S(e0.z));
				pair4(y1, z1, S(e1.y), S(e1.z));
			}
			if (t < end)
			{
				const ushort4 e0 = e[t];
				const T y0 = M(e0.y), z0 = M(e0.z);
				pair4(y0, z0, S(e0.y), S(e0.z));
			}
		}
		if (n <= a.L - 2) rows(n, false, 4);
		if (n >= 2) rows(n - 2, true, 7);
	}
	else if (shift < 0)
		for (unsigned t = a.pstart[n - 2] + t0; t < (unsigned)a.pstart[n - 1]; t += st)
		{
			const ushort4 r = e[t];
			const T m0 = M(DT ? r.x : r.w), s0 = S(DT ? r.w : r.x);
			P::acc_mul_add_short(acc[6], DT ? s0 : m0, DT ? m0 : s0);
		}
	else
		for (unsigned t = a.pstart[n] + t0; t < (unsigned)a.pstart[n + 1]; t += st)
		{
			const ushort4 r = e[t];
			const T m0 = M(DT ? r.w : r.x), s0 = S(DT ? r.x : r.w);
			P::acc_mul_add_short(acc[5], DT ? s0 : m0, DT ? m0 : s0);
		}
}

// the tile gains the move of entry x (see fit_move) of the cached state of sector n
template <class P>
__device__ __forceinline__ void ws_move(const WsArgs<P>& a, int pair, int n, int x, unsigned tb, const typename P::T* __restrict__ ym)
{
	typedef typename P::T T;
	const int m = x < 4 ? n - 1 : (x == 5 || x == 7) ? n - 2 : n;   // other wires' ones
	if (m < 0 || m > a.L - 2) return;
	const ushort4* e = a.pairs + ((size_t)pair << (a.L - 2)) + a.pstart[m];
	const unsigned cnt = (unsigned)(a.pstart[m + 1] - a.pstart[m]) << a.ln, cm = (1u << a.ln) - 1u;
	for (unsigned t = threadIdx.x; t < cnt; t += WS_NT)
	{
		const ushort4 r = e[t >> a.ln];
		const unsigned to = x < 4 ? ((x & 2) ? r.z : r.y) : ((x & 2) ? r.w : r.x);
		const unsigned from = x < 4 ? ((x & 1) ? r.z : r.y) : ((x & 1) ? r.w : r.x);
		const unsigned ad = tb + ((to << a.ln) | (t & cm)) * (unsigned)sizeof(T);
		sts<T>(ad, P::add(lds<T>(ad), ym[(from << a.ln) | (t & cm)]));
	}
}

// sector and first row of a column group
template <class P>
__device__ __forceinline__ WsSec ws_sector(const WsArgs<P>& a, long grp)
{
	int s = 0;
	while (s + 1 < a.nsec && a.sec[s + 1].first <= grp) s++;
	return a.sec[s];
}

template <class P, bool QC>
__global__ void __launch_bounds__(WS_NT, 2) k_ws_grad(WsArgs<P> a)
{
	typedef typename P::T T;
	extern __shared__ __align__(16) char smem_raw[];
	__shared__ double red[2 * (WS_NT / 32) * 16];
	const unsigned tb = smem_u32(smem_raw);
	typename P::Acc acc[8];
#pragma unroll
	for (int e = 0; e < 8; e++) acc[e] = P::acc_zero();
	int nred = 0;
	for (long grp = blockIdx.x; grp < a.ngroups; grp += gridDim.x)
	{
		const WsSec I = ws_sector(a, grp);
		const int n = I.n, r0 = I.rlo + (int)((grp - I.first) << a.ln), ncol = min(1 << a.ln, I.rhi - r0);
		const unsigned d = a.rstart[n + 1] - a.rstart[n], cnt = d << a.ln, cm = (1u << a.ln) - 1u;
		T* yc = a.ycache + (size_t)grp * a.nlev * ((size_t)a.dmax << a.ln);
		T* ec = a.ecache + (size_t)grp * a.nlev * ((size_t)a.dmax << a.ln);
		const size_t ls = (size_t)a.dmax << a.ln;
		__syncthreads();
		for (unsigned t = threadIdx.x; t < cnt; t += WS_NT) sts<T>(tb + t * (unsigned)sizeof(T), P::zero());
		__syncthreads();
		if ((int)threadIdx.x < ncol) sts<T>(tb + ((((unsigned)(r0 + threadIdx.x)) << a.ln) + threadIdx.x) * (unsigned)sizeof(T), P::make(1.0, 0.0));
		__syncthreads();
		for (int l = 0; l < a.nlev; l++)
		{
			const WsLevel V = a.levels[l];
			ws_flush<P>(a, l, n, tb);
			__syncthreads();
			for (int g = V.gbeg; g < V.gend; g++) { ws_rotate<P, QC, false>(a, a.gates[g], n, tb); __syncthreads(); }
			for (unsigned t = threadIdx.x; t < cnt; t += WS_NT) yc[l * ls + t] = lds<T>(tb + t * (unsigned)sizeof(T));
			__syncthreads();
		}
		const unsigned* rows = a.rows + a.rstart[n];
		const T* fin = a.tables + ((size_t)a.nlev << a.L) + a.rstart[n];
		for (unsigned t = threadIdx.x; t < cnt; t += WS_NT)
		{
			const unsigned r = t >> a.ln, c = t & cm;
			sts<T>(tb + t * (unsigned)sizeof(T), (int)c < ncol
				? P::mul(fin[r], a.dense[(size_t)((long)rows[r0 + c] - a.dense_b0) * a.S + (rows[r] >> 1)]) : P::zero());
		}
		__syncthreads();
		for (int l = a.nlev - 1; l >= 0; l--)
		{
			const WsLevel V = a.levels[l];
			for (unsigned t = threadIdx.x; t < cnt; t += WS_NT) ec[l * ls + t] = lds<T>(tb + t * (unsigned)sizeof(T));
			for (int g = V.gend - 1; g >= V.gbeg; g--)
			{
				ws_contract<P, true>(a, a.gates[g].pair, n, 0, tb, yc + l * ls, acc);
				if (g > V.gbeg && a.gates[g - 1].blk == a.gates[g].blk)
				{
#pragma unroll
					for (int e = 0; e < 8; e++) P::acc_norm(acc[e]);
					continue;
				}
				block_reduce8<P>(acc, red, a.part + ((size_t)blockIdx.x * a.nblocks + a.gates[g].blk) * 16, 1.0, nred);
#pragma unroll
				for (int e = 0; e < 8; e++) acc[e] = P::acc_zero();
			}
			if (l == 0) break;
			__syncthreads();
			for (int g = V.gend - 1; g >= V.gbeg; g--) { ws_rotate<P, QC, true>(a, a.gates[g], n, tb); __syncthreads(); }
			ws_flush<P>(a, l, n, tb);
			__syncthreads();
		}
	}
}

template <class P, bool QC>
__global__ void __launch_bounds__(WS_NT, 2) k_ws_hess(WsArgs<P> a, long nitems)
{
	typedef typename P::T T;
	extern __shared__ __align__(16) char smem_raw[];
	__shared__ double red[2 * (WS_NT / 32) * 16];
	__shared__ WsGate<T> gs[WS_MAXG];
	const unsigned tb = smem_u32(smem_raw);
	double* parth = a.part_h + (size_t)blockIdx.x * a.mdim * a.mdim * 2;
	for (int i = threadIdx.x; i < a.ngates; i += WS_NT) gs[i] = a.gates[i];
	typename P::Acc acc[8];
#pragma unroll
	for (int e = 0; e < 8; e++) acc[e] = P::acc_zero();
	int nred = 0;
	for (long it = blockIdx.x; it < nitems; it += gridDim.x)
	{
		const int x = (int)(it & 7);
		const long rest = it >> 3;
		const int p = (int)(a.placewise ? rest / a.placewise : rest % a.nplace);
		const long grp = a.placewise ? rest % a.placewise : rest / a.nplace;
		const WsSec I = ws_sector(a, grp);
		const int n = I.n, shift = x == 5 ? -1 : x == 6 ? 1 : 0, m = n + 2 * shift;   // the tangent's sector
		if (m < 0 || m > a.L) continue;
		const unsigned cnt = (unsigned)(a.rstart[m + 1] - a.rstart[m]) << a.ln;
		const size_t ls = (size_t)a.dmax << a.ln;
		const T* yc = a.ycache + (size_t)grp * a.nlev * ls;
		const T* ec = a.ecache + (size_t)grp * a.nlev * ls;
		const int k = a.place[p], l0 = a.place_level[p], kb = a.block[k], own = a.hgroup ? kb : -1;
		const double* wrow = a.place_w + (size_t)p * a.ngates;
		double* hrow = parth + (size_t)(kb * 8 + x) * a.mdim * 2;
		int cblk = -1;
		double cw = 0;
		auto flush = [&]() {
			if (cblk < 0) return;
			block_reduce8<P>(acc, red, hrow + (size_t)cblk * 16, cw, nred);
#pragma unroll
			for (int e = 0; e < 8; e++) acc[e] = P::acc_zero();
			cblk = -1;
		};
		__syncthreads();
		for (unsigned t = threadIdx.x; t < cnt; t += WS_NT) sts<T>(tb + t * (unsigned)sizeof(T), P::zero());
		__syncthreads();
		for (int l = l0; l < a.nlev; l++)
		{
			const WsLevel V = a.levels[l];
			if (l > l0)
			{
				ws_flush<P>(a, l, m, tb);
				__syncthreads();
				for (int g = V.gbeg; g < V.gend; g++) { ws_rotate<P, QC, false>(a, gs[g], m, tb); __syncthreads(); }
			}
			for (int g = l == l0 ? k : V.gbeg; g < V.gend; g++)
			{
				const int blk = gs[g].blk;
				if (g != k)
				{
					const double wg = wrow[g];
					if (cblk != blk || cw != wg) flush();
					else
					{
#pragma unroll
						for (int e = 0; e < 8; e++) P::acc_norm(acc[e]);
					}
					cblk = blk; cw = wg;
					ws_contract<P, false>(a, gs[g].pair, n, shift, tb, ec + l * ls, acc);
				}
				if (g == k || blk == own)
				{
					__syncthreads();
					ws_move<P>(a, gs[g].pair, n, x, tb, yc + l * ls);
					__syncthreads();
				}
			}
			__syncthreads();
		}
		flush();
	}
}

// the level tables by row position (level nlev: the factors after the last gate)
template <class P>
__global__ void k_ws_tables(const FitDiag* __restrict__ diag, const int* __restrict__ beg, int nlev, int L, const unsigned* __restrict__ rows,
	typename P::T* __restrict__ tables)
{
	for (long q = blockIdx.x * (long)blockDim.x + threadIdx.x; q < ((long)(nlev + 1) << L); q += (long)gridDim.x * blockDim.x)
	{
		const int l = (int)(q >> L);
		tables[q] = fit_table_entry<P>(diag, beg[l], beg[l + 1], rows[q & ((1L << L) - 1)]);
	}
}
