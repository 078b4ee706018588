// Sector sweep (k_sector): -conj(U e_b) of targets whose gates conserve particle numbers, with
// the whole column kept in shared memory.  Included by mgcu_engine.cu inside its anonymous
// namespace (uses its precision policies, block kinds and shared-memory accessors).
//
// When every corner block of a target is diagonal, the wires split into components joined by
// the gates whose center block moves amplitudes, and U conserves the number of ones on each
// component (a chain of spinless fermions: one component; spinful Hubbard: one per spin).
// U e_b then lives on the basis indices with b's numbers, its sector: d amplitudes, at most
// C(L/2, L/4)^2 (4900 at L=16) for two components or C(L, L/2) (12870) for one, against
// 2^(L-1) in the parity sector.  A sector of 16-byte amplitudes up to d = 14000 fits in the
// shared memory of one block, so a column needs no passes, no tile transfers and no zero
// amplitudes: every gate of the circuit runs on it back to back.  The rows that a gate pairs
// are the same for every column of a sector: they are listed on the host once per (sector,
// wire pair) as 4-byte entries (y row, z row, sign of the gate's Jordan-Wigner string), which
// replaces all per-quartet index arithmetic by one coalesced read.
//
// A block runs the program in steps, one per gate (more for gates whose diagonal entries touch
// several row classes): the center pairs and the rows of one diagonal entry, disjoint rows.
// Steps are staged in shared memory SEC_STAGE at a time.
//
// A block holds 2^ln columns of one sector, row-major with the columns adjacent, so small
// sectors share each entry between up to 8 columns.  The entries are ordered on the host so
// that the lanes of one shared-memory wavefront touch distinct banks (see sector_order).
// The arithmetic per amplitude and the order of the gates are those of k_target: bit-identical.
//
// Bound: shared-memory bandwidth and issue in float-float (a hop pair moves 64 bytes, 16 cycles
// of shared memory per warp, and issues about 76 instructions, 19 cycles), the FP64 pipe in
// complex128.  Measured against the tiled sweep that it replaces (k_target_w, which stays for
// sectors too large for shared memory): L=16 spinful, 6001 columns, float-float 267 -> 27.6 ms;
// L=14 spinful, whole trace, float-float 147 -> 16.6 ms; L=12 spinless (3606 gates), complex128
// 101 -> 75 ms (FP64 pipe 87 % busy); L=12 spinful, complex128 18.2 -> 5.3 ms.  Reading each
// thread's first entries before the barrier, or one task list for pairs and rows, measured
// slower (33.4 and 22.4 ms for the first two): the sweep is not bound by the entries' latency.

constexpr int SEC_STAGE = 64;          // steps staged at a time

// one step of the program: kc, kr: lists of the center pairs and of the rows (-1: none); kind:
// the gate's kind word; mat: its matrix; flags: entry of the row factor | SEC_NEG | SEC_SYNC
struct SecStep { int kc, kr, kind, mat, flags; };
constexpr int SEC_NEG = 16, SEC_SYNC = 32;

struct SecItem { int first, d, ln, row0, offs, rlo, rhi, pad; };   // one sector's blocks start at `first`

// a staged step: its lists in the block's sector
struct SecRec { int cbeg, ccnt, rbeg, rcnt, kind, mat, flags, pad; };

template <class P>
struct SecArgs
{
	typedef typename P::T T;
	const SecItem* items;
	int nitems;
	const SecStep* steps;
	int nsteps;
	const T* mats;
	const unsigned* list;      // entries of all lists
	const int* offs;           // per sector: list k = list[offs[k], offs[k + 1])
	const unsigned* rows;      // full basis index of each sector row, ascending within a sector
	T* ucols;
	long b0, S;
};

// center block of kind `kind` on the pair (a, b); sg: off-diagonal entries negated (k_target's
// arithmetic, tgt_block / tgt_hop; diagonal center blocks are row steps)
template <class P>
__device__ __forceinline__ void sec_block(int kind, unsigned rot, const typename P::T* __restrict__ m, unsigned sg,
	typename P::T& a, typename P::T& b)
{
	typedef typename P::T T;
	const T x = a, y = b;
	switch (kind)
	{
	case BK_SWAP: a = P::negif(y, sg); b = P::negif(x, sg); return;
	case BK_ANTI: a = P::mul(m[1], P::negif(y, sg)); b = P::mul(m[2], P::negif(x, sg)); return;
	case BK_RI:
		a = P::madd2_ri(m[0], rot & 1, x, m[1], rot & 2, P::negif(y, sg));
		b = P::madd2_ri(m[2], rot & 4, P::negif(x, sg), m[3], rot & 8, y);
		return;
	default:
		a = P::madd2(m[0], x, m[1], P::negif(y, sg));
		b = P::madd2(m[2], P::negif(x, sg), m[3], y);
	}
}

template <class P, int NT, int NB>
__global__ void __launch_bounds__(NT, NB) k_sector(SecArgs<P> a)
{
	typedef typename P::T T;
	constexpr unsigned ES = sizeof(T);
	extern __shared__ __align__(16) char smem_raw[];
	__shared__ SecRec stage[SEC_STAGE];
	const unsigned tb = smem_u32(smem_raw);
	// this block's sector: the last whose first block is not after it
	int lo = 0, hi = a.nitems - 1;
	while (lo < hi)
	{
		const int mid = (lo + hi + 1) >> 1;
		if (a.items[mid].first <= (int)blockIdx.x) lo = mid; else hi = mid - 1;
	}
	const SecItem I = a.items[lo];
	const int ln = I.ln, nc = 1 << ln, cm = nc - 1;
	const int r0 = I.rlo + (((int)blockIdx.x - I.first) << ln);   // first column: row r0 of the sector
	const int ncol = min(nc, I.rhi - r0);
	const unsigned n = (unsigned)I.d << ln;
	const int* offs = a.offs + I.offs;

	for (unsigned e = threadIdx.x; e < n; e += NT) sts<T>(tb + e * ES, P::zero());
	__syncthreads();
	if ((int)threadIdx.x < ncol) sts<T>(tb + ((((unsigned)(r0 + threadIdx.x)) << ln) + threadIdx.x) * ES, P::make(1.0, 0.0));

	const unsigned cb = tb + (threadIdx.x & cm) * ES;         // this thread's column
	const unsigned p0 = threadIdx.x >> ln, ps = NT >> ln;      // first task and stride
	const unsigned sh = ln + (ES == 16 ? 4 : 3);
	for (int s0 = 0; s0 < a.nsteps; s0 += SEC_STAGE)
	{
		const int ns = min(SEC_STAGE, a.nsteps - s0);
		__syncthreads();
		if ((int)threadIdx.x < ns)
		{
			const SecStep S = a.steps[s0 + threadIdx.x];
			SecRec R;
			R.cbeg = R.ccnt = R.rbeg = R.rcnt = 0;
			if (S.kc >= 0) { R.cbeg = offs[S.kc]; R.ccnt = offs[S.kc + 1] - R.cbeg; }
			if (S.kr >= 0) { R.rbeg = offs[S.kr]; R.rcnt = offs[S.kr + 1] - R.rbeg; }
			R.kind = S.kind; R.mat = S.mat; R.flags = S.flags; R.pad = 0;
			stage[threadIdx.x] = R;
		}
		__syncthreads();
		for (int s = 0; s < ns; s++)
		{
			const SecRec R = stage[s];
			const unsigned* li = a.list + R.cbeg;
			const T* m = a.mats + (size_t)R.mat * 8;
			unsigned p = p0;
			if (kw_hop_center(R.kind))
			{
				const T c0 = m[0], c1 = m[1];
				for (; p + ps < (unsigned)R.ccnt; p += 2 * ps)
				{
					const unsigned f0 = li[p], f1 = li[p + ps];
					const unsigned ay0 = cb + ((f0 & 0x7fffu) << sh), az0 = cb + ((f0 >> 16) << sh);
					const unsigned ay1 = cb + ((f1 & 0x7fffu) << sh), az1 = cb + ((f1 >> 16) << sh);
					T y0 = lds<T>(ay0), z0 = lds<T>(az0), y1 = lds<T>(ay1), z1 = lds<T>(az1);
					P::hop(c0, c1, (f0 >> 15) & 1u, y0, z0);
					P::hop(c0, c1, (f1 >> 15) & 1u, y1, z1);
					sts<T>(ay0, y0); sts<T>(az0, z0); sts<T>(ay1, y1); sts<T>(az1, z1);
				}
				if (p < (unsigned)R.ccnt)
				{
					const unsigned f = li[p], ay = cb + ((f & 0x7fffu) << sh), az = cb + ((f >> 16) << sh);
					T y = lds<T>(ay), z = lds<T>(az);
					P::hop(c0, c1, (f >> 15) & 1u, y, z);
					sts<T>(ay, y); sts<T>(az, z);
				}
			}
			else
				for (; p < (unsigned)R.ccnt; p += ps)
				{
					const unsigned f = li[p], ay = cb + ((f & 0x7fffu) << sh), az = cb + ((f >> 16) << sh);
					T y = lds<T>(ay), z = lds<T>(az);
					sec_block<P>(R.kind & 7, (unsigned)(R.kind >> 6) & 15u, m, (f >> 15) & 1u, y, z);
					sts<T>(ay, y); sts<T>(az, z);
				}
			if (R.rcnt)
			{
				// from the last thread down: the threads that had fewer pairs start
				const T c = m[R.flags & 7];
				li = a.list + R.rbeg;
				for (p = ps - 1 - p0; p < (unsigned)R.rcnt; p += ps)
				{
					const unsigned ay = cb + (li[p] << sh);
					const T y = lds<T>(ay);
					sts<T>(ay, (R.flags & SEC_NEG) ? P::neg(y) : P::mul(c, y));
				}
			}
			if (R.flags & SEC_SYNC) __syncthreads();
		}
	}
	__syncthreads();

	// -conj of each column into its parity-sector slot: zeros, then the sector's rows
	const unsigned* rows = a.rows + I.row0;
	for (int c = 0; c < ncol; c++)
	{
		T* out = a.ucols + (size_t)((long)rows[r0 + c] - a.b0) * a.S;
		for (long e = threadIdx.x; e < a.S; e += NT) out[e] = P::zero();
	}
	__syncthreads();
	for (unsigned e = threadIdx.x; e < n; e += NT)
	{
		const unsigned r = e >> ln, c = e & cm;
		if ((int)c < ncol)
			a.ucols[(size_t)((long)rows[r0 + c] - a.b0) * a.S + (rows[r] >> 1)] = P::negconj(lds<T>(tb + e * ES));
	}
}
