// Fitted circuit in factored form (k_fit): f and block gradients of the columns whose
// -conj(U e_b) are given.  Included by mgcu_engine.cu inside its anonymous namespace.
//
// Each 2x2 block is factored as diag(l0, l1) M diag(1, r1) with M = [[1, p], [q, 1]] or, when
// the off-diagonal entries dominate, [[p, 1], [1, q]]: p is real, and q is real too for unitary
// blocks (up to rounding, which q keeps in complex128).  M takes one real multiply-add per real
// number instead of four, and the diagonal factors of all gates between two uses of a wire are
// merged into one table with an entry per amplitude (a "flush": one complex multiply per
// amplitude and brickwall layer).  Per gate and amplitude that is 24 FP32 operations in
// float-float (80 unfactored) or 3 FP64 operations (8).
//
// Gates are applied in groups of up to two with disjoint wires: a thread owns the 16
// amplitudes ("registers" 0..15) of the group's four tile bits, so there is one barrier and one
// cached state per two gates, and the cache is stored in the order in which the threads own the
// amplitudes.  A gate on the dropped qubit pairs along one tile bit, corner or center by the
// parity of the rest; it takes a fourth, free bit by which each thread relabels its amplitudes
// so that register 0 has even parity.
//
// Gradients: with Y the state and E the derivative after a gate's M, R[r][u] = sum E_r Y_u over
// all columns determines the gradient of the gate: dG[r][t] = sum_u R[r][u] Minv[t][u] /
// (l_r r_t), applied once at the end (k_fit_finish).  R of all gates of a parameter block are
// summed, and f is the trace of R.
//
// Bound: issue (58 %) and the latency of the cached states in float-float, the FP64 pipe in
// complex128.  Measured against k_columns (which stays for small sectors, FP32 Hessians and
// gates that do not factor): float-float L=12, 7 layers 5.17 -> 2.88 ms; L=14, 9 layers
// 122 -> 73 ms; L=16, 5 layers, 6001 columns 119 -> 81 ms; complex128 L=12, 5 layers
// 12.2 -> 6.4 ms.

constexpr int FIT_RENORM = 64;     // quartets per thread between renormalisations of the sums

// register bits 0, 1: wires j, i of gate a; bits 2, 3: wires j, i of gate b (kind_b 1), or bit 2:
// the compact wire of a gate on the dropped qubit and bit 3 free (kind_b 2)
struct FitGroup
{
	unsigned m[4];        // byte offsets (swizzled) of the register bits
	int cbit[14];         // compact bits: register bits 0..3, then the unit-index bits
	int ga, gb, kind_b;   // gates (-1: none)
	int rev;              // gate b is on the dropped qubit as wire i: its center pair is (z, y)
	int order;            // 1: gate b comes before gate a in the sequence
	int blk_a, blk_b;
	int blk_next;         // block of the first sum of the group before (gate b's, if it has one)
	int flush;            // table multiplied in before the gates (-1: none)
	int pass;
	// per gate (a, b) and quartet: registers of |00>, |01>, |10>, |11> as byte offsets in the
	// tile (swizzled, XOR) and in a unit's cached state
	uint4 qs[2][4], qy[2][4];
};

// QC: how a group's gates are applied -- 0: M with a real q, 1: with a complex q, 2: unfactored
// (the whole blocks, in k_columns' and k_target's arithmetic)
template <class T> struct FitGate { T pc, qc, pk, qk; int swc, swk, pad[2]; };
template <class T> struct FitWhole { T c[4], k[4]; };
template <class T, int QC> struct FitGateOf { typedef FitGate<T> type; };
template <class T> struct FitGateOf<T, 2> { typedef FitWhole<T> type; };
// what k_fit makes: f; f and gradients; -conj of the columns; f and gradients, with states and
// derivatives cached per column (Hessian plans)
enum { FIT_VALUE = 0, FIT_GRAD = 1, FIT_COLS = 2, FIT_HESS = 3 };

struct FitPass { int gbeg, gend; };

// a group's record and gates in shared memory, copied asynchronously one group ahead
template <class G> struct __align__(16) FitStage { FitGroup g; G gate[2]; };

template <class G>
__device__ __forceinline__ void fit_stage(FitStage<G>& d, const FitGroup* __restrict__ g, const G* __restrict__ gates)
{
	constexpr unsigned NG = sizeof(FitGroup) / 16, NT = 2 * sizeof(G) / 16;
	const unsigned i = threadIdx.x;
	if (i < NG + NT)
	{
		const char* src = i < NG ? reinterpret_cast<const char*>(g) + 16 * i : reinterpret_cast<const char*>(gates) + 16 * (i - NG);
		const unsigned dst = smem_u32(&d) + 16 * i;
		asm volatile("cp.async.ca.shared.global [%0], [%1], 16;" :: "r"(dst), "l"(src) : "memory");
	}
}
__device__ __forceinline__ void fit_stage_wait() { asm volatile("cp.async.wait_all;" ::: "memory"); }

template <class P>
struct FitArgs
{
	typedef typename P::T T;
	int L, nb, kt, npass, ngroups, nc, ncs;   // nc, ncs: columns per block and per cache slot
	long S;
	const PassRec* pass;        // tiles of the passes
	const FitPass* groups_of;
	const FitGroup* groups;
	const unsigned* bases;      // [group][unit]: byte offset (swizzled) of register 0
	const void* gates;          // [group][2], FitGate or FitWhole
	const T* tables;            // [flush][parity][S], in thread order of the flush's group
	const T* final;             // [parity][S]: the diagonal factors after the last gate
	const T* dense;
	long dense_b0, b0, b1;
	T* ucols;                   // FIT_COLS: output columns [b - b0][S]
	T* su;
	T* sw;
	T* cache;                   // [slot][group][column of the block][S]; slot: the block, or (FIT_HESS) its columns from b0
	T* dcache;                  // the derivatives, alike (FIT_HESS)
	double* part;               // [block][nblocks][16] (gradient) or [block][2]
	double* part_f;             // [block][2]: f beside a gradient of whole blocks
	int nblocks;
};

// swizzled slot of a tile index: its low bits XORed with the higher groups of bits, so that the
// lanes of a wavefront hit distinct banks whenever their bits differ mod 3 (mod 4 for 8 bytes)
template <int ES>
__host__ __device__ __forceinline__ unsigned fsw(unsigned e)
{
	return ES == 16 ? e ^ ((e >> 3) & 7u) ^ ((e >> 6) & 7u) ^ ((e >> 9) & 7u)
	                : e ^ ((e >> 4) & 15u) ^ ((e >> 8) & 15u) ^ ((e >> 12) & 15u);
}

// M (or its transpose) on the pair (f, s); sw: M = [[p, 1], [1, q]]
template <class P, bool QC, bool TR>
__device__ __forceinline__ void fit_pair(typename P::T& f, typename P::T& s, const typename P::T& p, const typename P::T& q, bool sw)
{
	typedef typename P::T T;
	const T x = f, y = s;
	if (sw)
	{
		f = P::axpy(y, p, x);
		s = QC ? P::axpyc(x, q, y) : P::axpy(x, q, y);
	}
	else if (!TR)
	{
		f = P::axpy(x, p, y);
		s = QC ? P::axpyc(y, q, x) : P::axpy(y, q, x);
	}
	else
	{
		f = QC ? P::axpyc(x, q, y) : P::axpy(x, q, y);
		s = P::axpy(y, p, x);
	}
}

// byte offset in the tile of register k of a unit whose register 0 is at `base`
__device__ __forceinline__ unsigned fit_off(const FitGroup& G, unsigned base, int k)
{
	return base ^ ((k & 1) ? G.m[0] : 0u) ^ ((k & 2) ? G.m[1] : 0u) ^ ((k & 4) ? G.m[2] : 0u) ^ ((k & 8) ? G.m[3] : 0u);
}

// byte offset of register 0 of unit u; tpar: parity of the column and of the tile's nonlocal bits
__device__ __forceinline__ unsigned fit_base(const FitGroup& G, const unsigned* __restrict__ bases, unsigned u, int tpar)
{
	const unsigned b = bases[u];
	return (G.kind_b == 2 && ((__popc(u) + tpar) & 1)) ? b ^ G.m[3] : b;
}

// the corner or center block of a gate on a pair, whole or as M
template <class P, int QC>
__device__ __forceinline__ void fit_apply(typename P::T& f, typename P::T& s, const typename FitGateOf<typename P::T, QC>::type& g, bool corner)
{
	typedef typename P::T T;
	if constexpr (QC == 2)
	{
		const T* m = corner ? g.k : g.c;
		const T x = f, y = s;
		f = P::madd2(m[0], x, m[1], y);
		s = P::madd2(m[2], x, m[3], y);
	}
	else if (corner) fit_pair<P, QC == 1, false>(f, s, g.pk, g.qk, g.swk);
	else fit_pair<P, QC == 1, false>(f, s, g.pc, g.qc, g.swc);
}

template <class P, int QC>
__device__ __forceinline__ void fit_gate_a(typename P::T (&v)[16], const typename FitGateOf<typename P::T, QC>::type& g)
{
#pragma unroll
	for (int k = 0; k < 4; k++) fit_apply<P, QC>(v[4 * k], v[4 * k + 3], g, true);
#pragma unroll
	for (int k = 0; k < 4; k++) fit_apply<P, QC>(v[4 * k + 1], v[4 * k + 2], g, false);
}

template <class P, int QC>
__device__ __forceinline__ void fit_gate_b(typename P::T (&v)[16], const FitGroup& G, const typename FitGateOf<typename P::T, QC>::type& g)
{
	if (G.kind_b == 1)
	{
#pragma unroll
		for (int k = 0; k < 4; k++) fit_apply<P, QC>(v[k], v[k + 12], g, true);
#pragma unroll
		for (int k = 0; k < 4; k++) fit_apply<P, QC>(v[k + 4], v[k + 8], g, false);
		return;
	}
	// pairs along bit 2: corner where the other bits (0, 1, 3) have even parity
	fit_apply<P, QC>(v[0], v[4], g, true);
	fit_apply<P, QC>(v[3], v[7], g, true);
	fit_apply<P, QC>(v[9], v[13], g, true);
	fit_apply<P, QC>(v[10], v[14], g, true);
	if (!G.rev)
	{
		fit_apply<P, QC>(v[1], v[5], g, false);
		fit_apply<P, QC>(v[2], v[6], g, false);
		fit_apply<P, QC>(v[8], v[12], g, false);
		fit_apply<P, QC>(v[11], v[15], g, false);
	}
	else
	{
		fit_apply<P, QC>(v[5], v[1], g, false);
		fit_apply<P, QC>(v[6], v[2], g, false);
		fit_apply<P, QC>(v[12], v[8], g, false);
		fit_apply<P, QC>(v[15], v[11], g, false);
	}
}

// one group on a unit, all 16 amplitudes in registers: one shared-memory round trip for both
// gates.  For the forward sweep of f alone; beside the gradient sums' registers it spills
// (float-float L=12, 42 gates: 3.8 ms against 3.3 ms quartet by quartet)
template <class P, int QC>
__device__ __forceinline__ void fit_group16(const FitGroup& G, const typename FitGateOf<typename P::T, QC>::type* gates, unsigned tc, unsigned base,
	unsigned U, const typename P::T* __restrict__ tab)
{
	typedef typename P::T T;
	T v[16];
#pragma unroll
	for (int k = 0; k < 16; k++) v[k] = lds<T>(tc + fit_off(G, base, k));
	if (QC != 2 && tab)
	{
#pragma unroll
		for (int k = 0; k < 16; k++) v[k] = P::mul(tab[k * U], v[k]);
	}
	// in sequence order (it matters to the rounding of whole blocks only)
	if (QC == 2 && G.order) fit_gate_b<P, QC>(v, G, gates[1]);
	if (G.ga >= 0) fit_gate_a<P, QC>(v, gates[0]);
	if (G.kind_b && !(QC == 2 && G.order)) fit_gate_b<P, QC>(v, G, gates[1]);
#pragma unroll
	for (int k = 0; k < 16; k++) sts<T>(tc + fit_off(G, base, k), v[k]);
}

// both gates of a group on a unit, quartet by quartet in the tile.  Forward: flush (tab or null)
// with the first gate, the state to the cache (out or null) with the last; transposed (TR):
// flush with the last
// SP: threads per unit, 1 or 4 (one quartet each, part = 0..3)
template <class P, int QC, bool TR, int SP>
__device__ __forceinline__ void fit_group(const FitGroup& G, const FitGate<typename P::T>* gates, unsigned tc, unsigned base,
	const typename P::T* __restrict__ tab, typename P::T* __restrict__ out, int part)
{
	typedef typename P::T T;
	const int w0 = G.ga >= 0 ? 0 : 1, w1 = G.kind_b ? 1 : 0;
#pragma unroll 1
	for (int w = w0; w <= w1; w++)
	{
		const FitGate<T>& g = gates[w];
		const T pk = g.pk, qk = g.qk, pc = g.pc, qc = g.qc;
		const bool sk = g.swk, sc = g.swc;
		const char* tb = (w == (TR ? w1 : w0)) ? reinterpret_cast<const char*>(tab) : nullptr;
		char* ob = (!TR && w == w1) ? reinterpret_cast<char*>(out) : nullptr;
		if (SP > 1) __syncwarp();   // the other threads' quartets of the unit
#pragma unroll 1
		for (int i = part; i < 4; i += SP)
		{
			const uint4 o = G.qs[w][i], q = G.qy[w][i];
			const unsigned ax = tc + (base ^ o.x), ay = tc + (base ^ o.y), az = tc + (base ^ o.z), aw = tc + (base ^ o.w);
			T x = lds<T>(ax), y = lds<T>(ay), z = lds<T>(az), v = lds<T>(aw);
			T tx, ty, tz, tv;
			if (tb)
			{
				tx = *reinterpret_cast<const T*>(tb + q.x); ty = *reinterpret_cast<const T*>(tb + q.y);
				tz = *reinterpret_cast<const T*>(tb + q.z); tv = *reinterpret_cast<const T*>(tb + q.w);
			}
			if (!TR && tb) { x = P::mul(tx, x); y = P::mul(ty, y); z = P::mul(tz, z); v = P::mul(tv, v); }
			fit_pair<P, QC == 1, TR>(x, v, pk, qk, sk);
			fit_pair<P, QC == 1, TR>(y, z, pc, qc, sc);
			if (TR && tb) { x = P::mul(tx, x); y = P::mul(ty, y); z = P::mul(tz, z); v = P::mul(tv, v); }
			sts<T>(ax, x); sts<T>(ay, y); sts<T>(az, z); sts<T>(aw, v);
			if (ob)
			{
				*reinterpret_cast<T*>(ob + q.x) = x; *reinterpret_cast<T*>(ob + q.y) = y;
				*reinterpret_cast<T*>(ob + q.z) = z; *reinterpret_cast<T*>(ob + q.w) = v;
			}
		}
	}
}

// The gradient sweeps with whole blocks (FP32), gate by gate in k_columns' arithmetic: forward
// keeps each gate's input (cache: two slots per group, `slot` apart), backward sums the
// derivative against it and applies the transpose, one quartet per iteration, the inputs read
// one quartet ahead.
template <class P>
__device__ __forceinline__ void fit_whole_forward(const FitGroup& G, int w, const FitWhole<typename P::T>& g, unsigned tc, unsigned base,
	typename P::T* __restrict__ out)
{
	typedef typename P::T T;
	char* ob = reinterpret_cast<char*>(out);
	const T c0 = g.c[0], c1 = g.c[1], c2 = g.c[2], c3 = g.c[3], k0 = g.k[0], k1 = g.k[1], k2 = g.k[2], k3 = g.k[3];
#pragma unroll 2
	for (int i = 0; i < 4; i++)
	{
		const uint4 o = G.qs[w][i], q = G.qy[w][i];
		const unsigned ax = tc + (base ^ o.x), ay = tc + (base ^ o.y), az = tc + (base ^ o.z), aw = tc + (base ^ o.w);
		const T x = lds<T>(ax), y = lds<T>(ay), z = lds<T>(az), v = lds<T>(aw);
		*reinterpret_cast<T*>(ob + q.x) = x; *reinterpret_cast<T*>(ob + q.y) = y;
		*reinterpret_cast<T*>(ob + q.z) = z; *reinterpret_cast<T*>(ob + q.w) = v;
		sts<T>(ax, P::madd2(k0, x, k1, v)); sts<T>(aw, P::madd2(k2, x, k3, v));
		sts<T>(ay, P::madd2(c0, y, c1, z)); sts<T>(az, P::madd2(c2, y, c3, z));
	}
}

template <class P>
__device__ __forceinline__ void fit_whole_backward(const FitGroup& G, int w, const FitWhole<typename P::T>& g, unsigned tc, unsigned base,
	const typename P::T* __restrict__ ct, typename P::Acc (&acc)[8])
{
	typedef typename P::T T;
	const char* cb = reinterpret_cast<const char*>(ct);
	const T c0 = g.c[0], c1 = g.c[1], c2 = g.c[2], c3 = g.c[3], k0 = g.k[0], k1 = g.k[1], k2 = g.k[2], k3 = g.k[3];
	uint4 q = G.qy[w][0];
	T nx = *reinterpret_cast<const T*>(cb + q.x), ny = *reinterpret_cast<const T*>(cb + q.y);
	T nz = *reinterpret_cast<const T*>(cb + q.z), nv = *reinterpret_cast<const T*>(cb + q.w);
#pragma unroll 2
	for (int i = 0; i < 4; i++)
	{
		const uint4 o = G.qs[w][i];
		const unsigned ax = tc + (base ^ o.x), ay = tc + (base ^ o.y), az = tc + (base ^ o.z), aw = tc + (base ^ o.w);
		const T x = nx, y = ny, z = nz, v = nv;
		q = G.qy[w][min(i + 1, 3)];
		nx = *reinterpret_cast<const T*>(cb + q.x); ny = *reinterpret_cast<const T*>(cb + q.y);
		nz = *reinterpret_cast<const T*>(cb + q.z); nv = *reinterpret_cast<const T*>(cb + q.w);
		const T dx = lds<T>(ax), dy = lds<T>(ay), dz = lds<T>(az), dv = lds<T>(aw);
		contract_quartet<P>(acc, dx, dv, dy, dz, x, v, y, z);
		// transpose (no conjugation): reference src/gate.c:725-728
		sts<T>(ax, P::madd2(k0, dx, k2, dv)); sts<T>(aw, P::madd2(k1, dx, k3, dv));
		sts<T>(ay, P::madd2(c0, dy, c2, dz)); sts<T>(az, P::madd2(c1, dy, c3, dz));
	}
}

// R sums of the gates first..last (1: b, 0: a) of a group over the quartets of a unit: the
// derivative in the tile and the cached state ct, read one quartet ahead.  One loop for every
// kind of gate, not unrolled: with each gate's quartets unrolled the kernel's code outgrew the
// instruction caches (a third of its stalls).
// EOUT: the derivative also to its cache eout, with the last gate.  SW: the tile holds the
// state and ct the derivative (Hessian items)
template <class P, bool SW, bool EOUT, int SP>
__device__ __forceinline__ void fit_contract(const FitGroup& G, int first, int last, unsigned tc, unsigned base,
	const typename P::T* __restrict__ ct, typename P::Acc (&acc)[8], typename P::T* __restrict__ eout, int part)
{
	typedef typename P::T T;
	const char* cb = reinterpret_cast<const char*>(ct);
	const uint4 *qs = &G.qs[0][0], *qy = &G.qy[0][0];
	int i = 4 * first + part;
	uint4 oy = qy[i];
	T cx = *reinterpret_cast<const T*>(cb + oy.x), cy = *reinterpret_cast<const T*>(cb + oy.y);
	T cz = *reinterpret_cast<const T*>(cb + oy.z), cw = *reinterpret_cast<const T*>(cb + oy.w);
#pragma unroll 1
	for (int k = 4 * (first - last + 1); k > 0; k -= SP)
	{
		const uint4 o = qs[i];
		const T x = lds<T>(tc + (base ^ o.x)), y = lds<T>(tc + (base ^ o.y)), z = lds<T>(tc + (base ^ o.z)), v = lds<T>(tc + (base ^ o.w));
		const T sx = cx, sy = cy, sz = cz, sv = cw;
		if (EOUT && (i >> 2) == last)
		{
			const uint4 q = qy[i];
			char* eb = reinterpret_cast<char*>(eout);
			*reinterpret_cast<T*>(eb + q.x) = x; *reinterpret_cast<T*>(eb + q.y) = y;
			*reinterpret_cast<T*>(eb + q.z) = z; *reinterpret_cast<T*>(eb + q.w) = v;
		}
		i = (i + SP) & 7;   // gate b's quartets 4..7, then gate a's 0..3
		if (k > SP)
		{
			oy = qy[i];
			cx = *reinterpret_cast<const T*>(cb + oy.x); cy = *reinterpret_cast<const T*>(cb + oy.y);
			cz = *reinterpret_cast<const T*>(cb + oy.z); cw = *reinterpret_cast<const T*>(cb + oy.w);
		}
		if (SW) contract_quartet<P>(acc, sx, sv, sy, sz, x, v, y, z);
		else contract_quartet<P>(acc, x, v, y, z, sx, sv, sy, sz);
	}
}

// threads per block: 128, or 256 where a tile has that many units; four (two) blocks per SM
// (registers), three of 128 in complex128, whose pipe is the bound.  In FP32 f and columns keep
// one state per thread and fit 768 threads on 80 registers: f at L=13, 8192 columns 4.95 ->
// 4.63 ms (gradients, whose sums spill there, keep 512).  SP 4 (gradients of few columns, see
// fit_build): four threads per unit
constexpr int fit_blocks(int prec, int mode, int nt)
{
	if (prec == MG_PREC_FP32_ID && mode != FIT_GRAD) return 768 / nt;
	return nt == 512 ? 1 : nt == 256 ? 2 : prec == MG_PREC_FP64_ID ? 3 : 4;
}
template <class P, int QC, int MODE, int FIT_NT, int SP>
__global__ void __launch_bounds__(FIT_NT, fit_blocks(P::kId, MODE, FIT_NT)) k_fit(FitArgs<P> a)
{
	typedef typename P::T T;
	constexpr unsigned ES = sizeof(T);
	extern __shared__ __align__(16) char smem_raw[];
	typedef typename FitGateOf<T, QC>::type Gate;
	constexpr bool GRAD = MODE == FIT_GRAD || MODE == FIT_HESS;
	__shared__ FitStage<Gate> stage[2];
	const int kt = a.kt, nu = kt - 4;
	const unsigned U = 1u << nu, n = 1u << kt;
	const int nc = a.nc;
	// units per thread (none for the threads beyond the block's units)
	const unsigned its = U > FIT_NT ? U / FIT_NT : threadIdx.x < U * nc * SP ? 1 : 0;
	const unsigned tb = smem_u32(smem_raw);
	Smem s;
	s.dlo = reinterpret_cast<unsigned*>(smem_raw + (size_t)ES * n * nc);
	s.dhi = s.dlo + 128;
	s.red = reinterpret_cast<double*>(s.dhi + 128);
	s.h = kt / 2;
	const long S = a.S;
	const unsigned tu = threadIdx.x / SP, mycol = min(tu >> nu, (unsigned)nc - 1), u0 = (nc > 1 || SP > 1) ? (tu & (U - 1)) : tu;
	const int part = SP > 1 ? (int)(threadIdx.x % SP) : 0;
	const unsigned colb = mycol * n * ES;
	const size_t cstride = (size_t)(MODE == FIT_HESS ? a.ncs : nc) * S * (QC == 2 ? 2 : 1);
	typename P::Acc acc[8];
#pragma unroll
	for (int e = 0; e < 8; e++) acc[e] = P::acc_zero();
	typename P::Acc facc = P::acc_zero();
	int nred = 0;

	for (long cb = a.b0 + (long)blockIdx.x * nc; cb < a.b1; cb += (long)gridDim.x * nc)
	{
		// this thread's column (the last one again past the range: its derivative is zero)
		const long b = min(cb + (long)mycol, a.b1 - 1);
		const int par = __popcll(b) & 1;
		const size_t coff = MODE == FIT_HESS ? (size_t)((cb - a.b0) / a.ncs) * a.ngroups * cstride + (size_t)((cb - a.b0) % a.ncs + mycol) * S
			: (size_t)blockIdx.x * a.ngroups * cstride + (size_t)mycol * S;
		T* cache = GRAD ? a.cache + coff : nullptr;
		// the state between passes (one column per block then): the output column itself, or a slot
		auto between = [&]() { return MODE == FIT_COLS ? a.ucols + (size_t)(cb - a.b0) * S : a.sw + (size_t)blockIdx.x * S; };
		for (int p = 0; p < a.npass; p++)
		{
			const PassRec& pr = a.pass[p];
			const FitPass fp = a.groups_of[p];
			__syncthreads();
			setup_pass(pr, kt, s);
			__syncthreads();
			const bool last = p == a.npass - 1;
			for (unsigned tau = 0; tau < (1u << pr.nnl); tau++)
			{
				const unsigned nlb = nl_base(pr, tau);
				const int tpar = (__popc(nlb) + par) & 1;
				fit_stage<Gate>(stage[fp.gbeg & 1], a.groups + fp.gbeg, static_cast<const Gate*>(a.gates) + 2 * fp.gbeg);
				for (unsigned e = threadIdx.x; e < n * nc; e += FIT_NT)
				{
					const unsigned c = gidx(s, nlb, e & (n - 1));
					T v;
					if (p == 0) v = c == (unsigned)(min(cb + (long)(e >> kt), a.b1 - 1) >> 1) ? P::make(1.0, 0.0) : P::zero();
					else v = between()[c];
					sts<T>(tb + ((e & ~(n - 1)) + fsw<ES>(e & (n - 1))) * ES, v);
				}
				fit_stage_wait();
				__syncthreads();
				for (int g = fp.gbeg; g < fp.gend; g++)
				{
					const FitGroup& G = stage[g & 1].g;
					if (g + 1 < fp.gend) fit_stage<Gate>(stage[(g + 1) & 1], a.groups + g + 1, static_cast<const Gate*>(a.gates) + 2 * (g + 1));
					for (unsigned i = 0; i < its; i++)
					{
						const unsigned u = u0 + i * FIT_NT, base = fit_base(G, a.bases + (size_t)g * U, u, tpar);
						const T* tab = G.flush >= 0 ? a.tables + ((size_t)(2 * G.flush + par) * S + ((size_t)tau << kt) + u) : nullptr;
						T* out = GRAD ? cache + (size_t)g * cstride + ((size_t)tau << kt) + u : nullptr;
						if constexpr (GRAD && QC == 2)
						{
							const int ngt = (G.ga >= 0 && G.kind_b) ? 2 : 1, w0 = ngt == 2 ? G.order : (G.ga >= 0 ? 0 : 1);
#pragma unroll 1
							for (int st = 0; st < ngt; st++)
								fit_whole_forward<P>(G, w0 ^ st, stage[g & 1].gate[w0 ^ st], tb + colb, base, out + (size_t)(w0 ^ st) * nc * S);
						}
						else if constexpr (GRAD) fit_group<P, QC, false, SP>(G, stage[g & 1].gate, tb + colb, base, tab, out, part);
						else fit_group16<P, QC>(G, stage[g & 1].gate, tb + colb, base, U, tab);
					}
					fit_stage_wait();
					__syncthreads();
				}
				if (MODE == FIT_COLS && last)
				{
					for (unsigned e = threadIdx.x; e < n * nc; e += FIT_NT)
					{
						const unsigned c = gidx(s, nlb, e & (n - 1));
						const long be = cb + (long)(e >> kt);
						if (be >= a.b1) continue;
						T v = lds<T>(tb + ((e & ~(n - 1)) + fsw<ES>(e & (n - 1))) * ES);
						if (QC != 2) v = P::mul(a.final[(size_t)(__popcll(be) & 1) * S + c], v);
						a.ucols[(size_t)(be - a.b0) * S + c] = P::negconj(v);
					}
				}
				if ((MODE == FIT_VALUE || (GRAD && QC == 2)) && last)
				{
					for (unsigned e = threadIdx.x; e < n * nc; e += FIT_NT)
					{
						const unsigned c = gidx(s, nlb, e & (n - 1));
						const long be = cb + (long)(e >> kt);
						if (be >= a.b1) continue;
						T d = a.dense[(size_t)(be - a.dense_b0) * S + c];
						if (QC != 2) d = P::mul(a.final[(size_t)(__popcll(be) & 1) * S + c], d);
						P::acc_mul_add(facc, d, lds<T>(tb + ((e & ~(n - 1)) + fsw<ES>(e & (n - 1))) * ES));
					}
				}
				if (!last)
					for (unsigned e = threadIdx.x; e < n; e += FIT_NT) between()[gidx(s, nlb, e)] = lds<T>(tb + fsw<ES>(e) * ES);
				__syncthreads();
			}
		}
		if constexpr (GRAD)
		{
		for (int p = a.npass - 1; p >= 0; p--)
		{
			const PassRec& pr = a.pass[p];
			const FitPass fp = a.groups_of[p];
			__syncthreads();
			setup_pass(pr, kt, s);
			__syncthreads();
			const bool last = p == a.npass - 1;
			for (unsigned tau = 0; tau < (1u << pr.nnl); tau++)
			{
				const unsigned nlb = nl_base(pr, tau);
				const int tpar = (__popc(nlb) + par) & 1;
				fit_stage<Gate>(stage[(fp.gend - 1) & 1], a.groups + fp.gend - 1, static_cast<const Gate*>(a.gates) + 2 * (fp.gend - 1));
				for (unsigned e = threadIdx.x; e < n * nc; e += FIT_NT)
				{
					const unsigned c = gidx(s, nlb, e & (n - 1));
					T v;
					if (last)
					{
						const long be = cb + (long)(e >> kt);
						v = be < a.b1 ? a.dense[(size_t)(be - a.dense_b0) * S + c] : P::zero();
						if (QC != 2 && be < a.b1) v = P::mul(a.final[(size_t)(__popcll(be) & 1) * S + c], v);
					}
					else v = a.su[(size_t)blockIdx.x * S + c];
					sts<T>(tb + ((e & ~(n - 1)) + fsw<ES>(e & (n - 1))) * ES, v);
				}
				fit_stage_wait();
				__syncthreads();
				if constexpr (QC == 2)
				{
					int cblk = -1, merged = 0;   // the parameter block of the sums in acc
					auto flush = [&]() {
						if (cblk < 0) return;
						block_reduce8<P>(acc, s.red, a.part + ((size_t)blockIdx.x * a.nblocks + cblk) * 16, 1.0, nred);
#pragma unroll
						for (int e = 0; e < 8; e++) acc[e] = P::acc_zero();
						cblk = -1;
						merged = 0;
					};
					for (int g = fp.gend - 1; g >= fp.gbeg; g--)
					{
						const FitGroup& G = stage[g & 1].g;
						if (g > fp.gbeg) fit_stage<Gate>(stage[(g - 1) & 1], a.groups + g - 1, static_cast<const Gate*>(a.gates) + 2 * (g - 1));
						const T* cg = cache + (size_t)g * cstride + ((size_t)tau << kt) + u0;
						if (g > fp.gbeg)
						{
							// the next group's cached inputs to L2, a 128-byte line per thread and slot
							const T* nx = cg - cstride - (threadIdx.x & 15) + (size_t)(threadIdx.x & 15) * U;
							for (unsigned i = 0; i < its; i++)
							{
								asm volatile("prefetch.global.L2 [%0];" :: "l"(nx + i * FIT_NT));
								asm volatile("prefetch.global.L2 [%0];" :: "l"(nx + (size_t)nc * S + i * FIT_NT));
							}
						}
						const int ngt = (G.ga >= 0 && G.kind_b) ? 2 : 1, w0 = ngt == 2 ? G.order : (G.ga >= 0 ? 0 : 1);
#pragma unroll 1
						for (int st = ngt - 1; st >= 0; st--)
						{
							const int w = w0 ^ st, blk = w ? G.blk_b : G.blk_a;
							if (cblk != blk) flush();
							cblk = blk;
							merged += 4 * (int)max(its, 1u);
							for (unsigned i = 0; i < its; i++)
								fit_whole_backward<P>(G, w, stage[g & 1].gate[w], tb + colb, fit_base(G, a.bases + (size_t)g * U, u0 + i * FIT_NT, tpar),
									cg + (size_t)w * nc * S + i * FIT_NT, acc);
							if (merged >= FIT_RENORM)
							{
#pragma unroll
								for (int e = 0; e < 8; e++) P::acc_norm(acc[e]);
								merged = 0;
							}
						}
						fit_stage_wait();
						__syncthreads();
					}
					flush();
				}
				else
				{
				int merged = 0;
				for (int g = fp.gend - 1; g >= fp.gbeg; g--)
				{
					// the state is the one after both gates: both sums come before the
					// transposed gates
					const FitGroup& G = stage[g & 1].g;
					if (g > fp.gbeg) fit_stage<Gate>(stage[(g - 1) & 1], a.groups + g - 1, static_cast<const Gate*>(a.gates) + 2 * (g - 1));
					const T* cg = cache + (size_t)g * cstride + ((size_t)tau << kt) + u0;
					T* eg = MODE == FIT_HESS ? a.dcache + coff + (size_t)g * cstride + ((size_t)tau << kt) + u0 : nullptr;
					const T* tab = G.flush >= 0 ? a.tables + ((size_t)(2 * G.flush + par) * S + ((size_t)tau << kt) + u0) : nullptr;
					const int blk = G.ga >= 0 ? G.blk_a : G.blk_b;
					if (SP == 1 && g > fp.gbeg)
					{
						// the next group's cached state to L2: two of the sixteen 128-byte lines that
						// eight threads' registers take
						const T* nx = cg - cstride - (threadIdx.x & 7);
						for (unsigned i = 0; i < its; i++)
							for (unsigned k = threadIdx.x & 7; k < 16; k += 8)
								asm volatile("prefetch.global.L2 [%0];" :: "l"(nx + i * FIT_NT + k * U));
					}
					const bool split = G.ga >= 0 && G.kind_b && G.blk_b != blk;
					if (split)
					{
						for (unsigned i = 0; i < its; i++)
							fit_contract<P, false, false, SP>(G, 1, 1, tb + colb, fit_base(G, a.bases + (size_t)g * U, u0 + i * FIT_NT, tpar), cg + i * FIT_NT, acc, nullptr, part);
						block_reduce8<P>(acc, s.red, a.part + ((size_t)blockIdx.x * a.nblocks + G.blk_b) * 16, 1.0, nred);
#pragma unroll
						for (int e = 0; e < 8; e++) acc[e] = P::acc_zero();
					}
					for (unsigned i = 0; i < its; i++)
						fit_contract<P, false, MODE == FIT_HESS, SP>(G, (G.kind_b && !split) ? 1 : 0, G.ga >= 0 ? 0 : 1, tb + colb,
							fit_base(G, a.bases + (size_t)g * U, u0 + i * FIT_NT, tpar), cg + i * FIT_NT, acc, eg + i * FIT_NT, part);
					if (g > 0)   // nothing uses the derivative before the first group
						for (unsigned i = 0; i < its; i++)
							fit_group<P, QC, true, SP>(G, stage[g & 1].gate, tb + colb, fit_base(G, a.bases + (size_t)g * U, u0 + i * FIT_NT, tpar),
								tab ? tab + i * FIT_NT : nullptr, nullptr, part);
					merged += 8 * (int)max(its, 1u);
					fit_stage_wait();
					// the next group continues this sum when its gates are of the same block
					bool more = false;
					if (g > fp.gbeg)
					{
						more = G.blk_next == blk;
					}
					if (!more)
					{
						block_reduce8<P>(acc, s.red, a.part + ((size_t)blockIdx.x * a.nblocks + blk) * 16, 1.0, nred);
#pragma unroll
						for (int e = 0; e < 8; e++) acc[e] = P::acc_zero();
						merged = 0;
					}
					else
					{
						if (merged >= FIT_RENORM)
						{
#pragma unroll
							for (int e = 0; e < 8; e++) P::acc_norm(acc[e]);
							merged = 0;
						}
						__syncthreads();
					}
				}
				}
				if (p > 0)
					for (unsigned e = threadIdx.x; e < n; e += FIT_NT) a.su[(size_t)blockIdx.x * S + gidx(s, nlb, e)] = lds<T>(tb + fsw<ES>(e) * ES);
				__syncthreads();
			}
		}
		}
	}
	if (MODE == FIT_VALUE) block_reduce1<P>(facc, s.red, a.part + (size_t)blockIdx.x * 2);
	if (GRAD && QC == 2) block_reduce1<P>(facc, s.red, a.part_f + (size_t)blockIdx.x * 2);
}

// ------------------------------------------------------------------------------------
// Hessian items in factored form.  An item (placement, entry (r, u), a block's columns) carries
// the tangent state B of moving amplitude u of the placement gate's pair onto r after its M:
// B starts as that move of the cached state, passes through the later groups, and at each later
// gate sum E_r' B_u' with the cached derivative gives the second derivative between the two
// moves.  Grouped placements (see k_hessian): every gate of the placement's block adds its move,
// after its own sum.  k_fit_hess_finish turns moves into gate entries.  Per gate and amplitude
// 124 FP32 operations in float-float (176 unfactored) or 10.7 FP64 operations (16).  Measured
// against k_hessian (which stays for FP32, several tiles and gates that do not factor):
// translation-invariant L=12, 9 layers, float-float 152 -> 101 ms; per-layer L=12, 5 layers,
// complex128 169 -> 128 ms; per-gate L=9, 19 gates, float-float 3.97 -> 2.45 ms.  With the items
// in balanced order (item_grid) the last two take 113 ms (FP64 pipe 95 % busy) and 1.30 ms.
// ------------------------------------------------------------------------------------
template <class P>
struct FitHessArgs
{
	FitArgs<P> f;
	const int* place;          // placement gates
	const int* place_group;    // their groups
	const double* place_w;     // [nplace][ngates]
	const int* block;          // [ngates]
	int nplace, ngates, mdim, hgroup;
	long placewise;            // column groups when the items run placement by placement (0: group by group)
	double* part_h;            // [grid][mdim][mdim][2]
};

// adds (init: sets, the rest of the unit zero) the move of entry x of gate w: one amplitude of
// each quartet gains another of the cached state
template <class P>
__device__ __forceinline__ void fit_move(const FitGroup& G, int w, int x, unsigned tc, unsigned base, const typename P::T* __restrict__ ct, bool init)
{
	typedef typename P::T T;
	const char* cb = reinterpret_cast<const char*>(ct);
#pragma unroll 1
	for (int i = 0; i < 4; i++)
	{
		const uint4 o = G.qs[w][i], q = G.qy[w][i];
		const unsigned to = x < 4 ? ((x & 2) ? o.z : o.y) : ((x & 2) ? o.w : o.x);
		const unsigned from = x < 4 ? ((x & 1) ? q.z : q.y) : ((x & 1) ? q.w : q.x);
		const T v = *reinterpret_cast<const T*>(cb + from);
		if (init)
		{
			const T zero = P::zero();
			sts<T>(tc + (base ^ o.x), zero); sts<T>(tc + (base ^ o.y), zero);
			sts<T>(tc + (base ^ o.z), zero); sts<T>(tc + (base ^ o.w), zero);
			sts<T>(tc + (base ^ to), v);
		}
		else sts<T>(tc + (base ^ to), P::add(lds<T>(tc + (base ^ to)), v));
	}
}

template <class P, int QC, int FIT_NT>
__global__ void __launch_bounds__(FIT_NT, FIT_NT == 512 ? 1 : FIT_NT == 256 ? 2 : P::kId == MG_PREC_FP64_ID ? 3 : 4) k_fit_hess(FitHessArgs<P> h, long nitems)
{
	typedef typename P::T T;
	constexpr unsigned ES = sizeof(T);
	extern __shared__ __align__(16) char smem_raw[];
	typedef FitGate<T> Gate;
	__shared__ FitStage<Gate> stage[2];
	const FitArgs<P>& a = h.f;
	const int kt = a.kt, nu = kt - 4, nc = a.nc;
	const unsigned U = 1u << nu, n = 1u << kt;
	const unsigned its = U > FIT_NT ? U / FIT_NT : threadIdx.x < U * nc ? 1 : 0;
	const unsigned tb = smem_u32(smem_raw);
	double* red = reinterpret_cast<double*>(smem_raw + (size_t)ES * n * nc + 256 * sizeof(unsigned));
	const unsigned mycol = min(threadIdx.x >> nu, (unsigned)nc - 1), u0 = nc > 1 ? (threadIdx.x & (U - 1)) : threadIdx.x;
	const unsigned tc = tb + mycol * n * ES;
	const size_t cstride = (size_t)nc * a.S;
	double* parth = h.part_h + (size_t)blockIdx.x * h.mdim * h.mdim * 2;
	typename P::Acc acc[8];
#pragma unroll
	for (int e = 0; e < 8; e++) acc[e] = P::acc_zero();
	int nred = 0;

	for (long it = blockIdx.x; it < nitems; it += gridDim.x)
	{
		const int x = (int)(it & 7);
		const long rest = it >> 3;
		const int p = (int)(h.placewise ? rest / h.placewise : rest % h.nplace);
		const long cgi = h.placewise ? rest % h.placewise : rest / h.nplace;
		const long b = min(a.b0 + cgi * nc + (long)mycol, a.b1 - 1);
		const int par = __popcll(b) & 1;
		const int k = h.place[p], g0 = h.place_group[p];
		const int grp = h.hgroup ? h.block[k] : -1;
		const double* wrow = h.place_w + (size_t)p * h.ngates;
		double* hrow = parth + (size_t)(h.block[k] * 8 + x) * h.mdim * 2;
		const size_t coff = (size_t)cgi * a.ngroups * cstride + (size_t)mycol * a.S + u0;
		// the sums in acc: of gates of block cblk with weight cw (none: -1)
		int cblk = -1, merged = 0;
		double cw = 0;
		auto flush = [&]() {
			if (cblk < 0) return;
			block_reduce8<P>(acc, red, hrow + (size_t)cblk * 16, cw, nred);
#pragma unroll
			for (int e = 0; e < 8; e++) acc[e] = P::acc_zero();
			cblk = -1;
			merged = 0;
		};
		__syncthreads();   // the previous item's last reads
		fit_stage<Gate>(stage[g0 & 1], a.groups + g0, static_cast<const Gate*>(a.gates) + 2 * g0);
		fit_stage_wait();
		__syncthreads();
		for (int g = g0; g < a.ngroups; g++)
		{
			const FitGroup& G = stage[g & 1].g;
			if (g + 1 < a.ngroups) fit_stage<Gate>(stage[(g + 1) & 1], a.groups + g + 1, static_cast<const Gate*>(a.gates) + 2 * (g + 1));
			const T* cg = a.cache + coff + (size_t)g * cstride;
			const T* eg = a.dcache + coff + (size_t)g * cstride;
			const unsigned* bs = a.bases + (size_t)g * U;
			// the group's gates in sequence order; in the first group those after the placement
			const int ngt = (G.ga >= 0 && G.kind_b) ? 2 : 1, w0 = ngt == 2 ? G.order : (G.ga >= 0 ? 0 : 1);
			int st = 0;
			if (g == g0)
			{
				const int w = G.ga == k ? 0 : 1;
				for (unsigned i = 0; i < its; i++)
					fit_move<P>(G, w, x, tc, fit_base(G, bs, u0 + i * FIT_NT, par), cg + i * FIT_NT, true);
				st = w == w0 ? 1 : 2;
			}
			else
			{
				const T* tab = G.flush >= 0 ? a.tables + (size_t)(2 * G.flush + par) * a.S + u0 : nullptr;
				for (unsigned i = 0; i < its; i++)
					fit_group<P, QC, false, 1>(G, stage[g & 1].gate, tc, fit_base(G, bs, u0 + i * FIT_NT, par), tab ? tab + i * FIT_NT : nullptr, nullptr, 0);
			}
#pragma unroll 1
			for (; st < ngt; st++)
			{
				const int w = w0 ^ st;
				const int blk = w ? G.blk_b : G.blk_a;
				const double wg = wrow[w ? G.gb : G.ga];
				if (cblk != blk || cw != wg) flush();
				if (merged >= FIT_RENORM)
				{
#pragma unroll
					for (int e = 0; e < 8; e++) P::acc_norm(acc[e]);
					merged = 0;
				}
				cblk = blk; cw = wg;
				merged += 4 * (int)max(its, 1u);
				for (unsigned i = 0; i < its; i++)
				{
					const unsigned base = fit_base(G, bs, u0 + i * FIT_NT, par);
					fit_contract<P, true, false, 1>(G, w, w, tc, base, eg + i * FIT_NT, acc, nullptr, 0);
					if (blk == grp) fit_move<P>(G, w, x, tc, base, cg + i * FIT_NT, false);
				}
			}
			fit_stage_wait();
			__syncthreads();
		}
		flush();
	}
}

// complex products in double-double, for the factors (on the host) and the tables of complex128
// (every entry correctly rounded to a few 2^-100, so that the tables carry no common rounding
// error into all columns)
struct Dd { double h, l; };
__host__ __device__ __forceinline__ Dd dd_add(Dd a, Dd b)
{
	const double s = a.h + b.h, bb = s - a.h, e = (a.h - (s - bb)) + (b.h - bb) + (a.l + b.l);
	Dd r;
	r.h = s + e;
	r.l = e - (r.h - s);
	return r;
}
__host__ __device__ __forceinline__ Dd dd_mul(Dd a, Dd b)
{
	const double p = a.h * b.h, e = fma(a.h, b.h, -p) + (a.h * b.l + a.l * b.h);
	Dd r;
	r.h = p + e;
	r.l = e - (r.h - p);
	return r;
}
__host__ __device__ __forceinline__ Dd dd_neg(Dd a) { a.h = -a.h; a.l = -a.l; return a; }

// one diagonal factor: entry 2 bit_i + bit_j (bits si, sj of the full index), (re, im) as
// double-double
struct FitDiag { double v[4][4]; int si, sj; };

// product of the factors beg..end at a full basis index
template <class P>
__device__ __forceinline__ typename P::T fit_table_entry(const FitDiag* __restrict__ diag, int beg, int end, unsigned long full)
{
	Dd re = { 1, 0 }, im = { 0, 0 };
	for (int d = beg; d < end; d++)
	{
		const FitDiag& D = diag[d];
		const double* v = D.v[2 * ((full >> D.si) & 1) + ((full >> D.sj) & 1)];
		if (P::kId == MG_PREC_FP64_ID)
		{
			const Dd a = { v[0], v[1] }, b = { v[2], v[3] };
			const Dd r = dd_add(dd_mul(re, a), dd_neg(dd_mul(im, b)));
			im = dd_add(dd_mul(re, b), dd_mul(im, a));
			re = r;
		}
		else
		{
			const double r = re.h * v[0] - im.h * v[2];
			im.h = re.h * v[2] + im.h * v[0];
			re.h = r;
		}
	}
	return P::make(re.h, im.h);
}

// entry (parity, position) of every flush's table and of the final one (flush == nflush)
template <class P>
__global__ void k_fit_tables(const FitDiag* __restrict__ diag, const int* __restrict__ beg, int nflush, const int* __restrict__ group_of,
	const FitGroup* __restrict__ groups, const PassRec* __restrict__ pass, int kt, long S, typename P::T* __restrict__ tables)
{
	const int nu = kt - 4;
	for (long q = blockIdx.x * (long)blockDim.x + threadIdx.x; q < 2 * S * (nflush + 1); q += (long)gridDim.x * blockDim.x)
	{
		const int f = (int)(q / (2 * S));
		const long rest = q - f * 2 * S;
		const int par = rest >= S;
		unsigned c = (unsigned)(rest - par * S);
		if (f < nflush)
		{
			// thread order of the flush's group: (tile, register, unit)
			const FitGroup& G = groups[group_of[f]];
			const PassRec& pr = pass[G.pass];
			const unsigned tau = c >> kt, u = c & ((1u << nu) - 1u);
			unsigned k = (c >> nu) & 15u;
			c = nl_base(pr, tau);
			if (G.kind_b == 2 && ((__popc(u) + __popc(c) + par) & 1)) k ^= 8u;
			for (int j = 0; j < 4; j++) c |= ((k >> j) & 1u) << G.cbit[j];
			for (int j = 0; j < nu; j++) c |= ((u >> j) & 1u) << G.cbit[4 + j];
		}
		const unsigned long full = ((unsigned long)c << 1) | ((__popc(c) + par) & 1);
		tables[q] = fit_table_entry<P>(diag, beg[f], beg[f + 1], full);
	}
}

// block gradients and f from the summed R: one block of threads per parameter block, the rows of
// the parts summed by FIT_FIN threads each in a fixed order
constexpr int FIT_FIN = 32;
struct FitBlock { double minv[8][2]; double scale[8][2]; int ngates, pad; };   // see mgcu_fit_build.cuh

__global__ void __launch_bounds__(FIT_FIN * 16) k_fit_finish(const double* __restrict__ part, int nparts, int nblocks, const FitBlock* __restrict__ fb,
	double* __restrict__ out_f, double* __restrict__ out_blk)
{
	__shared__ double sum[FIT_FIN][16];
	const int blk = blockIdx.x, e = threadIdx.x & 15, w = threadIdx.x >> 4;
	double s = 0;
#pragma unroll 4
	for (int r = w; r < nparts; r += FIT_FIN) s += part[((size_t)r * nblocks + blk) * 16 + e];
	sum[w][e] = s;
	__syncthreads();
	if (threadIdx.x >= 16) return;
	s = 0;
	for (int r = 0; r < FIT_FIN; r++) s += sum[r][threadIdx.x];
	__syncwarp(0xffffu);
	sum[0][threadIdx.x] = s;
	__syncwarp(0xffffu);
	const double* R = sum[0];
	// entry q = 4 (corner) + 2 r + t
	if (threadIdx.x < 8)
	{
		const int q = threadIdx.x, h = q & 4, r = (q >> 1) & 1, t = q & 1;
		const FitBlock& B = fb[blk];
		double gr = 0, gi = 0;
		for (int k = 0; k < 2; k++)
		{
			const double* x = R + 2 * (h + 2 * r + k);
			const double* m = B.minv[h + 2 * t + k];
			gr += x[0] * m[0] - x[1] * m[1];
			gi += x[0] * m[1] + x[1] * m[0];
		}
		const double* c = B.scale[q];
		out_blk[blk * 16 + 2 * q] = gr * c[0] - gi * c[1];
		out_blk[blk * 16 + 2 * q + 1] = gr * c[1] + gi * c[0];
	}
	if (blk == 0 && threadIdx.x >= 8 && threadIdx.x < 10 && fb[0].ngates > 0)   // (whole blocks: f has its own sums)
	{
		const int c = threadIdx.x - 8;
		out_f[c] = ((R[0 + c] + R[6 + c]) + (R[8 + c] + R[14 + c])) / fb[0].ngates;
	}
}

// summed parts of the Hessian in moves -> gate entries: both indices transformed as the gradient
__global__ void k_fit_hess_finish(const double2* __restrict__ A, int nb, const FitBlock* __restrict__ fb, double2* __restrict__ H)
{
	const int m = nb * 8;
	for (int q = blockIdx.x * blockDim.x + threadIdx.x; q < m * m; q += gridDim.x * blockDim.x)
	{
		const int r = q / m, c = q % m, bi = r >> 3, bj = c >> 3, x = r & 7, y = c & 7;
		double sr = 0, si = 0;
		for (int u = 0; u < 2; u++)
		{
			const double* mu = fb[bi].minv[(x & 4) + 2 * (x & 1) + u];
			for (int v = 0; v < 2; v++)
			{
				const double* mv = fb[bj].minv[(y & 4) + 2 * (y & 1) + v];
				const double2 e = A[(long)(bi * 8 + (x & 6) + u) * m + bj * 8 + (y & 6) + v];
				const double wr = mu[0] * mv[0] - mu[1] * mv[1], wi = mu[0] * mv[1] + mu[1] * mv[0];
				sr += e.x * wr - e.y * wi;
				si += e.x * wi + e.y * wr;
			}
		}
		const double *ci = fb[bi].scale[x], *cj = fb[bj].scale[y];
		const double wr = ci[0] * cj[0] - ci[1] * cj[1], wi = ci[0] * cj[1] + ci[1] * cj[0];
		H[q] = make_double2(sr * wr - si * wi, sr * wi + si * wr);
	}
}
