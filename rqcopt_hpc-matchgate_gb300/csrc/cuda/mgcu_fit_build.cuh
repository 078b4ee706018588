// Host side of the factored fitted circuit (mgcu_fit.cuh): groups, flushes, factors.
// Included by mgcu_engine.cu.

// most bytes of a program's tables before the final one: of a target's, which live as long as the
// target (64 tables at 18 qubits, where one takes 4 MB), and of a plan's or batch's, a quarter of
// the room in which those stage target columns (512 at 18 qubits)
constexpr size_t FIT_TABLES = (size_t)256 << 20, FIT_PLAN_TABLES = (size_t)2 << 30;

// wires of gate g as a mask
static unsigned fit_wires(const int* w, int g) { return (1u << w[2 * g]) | (1u << w[2 * g + 1]); }

// Passes as for the other sweeps (reordered: commuting gates only), then groups of up to two
// gates within a pass, then flushes: before a group whose right factors are not merged yet, one
// table of all pending left factors and of the right factors of every gate that comes next on
// both of its wires (one flush per brickwall layer when the sector is one tile).  ordered
// (Hessians, unfactored gates): the groups keep the sequence of the gates; unfactored: no flushes.
// Tables of more than `room` bytes are not made: f.built stays false and nothing is kept.
static int fit_build(int L, int kt, const int* wires, int ng, const int* block, int nblocks, int es, bool ordered, bool factored, FitProg& f,
	size_t room, const std::vector<int>& place = {})
{
	const int nb = L - 1;
	const size_t table = (size_t)es * 2 << nb;   // bytes of one table
	f.built = false;
	schedule(L, kt, wires, ng, !ordered, f.sched, es >= 16 ? 1 : 2);
	f.nflush = 0;
	std::vector<std::vector<int>> onq(L);
	for (int g = 0; g < ng; g++) { onq[wires[2 * g]].push_back(g); onq[wires[2 * g + 1]].push_back(g); }
	std::vector<size_t> next(L, 0);
	std::vector<unsigned> bases;
	std::vector<char> cdone(ng, 0);
	std::vector<int> pending;
	f.group.clear(); f.pass_groups.clear(); f.diag.clear(); f.beg.assign(1, 0); f.group_of.clear();
	f.group_of_gate.assign(ng, 0);
	const unsigned pers = es == 16 ? 3 : 4;   // swizzle period of the tile bits
	for (size_t p = 0; p < f.sched.pass.size(); p++)
	{
		const PassRec& pr = f.sched.pass[p];
		FitPass fp;
		fp.gbeg = (int)f.group.size();
		std::vector<int> rest;
		std::vector<const GateRec*> rec(ng, nullptr);
		for (int i = pr.gbeg; i < pr.gend; i++) { rest.push_back(f.sched.gate[i].g); rec[f.sched.gate[i].g] = &f.sched.gate[i]; }
		while (!rest.empty())
		{
			int a = rest[0], b = -1;
			unsigned used = fit_wires(wires, a);
			size_t at = 0;
			for (size_t i = 1; i < rest.size() && b < 0; i++)
			{
				if (!(fit_wires(wires, rest[i]) & used)) { b = rest[i]; at = i; }
				used |= fit_wires(wires, rest[i]);
				if (ordered) break;
			}
			if (b >= 0) rest.erase(rest.begin() + at);
			rest.erase(rest.begin());
			// a gate on the dropped qubit is gate b
			if (rec[a]->type != 0) std::swap(a, b);
			FitGroup G;
			memset(&G, 0, sizeof(G));
			G.ga = a; G.gb = b;
			G.blk_a = a >= 0 ? block[a] : -1;
			G.blk_b = b >= 0 ? block[b] : -1;
			G.kind_b = b < 0 ? 0 : (rec[b]->type == 0 ? 1 : 2);
			G.rev = b >= 0 && rec[b]->type == 2;
			G.pass = (int)p;
			G.order = a >= 0 && b >= 0 && b < a;
			G.blk_next = f.group.empty() ? -1 : (f.group.back().kind_b ? f.group.back().blk_b : f.group.back().blk_a);
			int bits[14], n = 0;
			unsigned in = 0;
			auto take = [&](int lb) { bits[n++] = lb; in |= 1u << lb; };
			int rb[4] = { -1, -1, -1, -1 };
			if (a >= 0) { rb[0] = rec[a]->lb; rb[1] = rec[a]->la; }
			if (G.kind_b == 1) { rb[2] = rec[b]->lb; rb[3] = rec[b]->la; }
			if (G.kind_b == 2) rb[2] = rec[b]->type == 1 ? rec[b]->la : rec[b]->lb;
			for (int j = 0; j < 4; j++) if (rb[j] >= 0) in |= 1u << rb[j];
			for (int j = 0; j < 4; j++)
				if (rb[j] < 0)
				{
					// a free bit: the highest, which the lanes of a wavefront need least
					int q = kt - 1;
					while (in & (1u << q)) q--;
					rb[j] = q;
					in |= 1u << q;
				}
			for (int j = 0; j < 4; j++) bits[n++] = rb[j];
			// unit bits: first the lowest ones of distinct swizzle classes, then the others
			unsigned cls = 0;
			for (int lb = 0; lb < kt; lb++)
				if (!(in & (1u << lb)) && !(cls & (1u << (lb % pers)))) { cls |= 1u << (lb % pers); take(lb); }
			for (int lb = 0; lb < kt; lb++) if (!(in & (1u << lb))) take(lb);
			unsigned tm[10];
			for (int j = 0; j < kt; j++)
			{
				G.cbit[j] = pr.lbits[bits[j]];
				const unsigned off = (es == 16 ? fsw<16>(1u << bits[j]) : fsw<8>(1u << bits[j])) * (unsigned)es;
				if (j < 4) G.m[j] = off; else tm[j - 4] = off;
			}
			for (unsigned u = 0; u < (1u << (kt - 4)); u++)
			{
				unsigned o = 0;
				for (int j = 0; j < kt - 4; j++) if (u & (1u << j)) o ^= tm[j];
				bases.push_back(o);
			}
			auto slot = [&](int k) {
				unsigned o = 0;
				for (int j = 0; j < 4; j++) if (k & (1 << j)) o ^= G.m[j];
				return o;
			};
			for (int w = 0; w < 2; w++)
				for (int i = 0; i < 4; i++)
				{
					int k[4];   // registers of |00>, |01>, |10>, |11>
					if (w == 0) for (int j = 0; j < 4; j++) k[j] = 4 * i + j;
					else if (G.kind_b != 2) for (int j = 0; j < 4; j++) k[j] = i + 4 * j;
					else
					{
						// pairs along bit 2: corner where bits 0, 1, 3 have even parity
						k[0] = (0xA930 >> (4 * i)) & 15;
						k[3] = k[0] | 4;
						k[1] = G.rev ? (k[0] ^ 5) : (k[0] ^ 1);
						k[2] = G.rev ? (k[0] ^ 1) : (k[0] ^ 5);
					}
					const unsigned us = (1u << (kt - 4)) * (unsigned)es;
					G.qs[w][i] = make_uint4(slot(k[0]), slot(k[1]), slot(k[2]), slot(k[3]));
					G.qy[w][i] = make_uint4(k[0] * us, k[1] * us, k[2] * us, k[3] * us);
				}
			// flush
			G.flush = -1;
			bool need = false;
			for (int s : { a, b })
				if (s >= 0) need = need || (factored && !cdone[s]);
			if (need)
			{
				G.flush = f.nflush++;
				if (f.nflush * table > room) { f.release(); return 0; }
				f.group_of.push_back((int)f.group.size());
				for (int s : pending) f.diag.push_back({ s, 0 });
				pending.clear();
				for (int q = 0; q < L; q++)
				{
					if (next[q] >= onq[q].size()) continue;
					const int s = onq[q][next[q]], o = wires[2 * s] == q ? wires[2 * s + 1] : wires[2 * s];
					if (cdone[s] || next[o] >= onq[o].size() || onq[o][next[o]] != s) continue;
					cdone[s] = 1;
					f.diag.push_back({ s, 1 });
				}
				f.beg.push_back((int)f.diag.size());
			}
			for (int s : { a, b })
				if (s >= 0)
				{
					f.group_of_gate[s] = (int)f.group.size();
					pending.push_back(s);
					next[wires[2 * s]]++; next[wires[2 * s + 1]]++;
				}
			f.group.push_back(G);
		}
		fp.gend = (int)f.group.size();
		f.pass_groups.push_back(fp);
	}
	for (int s : pending) f.diag.push_back({ s, 0 });
	f.beg.push_back((int)f.diag.size());
	f.block_gates.assign(nblocks, 0);
	for (int g = 0; g < ng; g++) f.block_gates[block[g]]++;
	const int U = 1 << (kt - 4);
	f.threads = (U >= 512 && es == 16) ? 512 : U >= 256 ? 256 : 128;
	f.kt = kt;
	f.factored = factored;
	f.nc = (U < 128 && nb <= kt) ? 128 / U : 1;   // small sectors share a block
	// gradients of few columns: four threads per unit and a fourth of the columns per block, while
	// that leaves blocks unused otherwise
	f.split = (factored && nb <= kt && U <= 32 && (1L << L) / f.nc < mgcu_ctx()->nsm) ? 4 : 1;
	f.ncb = f.split > 1 ? f.nc / f.split : f.nc;
	f.smem = (size_t)f.nc * ((size_t)1 << kt) * es + 2 * 128 * sizeof(unsigned) + red_bytes(f.threads);
	std::vector<int> pg;
	for (int q : place) pg.push_back(f.group_of_gate[q]);
	Arena ar(f.fixed);
	ar.add(f.d_pass, f.sched.pass.data(), sizeof(PassRec) * f.sched.pass.size());
	ar.add(f.d_group, f.group.data(), sizeof(FitGroup) * f.group.size());
	ar.add(f.d_pgroups, f.pass_groups.data(), sizeof(FitPass) * f.pass_groups.size());
	ar.add(f.d_beg, f.beg.data(), sizeof(int) * f.beg.size());
	ar.add(f.d_gof, f.group_of.data(), sizeof(int) * f.group_of.size());
	ar.add(f.d_bases, bases.data(), sizeof(unsigned) * bases.size());
	ar.add(f.d_pgroup, pg.data(), sizeof(int) * pg.size());
	int e = ar.up();
	if (!e) e = f.d_tab.alloc(table * (f.nflush + 1));
	if (e) return e;
	MGCU_TRY(cudaStreamSynchronize(mgcu_stream()));
	f.built = true;
	return 0;
}

// complex arithmetic in double-double for the factors
static Dd hdd(double x) { return { x, 0 }; }
static Dd hdiv(Dd a, Dd b)
{
	const double q = a.h / b.h;
	const Dd r = dd_add(a, dd_neg(dd_mul(hdd(q), b)));
	const double q2 = r.h / b.h;
	const double s = q + q2;
	return { s, q2 - (s - q) };
}
struct Hcx { Dd re, im; };
static Hcx hcx(mgc z) { return { hdd(z.re), hdd(z.im) }; }
static Hcx cmul(Hcx a, Hcx b)
{
	return { dd_add(dd_mul(a.re, b.re), dd_neg(dd_mul(a.im, b.im))), dd_add(dd_mul(a.re, b.im), dd_mul(a.im, b.re)) };
}
static Hcx cscale(Hcx a, double s) { return { dd_mul(a.re, hdd(s)), dd_mul(a.im, hdd(s)) }; }
static Hcx cdiv(Hcx a, Hcx b)
{
	const Dd d = dd_add(dd_mul(b.re, b.re), dd_mul(b.im, b.im));
	const Hcx n = cmul(a, { b.re, dd_neg(b.im) });
	return { hdiv(n.re, d), hdiv(n.im, d) };
}

struct FitFactor { double p; mgc q; int sw; Hcx l[2], r[2]; };

// diag(l) M diag(r) of a 2x2 block (entries a, b, c, d), r[0] = 1; false (general kernels) when an
// entry is not finite or far from one, when an entry that M is scaled by is small (under a
// quarter of the largest; at least 0.7 in a unitary block) or M is near singular.  p has 64
// candidates around |b / a| (|a / b| when swapped): p q = bc / (ad) is fixed, and the candidate
// whose q rounds best leaves no rounding of the factors common to all amplitudes.
static bool fit_factor(const mgc* e, FitFactor& F)
{
	double ab[4], mx = 0;
	for (int k = 0; k < 4; k++)
	{
		ab[k] = std::hypot(e[k].re, e[k].im);
		if (!(ab[k] < 1e3)) return false;   // infinities and NaN too
		mx = std::max(mx, ab[k]);
	}
	if (mx < 1e-3) return false;
	F.sw = ab[1] * ab[2] > ab[0] * ab[3];
	// pivots (u, v) scaled to 1 and the others: unswapped M = [[1, p], [q, 1]], u = a, v = d
	const int iu = F.sw ? 1 : 0, iv = F.sw ? 2 : 3, ip = F.sw ? 0 : 1, iq = F.sw ? 3 : 2;
	if (ab[iu] < mx / 4 || ab[iv] < mx / 4) return false;
	const Hcx u = hcx(e[iu]), v = hcx(e[iv]), ep = hcx(e[ip]), eq = hcx(e[iq]);
	const Hcx one = { hdd(1), hdd(0) };
	const Hcx k = cdiv(cmul(ep, eq), cmul(u, v));   // p q
	F.p = 0;
	if (ab[ip] > 1e-100)
	{
		const double p0 = ab[ip] / ab[iu];
		double best = -1, p = p0;
		for (int c = 0; c < 64; c++)
		{
			const double q = k.re.h / p, r = std::fabs(std::fma(-q, p, k.re.h) + k.re.l);
			if (best < 0 || r < best) { best = r; F.p = p; }
			p = std::nextafter(p, 2 * p0);
		}
	}
	F.r[0] = one;
	if (!F.sw)
	{
		// a = l0, b = l0 p r1, c = l1 q, d = l1 r1
		F.l[0] = u;
		F.r[1] = F.p > 0 ? cdiv(ep, cscale(u, F.p)) : one;
		F.l[1] = cdiv(v, F.r[1]);
	}
	else
	{
		// a = l0 p, b = l0 r1, c = l1, d = l1 q r1
		F.l[1] = v;
		F.r[1] = F.p > 0 ? cdiv(cscale(u, F.p), ep) : one;
		F.l[0] = cdiv(u, F.r[1]);
	}
	const Hcx q = cdiv(eq, F.sw ? cmul(F.l[1], F.r[1]) : F.l[1]);
	F.q = mgc_make(q.re.h, q.im.h);
	const double dr = 1 - F.p * F.q.re, di = -F.p * F.q.im;
	return std::hypot(dr, di) > 0.125 && std::hypot(F.q.re, F.q.im) < 8 && F.p < 8;
}

// Levels, pair tables and row positions for the number sectors (see mgcu_wsec.cuh): w.built when
// the largest sector leaves two blocks per SM (L <= 14) and the gates fit in shared memory.
// Columns per block: up to eight, as many as fit.
template <class P>
static int ws_build(int L, const int* wires, int ng, const std::vector<int>& place, WsProg& w)
{
	typedef typename P::T T;
	if (L > 14 || L < 4 || ng > WS_MAXG) return 0;
	auto bit = [&](int q) { return 1u << (L - 1 - q); };
	const unsigned N = 1u << L;
	// rows by (ones, index)
	w.rstart.assign(L + 2, 0);
	for (unsigned a = 0; a < N; a++) w.rstart[__builtin_popcount(a) + 1]++;
	for (int n = 0; n <= L; n++) w.rstart[n + 1] += w.rstart[n];
	w.rows.assign(N, 0);
	std::vector<int> row(N), fill(w.rstart);
	for (unsigned a = 0; a < N; a++)
	{
		const int n = __builtin_popcount(a), q = fill[n]++;
		w.rows[q] = a;
		row[a] = q - w.rstart[n];
	}
	w.dmax = 0;
	for (int n = 0; n <= L; n++) w.dmax = std::max(w.dmax, w.rstart[n + 1] - w.rstart[n]);
	const size_t room = 107000;
	w.ln = 0;
	while (w.ln < 3 && ((size_t)w.dmax << (w.ln + 1)) * sizeof(T) <= room) w.ln++;
	w.smem = ((size_t)w.dmax << w.ln) * sizeof(T);
	if (w.smem > room) return 0;
	// other wires' values by (ones, value)
	w.pstart.assign(L, 0);
	std::vector<unsigned> order(N >> 2);
	for (unsigned q = 0; q < (N >> 2); q++) order[q] = q;
	std::stable_sort(order.begin(), order.end(), [](unsigned x, unsigned y) { return __builtin_popcount(x) < __builtin_popcount(y); });
	for (unsigned q = 0; q < (N >> 2); q++) w.pstart[__builtin_popcount(q) + 1]++;
	for (int m = 0; m + 1 < L; m++) w.pstart[m + 1] += w.pstart[m];
	std::map<std::pair<int, int>, int> id;
	std::vector<ushort4> pairs;
	w.pair_of.assign(ng, 0);
	for (int g = 0; g < ng; g++)
	{
		const auto ins = id.emplace(std::make_pair(wires[2 * g], wires[2 * g + 1]), (int)id.size());
		w.pair_of[g] = ins.first->second;
		if (!ins.second) continue;
		const unsigned bi = bit(wires[2 * g]), bj = bit(wires[2 * g + 1]), lo = std::min(bi, bj), hi = std::max(bi, bj);
		for (unsigned q : order)
		{
			unsigned a = ((q & ~(lo - 1)) << 1) | (q & (lo - 1));
			a = ((a & ~(hi - 1)) << 1) | (a & (hi - 1));
			pairs.push_back(make_ushort4((unsigned short)row[a], (unsigned short)row[a | bj], (unsigned short)row[a | bi], (unsigned short)row[a | bi | bj]));
		}
	}
	// levels: runs of gates on disjoint wires; each level's table holds the left factors of the
	// level before and its own right factors
	std::vector<WsLevel> lev;
	w.level_of.assign(ng, 0);
	w.diag.clear();
	w.beg.assign(1, 0);
	for (int g = 0; g < ng;)
	{
		WsLevel V;
		V.gbeg = g;
		unsigned used = 0;
		while (g < ng && !(fit_wires(wires, g) & used)) { used |= fit_wires(wires, g); w.level_of[g++] = (int)lev.size(); }
		V.gend = g;
		if (!lev.empty()) for (int s = lev.back().gbeg; s < lev.back().gend; s++) w.diag.push_back({ s, 0 });
		for (int s = V.gbeg; s < V.gend; s++) w.diag.push_back({ s, 1 });
		w.beg.push_back((int)w.diag.size());
		lev.push_back(V);
	}
	for (int s = lev.back().gbeg; s < lev.back().gend; s++) w.diag.push_back({ s, 0 });
	w.beg.push_back((int)w.diag.size());
	w.nlev = (int)lev.size();
	std::vector<int> pl;
	for (int q : place) pl.push_back(w.level_of[q]);
	Arena ar(w.fixed);
	ar.add(w.d_levels, lev.data(), sizeof(WsLevel) * lev.size());
	ar.add(w.d_pairs, pairs.data(), sizeof(ushort4) * pairs.size());
	ar.add(w.d_rows, w.rows.data(), sizeof(unsigned) * N);
	ar.add(w.d_beg, w.beg.data(), sizeof(int) * w.beg.size());
	ar.add(w.d_plevel, pl.data(), sizeof(int) * pl.size());
	int e = ar.up();
	if (!e) e = w.d_tab.alloc(sizeof(T) * (size_t)N * (w.nlev + 1));
	if (!e) e = w.d_sec.alloc(sizeof(WsSec) * (L + 1));
	if (e) return e;
	MGCU_TRY(cudaStreamSynchronize(mgcu_stream()));
	for (auto k : { k_ws_grad<P, true>, k_ws_grad<P, false> }) MGCU_TRY(cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)room));
	for (auto k : { k_ws_hess<P, true>, k_ws_hess<P, false> }) MGCU_TRY(cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)room));
	w.built = true;
	return 0;
}

// one diagonal factor of a gate for the tables (side 0: left, 1: right)
static FitDiag fit_diag(const FitFactor& c, const FitFactor& k, int side, int wi, int wj, int L)
{
	const Hcx* fc = side ? c.r : c.l;
	const Hcx* fk = side ? k.r : k.l;
	const Hcx ent[4] = { fk[0], fc[0], fc[1], fk[1] };   // |00>, |01>, |10>, |11>
	FitDiag d;
	for (int q = 0; q < 4; q++)
	{
		d.v[q][0] = ent[q].re.h; d.v[q][1] = ent[q].re.l;
		d.v[q][2] = ent[q].im.h; d.v[q][3] = ent[q].im.l;
	}
	d.si = L - 1 - wi; d.sj = L - 1 - wj;
	return d;
}

// the number sectors' gates and tables; w.ok when every corner block is exactly diagonal
template <class P>
static int ws_set_gates(const mgg* gates, int ng, const int* block, int L, const int* wires, const std::vector<FitFactor>& fac, WsProg& w)
{
	typedef typename P::T T;
	w.ok = false;
	for (int g = 0; g < ng; g++)
		if (gates[g].k[1].re != 0 || gates[g].k[1].im != 0 || gates[g].k[2].re != 0 || gates[g].k[2].im != 0) return 0;
	std::vector<WsGate<T>> hg(ng);
	for (int g = 0; g < ng; g++)
	{
		const FitFactor& c = fac[2 * block[g]];
		hg[g].p = P::make(c.p, 0); hg[g].q = P::make(c.q.re, c.q.im);
		hg[g].sw = c.sw; hg[g].pair = w.pair_of[g]; hg[g].blk = block[g]; hg[g].pad = 0;
	}
	std::vector<FitDiag> hd;
	for (const auto& d : w.diag) hd.push_back(fit_diag(fac[2 * block[d[0]]], fac[2 * block[d[0]] + 1], d[1], wires[2 * d[0]], wires[2 * d[0] + 1], L));
	cudaStream_t st = mgcu_stream();
	Arena av(w.values);
	av.add(w.d_gates, hg.data(), sizeof(WsGate<T>) * ng);
	av.add(w.d_diag, hd.data(), sizeof(FitDiag) * hd.size());
	const int ev = av.up();
	if (ev) return ev;
	k_ws_tables<P><<<grid_cap((long)(w.nlev + 1) << L, 128), 128, 0, st>>>(w.d_diag.as<FitDiag>(), w.d_beg.as<int>(), w.nlev, L, w.d_rows.as<unsigned>(),
		w.d_tab.as<T>());
	MGCU_LAUNCHED();
	w.ok = true;
	return 0;
}

// factors, tables and end transforms of the current gates; f.ok tells whether they factor
template <class P>
static int fit_set_gates(const mgg* gates, int ng, const int* block, int nblocks, int L, int kt, const int* wires, FitProg& f)
{
	typedef typename P::T T;
	f.ok = false;
	if (!f.factored)
	{
		std::vector<FitWhole<T>> hw(2 * f.group.size());
		memset(hw.data(), 0, sizeof(FitWhole<T>) * hw.size());
		for (size_t i = 0; i < hw.size(); i++)
		{
			const int g = i & 1 ? f.group[i / 2].gb : f.group[i / 2].ga;
			if (g < 0) continue;
			for (int q = 0; q < 4; q++)
			{
				hw[i].c[q] = P::make(gates[g].c[q].re, gates[g].c[q].im);
				hw[i].k[q] = P::make(gates[g].k[q].re, gates[g].k[q].im);
			}
		}
		std::vector<FitBlock> fb(nblocks);
		memset(fb.data(), 0, sizeof(FitBlock) * nblocks);   // the sums are the gradients
		for (FitBlock& b : fb)
			for (int h = 0; h < 8; h++) { b.scale[h][0] = 1; b.minv[h][0] = (h & 3) == 0 || (h & 3) == 3; }
		Arena av(f.values);
		av.add(f.d_gates, hw.data(), sizeof(FitWhole<T>) * hw.size());
		av.add(f.d_blk, fb.data(), sizeof(FitBlock) * nblocks);
		const int e = av.up();
		f.qc = 2;
		f.ok = e == 0;
		return e;
	}
	std::vector<int> first(nblocks, -1);
	for (int g = 0; g < ng; g++)
	{
		if (first[block[g]] < 0) first[block[g]] = g;
		else if (memcmp(&gates[g], &gates[first[block[g]]], sizeof(mgg))) return 0;   // a block's gates must be equal
	}
	std::vector<FitFactor> fac(2 * nblocks);
	double qi = 0;
	std::vector<FitBlock> fb(nblocks);
	memset(fb.data(), 0, sizeof(FitBlock) * nblocks);
	for (int b = 0; b < nblocks; b++)
	{
		if (first[b] < 0) continue;
		fb[b].ngates = f.block_gates[b];
		for (int h = 0; h < 2; h++)
		{
			FitFactor& F = fac[2 * b + h];
			if (!fit_factor(h ? gates[first[b]].k : gates[first[b]].c, F)) return 0;
			qi = std::max(qi, std::fabs(F.q.im));
			// inverse of M and 1 / (l_r r_t)
			const mgc det = mgc_make(1 - F.p * F.q.re, -F.p * F.q.im);
			const double d2 = det.re * det.re + det.im * det.im;
			const mgc id = mgc_make(det.re / d2, -det.im / d2), one = mgc_make(1, 0), p = mgc_make(F.p, 0);
			auto neg = [](mgc z) { return mgc_make(-z.re, -z.im); };
			const mgc mi[4] = { F.sw ? neg(F.q) : one, F.sw ? one : neg(p), F.sw ? one : neg(F.q), F.sw ? neg(p) : one };
			for (int k = 0; k < 4; k++)
			{
				const mgc m = mgc_mul(mi[k], id);
				fb[b].minv[4 * h + k][0] = m.re; fb[b].minv[4 * h + k][1] = m.im;
				const Hcx s = cdiv({ hdd(1), hdd(0) }, cmul(F.l[k >> 1], F.r[k & 1]));
				fb[b].scale[4 * h + k][0] = s.re.h; fb[b].scale[4 * h + k][1] = s.im.h;
			}
		}
	}
	// beyond the rounding of a unitary block q keeps its imaginary part (complex128: always)
	f.qc = qi > (P::kId == MG_PREC_FP64_ID ? 0.0 : 1e-15);
	std::vector<FitGate<T>> hg(2 * f.group.size());
	memset(hg.data(), 0, sizeof(FitGate<T>) * hg.size());
	for (size_t i = 0; i < hg.size(); i++)
	{
		const int g = i & 1 ? f.group[i / 2].gb : f.group[i / 2].ga;
		if (g < 0) continue;
		const FitFactor &c = fac[2 * block[g]], &k = fac[2 * block[g] + 1];
		hg[i].pc = P::make(c.p, 0); hg[i].qc = P::make(c.q.re, c.q.im);
		hg[i].pk = P::make(k.p, 0); hg[i].qk = P::make(k.q.re, k.q.im);
		hg[i].swc = c.sw; hg[i].swk = k.sw;
	}
	std::vector<FitDiag> hd(f.diag.size());
	for (size_t i = 0; i < hd.size(); i++)
	{
		const int g = f.diag[i][0];
		hd[i] = fit_diag(fac[2 * block[g]], fac[2 * block[g] + 1], f.diag[i][1], wires[2 * g], wires[2 * g + 1], L);
	}
	cudaStream_t st = mgcu_stream();
	Arena av(f.values);
	av.add(f.d_gates, hg.data(), sizeof(FitGate<T>) * hg.size());
	av.add(f.d_diag, hd.data(), sizeof(FitDiag) * hd.size());
	av.add(f.d_blk, fb.data(), sizeof(FitBlock) * nblocks);
	const int ev = av.up();
	if (ev) return ev;
	f.ws.ok = false;
	if constexpr (P::kId != MG_PREC_FP32_ID)
		if (f.ws.built)
		{
			const int e = ws_set_gates<P>(gates, ng, block, L, wires, fac, f.ws);
			if (e) return e;
		}
	const long S = 1L << (L - 1);
	k_fit_tables<P><<<grid_cap(2 * S * (f.nflush + 1), 128), 128, 0, st>>>(f.d_diag.as<FitDiag>(), f.d_beg.as<int>(), f.nflush, f.d_gof.as<int>(),
		f.d_group.as<FitGroup>(), f.d_pass.as<PassRec>(), kt, S, f.d_tab.as<T>());
	MGCU_LAUNCHED();
	f.ok = true;
	return 0;
}

template <class P, int NT, int SP>
static void (*fit_kernel_nt(int qc, int mode))(FitArgs<P>)
{
	if constexpr (P::kId == MG_PREC_FP32_ID)
		return mode == FIT_COLS ? k_fit<P, 2, FIT_COLS, NT, 1> : mode == FIT_GRAD ? k_fit<P, 2, FIT_GRAD, NT, 1> : k_fit<P, 2, FIT_VALUE, NT, 1>;
	else if (qc)
		return mode == FIT_COLS ? k_fit<P, 1, FIT_COLS, NT, 1> : mode == FIT_GRAD ? k_fit<P, 1, FIT_GRAD, NT, SP>
			: mode == FIT_HESS ? k_fit<P, 1, FIT_HESS, NT, SP> : k_fit<P, 1, FIT_VALUE, NT, 1>;
	else
		return mode == FIT_COLS ? k_fit<P, 0, FIT_COLS, NT, 1> : mode == FIT_GRAD ? k_fit<P, 0, FIT_GRAD, NT, SP>
			: mode == FIT_HESS ? k_fit<P, 0, FIT_HESS, NT, SP> : k_fit<P, 0, FIT_VALUE, NT, 1>;
}
template <class P>
static void (*fit_kernel(int qc, int mode, int threads, int split = 1))(FitArgs<P>)
{
	return threads == 512 ? fit_kernel_nt<P, 512, 1>(qc, mode) : threads == 256 ? fit_kernel_nt<P, 256, 1>(qc, mode)
		: split > 1 ? fit_kernel_nt<P, 128, 4>(qc, mode) : fit_kernel_nt<P, 128, 1>(qc, mode);
}

// k_fit's arguments that come from a program
template <class P>
static FitArgs<P> fit_args(const FitProg& f, int L)
{
	typedef typename P::T T;
	FitArgs<P> w;
	memset(&w, 0, sizeof(w));
	w.L = L; w.nb = L - 1; w.kt = f.kt; w.npass = (int)f.sched.pass.size(); w.ngroups = (int)f.group.size(); w.nc = w.ncs = f.nc;
	w.S = 1L << (L - 1);
	w.pass = f.d_pass.as<PassRec>(); w.groups_of = f.d_pgroups.as<FitPass>(); w.groups = f.d_group.as<FitGroup>();
	w.bases = f.d_bases.as<unsigned>();
	w.gates = f.d_gates.as<char>(); w.tables = f.d_tab.as<T>(); w.final = w.tables + (size_t)2 * w.S * f.nflush;
	return w;
}

// The columns of a circuit target by k_fit, for targets that don't conserve particle numbers:
// factored blocks in complex128 and float-float; in FP32 whole blocks in k_target's order (the
// same bits), when every block is general there.  f.grid: resident blocks.  Where it does not
// apply (f.built stays false: gates that do not factor, tables past FIT_TABLES or with no memory
// left for them) the tiled sweep runs, which needs none of it, and nothing is kept here.
template <class P>
static int target_fit(mgcu_target* t, TargetProg& tp, FitProg& f)
{
	constexpr int es = sizeof(typename P::T);
	if (f.built || f.tried) return 0;
	f.tried = true;
	const int ng = (int)tp.sched.gate.size();
	if (ng < 1 || t->L > 18 || t->L < 10) return 0;
	for (unsigned m : t->smask) if (m) return 0;
	const bool factored = P::kId != MG_PREC_FP32_ID;
	std::vector<mgg> g(ng);
	std::vector<int> w(2 * ng), block(ng);
	std::map<int, int> id;
	for (int i = 0; i < ng; i++)
	{
		const int q = tp.sched.gate[i].g;
		g[i] = t->sg[q];
		w[2 * i] = t->sw[2 * q]; w[2 * i + 1] = t->sw[2 * q + 1];
		block[i] = id.emplace(tp.first[q], (int)id.size()).first->second;
		if (!factored && ((tp.kw[q] & 7) != BK_GEN || ((tp.kw[q] >> 3) & 7) != BK_GEN)) return 0;
	}
	const int nb = t->L - 1;
	int e = fit_build(t->L, std::min(nb, es == 16 ? (nb <= 13 ? 13 : 12) : 13), w.data(), ng, block.data(), (int)id.size(), es, !factored, factored, f, FIT_TABLES);
	if (!e && !f.built) return 0;
	if (!e) e = fit_set_gates<P>(g.data(), ng, block.data(), (int)id.size(), t->L, f.kt, w.data(), f);
	if (e || !f.ok)
	{
		f.release();
		if (e == MG_ERR_ALLOC) { cudaGetLastError(); e = 0; }
		return e;
	}
	int per = 0;
	const int lim = (int)std::min<size_t>(mgcu_ctx()->smem_optin, 227 * 1024) - 4096;
	MGCU_TRY(cudaFuncSetAttribute(fit_kernel<P>(f.qc, FIT_COLS, f.threads), cudaFuncAttributeMaxDynamicSharedMemorySize, lim));
	MGCU_TRY(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per, fit_kernel<P>(f.qc, FIT_COLS, f.threads), f.threads, f.smem));
	f.grid = mgcu_ctx()->nsm * std::max(per, 1);
	MGCU_TRY(cudaStreamSynchronize(mgcu_stream()));   // kept on the target: other threads' streams use it too
	return 0;
}

template <class P>
static void (*fit_hess_kernel(int qc, int threads))(FitHessArgs<P>, long)
{
	return threads == 512 ? (qc ? k_fit_hess<P, 1, 512> : k_fit_hess<P, 0, 512>)
		: threads == 256 ? (qc ? k_fit_hess<P, 1, 256> : k_fit_hess<P, 0, 256>)
		: (qc ? k_fit_hess<P, 1, 128> : k_fit_hess<P, 0, 128>);
}
