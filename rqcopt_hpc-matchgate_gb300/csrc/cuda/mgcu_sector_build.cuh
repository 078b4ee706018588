// Host side of the sector sweep (mgcu_sector.cuh): sectors, row lists and gate program of a
// target.  Included by mgcu_engine.cu.

template <class P>
static void (*sector_kernel(int threads))(SecArgs<P>)
{
	return threads == 1024 ? k_sector<P, 1024, 1> : threads == 512 ? k_sector<P, 512, 2> : k_sector<P, 256, 4>;
}

// Order the entries of a list so that each run of m (the list entries that one shared-memory
// wavefront touches) has distinct rows mod m for both of its members: entries are bucketed by
// (y mod m, z mod m) and each run takes, for every y class, the fullest bucket of a z class not
// yet in the run; what does not match fills up the run.  Lists of single rows have z = y.
static void sector_order(std::vector<unsigned>& v, size_t beg, size_t end, int m, bool pairs)
{
	if (m <= 1 || end - beg <= (size_t)m) return;
	std::vector<std::vector<unsigned>> bucket(m * m);
	for (size_t i = beg; i < end; i++)
	{
		const int y = (int)((v[i] & 0x7fffu) % m), z = pairs ? (int)((v[i] >> 16) % m) : y;
		bucket[y * m + z].push_back(v[i]);
	}
	size_t o = beg;
	int rot = 0;
	while (o < end)
	{
		unsigned usedz = 0;
		int got = 0;
		for (int k = 0; k < m; k++)
		{
			const int y = (k + rot) % m;
			int best = -1;
			for (int z = 0; z < m; z++)
				if (!(usedz & (1u << z)) && !bucket[y * m + z].empty() && (best < 0 || bucket[y * m + z].size() > bucket[y * m + best].size()))
					best = z;
			if (best < 0) continue;
			v[o++] = bucket[y * m + best].back();
			bucket[y * m + best].pop_back();
			usedz |= 1u << best;
			got++;
		}
		rot++;
		while (got < m && o < end)
		{
			size_t big = 0;
			for (size_t q = 1; q < bucket.size(); q++) if (bucket[q].size() > bucket[big].size()) big = q;
			if (bucket[big].empty()) break;
			v[o++] = bucket[big].back();
			bucket[big].pop_back();
			got++;
		}
	}
}

// columns per block (log2) of a sector of d rows: as many as fit in `room` amplitudes, up to 8,
// within `share` amplitudes
static int sector_columns(long d, size_t room, double share)
{
	int ln = 0;
	while (ln < 3 && ((size_t)d << (ln + 1)) <= room && (double)(d << (ln + 1)) <= share) ln++;
	return ln;
}

// The amplitudes a block may hold: a resident block's share of the trace (slots: resident
// blocks) times 2, 1, 1/2 or 1/4.  More columns per block cost a gate's fixed overhead (worth
// `fixed` amplitudes: barrier, step record; little in FP64, whose pipe hides it) less often,
// fewer leave smaller last blocks: the choice is the one whose blocks, handed out largest
// first, finish first.  Measured on whole traces (per sweep, share factor 2 / 1 / 1/2 / 1/4):
// spinless L=10 float-float 0.54 / 0.74 / 0.78 / 0.78 ms, spinful L=12 complex128 6.4 / 5.3 /
// 5.4 / 6.1 ms.  Traces of many more blocks than slots take factor 1.
static double sector_share(const std::vector<int>& order, const std::vector<int>& dim, size_t room, int slots, long fixed)
{
	double work = 0;
	for (int k : order) work += (double)dim[k] * dim[k];
	const double share = work / slots;
	double best = -1, pick = share;
	for (double f : { 1.0, 2.0, 0.5, 0.25 })
	{
		long blocks = 0;
		for (int k : order) blocks += (dim[k] + (1 << sector_columns(dim[k], room, f * share)) - 1) >> sector_columns(dim[k], room, f * share);
		if (blocks > 8L * slots) break;
		std::priority_queue<long, std::vector<long>, std::greater<long>> end;
		for (int i = 0; i < slots; i++) end.push(0);
		long last = 0;
		for (int k : order)
		{
			const int ln = sector_columns(dim[k], room, f * share);
			for (int i = 0; i < (dim[k] + (1 << ln) - 1) >> ln; i++)
			{
				const long t = end.top() + fixed + ((long)dim[k] << ln);
				end.pop();
				end.push(t);
				last = std::max(last, t);
			}
		}
		if (best < 0 || last < best) { best = last; pick = f * share; }
	}
	return pick;
}

// Build the target's sector program (sp.state 1), or find that it does not apply (0): a sector
// must fit in one block's shared memory, and the tables stay small (at most 4096 sectors and
// 2^24 basis indices listed, about 20 ms of host work).  Block shape by the largest sector:
// four blocks of 256 threads per SM while a column takes at most 54 KB, two of 512 up to
// 111 KB, one of 1024 up to 225 KB, always 1024 threads of at most 64 registers per SM.
template <class P>
static int build_sector(mgcu_target* t, TargetProg& tp, SectorProg& sp)
{
	constexpr size_t ES = sizeof(typename P::T);
	sp.state = 0;
	const int L = t->L;
	if (!tp.wcons || L > 18) return 0;
	const std::vector<mgg>& gates = t->sg;
	const int ng = (int)gates.size();
	const unsigned N = 1u << L;
	auto bit = [&](int q) { return 1u << (L - 1 - q); };
	auto diag = [](int k) { return k == BK_ID || k == BK_D1 || k == BK_NEG1 || k == BK_DIAG; };
	// components of wires joined by center blocks that move amplitudes
	std::vector<int> comp(L);
	for (int q = 0; q < L; q++) comp[q] = q;
	auto find = [&](int q) { while (comp[q] != q) q = comp[q]; return q; };
	for (int g = 0; g < ng; g++)
		if (!diag(tp.kw[g] & 7)) comp[find(t->sw[2 * g])] = find(t->sw[2 * g + 1]);
	std::vector<unsigned> cmask;
	std::vector<int> radix;
	long nkey = 1;
	for (int q = 0; q < L; q++)
		if (find(q) == q)
		{
			unsigned m = 0;
			for (int r = 0; r < L; r++) if (find(r) == q) m |= bit(r);
			cmask.push_back(m);
			radix.push_back((int)nkey);
			nkey *= __builtin_popcount(m) + 1;
			if (nkey > 4096) return 0;
		}
	// sector and row of every basis index
	std::vector<int> sid(N), rank(N), dim(nkey, 0);
	for (unsigned a = 0; a < N; a++)
	{
		int k = 0;
		for (size_t c = 0; c < cmask.size(); c++) k += radix[c] * __builtin_popcount(a & cmask[c]);
		sid[a] = k;
		rank[a] = dim[k]++;
	}
	int dmax = 0;
	for (int d : dim) dmax = std::max(dmax, d);
	const size_t col = (size_t)dmax * ES;
	size_t budget;
	if (col <= 55296) { sp.threads = 256; sp.blocks = 4; budget = 55296; }
	else if (col <= 113664) { sp.threads = 512; sp.blocks = 2; budget = 113664; }
	else if (col <= 230400) { sp.threads = 1024; sp.blocks = 1; budget = 230400; }
	else return 0;
	if (budget > mgcu_ctx()->smem_optin || dmax >= 32768) return 0;
	// the lists the steps need: center pairs by (wires, string); rows by (wires, their values)
	std::map<std::array<unsigned, 4>, int> keys;
	std::vector<SecStep> sg;
	auto key_of = [&](int type, unsigned bi, unsigned bj, unsigned mask) {
		return keys.emplace(std::array<unsigned, 4>{ (unsigned)type, bi, bj, mask }, (int)keys.size()).first->second;
	};
	for (const GateRec& r : tp.sched.gate)
	{
		const int g = r.g, kc = tp.kw[g] & 7, kk = (tp.kw[g] >> 3) & 7;
		const unsigned bi = bit(t->sw[2 * g]), bj = bit(t->sw[2 * g + 1]);
		unsigned mask = 0;
		for (int q = 0; q < L; q++) if (t->smask[g] & (1u << q)) mask |= bit(q);
		SecStep base = { -1, -1, tp.kw[g], tp.first[g], 0 };
		const size_t first = sg.size();
		if (!diag(kc)) base.kc = key_of(0, bi, bj, mask);
		// diagonal entries: |01>, |10> of a diagonal center block, |00>, |11> of the corner block
		const int entry[4] = { 0, 3, 4, 7 };
		for (int q = 0; q < 4; q++)
		{
			const int k = q < 2 ? kc : kk;
			if (!diag(k) || k == BK_ID || (q % 2 == 0 && k != BK_DIAG)) continue;
			SecStep s = base;
			s.kr = key_of(1, bi | bj, q == 0 ? bj : q == 1 ? bi : q == 2 ? 0 : (bi | bj), 0);
			s.flags = entry[q] | (k == BK_NEG1 ? SEC_NEG : 0);
			sg.push_back(s);
			base.kc = -1;
		}
		if (base.kc >= 0) sg.push_back(base);
		if (sg.size() > first) sg.back().flags |= SEC_SYNC;
	}
	const int nk = (int)keys.size();
	if ((size_t)std::max(nk, 1) * N > (1u << 24)) return 0;
	// sectors, largest first, and columns per block
	std::vector<int> order;
	for (int k = 0; k < (int)nkey; k++) if (dim[k]) order.push_back(k);
	std::stable_sort(order.begin(), order.end(), [&](int x, int y) { return dim[x] > dim[y]; });
	const double frac = sector_share(order, dim, budget / ES, mgcu_ctx()->nsm * sp.blocks, P::kId == MG_PREC_FP64_ID ? 64 : 512);
	std::vector<int> pos(nkey, -1);
	sp.sec.clear();
	int row0 = 0;
	size_t smem = 16;
	for (int k : order)
	{
		SectorProg::Sec s;
		s.d = dim[k]; s.row0 = row0; s.offs = (int)sp.sec.size() * (nk + 1);
		s.ln = sector_columns(s.d, budget / ES, frac);
		row0 += s.d;
		smem = std::max(smem, ((size_t)s.d << s.ln) * ES);
		pos[k] = (int)sp.sec.size();
		sp.sec.push_back(s);
	}
	sp.smem = smem;
	sp.rows.assign(N, 0);
	for (unsigned a = 0; a < N; a++) sp.rows[sp.sec[pos[sid[a]]].row0 + rank[a]] = a;
	// lists, sector by sector
	const size_t nsec = sp.sec.size();
	std::vector<int> offs(nsec * (nk + 1), 0);
	auto each = [&](const std::array<unsigned, 4>& key, auto&& fn) {
		// every base index with both wires clear; pairs list their |01> member
		const unsigned both = key[0] == 0 ? key[1] | key[2] : key[1], hi = 1u << (31 - __builtin_clz(both)), lo = both ^ hi;
		for (unsigned q = 0; q < (N >> 2); q++)
		{
			unsigned a = ((q & ~(lo - 1)) << 1) | (q & (lo - 1));
			a = ((a & ~(hi - 1)) << 1) | (a & (hi - 1));
			fn(a | key[2]);
		}
	};
	for (const auto& kv : keys)
		each(kv.first, [&](unsigned a) { offs[(size_t)sp.sec[pos[sid[a]]].offs + kv.second + 1]++; });
	int total = 0;
	for (size_t s = 0; s < nsec; s++)
	{
		int* o = offs.data() + s * (nk + 1);
		o[0] = total;
		for (int k = 0; k < nk; k++) o[k + 1] += o[k];
		total = o[nk];
	}
	std::vector<unsigned> list(std::max(total, 1));
	std::vector<int> fill(offs);
	for (const auto& kv : keys)
		each(kv.first, [&](unsigned a) {
			int& f = fill[(size_t)sp.sec[pos[sid[a]]].offs + kv.second];
			if (kv.first[0] == 0)
				list[f++] = (unsigned)rank[a] | (unsigned)(__builtin_popcount(a & kv.first[3]) & 1) << 15
					| (unsigned)rank[a ^ kv.first[1] ^ kv.first[2]] << 16;
			else list[f++] = (unsigned)rank[a];
		});
	for (const auto& kv : keys)
		for (const SectorProg::Sec& s : sp.sec)
			sector_order(list, offs[s.offs + kv.second], offs[s.offs + kv.second + 1], (ES == 16 ? 8 : 16) >> s.ln, kv.first[0] == 0);
	sp.nsteps = (int)sg.size();
	Arena ar(sp.fixed);
	ar.add(sp.steps, sg.data(), sizeof(SecStep) * sg.size());
	ar.add(sp.list, list.data(), sizeof(unsigned) * list.size());
	ar.add(sp.offs, offs.data(), sizeof(int) * offs.size());
	ar.add(sp.drows, sp.rows.data(), sizeof(unsigned) * N);
	const int e = ar.up();
	if (e) return e;
	MGCU_TRY(cudaStreamSynchronize(mgcu_stream()));
	MGCU_TRY(cudaFuncSetAttribute(sector_kernel<P>(sp.threads), cudaFuncAttributeMaxDynamicSharedMemorySize, (int)budget));
	sp.state = 1;
	return 0;
}

template <class P>
static int sector_prog(mgcu_target* t, TargetProg& tp)
{
	return tp.sector.state < 0 ? build_sector<P>(t, tp, tp.sector) : 0;
}

template <class P>
static int plan_sector(mgcu_target* t, int kt, bool& use)
{
	TargetProg* tp = nullptr;
	int e = target_prog<P>(t, kt, 128, tp);
	if (!e) e = sector_prog<P>(t, *tp);
	if (!e) use = tp->sector.state == 1;
	return e;
}
