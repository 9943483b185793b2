// Host side of the granule pass (gran.cuh): which columns one pass takes, the register program, the
// address maps and the output order; and the pass on host memory for the scheduler's CPU tests.
// Included by dense.cu after HostOp and RowInfo.
#pragma once

namespace tg {

#define GP_MINW 9            // narrowest table of a pass (input and output)
#define GP_MAXBITS 32        // widest, in granules: the kernel's offsets are 32-bit granule numbers
// An in-granule row that closes within GP_EVICT_OPS ops leaves the granule, for a row that lives GP_EVICT_GAIN
// ops longer at least.  A 300 x 600 sweep at 10 / 20 / 40 / 80 / 160 ops: uint8 30 bits 5.93 / 3.93 / 3.68 /
// 3.74 / 4.09 ms, 26 bits 0.81 / 0.76 / 0.74 / 0.75 / 0.76; uint16 26 bits 1.10 / 1.02 / 1.01 / 0.95 / 0.94.
// The gain: 1, 8, 16 and 32 within 2 % of each other, 64 5 % slower at 30 bits (a row stays that should leave).
#define GP_EVICT_OPS 40
#define GP_EVICT_GAIN 16

// value of a row as a parity of register slots, coset-number bits and a constant
struct RowExpr {
    uint32_t z = 0;
    uint64_t k = 0;
    uint32_t c = 0;
    void add(const RowExpr &o) { z ^= o.z; k ^= o.k; c ^= o.c; }
};

struct GranCol {
    int type;                // GC_N, GC_C, GC_O, GC_A or GC_I1
    uint64_t h;              // rows of the column (local numbers)
    uint64_t D = 0;          // N, C: direction over the input rows
    uint32_t hit = 0;        // N, C: earlier columns of the pass whose opened row D was reduced by
    int w, r = -1, c = -1, t = 0, slot = -1;
};

// Builds the pass that starts at op i0 on the table with rows `phys` (canonical order `canon`);
// ops before `limit` may be taken.  Returns the first op not taken, with canon / phys brought to the
// pass's output (i0 when only rows changed places); -1 when the form does not apply (tables of more than
// 2^GP_MAXBITS granules, read or written, take the other forms); -2 on an internal
// inconsistency.  nupd: updates taken.
//
// Local row numbers: input rows by physical position, then the rows opened in the pass.  With column
// m's use as variable z_m, a state is s_base + sum z_m h_m.  A column that opens a row has no free
// variable before it (the row is 0 there), so the direction D_j of a later column j is h_j reduced by
// the columns that opened rows of it; a column that closes a row has none after it.
static int64_t build_gran(const std::vector<HostOp> &hops, const RowInfo &RI, int64_t i0, int64_t limit, int eb,
                          std::vector<int> &canon, std::vector<int> &phys, GranParams &gp, int &nupd) {
    const int G = eb == 1 ? 2 : 1, w_in = (int)phys.size();
    if (w_in < GP_MINW || w_in > GP_MAXBITS + G) return -1;
    static thread_local std::vector<int> where;          // row -> local number
    if (where.size() < RI.uses.size()) where.resize(RI.uses.size());
    int rowid[64];
    for (int p = 0; p < w_in; p++) { rowid[p] = phys[p]; where[phys[p]] = p; }
    int nrow = w_in;
    int cpos[64], nc_rows = w_in;                        // canonical position -> local number
    for (int p = 0; p < w_in; p++) cpos[p] = where[canon[p]];
    auto life = [&](int l) { return RI.close_op[rowid[l]]; };
    const uint64_t lowm = (1ull << G) - 1, gmask = ((1ull << w_in) - 1) & ~lowm;

    // loaded directions in echelon form (distinct top bits)
    uint64_t basis[GP_SLOTS];
    int nb = 0;
    auto top = [](uint64_t v) { return 63 - __builtin_clzll(v); };
    auto reduce = [&](uint64_t v) {
        for (int q = 0; q < nb; q++)
            if ((v >> top(basis[q])) & 1ull) v ^= basis[q];
        return v;
    };
    auto insert = [&](uint64_t v) {                      // v reduced and nonzero; kept by descending top
        int q = nb++;
        while (q > 0 && basis[q - 1] < v) { basis[q] = basis[q - 1]; q--; }
        basis[q] = v;
    };
    int L = 0, bal = 0, M = 0;                           // loaded slots, opened - closed, its maximum
    // in-granule rows about to close change places with the longest-living row outside the lowest
    // three granule positions (those keep a warp's sectors whole)
    struct Swap { int g, row, slot; } sw[2];
    int nsw = 0;
    for (int g = 0; g < G; g++) {
        if (life(g) == INT64_MAX || life(g) - i0 >= GP_EVICT_OPS) continue;
        int best = -1;
        for (int p = G + 3; p < w_in; p++)
            if ((best < 0 || life(p) > life(best)) && !(nsw && sw[0].row == p)) best = p;
        if (best < 0 || (life(best) != INT64_MAX && life(best) < life(g) + GP_EVICT_GAIN)) continue;
        sw[nsw++] = {g, best, -1};
        insert(1ull << best);
        L++;
    }
    // a pass takes no column that closes an in-granule row
    bool blocked = false;
    uint64_t fixed = 0, fixed1 = 0;
    int64_t j = i0;
    while (j < limit && hops[j].code == 2 && nc_rows > GP_MINW) {     // rows closed before any column
        const int l = cpos[hops[j].a];
        if (l < G) { blocked = true; break; }
        bool used = false;
        for (int s = 0; s < nsw; s++) used |= sw[s].row == l;
        if (used) break;
        fixed |= 1ull << l;
        if (hops[j].b) fixed1 |= 1ull << l;
        for (int p = (int)hops[j].a; p + 1 < nc_rows; p++) cpos[p] = cpos[p + 1];
        nc_rows--;
        j++;
    }
    GranCol cols[GP_MAXOPS];
    int nc = 0;
    while (!blocked && j < limit && nc + nsw < GP_MAXOPS && nrow < 62) {
        int64_t k = j;
        const bool open = hops[k].code == 0;
        if (open) {
            k++;
            if (k >= limit || hops[k].code != 1 || !((hops[k].a >> nc_rows) & 1ull)) break;
        }
        if (hops[k].code != 1) break;
        GranCol C;
        C.h = 0;
        for (uint64_t a = hops[k].a; a; a &= a - 1) {
            const int p = __builtin_ctzll(a);
            C.h |= 1ull << (p < nc_rows ? cpos[p] : nrow);
        }
        C.w = (int)hops[k].b;
        if (open) C.r = nrow;
        int64_t kn = k + 1;
        int cp = -1;
        if (kn < limit && hops[kn].code == 2) {
            cp = (int)hops[kn].a;
            const int l = cp < nc_rows ? cpos[cp] : nrow;
            if (l < G) { blocked = true; break; }
            if (((C.h >> l) & 1ull) && l != C.r) { C.c = l; C.t = (int)hops[kn].b; kn++; }
        }
        C.type = open ? (C.c >= 0 ? GC_A : GC_O) : (C.c >= 0 ? GC_C : GC_N);
        const int w_next = nc_rows + (open ? 1 : 0) - (C.c >= 0 ? 1 : 0);
        if (w_next < GP_MINW || w_next > GP_MAXBITS + G) break;
        int L2 = L, M2 = M;
        uint64_t red = 0;
        if (!open) {
            C.D = C.h;
            for (int m = nc - 1; m >= 0; m--)
                if (cols[m].r >= 0 && ((C.D >> cols[m].r) & 1ull)) { C.D ^= cols[m].h; C.hit |= 1u << m; }
            if (C.D >> w_in) return -2;
            if ((C.D & gmask) == 0) {
                if (C.type != GC_N || (C.h & ~lowm)) break;
                C.type = GC_I1;
            } else {
                red = reduce(C.D & gmask);
                if (!red) break;                         // depends on the pass's other directions
                L2++;
            }
        }
        if (C.type == GC_O) M2 = std::max(M, bal + 1);
        if (L2 + M2 > GP_SLOTS) break;
        if (red) insert(red);
        L = L2;
        M = M2;
        bal += (C.type == GC_O) - (C.type == GC_C);
        if (open) { cpos[nc_rows++] = nrow; rowid[nrow] = RI.exp_row[j]; nrow++; }
        if (C.c >= 0) {
            for (int p = cp; p + 1 < nc_rows; p++) cpos[p] = cpos[p + 1];
            nc_rows--;
        }
        cols[nc++] = C;
        j = kn;
    }
    if (j == i0 && !(blocked && nsw)) return -1;

    // ---- slots.  The loaded ones are 0 .. L - 1 (rows that change places first), an opening column takes
    // the lowest free one; of the orders of the loaded columns, the one whose program goes through the
    // fewest members (an op leaves out the highest slots while they are dead)
    for (int s = 0; s < nsw; s++) sw[s].slot = s;
    int loaded[GP_SLOTS], nl = 0;
    for (int m = 0; m < nc; m++)
        if (cols[m].type == GC_N || cols[m].type == GC_C) loaded[nl++] = m;
    if (nl + nsw != L) return -2;
    int lims[GP_MAXOPS];
    uint32_t live_slots = 0;
    // assigns the opening columns' slots and fills lims; returns the members gone through, or -1 once
    // they reach `bound`
    auto assign = [&](int bound) {
        int work = 0;
        uint32_t m = (1u << L) - 1u;                     // live slots
        for (int c = 0; c < nc; c++) {
            GranCol &C = cols[c];
            if (C.type == GC_O) C.slot = __builtin_ctz(~m);
            int n;                                       // the highest live slot decides
            if (C.type == GC_I1) {
                n = 32;
                work += n;
            } else if (C.type == GC_A) {
                n = m >= 16 ? 32 : m >= 8 ? 16 : 8;
                work += n;
            } else {
                const uint32_t lo = m & ((1u << C.slot) - 1u), o = lo | ((m >> (C.slot + 1)) << C.slot);
                n = o >= 8 ? 16 : o >= 4 ? 8 : 4;
                work += 2 * n;
            }
            lims[c] = n;
            if (work >= bound) return -1;
            if (C.type == GC_O) m |= 1u << C.slot;
            if (C.type == GC_C) m &= ~(1u << C.slot);
        }
        live_slots = m;
        return work;
    };
    // orders of the loaded columns (the N columns among themselves keep theirs), from the one that puts the
    // first to close highest
    int perm[GP_SLOTS], best_perm[GP_SLOTS], best_work = INT32_MAX, nn = 0;
    for (int q = 0; q < nl; q++) nn += cols[loaded[q]].type == GC_N;
    std::stable_partition(loaded, loaded + nl, [&](int m) { return cols[m].type == GC_N; });
    std::reverse(loaded + nn, loaded + nl);
    for (int q = 0; q < nl; q++) perm[q] = q;
    do {
        bool skip = false;
        for (int q = 0; q + 1 < nn; q++) skip |= perm[q] > perm[q + 1];
        if (skip) continue;
        for (int q = 0; q < nl; q++) cols[loaded[q]].slot = nsw + perm[q];
        const int w = assign(best_work);
        if (w < 0) continue;
        best_work = w;
        std::copy(perm, perm + nl, best_perm);
    } while (std::next_permutation(perm, perm + nl));
    if (best_work == INT32_MAX) return -2;
    for (int q = 0; q < nl; q++) cols[loaded[q]].slot = nsw + best_perm[q];
    assign(INT32_MAX);
    bool busy[GP_SLOTS];
    for (int s = 0; s < GP_SLOTS; s++) busy[s] = (live_slots >> s) & 1u;
    // ---- coset-number bits: the input rows that are neither pivots nor fixed, by position
    uint64_t piv = 0;
    for (int q = 0; q < nb; q++) piv |= 1ull << top(basis[q]);
    int krow[64], nk = 0;
    for (int p = G; p < w_in; p++)
        if (!((piv >> p) & 1ull) && !((fixed >> p) & 1ull)) krow[nk++] = p;
    if (nk > GP_MAXK) return -1;
    uint32_t kin[GP_MAXK + 1], kout[GP_MAXK + 1];
    memset(&gp, 0, sizeof(gp));
    gp.ncosets = 1ull << nk;
    gp.nk = nk;
    gp.nload = L;
    RowExpr ex[64];
    for (int b = 0; b < nk; b++) { ex[krow[b]].k = 1ull << b; kin[b] = (uint32_t)(1ull << (krow[b] - G)); kout[b] = 0; }
    uint64_t dir[GP_SLOTS] = {0, 0, 0, 0, 0};
    for (int m = 0; m < nc; m++)
        if (cols[m].type == GC_N || cols[m].type == GC_C) dir[cols[m].slot] = cols[m].D;
    for (int s = 0; s < nsw; s++) dir[sw[s].slot] = 1ull << sw[s].row;
    for (int p = 0; p < w_in; p++) {
        for (int s = 0; s < L; s++) ex[p].z |= (uint32_t)((dir[s] >> p) & 1ull) << s;
        if ((fixed1 >> p) & 1ull) ex[p].c = 1;
    }
    gp.fin = (uint32_t)(fixed1 >> G);
    auto unpack_sel = [&](uint32_t sh, uint32_t par) -> uint32_t {   // lanes of register `par` of a granule
        if (eb == 2) return sh & 1u ? 0x1032u : 0x3210u;
        const uint32_t p = par ^ (sh & 1u), l = sh >> 1;
        return (p + 2 * l) | 0x40u | ((p + 2 * (1u - l)) << 8) | 0x4000u;
    };
    auto parity = [](uint32_t v) { return (uint32_t)__builtin_parity(v); };
    for (uint32_t z = 0; z < GP_MEMBERS; z++) {
        uint64_t o = 0;
        for (int s = 0; s < L; s++)
            if ((z >> s) & 1u) o ^= dir[s];
        const uint32_t sh = (uint32_t)(o & lowm);
        gp.xin[z] = (uint32_t)(o >> G);
        gp.usel[z] = make_uint2(unpack_sel(sh, 0), unpack_sel(sh, 1));
    }
    // ---- the register program, following every row's value
    uint64_t alive = (1ull << w_in) - 1;
    alive &= ~fixed;
    auto emit = [&](int code, int w, uint32_t zm, uint64_t km, uint32_t cst) {
        GranOp &O = gp.ops[gp.nops];
        O.lim = gp.nops < nc ? (uint32_t)lims[gp.nops] : 0;
        gp.nops++;
        O.code = (uint32_t)code;
        O.cst = cst & 1u;
        O.w2 = (uint32_t)w | ((uint32_t)w << 16);
        for (int s = 0; s < 5; s++) O.d[s] = (zm >> s) & 1u ? O.w2 : 0u;
        O.kmask = (uint32_t)km;
    };
    auto plain = [&](const GranCol &C) {                 // flipping the slot flips exactly the column's rows
        for (uint64_t a = alive; a; a &= a - 1) {
            const int l = __builtin_ctzll(a);
            if (((ex[l].z >> C.slot) & 1u) != ((C.h >> l) & 1ull)) return false;
        }
        return true;
    };
    for (int m = 0; m < nc; m++) {
        const GranCol &C = cols[m];
        if (C.type == GC_N) {
            if (!plain(C)) return -2;
            emit(GC_N + C.slot, C.w, 0, 0, 0);
        } else if (C.type == GC_I1) {
            emit(GC_I1 + (int)(C.h & lowm) - 1, C.w, 0, 0, 0);
        } else if (C.type == GC_C) {
            if (!plain(C)) return -2;
            RowExpr P = ex[C.c];
            P.z ^= 1u << C.slot;
            P.c ^= (uint32_t)C.t;
            emit(GC_C + C.slot, C.w, P.z, P.k, P.c);
            alive &= ~(1ull << C.c);
            for (uint64_t a = alive; a; a &= a - 1) {
                RowExpr &e = ex[__builtin_ctzll(a)];
                if ((e.z >> C.slot) & 1u) { e.z ^= 1u << C.slot; e.add(P); }
            }
        } else {
            RowExpr P;
            if (C.type == GC_O) {
                RowExpr phi;
                for (int q = m + 1; q < nc; q++)
                    if ((cols[q].hit >> m) & 1u) phi.z ^= 1u << cols[q].slot;
                emit(GC_O + C.slot, C.w, phi.z, 0, 0);
                P = phi;
                P.z ^= 1u << C.slot;
            } else {
                P = ex[C.c];
                P.c ^= (uint32_t)C.t;
                emit(GC_A, C.w, P.z, P.k, P.c);
                alive &= ~(1ull << C.c);
            }
            alive |= 1ull << C.r;
            ex[C.r] = RowExpr();
            for (uint64_t a = C.h & alive; a; a &= a - 1) ex[__builtin_ctzll(a)].add(P);
        }
    }
    // ---- output order
    int gran_row[2] = {0, 1};
    for (int s = 0; s < nsw; s++) {
        const uint32_t bit = 1u << sw[s].slot;
        for (uint64_t a = alive; a; a &= a - 1) {
            const int l = __builtin_ctzll(a);
            if ((((ex[l].z & bit) != 0) != (l == sw[s].row))) return -2;
        }
        emit((eb == 1 && sw[s].g == 0 ? GC_T0 : GC_T1) + sw[s].slot, 0, 0, 0, 0);
        ex[sw[s].row].z ^= bit;                          // in the granule: its own bit, and the rest as a permutation
        ex[sw[s].g].z ^= bit;
        gran_row[sw[s].g] = sw[s].row;
    }
    int out[64], no = 0;
    uint64_t placed = 0;
    for (int g = 0; g < G; g++) { out[no++] = gran_row[g]; placed |= 1ull << gran_row[g]; }
    // the three longest-living of the lanes' rows stay lowest, the others follow by life
    for (int t = 0; t < 3; t++) {
        int best = -1;
        for (int b = 0; b < nk && b < 5; b++) {
            const int l = krow[b];
            if (!((alive >> l) & 1ull) || ((placed >> l) & 1ull)) continue;
            if (best < 0 || life(l) > life(best)) best = l;
        }
        if (best < 0) break;
        out[no++] = best;
        placed |= 1ull << best;
    }
    const int rest0 = no;
    for (uint64_t a = alive & ~placed; a; a &= a - 1) out[no++] = __builtin_ctzll(a);
    std::stable_sort(out + rest0, out + no, [&](int x, int y) { return life(x) > life(y); });
    if (no != nc_rows) return -2;
    // ---- output maps
    uint32_t live = 0;
    int nlive = 0;
    for (int s = 0; s < GP_SLOTS; s++) nlive += busy[s];
    for (uint32_t z = 0; z < GP_MEMBERS; z++) {
        bool ok = true;
        for (int s = 0; s < GP_SLOTS; s++) ok = ok && (busy[s] || !((z >> s) & 1u));
        if (ok) live |= 1u << z;
        uint32_t o = 0, sh = 0;
        for (int q = 0; q < no; q++) {
            const uint32_t v = parity(ex[out[q]].z & z) ^ (q < G ? ex[out[q]].c : 0u);
            if (q < G) sh |= v << q;
            else o |= v << (q - G);
        }
        uint32_t sel = 0;
        if (eb == 1)
            for (uint32_t e = 0; e < 4; e++) { const uint32_t q = e ^ sh; sel |= (4 * (q & 1u) + 2 * (q >> 1)) << (4 * e); }
        else sel = sh & 1u ? 0x1032u : 0x3210u;
        gp.mout[z] = make_uint2(o, sel);
    }
    if (nlive + nk != no - G) return -2;
    gp.live_out = live;
    for (int q = 0; q < no; q++) {
        const RowExpr &e = ex[out[q]];
        if (q == 0) gp.smask0 = (uint32_t)e.k;
        else if (q == 1 && G == 2) gp.smask1 = (uint32_t)e.k;
        if (q >= G) {
            for (int b = 0; b < nk; b++) kout[b] |= (uint32_t)((e.k >> b) & 1ull) << (q - G);
            gp.fout |= e.c << (q - G);
        }
    }
    for (int b = 0; b < nk && b < 8; b++) gp.klow[b] = make_uint2(kin[b], kout[b]);
    for (int b = 8; b < nk; b++)
        for (int v = 0; v < 16; v++)
            if ((v >> ((b - 8) & 3)) & 1) {
                gp.khigh[(b - 8) / 4][v].x ^= kin[b];
                gp.khigh[(b - 8) / 4][v].y ^= kout[b];
            }
    canon.clear();
    for (int p = 0; p < nc_rows; p++) canon.push_back(rowid[cpos[p]]);
    phys.clear();
    for (int q = 0; q < no; q++) phys.push_back(rowid[out[q]]);
    nupd = nc;
    return j;
}

// the granule pass on host memory, coset by coset, entry by entry (gran_step's maps and program)
template <typename E>
static void emulate_gran(const GranParams &P, const E *src, E *dst) {
    constexpr int EB = sizeof(E), NE = 4 / EB;            // entries per granule
    const uint32_t INF = Entry<E>::INF;
    auto g_drop = [](int z, int s) { return ((z >> (s + 1)) << s) | (z & ((1 << s) - 1)); };   // z without bit s
    auto minadd = [&](uint32_t a, uint32_t b, uint32_t w) { return std::min(a, std::min(INF, b + w)); };
    for (uint64_t k = 0; k < P.ncosets; k++) {
        uint32_t io = P.fin, oo = P.fout;
        for (int b = 0; b < 8; b++)
            if ((k >> b) & 1ull) { io ^= P.klow[b].x; oo ^= P.klow[b].y; }
        for (int g = 0; g < 6; g++) {
            io ^= P.khigh[g][(k >> (8 + 4 * g)) & 15u].x;
            oo ^= P.khigh[g][(k >> (8 + 4 * g)) & 15u].y;
        }
        // V[z][q]: register position q of member z (u8: q = parity + 2 * lane, u16: q = lane)
        uint32_t V[32][4];
        memset(V, 0, sizeof(V));
        for (int z = 0; z < (1 << P.nload); z++) {
            const E *g = src + (size_t)(io ^ P.xin[z]) * NE;
            const uint8_t *by = reinterpret_cast<const uint8_t *>(g);
            for (int q = 0; q < NE; q++) {
                if (EB == 1) {
                    const uint32_t sel = (q & 1) ? P.usel[z].y : P.usel[z].x;
                    V[z][q] = by[(sel >> (8 * (q >> 1))) & 3u];
                } else {
                    V[z][q] = g[((P.usel[z].x >> (8 * q)) & 3u) >> 1];
                }
            }
        }
        for (int u = 0; u < P.nops; u++) {
            const GranOp &O = P.ops[u];
            const uint32_t w = O.w2 & 0xFFFFu;
            const uint32_t kp = (__builtin_popcount((uint32_t)k & O.kmask) + O.cst) & 1;
            auto par = [&](int z) {
                int p = kp;
                for (int s = 0; s < 5; s++) p ^= ((z >> s) & 1) && O.d[s];
                return p;
            };
            const int code = (int)O.code;
            for (int z = 0; z < 32; z++) {
                if (code == GC_A) {
                    if (z >= (int)O.lim) continue;
                    for (int q = 0; q < NE; q++) V[z][q] = minadd(INF, V[z][q], par(z) ? w : 0);
                } else if (code >= GC_I1) {
                    const int mk = code - GC_I1 + 1;
                    uint32_t t[4];
                    for (int q = 0; q < NE; q++) t[q] = minadd(V[z][q], V[z][q ^ mk], w);
                    for (int q = 0; q < NE; q++) V[z][q] = t[q];
                } else {
                    const int s = code < GC_T0 ? code % 5 : (code - GC_T0) % 2, y = z | (1 << s);
                    if ((z >> s) & 1 || (code < GC_T0 && g_drop(z, s) >= (int)O.lim)) continue;
                    for (int q = 0; q < NE; q++) {
                        const uint32_t a = V[z][q], b = V[y][q];
                        if (code < GC_C) {
                            V[z][q] = minadd(a, b, w);
                            V[y][q] = minadd(b, a, w);
                        } else if (code < GC_O) {
                            V[z][q] = std::min(minadd(INF, a, par(z) ? w : 0), minadd(INF, b, par(z) ? 0 : w));
                        } else if (code < GC_A) {
                            V[z][q] = minadd(INF, a, par(z) ? w : 0);
                            V[y][q] = minadd(INF, a, par(z) ? 0 : w);
                        }
                    }
                    if (code >= GC_T0) {
                        const int bit = code < GC_T1 ? 1 : NE / 2;      // in-granule bit of register positions
                        for (int q = 0; q < NE; q++)
                            if (q & bit) std::swap(V[z][q], V[y][q ^ bit]);
                    }
                }
            }
        }
        const uint32_t ts = ((__builtin_popcount((uint32_t)k & P.smask0) & 1) ? (EB == 1 ? 0x4444u : 0x2222u) : 0u) ^
                            (EB == 1 && (__builtin_popcount((uint32_t)k & P.smask1) & 1) ? 0x2222u : 0u);
        for (int z = 0; z < 32; z++) {
            if (!((P.live_out >> z) & 1u)) continue;
            E *g = dst + (size_t)(oo ^ P.mout[z].x) * NE;
            const uint32_t sel = P.mout[z].y ^ ts;
            for (int e = 0; e < NE; e++) {
                if (EB == 1) {
                    const uint32_t nib = (sel >> (4 * e)) & 7u;
                    g[e] = (E)V[z][(nib >> 2) + (nib & 2u)];
                } else {
                    g[e] = (E)V[z][((sel >> (8 * e)) & 3u) >> 1];
                }
            }
        }
    }
}

}  // namespace tg
