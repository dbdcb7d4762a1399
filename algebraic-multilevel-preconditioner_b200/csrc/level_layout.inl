// Host layout of the level-synchronous sparse sweeps (level_sweep.cu), one triangular factor of one
// subdomain.  Included by capi.cu inside its anonymous namespace (HostCsr, chain_blocks).

// Rows are taken in blocks: runs of up to `cap` rows where each depends on the one solved just
// before it (a supernode).  A block B of two rows or more is solved in two steps,
//   s(B) = b(B) - M(B, outside) x,   x(B) = W^-1 s(B),   W = M(B, B),
// with W^-1 dense (k <= 64, inverted here), a single row in one, x = (b - M(row, :) x) / diagonal.
// The levels are those of the blocks, a level is one stage for the first step (A) and, if it holds
// blocks, one for the second (B).  Against folding W^-1 into the rows (chain_block 8) nothing fills
// in and the levels are a quarter: bubbles3d 100^3 / 64: 24 against 76, poisson2d 200^2 / 8: 19
// against 90, convdiff3d 48^3 / 12: 24 against 118.
struct LevelSweep {
    std::vector<int32_t> rhs_row;  // rows in the order of their right-hand sides: the n0 rows that are single and have
                                   // no entries (slots 0 .. n0 - 1), then per warp, task by task
    int n0 = 0;
    std::vector<int32_t> pos;      // row -> slot of x
    std::vector<double> dinv;      // per right-hand side: 1 / diagonal of a single row, 1 of a block's row
    std::vector<int32_t> col;      // per step 128: lane j's four columns at 4 j .. 4 j + 3
    std::vector<double> val;       // per step 128: value q of lane j at 32 q + j
    std::vector<uint4> task;       // descriptors (LevelFactor)
    std::vector<uint16_t> bout;    // slots of the block rows in the order of their stage-B tasks
    std::vector<int64_t> wtask, wstep, wrhs;  // per warp (nw + 1): first task, step, right-hand side (from n0 on)
    int nst = 0;                   // stages
    int smax = 0;                  // block rows of the largest level: slots of s
    int nlev = 0;
    int64_t real = 0, nblk = 0;
    // refactorization maps (when built with the factor position of every entry): per value its source
    // (-1 padding, -2 an entry of a W^-1), per right-hand side the diagonal's (-1: 1), per block its W
    // packed lower (-1: 0 off the diagonal, 1 on it) and where the entries of W^-1 go
    std::vector<int32_t> src, dsrc, wsrc;
    std::vector<int64_t> boff{0}, wpos;
    std::vector<int32_t> bk;
};

// cs CTAs of `warps` warps each; key: where a row's right-hand side is read from (rows that may be in any
// order are put in its order, so neighbouring lanes read neighbouring values); the slots (x, the zero slot T, s) fit 16 bits
void build_level_sweep(const HostCsr& M, int T, bool lower, bool unit_diag, int cs, int warps, int gmax, int epl, int cap,
                       const std::vector<int32_t>& key, LevelSweep& out, std::string& err,
                       const std::vector<int32_t>* mpos = nullptr)
{
    const bool track = mpos != nullptr;
    const int nw = cs * warps;
    std::vector<double> diag(T, 1.0);
    std::vector<int32_t> dpos(track ? T : 0, -1);
    for (int r = 0; r < T; ++r) {
        if (unit_diag) continue;
        for (int64_t e = M.rp[r]; e < M.rp[r + 1]; ++e)
            if (M.ci[e] == r) {
                diag[r] = M.v[e];
                if (track) dpos[r] = (*mpos)[e];
            }
        if (diag[r] == 0.0 || !std::isfinite(diag[r])) {
            err = "zero or non-finite diagonal in a triangular factor";
            return;
        }
    }
    const std::vector<std::vector<int32_t>> blocks = chain_blocks(M, T, lower, cap);
    std::vector<int32_t> blk(T, -1), in_blk(T, 0);
    for (size_t b = 0; b < blocks.size(); ++b)
        for (size_t i = 0; i < blocks[b].size(); ++i) {
            blk[blocks[b][i]] = (int32_t)b;
            in_blk[blocks[b][i]] = (int32_t)i;
        }
    // entries outside the blocks, and the levels of the blocks (blocks come in solve order)
    auto inside = [&](int c) { return lower ? c >= 0 : c < T; };
    std::vector<std::vector<int64_t>> rows(T);  // entry numbers of M
    std::vector<int32_t> level(blocks.size(), 0);
    out.nlev = 0;
    for (size_t b = 0; b < blocks.size(); ++b) {
        int lv = 0;
        for (int32_t r : blocks[b])
            for (int64_t e = M.rp[r]; e < M.rp[r + 1]; ++e) {
                const int c = M.ci[e];
                if ((lower ? c >= r : c <= r) || !inside(c) || blk[c] == (int32_t)b) continue;
                rows[r].push_back(e);
                lv = std::max(lv, level[blk[c]] + 1);
            }
        level[b] = lv;
        out.nlev = std::max(out.nlev, lv + 1);
    }
    std::vector<std::vector<int32_t>> lsingle(out.nlev), lblocks(out.nlev);
    for (size_t b = 0; b < blocks.size(); ++b) {
        if (blocks[b].size() == 1) lsingle[level[b]].push_back(blocks[b][0]);
        else lblocks[level[b]].push_back((int32_t)b);
    }
    // Lanes of a row of `len` entries when `n` rows share `w` warps: about epl entries per lane, and no
    // more lanes than it takes to give every warp a task.  (A task's sum over the lanes and its store
    // cost as much as three steps: a stage of many rows is done in few tasks of many rows each.)
    auto width = [&](int len, int n, int w) {
        int most = gmax;
        while (most > 1 && (int64_t)most * n > (int64_t)32 * w) most >>= 1;
        int g = 1;
        while (g < most && g * epl < len) g <<= 1;
        return g;
    };
    struct WarpOut {
        std::vector<uint4> task;
        std::vector<int32_t> col, src, rhs;
        std::vector<double> val;
        int64_t load = 0;
    };
    std::vector<WarpOut> wo(nw);
    out.pos.assign(T, -1);
    int slot = 0;
    // a task: R rows (G lanes each) of consecutive output slots; entries (column, value, source) by row
    struct Ent {
        int32_t c;
        double v;
        int32_t s;
    };
    struct Task {
        int G = 1, first = 0;     // lanes per row, first output slot (stage B: first of bout)
        int kept = 0;             // first slot that keeps its right-hand sides
        std::vector<std::vector<Ent>> rows;
        std::vector<int32_t> rhs; // rows whose right-hand side it reads (stage A)
        uint64_t flags = 0;
        int only = -1;            // the CTA it must run on (stage B), or any
        int ns = 0;               // steps
    };
    std::vector<Task> tasks;
    std::vector<int32_t> bid(blocks.size(), -1);
    auto place = [&](int stage) {
        for (Task& t : tasks) {
            size_t len = 0;
            for (const auto& r : t.rows) len = std::max(len, r.size());
            t.ns = ((int)((len + t.G - 1) / t.G) + 3) / 4;
        }
        std::vector<int> order(tasks.size());
        for (size_t i = 0; i < order.size(); ++i) order[i] = (int)i;
        std::stable_sort(order.begin(), order.end(), [&](int a, int b) { return tasks[a].ns > tasks[b].ns; });
        std::vector<int> now(nw, 0);  // work of this stage
        for (int i : order) {
            const Task& t = tasks[i];
            const int w0 = t.only < 0 ? 0 : t.only * warps, w1 = t.only < 0 ? nw : w0 + warps;
            int best = w0;
            for (int w = w0 + 1; w < w1; ++w)
                if (now[w] < now[best] || (now[w] == now[best] && wo[w].load < wo[best].load)) best = w;
            now[best] += t.ns + 3;
            wo[best].load += t.ns + 3;
            WarpOut& W = wo[best];
            const int R = (int)t.rows.size();
            int gl2 = 0;
            while ((1 << gl2) < t.G) ++gl2;
            const bool b = (t.flags & S2L_LTASK_NO_RHS) != 0;
            W.task.push_back(make_uint4((uint32_t)t.flags | (uint32_t)gl2 | ((uint32_t)R << 3) | ((uint32_t)stage << 16),
                                        (b ? 0u : (uint32_t)t.first) | ((uint32_t)t.ns << 16),
                                        (uint32_t)(b ? t.first : t.kept), 0u));
            if (t.ns > 65535) err = "a sparse row has too many entries";
            for (int st = 0; st < t.ns; ++st) {
                const size_t v0 = W.val.size();
                W.val.resize(v0 + 128, 0.0);
                W.col.resize(v0 + 128, T);
                if (track) W.src.resize(v0 + 128, -1);
                for (int q = 0; q < 4; ++q)
                    for (int lane = 0; lane < 32; ++lane) {
                        const int k = lane / t.G, e = (4 * st + q) * t.G + lane % t.G;
                        if (k >= R || e >= (int)t.rows[k].size()) continue;
                        const Ent& x = t.rows[k][e];
                        W.val[v0 + 32 * q + lane] = x.v;
                        W.col[v0 + 4 * lane + q] = x.c;
                        if (track) W.src[v0 + 32 * q + lane] = x.s;
                        ++out.real;
                    }
            }
            W.rhs.insert(W.rhs.end(), t.rhs.begin(), t.rhs.end());
        }
        tasks.clear();
    };
    // rows [i0, i1) of a list (same lanes) into tasks of 32 / G rows
    auto entries = [&](int r, double scale) {
        std::vector<Ent> v;
        v.reserve(rows[r].size());
        for (int64_t e : rows[r]) v.push_back({out.pos[M.ci[e]], M.v[e] * scale, track ? (*mpos)[e] : 0});
        return v;
    };
    int stage = 0;
    out.smax = 0;
    std::vector<int32_t> spos(T, -1);  // row -> slot of s
    for (int l = 0; l < out.nlev; ++l) {
        // slots of x: single rows by lanes and length, then the block rows by CTA, lanes and length of stage A
        std::vector<int32_t>& S = lsingle[l];
        int na = (int)S.size();  // rows of stage A
        for (int32_t b : lblocks[l]) na += (int)blocks[b].size();
        auto widtha = [&](int32_t r) { return width((int)rows[r].size(), na, nw); };
        auto shortera = [&](int32_t a, int32_t b) {
            const int ga = widtha(a), gb = widtha(b);
            return ga != gb ? ga < gb : rows[a].size() < rows[b].size();
        };
        auto by_key = [&](int32_t a, int32_t b) { return key[a] < key[b]; };
        std::sort(S.begin(), S.end(), by_key);
        std::stable_sort(S.begin(), S.end(), shortera);
        if (l == 0) {  // no entries: their x is their right-hand side
            out.n0 = (int)S.size();
            out.rhs_row = S;
        }
        for (size_t i0 = l == 0 ? S.size() : 0; i0 < S.size();) {
            const int G = widtha(S[i0]);
            size_t i1 = i0;
            while (i1 < S.size() && (int)(i1 - i0) < 32 / G && widtha(S[i1]) == G) ++i1;
            Task t;
            t.G = G;
            t.first = t.kept = slot + (int)i0;
            for (size_t i = i0; i < i1; ++i) {
                t.rows.push_back(entries(S[i], 1.0 / diag[S[i]]));
                t.rhs.push_back(S[i]);
            }
            tasks.push_back(std::move(t));
            i0 = i1;
        }
        for (size_t i = 0; i < S.size(); ++i) out.pos[S[i]] = slot + (int)i;
        slot += (int)S.size();
        if (lblocks[l].empty()) {
            place(stage++);
            continue;
        }
        // blocks to the CTAs, largest first
        std::vector<int32_t>& Bl = lblocks[l];
        std::stable_sort(Bl.begin(), Bl.end(), [&](int32_t a, int32_t b) { return blocks[a].size() > blocks[b].size(); });
        std::vector<int64_t> dense(cs, 0);
        std::vector<std::vector<int32_t>> own(cs);  // block rows per CTA
        std::vector<int32_t> brows;
        for (int32_t b : Bl) {
            int c = 0;
            for (int q = 1; q < cs; ++q)
                if (dense[q] < dense[c]) c = q;
            dense[c] += (int64_t)blocks[b].size() * (blocks[b].size() + 1);
            for (int32_t r : blocks[b]) own[c].push_back(r);
            bid[b] = (int32_t)out.nblk++;
        }
        int ns = 0;
        for (int c = 0; c < cs; ++c) {
            // stage A: s of the CTA's block rows, by lanes and length
            std::vector<int32_t> R = own[c];
            std::sort(R.begin(), R.end(), by_key);
            std::stable_sort(R.begin(), R.end(), shortera);
            for (size_t i0 = 0; i0 < R.size();) {
                const int G = widtha(R[i0]);
                size_t i1 = i0;
                while (i1 < R.size() && (int)(i1 - i0) < 32 / G && widtha(R[i1]) == G) ++i1;
                Task t;
                t.G = G;
                t.first = T + 1 + ns + (int)i0;
                t.kept = slot + ns + (int)i0;  // x of the block rows in the order of their s
                t.flags = S2L_LTASK_TO_S | ((uint64_t)c << 12);
                for (size_t i = i0; i < i1; ++i) {
                    t.rows.push_back(entries(R[i], 1.0));
                    t.rhs.push_back(R[i]);
                }
                tasks.push_back(std::move(t));
                i0 = i1;
            }
            for (size_t i = 0; i < R.size(); ++i) {
                spos[R[i]] = T + 1 + ns + (int)i;
                out.pos[R[i]] = slot + ns + (int)i;
            }
            ns += (int)R.size();
        }
        out.smax = std::max(out.smax, ns);
        slot += ns;
        place(stage++);
        // W^-1 of every block, by forward substitution column by column
        std::vector<std::vector<double>> winv(Bl.size());
        std::vector<int32_t> at(blocks.size(), -1);
        for (size_t q = 0; q < Bl.size(); ++q) {
            const std::vector<int32_t>& B = blocks[Bl[q]];
            const int k = (int)B.size();
            at[Bl[q]] = (int32_t)q;
            std::vector<double> W((size_t)k * k, 0.0), X((size_t)k * k, 0.0);
            std::vector<int32_t> Wp(track ? (size_t)k * k : 0, -1);
            for (int i = 0; i < k; ++i) {
                W[(size_t)i * k + i] = diag[B[i]];
                if (track) Wp[(size_t)i * k + i] = dpos[B[i]];
                for (int64_t e = M.rp[B[i]]; e < M.rp[B[i] + 1]; ++e) {
                    const int c = M.ci[e];
                    if ((lower ? c >= B[i] : c <= B[i]) || !inside(c) || blk[c] != Bl[q]) continue;
                    W[(size_t)i * k + in_blk[c]] = M.v[e];
                    if (track) Wp[(size_t)i * k + in_blk[c]] = (*mpos)[e];
                }
            }
            for (int j = 0; j < k; ++j)
                for (int i = j; i < k; ++i) {
                    double v = i == j ? 1.0 : 0.0;
                    for (int p = j; p < i; ++p) v -= W[(size_t)i * k + p] * X[(size_t)p * k + j];
                    X[(size_t)i * k + j] = v / W[(size_t)i * k + i];
                }
            winv[q].swap(X);
            if (track) {
                out.bk.push_back(k);
                for (int i = 0; i < k; ++i)
                    for (int j = 0; j <= i; ++j) out.wsrc.push_back(Wp[(size_t)i * k + j]);
                out.boff.push_back((int64_t)out.wsrc.size());
            }
        }
        // stage B: x of the block rows, on their CTA; row i of a block has i + 1 entries
        for (int c = 0; c < cs; ++c) {
            std::vector<int32_t> R = own[c];
            std::stable_sort(R.begin(), R.end(), [&](int32_t a, int32_t b) { return in_blk[a] < in_blk[b]; });
            auto widthb = [&](int32_t r) { return width(in_blk[r] + 1, (int)R.size(), warps); };
            for (size_t i0 = 0; i0 < R.size();) {
                const int G = widthb(R[i0]);
                size_t i1 = i0;
                while (i1 < R.size() && (int)(i1 - i0) < 32 / G && widthb(R[i1]) == G) ++i1;
                Task t;
                t.G = G;
                t.first = (int)out.bout.size();
                for (size_t i = i0; i < i1; ++i) out.bout.push_back((uint16_t)out.pos[R[i]]);
                t.flags = S2L_LTASK_NO_RHS;
                t.only = c;
                for (size_t i = i0; i < i1; ++i) {
                    const int32_t r = R[i], b = blk[r];
                    const int k = (int)blocks[b].size(), ri = in_blk[r];
                    std::vector<Ent> v;
                    for (int j = 0; j <= ri; ++j)  // source: -2 - (packed position in wsrc), resolved below
                        v.push_back({spos[blocks[b][j]], winv[at[b]][(size_t)ri * k + j],
                                     track ? (int32_t)(-2 - (out.boff[bid[b]] + (int64_t)ri * (ri + 1) / 2 + j)) : 0});
                    t.rows.push_back(std::move(v));
                }
                tasks.push_back(std::move(t));
                i0 = i1;
            }
        }
        place(stage++);
    }
    out.nst = stage;
    if (out.nst > 65535 || T + 1 + out.smax > 65535) {
        err = "level sweep: more than 65535 stages or slots";
        return;
    }
    out.wtask.assign(nw + 1, 0);
    out.wstep.assign(nw + 1, 0);
    out.wrhs.assign(nw + 1, 0);
    if (track) out.wpos.assign(out.wsrc.size(), -1);
    for (int w = 0; w < nw; ++w) {
        out.wtask[w] = (int64_t)out.task.size();
        out.wstep[w] = (int64_t)out.val.size() / 128;
        out.wrhs[w] = (int64_t)out.rhs_row.size() - out.n0;
        if (track)
            for (size_t e = 0; e < wo[w].src.size(); ++e) {
                if (wo[w].src[e] < -1) {
                    out.wpos[(size_t)(-2 - (int64_t)wo[w].src[e])] = 128 * out.wstep[w] + (int64_t)e;
                    wo[w].src[e] = -2;
                }
            }
        out.task.insert(out.task.end(), wo[w].task.begin(), wo[w].task.end());
        out.col.insert(out.col.end(), wo[w].col.begin(), wo[w].col.end());
        out.val.insert(out.val.end(), wo[w].val.begin(), wo[w].val.end());
        out.rhs_row.insert(out.rhs_row.end(), wo[w].rhs.begin(), wo[w].rhs.end());
        if (track) out.src.insert(out.src.end(), wo[w].src.begin(), wo[w].src.end());
    }
    out.wtask[nw] = (int64_t)out.task.size();
    out.wstep[nw] = (int64_t)out.val.size() / 128;
    out.wrhs[nw] = (int64_t)out.rhs_row.size() - out.n0;
    out.dinv.resize(out.rhs_row.size());
    if (track) out.dsrc.resize(out.rhs_row.size());
    for (size_t p = 0; p < out.rhs_row.size(); ++p) {
        const int r = out.rhs_row[p];
        const bool single = blocks[blk[r]].size() == 1;
        out.dinv[p] = single ? 1.0 / diag[r] : 1.0;
        if (track) out.dsrc[p] = single ? dpos[r] : -1;
    }
}
