// gemm_plan.h - the schedule of a group of products (gemm_group.cu), on the host: plain C++, no device code.
//
// Every product has a tile width and may be cut into pieces of its k range; the last tiles of a launch are cut when that shortens it.  The kernel comes in two
// classes: tiles of 128, 192 and 256 columns (five stages, two accumulators), and of 64 and 128 (eight and four).  The widest tile costs least per
// multiply-add; a narrower one pays where the wide tiles leave the last round mostly empty (2816 columns of 2048 rows are 96 tiles of 256 on 74
// pairs, two rounds, or 128 of 192: two shorter ones) and where one product's long k would outlast all others (a weight gradient over 2048 tokens
// beside an input gradient over 512 columns).  The cost of an item is its k blocks plus an epilogue that the next item's first two chunks hide
// part of; a launch is the greedy schedule of its items on the CTA pairs.  The constants (microseconds per k block of 64, per epilogue, for the
// fix-up launch) are measured.
//
// A schedule depends on tiles and k blocks only, so that is its key: rows by the 256 of a tile, columns by 64, the narrowest tile's.  Steps on batches of
// unequal length meet new keys all the time (a weight gradient's k blocks are the tokens / 64), between two launches: a search takes 1.5 to 8 us
// on the host (4 to 19 before bounds cut it short).
#pragma once
#include <stdint.h>
#include <stdlib.h>
#include <string.h>

#define GG_MAXP 10               // products per launch
#define GG_MAXE (2 * GG_MAXP)    // runs of items: whole tiles, then pieces, of each product
struct GgPlanRun { int prob, tile0, tiles, split; };
struct GgPlan { int bn, nruns, w[GG_MAXP]; GgPlanRun run[GG_MAXE]; };
struct GgPlanKey { int nprob, nt, G; int mnk[GG_MAXP][3]; };      // nt: passes; G: CTA pairs; of each product the rows / 256, columns / 64 and k / 64, rounded up
#define GG_NARROWER 1.03f                     // a plan with narrower tiles has to win by more than the constants are worth
static inline void gg_key_add(GgPlanKey* k, int M, int N, int kb) {
    int* e = k->mnk[k->nprob++];
    e[0] = (M + 255) / 256; e[1] = (N + 63) / 64; e[2] = kb;
}

struct GgWidth { int bn; float t_kb[2], t_epi; };      // t_kb: three passes, one pass
static const GgWidth gg_wide[3] = {{256, {1.00f, 0.47f}, 4.3f}, {192, {0.82f, 0.43f}, 3.5f}, {128, {0.64f, 0.38f}, 2.6f}};
static const GgWidth gg_narrow[2] = {{128, {0.52f, 0.31f}, 2.3f}, {64, {0.42f, 0.27f}, 2.0f}};
// the fix-up launch, and for each column of 256 rows that is written for it and read: in L2, and beyond 16 MB (512 x 256 columns: 130 us)
static const float gg_t_fix = 3.0f, gg_t_fix_col = 2.5e-4f, gg_t_fix_far = 8e-4f, gg_fix_near = 16384.f;

struct GgSim { float t[64]; int c[64]; int n; };
// `count` items of one cost, each to the pair that is free first
static void gg_sim_add(GgSim* s, int count, float cost, int G) {
    if (count > 4 * G) {                                         // whole rounds first
        const int rounds = count / G - 2;
        for (int i = 0; i < s->n; i++) s->t[i] += rounds * cost;
        count -= rounds * G;
    }
    while (count > 0) {
        int lo = 0;
        for (int i = 1; i < s->n; i++) if (s->t[i] < s->t[lo]) lo = i;
        const int a = count < s->c[lo] ? count : s->c[lo];
        const float nt = s->t[lo] + cost;
        count -= a; s->c[lo] -= a;
        int hit = -1;
        for (int i = 0; i < s->n; i++) if (s->t[i] == nt || (s->n >= 60 && s->t[i] > nt - 0.5f * cost && s->t[i] < nt + 0.5f * cost)) { hit = i; break; }
        if (hit >= 0) s->c[hit] += a;
        else if (s->c[lo] == 0) { s->t[lo] = nt; s->c[lo] = a; continue; }
        else { s->t[s->n] = nt; s->c[s->n] = a; s->n++; }
        if (s->c[lo] == 0) { s->n--; s->t[lo] = s->t[s->n]; s->c[lo] = s->c[s->n]; }
    }
}
// What a plan chooses for each product: its tiles' width (of the class's table) and the pieces every one of them is cut into.
struct GgPick { unsigned char w[GG_MAXP], s[GG_MAXP]; };
static bool gg_can_cut(int kb, int s) { const int per = (kb + s - 1) / s; return s == 1 || (per * (s - 1) < kb && per >= 2); }
// The products of a launch at each width of a class: tiles, and the cost of an item, whole or one of s pieces.
struct GgCosts {
    const GgWidth* tab;
    int tiles[GG_MAXP][3]; float cost[GG_MAXP][3][9];
    bool cut[GG_MAXP][9];
};
static void gg_costs(const GgPlanKey* k, const GgWidth* tab, int nw, GgCosts* t) {
    t->tab = tab;
    for (int i = 0; i < k->nprob; i++) {
        const int kb = k->mnk[i][2];
        for (int s = 1; s <= 8; s++) t->cut[i][s] = gg_can_cut(kb, s);
        for (int w = 0; w < nw; w++) {
            t->tiles[i][w] = k->mnk[i][0] * ((k->mnk[i][1] + tab[w].bn / 64 - 1) / (tab[w].bn / 64));
            for (int s = 1; s <= 8; s++) t->cost[i][w][s] = (kb + s - 1) / s * tab[w].t_kb[k->nt == 1] + tab[w].t_epi;
        }
    }
}
// The launch of these choices; tail: pieces of the tiles that its last round holds, taken from the shortest uncut products (1: they stay whole).
// Returns its time, and the runs where p is given, or -1 when there is no such plan or none below `limit` (0: no limit).
struct GgSeg1 { float cost; int count, prob, split; };      // items of one cost: whole tiles (split 1) or pieces of a product
static float gg_eval(const GgPlanKey* k, const GgCosts* t, const GgPick* c, int tail, float limit, GgPlan* p) {
    const int n = k->nprob, G = k->G;
    int tiles[GG_MAXP], spl[GG_MAXP], cut[GG_MAXP], items = 0;
    for (int i = 0; i < n; i++) {
        if (!t->cut[i][c->s[i]]) return -1.f;
        tiles[i] = t->tiles[i][c->w[i]];
        spl[i] = c->s[i];
        cut[i] = spl[i] > 1 ? tiles[i] : 0;
        items += tiles[i] * spl[i];
    }
    int order[GG_MAXP];                                          // by the cost of a whole item, the longest first
    for (int i = 0; i < n; i++) {
        const float ci = t->cost[i][c->w[i]][1];
        int j = i;
        for (; j > 0 && t->cost[order[j - 1]][c->w[order[j - 1]]][1] < ci; j--) order[j] = order[j - 1];
        order[j] = i;
    }
    if (tail > 1) {
        int left = items % G;
        bool any = false;
        for (int o = n - 1; o >= 0 && left > 0; o--) {
            const int i = order[o];
            if (spl[i] > 1) continue;
            if (!t->cut[i][tail]) return -1.f;
            spl[i] = tail; cut[i] = tiles[i] < left ? tiles[i] : left; left -= cut[i]; any = true;
            items += cut[i] * (tail - 1);
        }
        if (!any) return -1.f;
    }
    // the items, longest first, whole or pieces
    GgSeg1 seg[GG_MAXE];
    int ns = 0;
    float slots = 0.f, work = 0.f;
    for (int o = 0; o < n; o++) { const int i = order[o]; if (tiles[i] > cut[i]) seg[ns++] = {t->cost[i][c->w[i]][1], tiles[i] - cut[i], i, 1}; }
    for (int i = 0; i < n; i++) {
        if (!cut[i]) continue;
        const GgSeg1 e = {t->cost[i][c->w[i]][spl[i]], cut[i] * spl[i], i, spl[i]};
        int j = ns++;
        for (; j > 0 && seg[j - 1].cost < e.cost; j--) seg[j] = seg[j - 1];
        seg[j] = e;
        slots += (float)e.count * t->tab[c->w[i]].bn;
    }
    for (int a = 0; a < ns; a++) work += seg[a].count * seg[a].cost;
    const float fix = slots > 0.f ? gg_t_fix : 0.f;
    float time = seg[0].cost;                                    // one round of items, each on a pair of its own
    if (limit > 0.f && (work > time * G ? work / G : time) + fix >= limit) return -1.f;      // the longest item, or the work spread evenly: no schedule is shorter
    if (items > G) {
        // Some pair has r + 1 of the r G + 1 longest items: no less than the shortest r + 1 of those.
        const int r = (items - 1) / G;
        if (limit > 0.f && r <= 8) {
            float least = 0.f;
            for (int a = 0, left = r * G + 1, need = r + 1; need > 0; a++) {
                int last = left < seg[a].count ? left : seg[a].count;      // of this cost among the r G + 1
                left -= last;
                if (left >= need) continue;
                if (last > need - left) last = need - left;
                least += last * seg[a].cost; need -= last;
            }
            if (least * 0.9999f + fix >= limit) return -1.f;
        }
        GgSim q;
        q.n = 1; q.t[0] = 0.f; q.c[0] = G;
        for (int a = 0; a < ns; a++) gg_sim_add(&q, seg[a].count, seg[a].cost, G);
        time = 0.f;
        for (int i = 0; i < q.n; i++) if (q.t[i] > time) time = q.t[i];
    }
    if (slots > 0.f) time = (time + fix + slots * gg_t_fix_col + (slots > gg_fix_near ? (slots - gg_fix_near) * (gg_t_fix_far - gg_t_fix_col) : 0.f)) * 1.02f;
    if (p) {
        p->nruns = ns; p->bn = t->tab[0].bn;
        for (int a = 0; a < ns; a++) { const GgSeg1& e = seg[a]; const int i = e.prob; p->run[a] = {i, e.split > 1 ? tiles[i] - cut[i] : 0, e.count / e.split, e.split}; }
        for (int i = 0; i < n; i++) p->w[i] = t->tab[c->w[i]].bn;
    }
    return time;
}
static void gg_make_plan(const GgPlanKey* k, GgPlan* plan) {
    // products of one shape share their choice
    int kind_of[GG_MAXP], first[GG_MAXP], count_of[GG_MAXP], nk = 0;
    for (int i = 0; i < k->nprob; i++) {
        kind_of[i] = -1;
        for (int j = 0; j < i && kind_of[i] < 0; j++) if (memcmp(k->mnk[i], k->mnk[j], sizeof k->mnk[i]) == 0) kind_of[i] = kind_of[j];
        if (kind_of[i] < 0) { first[nk] = i; count_of[nk] = 0; kind_of[i] = nk++; }
        count_of[kind_of[i]]++;
    }
    static const unsigned char pieces[6] = {1, 2, 3, 4, 6, 8}, tails[6] = {2, 3, 4, 5, 6, 8};
    float best_t = 0.f;
    GgPick best;
    int best_tail = 1, best_cls = -1;
    GgCosts costs[2];
    for (int cls = 0; cls < 2; cls++) {
        const int nw = cls ? 2 : 3;
        GgCosts* tab = &costs[cls];
        gg_costs(k, cls ? gg_narrow : gg_wide, nw, tab);
        int total = 0;
        for (int i = 0; i < k->nprob; i++) total += tab->tiles[i][0];
        const bool many = total > 6 * k->G;                      // many rounds: no empty last one to speak of, and no product that outlasts the rest
        for (int base = 0; base < (many ? 1 : nw); base++) {
            GgPick c;
            memset(&c, 0, sizeof c);
            for (int i = 0; i < k->nprob; i++) { c.w[i] = (unsigned char)base; c.s[i] = 1; }
            const float off = cls || base ? GG_NARROWER : 1.f;
            float t = gg_eval(k, tab, &c, 1, 0.f, nullptr) * off;
            auto take = [&](const GgPick& v, int tail, float tv) { best = v; best_tail = tail; best_cls = cls; best_t = tv; };
            if (best_cls < 0 || t < best_t) take(c, 1, t);
            auto cut_tail = [&]() {
                float work = 0.f;                                // pieces only add to it
                for (int i = 0; i < k->nprob; i++) work += tab->tiles[i][c.w[i]] * c.s[i] * tab->cost[i][c.w[i]][c.s[i]];
                if ((work / k->G + gg_t_fix) * 0.999f >= best_t) return;
                for (int q = 0; q < 6; q++) {
                    const float tv = gg_eval(k, tab, &c, tails[q], best_t, nullptr) * off;
                    if (tv > 0.f && tv < best_t) take(c, tails[q], tv);
                }
            };
            cut_tail();
            // one kind of product after the other to its best choice beside the others'
            for (int sweep = 0; sweep < (many ? 0 : 2); sweep++) {
                bool moved = false;
                for (int kd = 0; kd < nk; kd++) {
                    float work = 0.f, longest = 0.f;             // the others'
                    bool fix = false;
                    for (int i = 0; i < k->nprob; i++) {
                        if (kind_of[i] == kd) continue;
                        const float ci = tab->cost[i][c.w[i]][c.s[i]];
                        work += tab->tiles[i][c.w[i]] * c.s[i] * ci;
                        if (ci > longest) longest = ci;
                        if (c.s[i] > 1) fix = true;
                    }
                    GgPick top = c;
                    const int f = first[kd];
                    for (int w = 0; w < nw; w++)
                        for (int q = 0; q < 6; q++) {
                            const int s = pieces[q];
                            if (!tab->cut[f][s] || (w == c.w[f] && s == c.s[f])) continue;
                            // no launch takes less than its longest item, or than its work spread evenly
                            const float cw = tab->cost[f][w][s], lo = (work + count_of[kd] * tab->tiles[f][w] * s * cw) / k->G, lb = lo > cw ? lo : cw;
                            const float narrower = cls || w || base ? GG_NARROWER : 1.f;
                            if (((lb > longest ? lb : longest) + (fix || s > 1 ? gg_t_fix : 0.f)) * narrower * 0.9999f >= t) continue;
                            GgPick v = c;
                            for (int i = 0; i < k->nprob; i++) if (kind_of[i] == kd) { v.w[i] = (unsigned char)w; v.s[i] = pieces[q]; }
                            const float tv = gg_eval(k, tab, &v, 1, t, nullptr) * narrower;
                            if (tv > 0.f && tv < t) { t = tv; top = v; moved = true; if (t < best_t) take(v, 1, t); }
                        }
                    c = top;
                }
                if (!moved) break;
            }
            if (!many) cut_tail();
        }
    }
    gg_eval(k, &costs[best_cls], &best, best_tail, 0.f, plan);
}

// Plans that were made before, by key: eight to a set, the oldest leaves.  The ten groups of a model's step have 5 x 32 forward and 5 x 128 backward keys over all
// lengths up to 8192 tokens; four to a set, a few sets held five and searched on and on.
#define GG_PLAN_SETS 512
#define GG_PLAN_WAYS 8
struct GgPlanEntry { GgPlanKey key; GgPlan plan; };
struct GgPlanTable { unsigned searches; unsigned char n[GG_PLAN_SETS], next[GG_PLAN_SETS]; GgPlanEntry e[GG_PLAN_SETS][GG_PLAN_WAYS]; };      // zeros: empty
static const GgPlan* gg_plan_find(GgPlanTable* t, const GgPlanKey* key) {
    uint64_t h = 1469598103934665603ull;
    const int* w = (const int*)key;
    for (size_t i = 0; i < sizeof *key / sizeof(int); i++) { h ^= (uint64_t)(uint32_t)w[i]; h *= 0x9E3779B97F4A7C15ull; h ^= h >> 29; }
    const unsigned set = (unsigned)(h % GG_PLAN_SETS);
    for (int i = 0; i < t->n[set]; i++) if (memcmp(&t->e[set][i].key, key, sizeof *key) == 0) return &t->e[set][i].plan;
    GgPlanEntry* e = &t->e[set][t->next[set]];
    t->next[set] = (t->next[set] + 1) % GG_PLAN_WAYS;
    if (t->n[set] < GG_PLAN_WAYS) t->n[set]++;
    gg_make_plan(key, &e->plan);
    e->key = *key;
    t->searches++;
    return &e->plan;
}
