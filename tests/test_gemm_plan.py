"""The schedule of grouped products (seraph_b200/csrc/gemm_plan.h), compiled for the host: every tile of every product is dealt once, in pieces that
hold k blocks; and a batch of another length costs a search only where tiles or k blocks differ."""
import os
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

DRIVER = r"""
#include "gemm_plan.h"
#include <stdio.h>
static GgPlanTable* table;
struct P { int M, N, K; };
static GgPlanKey key_of(const P* p, int n, int nt, int G) {
    GgPlanKey k;
    memset(&k, 0, sizeof k);
    k.nt = nt; k.G = G;
    for (int i = 0; i < n; i++) gg_key_add(&k, p[i].M, p[i].N, (p[i].K + 63) / 64);
    return k;
}
static int check(const P* p, int n, const GgPlan* plan) {
    static int seen[1 << 20];
    if (plan->nruns < 1 || plan->nruns > GG_MAXE || (plan->bn != 128 && plan->bn != 256)) return 1;
    for (int i = 0; i < n; i++) {
        const int bn = plan->w[i], kb = (p[i].K + 63) / 64;
        if (plan->bn == 256 ? bn != 128 && bn != 192 && bn != 256 : bn != 64 && bn != 128) return 2;
        const int tiles = (p[i].M + 255) / 256 * ((p[i].N + bn - 1) / bn);
        if (tiles > (1 << 20)) return 3;
        memset(seen, 0, tiles * sizeof(int));
        for (int r = 0; r < plan->nruns; r++) {
            const GgPlanRun* q = &plan->run[r];
            if (q->prob != i) continue;
            if (q->tiles < 1 || q->tile0 < 0 || q->tile0 + q->tiles > tiles || q->split < 1 || q->split > 8) return 4;
            const int per = (kb + q->split - 1) / q->split;
            if (q->split > 1 && per * (q->split - 1) >= kb) return 5;      // an empty piece
            for (int t = 0; t < q->tiles; t++) seen[q->tile0 + t]++;
        }
        for (int t = 0; t < tiles; t++) if (seen[t] != 1) return 6;
    }
    return 0;
}
static void clear() { memset(table, 0, sizeof *table); }
// the groups of a full training step: d, q and kv columns, F, V
static unsigned step(int T, int d, int qd, int kvd, int F, int V) {
    const unsigned before = table->searches;
    const P g[10][4] = {{{T, qd, d}, {T, kvd, d}, {T, kvd, d}}, {{T, d, qd}}, {{T, F, d}, {T, F, d}}, {{T, d, F}}, {{T, V, d}},
                        {{T, d, V}, {V, d, T}}, {{T, F, d}, {d, F, T}}, {{T, d, 2 * F}, {F, d, T}, {F, d, T}}, {{T, qd, d}, {d, qd, T}}, {{T, d, qd + 2 * kvd}, {qd, d, T}, {kvd, d, T}, {kvd, d, T}}};
    for (int i = 0; i < 10; i++) {
        int n = 0;
        while (n < 4 && g[i][n].M) n++;
        const GgPlanKey k = key_of(g[i], n, 3, 74);
        const GgPlan* p = gg_plan_find(table, &k);
        const int bad = check(g[i], n, p);
        if (bad) { printf("T %d group %d: plan fails check %d\n", T, i, bad); exit(1); }
    }
    return table->searches - before;
}
int main() {
    table = (GgPlanTable*)calloc(1, sizeof *table);
    srand(7);
    for (int r = 0; r < 20000; r++) {
        P p[GG_MAXP];
        const int n = 1 + rand() % GG_MAXP;
        for (int i = 0; i < n; i++) {
            int* e = &p[i].M;
            for (int j = 0; j < 3; j++) { const int b = 8 << rand() % 10; e[j] = b + rand() % b; }
            if (i && rand() % 3 == 0) p[i] = p[i - 1];
        }
        const GgPlanKey k = key_of(p, n, rand() % 2 ? 1 : 3, 1 + rand() % 74);
        const int bad = check(p, n, gg_plan_find(table, &k));
        if (bad) { printf("random group %d: plan fails check %d\n", r, bad); return 1; }
    }
    // a batch a few tokens longer or shorter: nothing new
    clear();
    const unsigned first = step(2048, 512, 512, 512, 1408, 8192), repeat = step(2048, 512, 512, 512, 1408, 8192);
    unsigned near = 0;
    for (int T = 2048 - 63; T < 2048; T++) near += step(T, 512, 512, 512, 1408, 8192);
    // batches of any length, twice over: a search for each count of row tiles or k blocks, and no more the second time
    clear();
    unsigned once = 0, again = 0;
    for (int i = 0; i < 8192; i++) once += step(1 + i * 2053 % 8192, 512, 512, 512, 1408, 8192);
    for (int i = 0; i < 8192; i++) again += step(1 + i * 2053 % 8192, 512, 512, 512, 1408, 8192);
    printf("%u %u %u %u %u\n", first, repeat, near, once, again);
    return 0;
}
"""


@pytest.fixture(scope="module")
def counts(tmp_path_factory):
    d = tmp_path_factory.mktemp("plan")
    src, exe = str(d / "driver.cpp"), str(d / "driver")
    with open(src, "w") as f:
        f.write(DRIVER)
    subprocess.run(["g++", "-O2", "-fsanitize=address,undefined", "-fno-sanitize-recover", "-I" + os.path.join(ROOT, "seraph_b200", "csrc"), src, "-o", exe], check=True)
    r = subprocess.run([exe], capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stdout + r.stderr
    return [int(x) for x in r.stdout.split()]


def test_every_tile_is_dealt_once_and_lengths_share_plans(counts):
    first, repeat, near, once, again = counts
    assert 0 < first <= 10 and repeat == 0
    assert near == 0                                  # the same row tiles and k blocks
    assert once <= 5 * 32 + 5 * 128                   # five groups know a length by its row tiles (256), five by its k blocks (64)
    assert again == 0
