"""The time the batch planner's item sizing takes (host logic, through
rfmf_debug_plan_items): it runs before the launches whose items it sizes, so a
class of many graphs that needs more than one round of its CTAs must be planned
in well under a millisecond, not by trying every graph at every step."""
import time

import numpy as np
import pytest


@pytest.mark.parametrize("graphs,chains,most_ms", [(64, 12, 1.5), (512, 64, 25.0)])
def test_many_graphs_are_planned_quickly(rfmf, graphs, chains, most_ms):
    rng = np.random.default_rng(graphs)
    level4 = np.exp(rng.uniform(np.log(2.0), np.log(9.0), graphs))
    ns = [[t * (l + 2) / 6 for l in (1, 2, 3, 4)] for t in level4]
    best = 1e9
    for _ in range(20):
        t0 = time.perf_counter()
        kg = rfmf.debug_plan_items([chains] * graphs, 4, 4, ns, 152)
        best = min(best, time.perf_counter() - t0)
    assert all(1 <= k <= 4 for k in kg)
    assert best * 1e3 < most_ms, best


def test_grouped_schedule_is_the_list_schedule(rfmf):
    # sizes chosen for a small class: no single step down from them shortens the
    # longest-first list schedule of single items
    rng = np.random.default_rng(3)
    for _ in range(20):
        G, slots = int(rng.integers(2, 7)), int(rng.integers(5, 30))
        chains = [int(c) for c in rng.integers(1, 60, G)]
        ns = [list(np.cumsum(rng.uniform(0.5, 2.0, 4))) for _ in range(G)]

        def makespan(kg):
            items = []
            for c, k, t in zip(chains, kg, ns):
                items += [t[k - 1]] * (c // k)
                if c % k:
                    items.append(t[c % k - 1])
            free = [0.0] * slots
            for t in sorted(items, reverse=True):
                free.sort()
                free[0] += t
            return max(free)

        kg = rfmf.debug_plan_items(chains, 4, 4, ns, slots)
        if sum(-(-c // k) for c, k in zip(chains, kg)) <= slots:
            continue   # one round: the makespan rule, tested elsewhere
        at = makespan(kg)
        for q in range(G):
            if kg[q] > 1:
                assert makespan(kg[:q] + [kg[q] - 1] + kg[q + 1:]) >= at * (1 - 1e-9)
