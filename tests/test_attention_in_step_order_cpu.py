"""The second fixed order of the attention backward's dQ additions (``csrc/attention.cu``, ``BWD_IN_STEP``), replayed on the
host like the first: key tiles ascending, query tiles descending with the heads of the group inside, a CTA waiting for the
key tiles below its own that touch the query tile.  With any number of resident CTAs every wait must be satisfiable by CTAs
handed out before, every counter must end at the number of key tiles that touch its query tile, and the additions must come
in strictly ascending key-tile order.  Here a turn passes on at once."""
import random

import pytest

from test_attention_order_cpu import TQ, replay, row_groups


def ctas_in_dispatch_order(lens_q, lens_k, causal, window, rep, grid_slack=3):
    n_tiles = [(lk + TQ - 1) // TQ for lk in lens_k]
    qtile_base, acc = [], 0
    for lq in lens_q:
        qtile_base.append(acc)
        acc += (lq + TQ - 1) // TQ
    out = []
    for tile in range(sum(n_tiles)):                  # blocks past the real tile count exit at once
        a = 0
        for seq, nt in enumerate(n_tiles):
            if tile < a + nt:
                break
            a += nt
        k0 = (tile - a) * TQ
        len_q, len_k = lens_q[seq], lens_k[seq]
        off, kr = len_k - len_q, min(TQ, len_k - k0)
        i_lo = max(0, k0 - off) if causal else 0
        i_hi = min(len_q, k0 + kr + window - 1 - off) if (causal and window > 0) else len_q
        i_lo = (i_lo // TQ) * TQ
        n_qt = (i_hi - i_lo + TQ - 1) // TQ if i_hi > i_lo else 0
        its, qt, h = [], i_lo + (n_qt - 1) * TQ, 0
        for _ in range(n_qt * rep):
            j_lo = max(0, qt + off - window + 1) // TQ if causal and window > 0 else 0
            its.append(((qtile_base[seq] + qt // TQ, h), k0 // TQ - j_lo, k0 // TQ, row_groups(len_q - qt)))
            h += 1
            if h == rep:
                h, qt = 0, qt - TQ
        out.append((seq, k0, its))
    return out


@pytest.mark.parametrize("seed", range(40))
def test_in_step_order_is_satisfiable_and_ascending(seed):
    rng = random.Random(seed)
    n = rng.randint(1, 4)
    causal = rng.random() < 0.8
    lens_q = [rng.randint(1, 900) for _ in range(n)]
    lens_k = [lq + rng.choice((0, 0, 1, 127, 128, 700)) for lq in lens_q]
    window = rng.choice((0, 0, 1, 100, 128, 129, 300)) if causal else 0
    ctas = ctas_in_dispatch_order(lens_q, lens_k, causal, window, rng.choice((1, 2, 4)))
    for resident in (1, 2, 5, 1000):
        done, sem, order = replay(ctas, resident, late=False)
        assert done
        for key, tiles in order.items():
            assert tiles == sorted(set(tiles)) and sem[key] == len(tiles)
        assert sum(map(len, order.values())) == sum(groups for c in ctas for *_, groups in c[2])
