"""Readouts of a sum against the oracle: patterns whose items start, end and run over the borders of
the plane words, with every item kind (position, star, repeat, repeat 0), on plain and lossy
sums; the largest weight against the weights of the exported terms."""

import numpy as np
import pytest

from ppvm_b200.paulisum import PauliSum

from tests.helpers import oracle_from
from tests.test_gpu_loss import gpu, lossy_oracle_from, random_lossy_terms

pytestmark = pytest.mark.gpu


def random_terms(rng, n, m):
    terms = {}
    for _ in range(m):
        p = rng.choice([0.02, 0.3, 0.9])
        w = "".join("XYZ"[int(rng.integers(3))] if rng.random() < p else "I" for _ in range(n))
        terms[w] = float(rng.uniform(-1, 1))
    return list(terms.items())


def random_pattern(rng, n):
    out = []
    for _ in range(int(rng.integers(1, 4))):
        acc = ["X", "Y", "Z", "_", "X?", "Z?", "[XY]", "[XZ]?", "[XYZ]", "[XYZ]?"][int(rng.integers(10))]
        pos = int(rng.choice([0, 1, n // 2, n - 1, 62, 63, 64, 65, int(rng.integers(0, n + 2))]))
        out.append(acc + ["*", "{%d}" % int(rng.integers(0, 4)), "{%d}" % max(pos, 0), str(pos)][int(rng.integers(4))])
    return "".join(out)


def patterns(rng, n, terms):
    pats = ["Z?*", "[XYZ]?*", "[XY]?*", "_*", "[XZ]?{%d}" % n, "_{%d}[XYZ]?*" % (n // 2), "X0", "Z%d" % (n - 1)]
    for w, _ in terms[:20]:  # patterns that match a term: its own letters by position, and by stretch
        at = [(i, c) for i, c in enumerate(w) if c != "I"]
        pats.append("".join(f"{c}{i}" for i, c in at) or "_*")
        if at:
            pats.append("_{%d}[XYZ]?{%d}" % (at[0][0], at[-1][0] - at[0][0] + 1))
    return pats + [random_pattern(rng, n) for _ in range(60)]


@pytest.mark.parametrize("n", [1, 5, 63, 64, 65, 127, 128, 129, 200])
def test_traces_match_the_oracle(n):
    rng = np.random.default_rng(n)
    terms = random_terms(rng, n, 300)
    g = PauliSum([w for w, _ in terms], n, [c for _, c in terms], min_abs_coeff=0.0)
    o = oracle_from(terms, n, 0.0)
    for pat in patterns(rng, n, [(w, c) for w, c in terms if set(w) <= set("IXYZ")]):
        assert abs(g.trace(pat) - o.trace(pat)) < 1e-10, pat
    assert g.current_max_weight() == max(w for _, w in g.weights())


@pytest.mark.parametrize("n", [3, 63, 64, 65, 200])
def test_lossy_traces_match_the_oracle(n):
    rng = np.random.default_rng(50 + n)
    terms = random_lossy_terms(rng, n, min(200, 5 ** n // 2))
    g, o = gpu(terms, n), lossy_oracle_from(terms, n, thr=0.0)
    for pat in patterns(rng, n, [(w, c) for w, c in terms if "L" not in w]):
        assert abs(g.trace(pat) - o.trace(pat)) < 1e-10, pat
    assert g.current_max_weight() == max(w for _, w in g.weights())
