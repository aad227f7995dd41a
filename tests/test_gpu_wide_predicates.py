"""Exact signs in wide integers (csrc/cmg_exact.cuh, orient3d_wide / insphere_wide) around
the spans they take: coplanar and cospherical integer queries with one zero coordinate
replaced by +-2^-j, so that the coordinates span from a few to 130 bits (beyond 100 the
expansions decide), at three scales (near the wide form's exponent limits too). Signs
equal the oracle's in both modes."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _queries(kind, n, scale_exp, seed):
    from cybermeshgenerator_gb300 import workloads as W
    S = W.predicate_stream(n, kind, degenerate=1.0, near=0.0, seed=seed)
    S = np.round(S * 2.0 ** 11)  # integers of at most 20 bits (the stream's scale is 2^-3..2^-11)
    rng = np.random.default_rng(seed)
    # move every query so that a coordinate of one point is zero, then set it to +-2^-j
    npt = S.shape[0] // 3
    row = rng.integers(0, npt, n) * 3 + rng.integers(0, 3, n)
    off = S[row, np.arange(n)]
    for k in range(S.shape[0]):
        S[k] -= np.where(k % 3 == row % 3, off, 0.0)
    S[row, np.arange(n)] = rng.choice([-1, 1], n) * 2.0 ** -rng.integers(0, 112, n).astype(np.float64)
    S[row[: n // 8], np.arange(n // 8)] = 0.0  # exact ties remain among them
    return np.ascontiguousarray(S * 2.0 ** scale_exp)


@pytest.mark.parametrize("kind,scale_exp", [("orient3d", 0), ("orient3d", -190), ("orient3d", 270),
                                            ("insphere", 0), ("insphere", -60), ("insphere", 150)])
def test_spans_match_oracle(cm, orc, kind, scale_exp):
    import oracle as O
    S = _queries(kind, 20_000, scale_exp, 71)
    fn = cm.orient3d_stream if kind == "orient3d" else cm.insphere_stream
    for mode, om in ((cm.PRED_COMPAT, O.COMPAT), (cm.PRED_EXACT, O.EXACT)):
        got, st = fn(S, mode)
        assert np.array_equal(got, orc.stream(kind, S, om))
        # some spans are beyond the wide integers, most are not
        assert st["expansion_queries"] < 0.4 * S.shape[1]


@pytest.mark.parametrize("kind", ["orient3d", "insphere"])
@pytest.mark.parametrize("n,first", [(255, 1), (257, 1), (1023, 0), (1025, 3), (70_001, 1)])
def test_columns_off_a_16_byte_boundary(cm, orc, kind, n, first):
    """Device columns whose starts are 0 or 8 bytes off a 16-byte boundary (rows of odd length
    in one matrix, from an odd or even first value): the bulk copies read the words around
    them and the signs equal the oracle's."""
    import torch
    import oracle as O
    from cybermeshgenerator_gb300 import workloads as W
    S = W.predicate_stream(n, kind, degenerate=0.1, near=0.1, seed=n)
    d = torch.full((S.shape[0] * n + 8,), float("nan"), dtype=torch.float64, device="cuda")
    d[first:first + S.size] = torch.from_numpy(S.ravel())
    out = torch.zeros(n, dtype=torch.int8, device="cuda")
    fn = cm.orient3d_stream if kind == "orient3d" else cm.insphere_stream
    _, st = fn(([d.data_ptr() + 8 * (first + k * n) for k in range(S.shape[0])], n, out.data_ptr()),
               cm.PRED_COMPAT, torch.cuda.current_stream().cuda_stream)
    assert np.array_equal(out.cpu().numpy(), orc.stream(kind, S, O.COMPAT))
    assert st["tma_reruns"] == 0
