"""The costs of the bench-size fixtures without the reference shim: the
product's own tap samples (measured equal to the shim's bit for bit) tell which
of the reference's values lie off the exact NCC of those samples, at most a
thousandth of a field; there the product is held to that exact value, elsewhere
to the reference and the oracle, by the bounds of ncc_split."""
import numpy as np
import pytest

import ncc_split
import oracle as orc
from test_gpu_parity_bench import K_ERR, _sample, case  # noqa: F401  (the fixture)

pytestmark = pytest.mark.gpu


def test_costs_against_their_own_samples_the_reference_and_the_oracle(case):  # noqa: F811
    name, g, c, ctx = case
    px = c["pixels"]
    for k, p in enumerate(c["planes"]):
        what = f"{name} field {k}"
        got = _sample(ctx.cost_vectors(p), px)
        samples, inside = ctx.tap_samples(p, px)
        exact = ncc_split.exact_costs(samples, inside, c["imgs"][0], px)
        ncc_split.check_exact(got, samples, inside, c["imgs"][0], px, f"{what} vs its samples")
        ocost, bound, acc, _ = orc.ncc_bounds(c["imgs"], c["cams"], p, K_ERR, pixels=px)
        ref = g["cost_vectors"][k]
        off = ncc_split.reference_self_inconsistent(ref, exact, bound + acc)
        print(what, [(int(i), float(ref.flat[i]), float(exact.flat[i]), float(got.flat[i])) for i in np.flatnonzero(off)])
        ncc_split.check_within_bound(got, ref, bound + acc, f"{what} vs reference", exact=exact, exempt=off)
        ncc_split.check_within_bound(got, ocost, bound + acc, f"{what} vs oracle", exempt=off)
