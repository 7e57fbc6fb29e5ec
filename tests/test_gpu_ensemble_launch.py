"""Ensemble launches set by hand: any z chunk of at least one plane is taken,
the largest int included (whole lattices, as a chunk of the members' height)."""
import numpy as np
import pytest

from entropicthreadsafe_b200 import capi, ensemble

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("zchunk", (1, 2 ** 31 - 64, 2 ** 31 - 1))
def test_any_z_chunk_gives_the_same_steps(zchunk):
    doms = ensemble.couette_droplets(n=3, seed=5)
    out = []
    for zc in (1 << 20, zchunk):
        with ensemble.Ensemble([d["params"] for d in doms], [d["dims"] for d in doms]) as ens:
            for i, d in enumerate(doms):
                ens.upload_moments(i, d["fields"])
            ens.set_launch(zc, 0)
            ens.step(2)
            ens.synchronize()
            out.append([ens.download(i) for i in range(len(doms))])
    for a, b in zip(*out):
        for k in capi.FIELDS:
            assert np.array_equal(a[k], b[k]), k   # the cut does not change a node's sums
