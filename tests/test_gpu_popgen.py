"""RS_populate's draws made on the device (rsc_popgen.cuh): the state
rsc_populate_upload leaves equals rsc_populate_host's, value for value, around
the sizes of its chunks of draws."""
import numpy as np
import pytest

from simradar_gb300 import synth

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("counts,concept,seed", [
    ([1], synth.CONCEPT_DBU, 1),
    ([4], 0, 0),
    ([1024, 1], synth.CONCEPT_DBU, 5),
    ([1025, 0, 30], 0, 0xFFFFFFFF),
    ([4097, 2047], synth.CONCEPT_DBU, 77),
    ([0, 5000], synth.CONCEPT_DBU, 9),
    ([70001], 0, 123456789),
])
def test_draws_equal_host(backend, counts, concept, seed):
    S = synth.make_scene(num_rain=1, les_count=1, with_tables=False)
    args = backend.PopulateArgs.make(seed, concept, S.box[:3], S.box[3:], counts, S.dsd_r, S.dsd_cdf)
    n = sum(counts) + 3
    host, pop_h = backend.populate_host(args, n)
    W = backend.Worker(0)
    W.malloc(n, S.range_start, S.range_delta, S.range_count)
    for _ in range(2):
        pop_d = backend.populate_upload(W, args)
        got = W.download(("pos", "vel", "ori", "tum", "aux", "rcs", "rnd"))
        for f, a in got.items():
            assert np.array_equal(a.view(np.uint32), host[f].view(np.uint32)), f
        assert np.array_equal(pop_d, pop_h)
    W.close()
