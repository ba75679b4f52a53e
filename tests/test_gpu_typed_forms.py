"""The typed forms of the frequent training ops (ready-queue kernel) against the general bodies (static kernel): the same bits on the same
input, at the sizes where a typed form changes its instance, its buffering or hands over to the general body."""
import numpy as np
import pytest

from kvm_b200.executor import CFG_DYNAMIC, CFG_STATIC, Executor
from kvm_b200.workloads.graph import Graph

pytestmark = pytest.mark.gpu


def same_bits(g):
    b = g.to_bundle()
    got = []
    for flags in (CFG_DYNAMIC, CFG_STATIC):
        with Executor(flags=flags) as ex:
            ex.load(b)
            assert ex.run().done == len(b.tasks)
            assert ex.plan_info()[0] == (flags == CFG_STATIC)
            got.append({s['name']: ex.read_buffer(s['name']) for s in b.buffers})
    for name, x in got[0].items():
        assert np.array_equal(x.view(np.uint32), got[1][name].view(np.uint32)), name
    return got[0]


def normal(seed, *shape):
    return np.random.default_rng(seed).standard_normal(shape).astype(np.float32)


# eight elements are the smallest typed range, 8192 a stage of the stream, four of them its depth; multiples of four only go to the general body
@pytest.mark.parametrize('n', [8, 12, 24, 4096, 8192, 8200, 32768, 40968])
def test_gradnorm_partial(kvm_lib, n):
    g = Graph('gradnorm')
    for i in range(6):
        g.data(f'g{i}', normal(i, 1, n + 8))
        g.buffer(f'p{i}', 1, 2)
        for slot in (0, 1):
            g.task('gradnorm_partial', {'g': f'g{i}', 'partial': f'p{i}', 'slot': slot, 'e0': 8 * slot, 'e1': n + 8 * slot}, [f'g{i}'], [(f'p{i}', (0, 1), (slot, slot + 1))])
    same_bits(g)
