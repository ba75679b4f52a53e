"""GPU parity at the sizes where the small-shape kernel forms can go wrong: 32x32 exact matmul tiles, attention of ragged sequences and every
head dimension, streamed decode rows that are no multiple of 256 columns and odd query-head groups."""
import numpy as np
import pytest

from tests.parity import compare, run_both
from tests.test_gpu_attention import attn_bundle
from tests.test_gpu_gemm import gemm_bundle

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize('flags', [0, 1, 2, 3])
@pytest.mark.parametrize('shape', [(1, 1, 1), (32, 32, 512), (31, 17, 33), (32, 10, 100), (7, 32, 200), (32, 32, 127)])
def test_matmul_tile_32_is_bit_exact(kvm_lib, flags, shape):
    M, N, K = shape
    ex, vm, res = run_both(gemm_bundle('matmul_tile', M, N, K, flags, 'f32', 'f32', bias=True))
    assert np.array_equal(ex.read_buffer('out'), vm.buffer('out').a)
    ex.close()


@pytest.mark.parametrize('case', [(1, 5, 1, 1, 16, 'f32'), (2, 17, 2, 1, 32, 'f32'), (1, 129, 3, 1, 64, 'f32'), (1, 257, 2, 2, 128, 'f32'), (1, 257, 2, 1, 64, 'bf16'),
                                  (1, 300, 2, 1, 128, 'bf16'), (3, 33, 1, 1, 32, 'bf16')])
def test_attention_ragged(kvm_lib, case):
    B, T, H, Hkv, hd, dt = case
    ex, vm, res = run_both(attn_bundle(B, T, H, Hkv, hd, dt))
    assert ex.tc_task_count() == 0
    compare(ex, vm, 2e-5 if dt == 'f32' else 6e-3)
    ex.close()


# hidden, heads, kv heads, head dim, ffn: seven query heads per key head; rows of 8 .. more than 12288 columns; one head each
@pytest.mark.parametrize('widths', [(448, 14, 2, 32, 712), (896, 14, 2, 64, 1096), (72, 1, 1, 128, 12552), (264, 6, 2, 64, 520), (128, 8, 1, 128, 136)])
@pytest.mark.parametrize('qk_norm', [False, True])
def test_decode_streams_odd_widths(kvm_lib, widths, qk_norm):
    from kvm_b200.executor import Executor
    from kvm_b200.workloads.decode import DecodeConfig, build_decode
    from oracle.vm_np import VM
    hidden, heads, kv, hd, ffn = widths
    b = build_decode(DecodeConfig(hidden=hidden, heads=heads, kv_heads=kv, head_dim=hd, ffn=ffn, vocab=304, ctx=70, init_std=0.05, qk_norm=qk_norm)).to_bundle()
    vm = VM(b).run()
    with Executor() as ex:
        ex.load(b)
        assert ex.run().done == len(b.tasks)
        assert ex.plan_info()[:2] == (True, True)
        for name in ('u0.logits', 'u0.l1.x2'):
            ref = vm.buffer(name).a
            assert np.abs(ex.read_buffer(name) - ref).max() <= 1e-2 * np.abs(ref).max(), name


# rows of masked logits: all columns -inf, NaN before them, and a single finite value, around the 8192 columns that a pass in pieces takes
@pytest.mark.parametrize('V', [8191, 8192, 8200, 16390])
def test_argmax_of_masked_rows(kvm_lib, V):
    from kvm_b200.workloads.graph import Graph
    rows = np.full((4, V), -np.inf, np.float32)
    rows[1, :100] = np.nan
    rows[2, V - 1] = 0.0
    rows[3, [5000, V - 2]] = 1.0
    g = Graph('argmax')
    g.data('l', rows), g.buffer('t', 4, 1, 'i32')
    g.task('argmax', {'logits': 'l', 'out': 't', 'r0': 0, 'r1': 4, 'V': V}, ['l'], ['t'])
    ex, vm, res = run_both(g.to_bundle())
    assert ex.read_buffer('t').ravel().tolist() == [0, 0, V - 1, 5000] == vm.buffer('t').a.ravel().tolist()
    ex.close()


# rows of two, three and four pieces per thread, normalised and plain: the loop over a thread's pieces with its remainder
@pytest.mark.parametrize('K', [4104, 8192, 12280, 12296])
def test_streamed_gemv_of_several_pieces(kvm_lib, K):
    from kvm_b200.workloads.graph import Graph
    rng = np.random.default_rng(K)
    g = Graph('pieces')
    g.data('x', rng.standard_normal((1, K)).astype(np.float32)), g.data('u', rng.standard_normal((1, K)).astype(np.float32))
    g.data('w', (rng.standard_normal((70, K)) * 0.02).astype(np.float32), 'bf16'), g.data('res', rng.standard_normal((1, 70)).astype(np.float32))
    for pro in (0, 1, 2):
        g.buffer(f'o{pro}', 1, 70)
        for n0, n1 in ((0, 33), (33, 70)):
            g.task('gemv_bf16', {'x': 'x', 'x2': 'u', 'gamma': 'u', 'w': 'w', 'out': f'o{pro}', 'res': 'res', 'n0': n0, 'n1': n1, 'K': K, 'pro': pro, 'eps': 1e-6},
                   ['x'], [(f'o{pro}', (0, 1), (n0, n1))])
    ex, vm, res = run_both(g.to_bundle())
    assert ex.plan_info()[:2] == (True, True)
    # an activation on a rounding tie of bf16 may fall on the other side: 2^-9 of one of K terms
    compare(ex, vm, 2.0 ** -9 / K ** 0.5 * 4)
    ex.close()
