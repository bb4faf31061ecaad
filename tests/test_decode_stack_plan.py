"""How the kernel of a decode step's layers divides its work, on the host."""
import ctypes

import pytest

SIZES = [(2560, 9728, 32, 8), (2048, 6144, 16, 8), (4096, 12288, 32, 8), (1024, 3072, 16, 8), (256, 1216, 4, 2),
         (320, 2432, 8, 1)]


@pytest.fixture(scope="module")
def lib():
    from grout_b200.kernels.build import module
    return module("decode_stack")


@pytest.mark.parametrize("blocks", [132, 144, 148, 160])
@pytest.mark.parametrize("sizes", SIZES, ids=str)
def test_every_row_is_one_blocks(lib, sizes, blocks):
    hidden, ff, nq, nkv = sizes
    if lib.gb_decode_stack_layer_bytes(*sizes, blocks) == 0:
        assert blocks != 148
        pytest.skip("no plan for this many blocks")
    for T in (1, 2, 4, 5, 8):
        out = (ctypes.c_int * 12)()
        rows, cols, halves = [], [], []
        for p in range(blocks):
            assert lib.gb_decode_stack_share(hidden, ff, nq, nkv, blocks, T, p, out) == 0
            q0, nq_rows, c0, nc, first, whole, half, slot, slots, at, kb_qkv, kb_o = out
            rows += range(q0, q0 + nq_rows)
            cols += range(c0, c0 + nc)
            halves += range(2 * first, 2 * (first + whole))
            if half >= 0:       # in front of the whole groups or behind them, in the other half of a neighbour's group
                assert half in (2 * first - 1, 2 * (first + whole))
                halves.append(half)
            gate_rows = 16 * whole + (8 if half >= 0 else 0)
            # a stage and its activations fit in a slot; the tiles of keys too
            assert 128 * max(gate_rows, nq_rows * kb_qkv, nc * kb_o) <= at and 16384 <= at and at % 1024 == 0
            assert at + 128 * T * max(kb_qkv, kb_o) <= slot and slot % 1024 == 0 and 6 <= slots <= 12
        assert rows == list(range((nq + 2 * nkv) * 128)) and cols == list(range(hidden))
        assert sorted(halves) == list(range(2 * ff // 8))


@pytest.mark.parametrize("sizes", [(2560, 9728, 32, 3), (2560, 9720, 32, 8), (100, 3072, 16, 8), (2560, 1024, 32, 8),
                                   (5120, 25600, 64, 8), (2048, 6144, 64, 4)], ids=str)
def test_sizes_without_a_plan_are_refused(lib, sizes):
    assert lib.gb_decode_stack_layer_bytes(*sizes, 148) == 0


@pytest.mark.parametrize("T", [1, 3, 8])
def test_fragment_order_is_a_permutation(lib, T):
    K = 128
    at = {lib.gb_decode_stack_fragment(k, t, T) for k in range(K) for t in range(T)}
    assert at == set(range(K * T))
    for k in range(K):          # lane c's eight values of 32 columns: the pairs 2c, 2c + 1 of every eight
        base = lib.gb_decode_stack_fragment(k, 0, T) % 32
        assert base // 8 == k % 8 // 2 and base % 8 == k % 32 // 8 * 2 + k % 2
