"""The streaming grouped product on the wide copy of an arena (csrc/q4b_wide.cu), and the one that decodes the tiles where
an arena has no such copy (csrc/q4b_few.cu), against the general CUDA-core kernel: row counts at the edges of their inner
forms (1 or 2 rows, fragments of 8, blocks of 16; 1 to 3 rows in registers), widths with 1, 2, 4, 8 super-blocks a row (bit
for bit) and others.  Then what keeps the wide copy and the tiles the same, and the tensor-core product on it
(csrc/q4b_wide_tc.cu) beyond the items that a block takes in at a time."""
import os

import numpy as np
import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
pytestmark = pytest.mark.gpu
IQ3_S = 21


@pytest.mark.parametrize("wide", [1, 0])
@pytest.mark.parametrize("H,F", [(2048, 512), (1024, 256), (2560, 768), (512, 256)])
@pytest.mark.parametrize("per", [[1, 2, 3, 0, 8, 9], [16, 17, 33, 1, 0, 70], [1, 1, 1, 1, 1, 1], [0, 0, 5, 0, 0, 0]])
def test_wide_product_equals_the_general_kernel(dev, pkg, monkeypatch, H, F, per, wide):
    monkeypatch.setenv("Q4B_WIDE", str(wide))
    rng = np.random.default_rng(H + F + sum(per))
    E, rows = len(per), sum(per)
    packs = pkg.synth.expert_packs(rng, E, H, F)
    layer = pkg.MoeLayer(dev, packs, None, np.zeros((E, H), np.float32), None, H, F, 1, arena=1)
    lib = dev.lib
    assert lib.q4_cuda_experts_wide_a(1) == wide
    bounds = dev.upload(np.concatenate([[0], np.cumsum(per)]).astype(np.int32))
    try:
        for w_rows, w_cols, off in ((2 * F, H, layer.og), (H, F, layer.od)):
            d_xq, d_dst = dev.malloc(lib.q4_mmq_q8_bytes(rows, w_cols)), dev.malloc(rows * w_rows * 4)
            x = rng.standard_normal((rows, w_cols)).astype(np.float32)
            assert lib.q4_mmq_quantize(dev.upload(x), None, d_xq, IQ3_S, w_cols, rows)
            got = {}
            for mode in (0, 2):
                dev.write(d_dst, np.full((rows, w_rows), 7.5, np.float32))
                assert lib.q4_cuda_mmq_tc_mode(mode)
                assert lib.q4_mmq_mul_id(layer.base + off, IQ3_S, w_rows, w_cols, layer.stride, E, d_xq, bounds,
                                         max(per), rows, d_dst, w_rows)
                got[mode] = dev.download(d_dst, (rows, w_rows), np.float32)
            if w_cols // 256 in (1, 2, 4, 8):
                assert np.array_equal(got[0].view(np.uint32), got[2].view(np.uint32))
            else:
                assert np.linalg.norm(got[0] - got[2]) <= 1e-6 * np.linalg.norm(got[2])
        assert lib.q4_cuda_device_error() == 0
    finally:
        lib.q4_cuda_mmq_tc_mode(-1)
        layer.close()


class _Bytes:
    """Device bytes as an array another library can write."""

    def __init__(self, ptr, n):
        self.__cuda_array_interface__ = {"shape": (n,), "typestr": "|u1", "data": (ptr, False), "version": 3}


@pytest.mark.parametrize("how", ["put", "retile", "copy", "h2d", "h2d_async", "fill", "memset", "part of a tile", "own copy"])
def test_bytes_written_into_a_tiled_arena_reach_both_forms(dev, pkg, how):
    """Packs that are put into a slot, and tiled bytes that are copied over it (a pack moved or duplicated), replace it for
    every kernel: the general one reads the tiles, the streaming and the tensor-core product the wide copy."""
    H, F, E, per = 2048, 512, 3, 24
    rng = np.random.default_rng(11)
    layer = pkg.MoeLayer(dev, pkg.synth.expert_packs(rng, E, H, F), None, np.zeros((E, H), np.float32), None, H, F, 1, arena=1)
    lib, n = dev.lib, layer.pack
    assert lib.q4_cuda_experts_wide_a(1) == 1
    src, dst = (lib.q4_hip_experts_dev_a(1, s) for s in (0, 2))
    x = rng.standard_normal((E * per, H)).astype(np.float32)
    d_x, d_xq = dev.upload(x), dev.malloc(lib.q4_mmq_q8_bytes(E * per, H))
    d_dst, bounds = dev.malloc(E * per * 2 * F * 4), dev.upload((np.arange(E + 1) * per).astype(np.int32))

    def products():
        out = []
        for mode in (2, 0, 1):       # general, streaming, tensor cores
            assert lib.q4_cuda_mmq_tc_mode(mode) and lib.q4_mmq_quantize(d_x, None, d_xq, IQ3_S, H, E * per)
            assert lib.q4_mmq_mul_id(layer.base, IQ3_S, 2 * F, H, layer.stride, E, d_xq, bounds, per, E * per, d_dst, 2 * F)
            out.append(dev.download(d_dst, (E, per, 2 * F), np.float32))
        return out
    try:
        before = products()[0]
        pack = dev.download(src, (n,), np.uint8)
        if how in ("put", "retile"):     # the wide copy is written by the kernel that writes the tiles
            eng, n0 = np.zeros(n, np.uint8), lib.q4_cuda_launch_count()
            assert lib.q4_cuda_experts_get_a(1, 0, eng.ctypes.data, n) and lib.q4_cuda_launch_count() == n0 + 1
            if how == "put":
                assert lib.q4_hip_experts_put_a(1, 2, eng.ctypes.data, n) and lib.q4_cuda_launch_count() == n0 + 2
            else:
                assert lib.q4_hip_h2d(dst, eng.ctypes.data, n)     # (widened as if they were tiles: one launch)
                assert lib.q4_cuda_experts_retile_a(1, 2, 1) and lib.q4_cuda_launch_count() == n0 + 3
            assert np.array_equal(dev.download(dst, (n,), np.uint8), pack)
        elif how == "copy":
            assert lib.q4_hip_copy_async(dst, src, n // 4)
        elif how == "h2d":
            assert lib.q4_hip_h2d(dst, pack.ctypes.data, n)
        elif how == "h2d_async":
            assert lib.q4_hip_h2d_async(dst, pack.ctypes.data, n)
        elif how == "fill":
            assert lib.q4_hip_fill(dst, 0.0, n // 4)
        elif how == "memset":            # on the upload stream
            assert lib.q4_hip_copy_memset(dst, 0, n)
            lib.q4_hip_copy_wait()
        elif how == "part of a tile":    # the tail of one tile, the next one, the head of a third; up to the arena's end too
            assert lib.q4_hip_copy_async(dst + 440, src + 440, (880 + 660) // 4)
            assert lib.q4_hip_copy_async(dst + n - 8, src + n - 8, 2)
        else:
            import torch
            torch.as_tensor(_Bytes(dst, n), device="cuda").copy_(torch.as_tensor(_Bytes(src, n), device="cuda"))
            torch.cuda.synchronize()
            assert lib.q4_cuda_experts_refresh_a(1, 2, 1)
        tiles, wide, tc = products()
        assert not np.array_equal(tiles[2], before[2])
        assert np.array_equal(tiles.view(np.uint32), wide.view(np.uint32))
        assert np.linalg.norm(tiles - tc) <= 1e-5 * np.linalg.norm(tiles)
        assert np.array_equal(tiles[0], before[0]) and np.array_equal(tiles[1], before[1])
        assert not lib.q4_cuda_experts_refresh_a(1, 3, 1) and not lib.q4_cuda_experts_refresh_a(1, 0, 0)
        assert lib.q4_cuda_device_error() == 0
    finally:
        lib.q4_cuda_mmq_tc_mode(-1)
        layer.close()


def test_gather_into_buffers_lent_from_an_arena(dev, pkg):
    """The expert-indexed buffers may be memory that the caller lends, slots of the arena among it: the products read there
    what was gathered.  In a child process: lending cannot be taken back."""
    import subprocess
    import sys
    code = """
import ctypes as C, sys
import numpy as np
sys.path.insert(0, %r)
import __graft_entry__ as entry
pkg = entry.load_package()
dev = pkg.Device()
lib, (H, F, E, per, ty) = dev.lib, (2048, 512, 3, 5, 21)
rng = np.random.default_rng(2)
layer = pkg.MoeLayer(dev, pkg.synth.expert_packs(rng, 2 * E + 2, H, F), None, np.zeros((2 * E + 2, H), np.float32), None, H, F, 1)
gu, d = layer.od, layer.pack - layer.od
slot = lambda i: layer.base + i * layer.stride
assert lib.q4_cuda_experts_wide_a(0) == 1
assert lib.q4_mmq_wbuf_lend(slot(E), E * gu, slot(2 * E), E * d)      # the slots from E on are lent
p, q = C.c_void_p(), C.c_void_p()
assert lib.q4_mmq_wbuf(gu, d, E, C.byref(p), C.byref(q))
order = np.array([2, 0, 1], np.int32)
assert lib.q4_mmq_gather(layer.base, layer.stride, 0, gu, layer.od, d, gu, d, dev.upload(np.arange(E, dtype=np.int32)),
                         dev.upload(order), E, p, q)
bounds = dev.upload((np.arange(E + 1) * per).astype(np.int32))
for w, want, rows, cols, stride in ((p, 0, 2 * F, H, gu), (q, layer.od, H, F, d)):
    x, xq = rng.standard_normal((E * per, cols)).astype(np.float32), dev.malloc(lib.q4_mmq_q8_bytes(E * per, cols))
    assert lib.q4_mmq_quantize(dev.upload(x), None, xq, ty, cols, E * per)
    out = dev.malloc(E * per * rows * 4)
    assert lib.q4_cuda_mmq_tc_mode(2)
    ref = np.zeros((E * per, rows), np.float32)
    for e in range(E):
        one = dev.upload(np.array([e * per, (e + 1) * per], np.int32))
        assert lib.q4_mmq_mul_id(slot(int(order[e])) + want, ty, rows, cols, 0, 1, xq, one, per, E * per, out, rows)
    ref = dev.download(out, (E * per, rows), np.float32)
    for mode in (0, 2):
        assert lib.q4_cuda_mmq_tc_mode(mode)
        assert lib.q4_mmq_mul_id(w, ty, rows, cols, stride, E, xq, bounds, per, E * per, out, rows)
        assert np.array_equal(dev.download(out, (E * per, rows), np.float32), ref), (mode, rows)
assert lib.q4_cuda_device_error() == 0
print("lent ok")
""" % ROOT
    r = subprocess.run([sys.executable, "-c", code], capture_output=True, text=True, timeout=300, cwd=ROOT)
    assert r.returncode == 0 and "lent ok" in r.stdout, r.stdout + r.stderr


@pytest.mark.parametrize("cols,tiles", [(256, 37), (512, 25)])
def test_tensor_core_product_with_several_batches_of_items(dev, pkg, cols, tiles):
    """A pair of CTAs takes in the descriptors of 128 work items at a time, and its pipeline runs on from one batch into the next.
    The launcher makes an item of as many pairs of 128-row tiles as take 16 steps of 128 k and divide their number; 19 and 13
    are prime, so an item is one: 263 and 180 a pair of CTAs on 148 SMs.  One entry in seven has two parts."""
    import torch
    n_exp, steps, pairs = 1023, cols // 128, (tiles + 1) // 2
    per = np.where(np.arange(n_exp) % 7 == 0, 80, 10)
    per[-1] += 20 * n_exp - per.sum()
    assert 0 < per.min() and per.max() <= 128                # a pass an entry
    mt = max(c for c in range(1, pairs + 1) if c == 1 or (c * steps <= 16 and pairs % c == 0))
    ctas = torch.cuda.get_device_properties(0).multi_processor_count // 2
    assert n_exp * (pairs // mt) > 128 * ctas                # more than one batch for every pair of CTAs
    _tensor_core_against_general(dev, pkg, cols, 128 * tiles, per, -1)


@pytest.mark.parametrize("cols,w_rows,n_exp", [(256, 256, 888), (256, 2816, 90), (512, 256, 600), (512, 384, 300), (2048, 128, 296)])
def test_tensor_core_product_with_passes_of_one_and_two_parts(dev, pkg, cols, w_rows, n_exp):
    """Entries of more than 64 rows (two parts) and of at most 64 (one part) in random order, several items to a pair of CTAs:
    the two sets of adding warps take every part of the first and every second tile of the second, and an accumulator goes
    from one set to the other.  Items of one super-block (256 columns, 256 and 2816 rows) up to eight."""
    rng = np.random.default_rng(cols + w_rows)
    per = np.where(rng.random(n_exp) < 0.5, rng.integers(1, 65, n_exp), rng.integers(65, 129, n_exp))
    _tensor_core_against_general(dev, pkg, cols, w_rows, per, 1)


def _tensor_core_against_general(dev, pkg, cols, w_rows, per, mode):
    """A call of mmq_wide_k and of the general kernel, per[e] rows of expert e.  The experts' matrices overlap (an expert starts one tile after the one
    before)."""
    import torch
    lib, n_exp, rows, rb = dev.lib, len(per), int(per.sum()), cols // 256 * 110
    rng = np.random.default_rng(cols)
    pack = pkg.synth.iq3s_blocks(rng, (w_rows * rb + (n_exp - 1) * 880) // 110).reshape(-1)
    lib.q4_cuda_set_tiled_default(2)
    try:
        assert lib.q4_hip_experts_alloc_a(1, 1, pack.nbytes)
    finally:
        lib.q4_cuda_set_tiled_default(1)
    try:
        assert lib.q4_hip_experts_put_a(1, 0, pack.ctypes.data, pack.nbytes) and lib.q4_cuda_experts_wide_a(1) == 1
        x, d_xq = rng.standard_normal((rows, cols)).astype(np.float32), dev.malloc(lib.q4_mmq_q8_bytes(rows, cols))
        bounds, out = dev.upload(np.concatenate([[0], np.cumsum(per)]).astype(np.int32)), []
        for m in (mode, 2):
            y = torch.full((rows, w_rows), 7.5, device="cuda")
            torch.cuda.synchronize()
            assert lib.q4_cuda_mmq_tc_mode(m) and lib.q4_mmq_quantize(dev.upload(x), None, d_xq, IQ3_S, cols, rows)
            assert lib.q4_mmq_mul_id(lib.q4_hip_experts_base_a(1), IQ3_S, w_rows, cols, 880, n_exp, d_xq, bounds, int(per.max()), rows,
                                     y.data_ptr(), w_rows)
            assert lib.q4_cuda_device_error() == 0
            out.append(y.view(rows, w_rows // 128, 128))
        off, ref = (out[0] - out[1]).norm(dim=2), out[1].norm(dim=2)
        assert (ref > 0).all() and (off <= 1e-5 * ref).all(), float((off / ref).max())
    finally:
        lib.q4_cuda_mmq_tc_mode(-1)
        lib.q4_hip_experts_free_a(1)


@pytest.mark.parametrize("H,F", [(2048, 512), (1024, 256), (2560, 768), (256, 256), (1280, 256)])
@pytest.mark.parametrize("per", [[1, 31, 32, 33, 0, 63], [64, 65, 128, 2, 129, 0], [0, 16, 0, 0, 0, 0], [200, 1, 1, 95, 96, 97]])
def test_tensor_core_product_at_the_edges_of_its_passes(dev, pkg, H, F, per):
    """Rows at the edges of the MMA's N (32), of a part (64) and of a pass (128), rows of 1 to 10 super-blocks.  (An odd
    number of 128-row tiles: the tests above.)
    Against the general kernel: activations carry 22 bits there (2^-23 of the row's largest group a term, of random
    sign) and the tensor core truncates eight additions of 24 bits per 128 k: a few 1e-7 of the result; bound 1e-5."""
    rng = np.random.default_rng(H + F + sum(per))
    E, rows = len(per), sum(per)
    packs = pkg.synth.expert_packs(rng, E, H, F)
    layer = pkg.MoeLayer(dev, packs, None, np.zeros((E, H), np.float32), None, H, F, 1, arena=1)
    lib = dev.lib
    assert lib.q4_cuda_experts_wide_a(1) == 1
    bounds = dev.upload(np.concatenate([[0], np.cumsum(per)]).astype(np.int32))
    try:
        for w_rows, w_cols, off in ((2 * F, H, layer.og), (H, F, layer.od)):
            d_xq, d_dst = dev.malloc(lib.q4_mmq_q8_bytes(rows, w_cols)), dev.malloc(rows * (w_rows + 3) * 4)
            x = rng.standard_normal((rows, w_cols)).astype(np.float32)
            assert lib.q4_mmq_quantize(dev.upload(x), None, d_xq, IQ3_S, w_cols, rows)
            got = {}
            for mode in (1, 2):
                dev.write(d_dst, np.full((rows, w_rows + 3), 7.5, np.float32))
                assert lib.q4_cuda_mmq_tc_mode(mode)
                assert lib.q4_mmq_mul_id(layer.base + off, IQ3_S, w_rows, w_cols, layer.stride, E, d_xq, bounds,
                                         max(per), rows, d_dst, w_rows + 3)
                got[mode] = dev.download(d_dst, (rows, w_rows + 3), np.float32)
            if w_cols // 256 in (1, 2, 4, 8):     # (else the call clears the rows whole)
                assert (got[1][:, w_rows:] == 7.5).all()
            diff, ref = np.linalg.norm(got[1] - got[2], axis=1), np.linalg.norm(got[2], axis=1)
            assert (diff <= 1e-5 * ref).all(), float((diff / ref).max())
        assert lib.q4_cuda_device_error() == 0
    finally:
        lib.q4_cuda_mmq_tc_mode(-1)
        layer.close()
