"""The streaming grouped product on the wide copy of an arena (csrc/q4b_wide.cu) against the general
CUDA-core kernel, which decodes the tiles themselves: row counts at the edges of its inner forms (1 or 2
rows, fragments of 8, blocks of 16), widths with 1, 2, 4, 8 super-blocks a row (bit for bit) and others."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu
IQ3_S = 21


@pytest.mark.parametrize("H,F", [(2048, 512), (1024, 256), (2560, 768), (512, 256)])
@pytest.mark.parametrize("per", [[1, 2, 3, 0, 8, 9], [16, 17, 33, 1, 0, 70], [1, 1, 1, 1, 1, 1], [0, 0, 5, 0, 0, 0]])
def test_wide_product_equals_the_general_kernel(dev, pkg, H, F, per):
    rng = np.random.default_rng(H + F + sum(per))
    E, rows = len(per), sum(per)
    packs = pkg.synth.expert_packs(rng, E, H, F)
    layer = pkg.MoeLayer(dev, packs, None, np.zeros((E, H), np.float32), None, H, F, 1, arena=1)
    lib = dev.lib
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
