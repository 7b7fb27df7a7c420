"""The streaming product on IQ4_NL / IQ4_XS rows (csrc/q4b_rows4.cu) against the kernel with a warp per weight
row, bit for bit: widths on either side of its lane splits (8, 16, 32, 64 groups a row and between), row counts
at the edges of its forms (1, 2, 8, 9, 16, 17 rows), short last chunks."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("ty,cols,w_rows", [(20, 128, 48), (20, 256, 144), (23, 256, 80), (20, 384, 64), (20, 512, 2048), (23, 512, 272),
                                            (23, 768, 96), (20, 1024, 208), (23, 2048, 1024), (20, 2048, 48),
                                            (23, 2560, 80), (20, 4096, 32)])
def test_streaming_product_equals_row_kernel(dev, pkg, ty, cols, w_rows):
    rng = np.random.default_rng(cols + w_rows + ty)
    per = [1, 2, 0, 3, 8, 9, 16, 17, 1, 35]
    E, rows = len(per), sum(per)
    rb = pkg.synth.row_bytes(ty, cols)
    w = pkg.synth.blocks_of(rng, ty, E * w_rows * rb)
    x = rng.standard_normal((rows, cols)).astype(np.float32)
    lib = dev.lib
    d_w, bounds = dev.upload(w), dev.upload(np.concatenate([[0], np.cumsum(per)]).astype(np.int32))
    d_xq, d_dst = dev.malloc(lib.q4_mmq_q8_bytes(rows, cols)), dev.malloc(rows * (w_rows + 4) * 4)
    assert lib.q4_mmq_quantize(dev.upload(x), None, d_xq, ty, cols, rows)
    got = {}
    try:
        for mode in (-1, 2):
            dev.write(d_dst, np.full((rows, w_rows + 4), 7.5, np.float32))
            assert lib.q4_cuda_mmq_tc_mode(mode)
            assert lib.q4_mmq_mul_id(d_w, ty, w_rows, cols, w_rows * rb, E, d_xq, bounds, max(per), rows, d_dst, w_rows + 4)
            got[mode] = dev.download(d_dst, (rows, w_rows + 4), np.uint32)
    finally:
        lib.q4_cuda_mmq_tc_mode(-1)
    assert np.array_equal(got[-1], got[2])
    assert lib.q4_cuda_device_error() == 0
