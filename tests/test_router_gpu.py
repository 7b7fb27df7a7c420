"""The router product of more than 256 tokens (csrc/q4b_router.cu: fp32 operands as three bf16 parts on the
tensor cores) against the product in double: edges of its tiles (128 tokens, 64 experts, 128 columns), one
row with an outlier, and error no larger than that of fp32 additions in sequence.  Below 512 tokens the modes
without tensor cores keep a row's bits independent of the batch."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n_tok,n_exp,n", [(257, 48, 1024), (300, 195, 2048), (512, 512, 2048), (641, 130, 2560), (259, 3, 132)])
def test_batch_router_product(dev, n_tok, n_exp, n):
    rng = np.random.default_rng(n_tok + n)
    x = rng.standard_normal((n_tok, n)).astype(np.float32)
    x[5, 7] = 4000.0
    w = (rng.standard_normal((n_exp, n)) * 0.02).astype(np.float32)
    d_y = dev.malloc(n_tok * n_exp * 4)
    dev.write(d_y, np.full((n_tok, n_exp), 7.5, np.float32))
    assert dev.lib.q4_hip_gemv_dd_n(0, dev.upload(w), n_exp, n, dev.upload(x), d_y, 0.5, n_tok)
    y = dev.download(d_y, (n_tok, n_exp), np.float32)
    want = 0.5 * x.astype(np.float64) @ w.astype(np.float64).T
    seq = np.zeros((n_tok, n_exp), np.float32)
    for h in range(n):
        seq += x[:, h:h + 1] * w[:, h]
    err, err_seq = np.abs(y - want), np.abs(0.5 * seq - want)
    plain = np.arange(n_tok) != 5                       # without the outlier's row
    print("router product: error %.3g (%.3g), of fp32 additions in sequence %.3g (%.3g)" %
          (err.max(), np.linalg.norm(err[plain]), err_seq.max(), np.linalg.norm(err_seq[plain])))
    assert err[5].max() <= max(err_seq[5].max(), 2.0 ** -21 * np.abs(want[5]).max())
    assert np.linalg.norm(err[plain]) <= np.linalg.norm(err_seq[plain])
    assert dev.lib.q4_cuda_device_error() == 0


@pytest.mark.parametrize("mode", [0, 2])
@pytest.mark.parametrize("n_tok", [257, 511])
def test_row_bits_without_tensor_cores(dev, n_tok, mode):
    n_exp, n = 130, 2048
    rng = np.random.default_rng(n_tok)
    d_w = dev.upload((rng.standard_normal((n_exp, n)) * 0.02).astype(np.float32))
    d_x, d_y, d_1 = dev.upload(rng.standard_normal((n_tok, n)).astype(np.float32)), dev.malloc(n_tok * n_exp * 4), dev.malloc(n_exp * 4)
    assert dev.lib.q4_cuda_mmq_tc_mode(mode)
    try:
        assert dev.lib.q4_hip_gemv_dd_n(0, d_w, n_exp, n, d_x, d_y, 1.0, n_tok)
    finally:
        assert dev.lib.q4_cuda_mmq_tc_mode(-1)
    y = dev.download(d_y, (n_tok, n_exp), np.float32)
    for t in (0, 128, n_tok - 1):
        assert dev.lib.q4_hip_gemv_dd(0, d_w, n_exp, n, d_x + t * n * 4, d_1, 1.0)
        assert np.array_equal(y[t].view(np.uint32), dev.download(d_1, (n_exp,), np.float32).view(np.uint32))


def test_infinite_operands_and_overflowing_parts(dev):
    """Infinities, NaN and values at the top of the fp32 range give what a sum of fp32 products gives, and leave the other
    logits alone."""
    lib, (n, e, h) = dev.lib, (300, 72, 512)
    rng = np.random.default_rng(3)
    x, w = rng.standard_normal((n, h)).astype(np.float32), rng.standard_normal((e, h)).astype(np.float32)
    x[5, 7], x[6, 8], x[9, 500] = np.inf, -np.inf, np.nan
    x[10, 3], w[3, 3] = 3.4e38, 0.5                       # rounds to infinity as a bf16 value
    w[:, 3] = np.where(np.arange(e) == 3, 0.5, 0.0)
    w[11, 100], w[12, 101] = -np.inf, np.nan
    x[20, :2], w[20, :] = 3e38, 0.0
    w[20, :2] = 1.0, -1.0
    with np.errstate(all="ignore"):
        want = (x[:, None, :].astype(np.float64) * w[None]).sum(2)
        want = np.where(np.abs(want) > np.finfo(np.float32).max, np.sign(want) * np.inf, want)
    d_y = dev.malloc(n * e * 4)
    assert lib.q4_hip_gemv_dd_n(0, dev.upload(w), e, h, dev.upload(x), d_y, 1.0, n)
    y = dev.download(d_y, (n, e), np.float32)
    keep = np.ones_like(y, bool)
    keep[20] = False                                      # fp32 sums of this token overflow or not by their order ...
    keep[20, 20] = True                                   # ... but for this expert
    assert np.array_equal(np.isnan(y)[keep], np.isnan(want)[keep])
    assert np.array_equal(y[keep & np.isinf(want)], want[keep & np.isinf(want)].astype(np.float32))
    fin = keep & np.isfinite(want)
    with np.errstate(all="ignore"):
        mag, off = np.abs(x[:, None, :].astype(np.float64) * w[None]).sum(2), np.abs(y - want)
    assert (off[fin] <= h * 2.0 ** -24 * mag[fin]).all()   # of h fp32 additions
    assert lib.q4_cuda_device_error() == 0
