"""Tiling of the tensor-core 32 -> 32 layers: bands of rows chosen by the batch
and tail items (16 rows x 8 columns) for the columns the 128-pixel segments
leave over.  Convolution outputs do not depend on the tiling (the same products
in the same order), so an image alone and the same image in a batch give the
same bits, and both match a float64 reference within the bf16 rounding of the
output (2^-9 relative, REL = 4e-3); the weight gradient matches a float64 sum
within REL_WG = 1e-4 (float32 sums of exact products)."""

import numpy as np
import pytest

from test_gpu_cnn_tc import REL, REL_WG, _bf16, _conv_ref, _rel

pytestmark = pytest.mark.gpu

# one column left, exactly the tail's width, one more, no segment at all; rows
# around the 16 of a tail item, a single row, more rows than slots hold bands
SHAPES = [(1, 1, 129), (1, 16, 136), (2, 17, 137), (3, 31, 5), (1, 33, 8), (2, 40, 264), (1, 257, 257), (40, 18, 130)]


@pytest.mark.parametrize("B,H,W", SHAPES)
def test_layers_do_not_depend_on_the_tiling(B, H, W):
    import torch

    from pararealml_gb300 import _native

    lib = _native.lib()
    rng = np.random.default_rng(B * 1000 + H * 10 + W)
    x = _bf16(rng.normal(0.0, 1.0, (B, H, W, 32))).cuda()
    g = _bf16(rng.normal(0.0, 1.0, (B, H, W, 32))).cuda()
    w = _bf16(rng.normal(0.0, 0.1, (9, 32, 32))).cuda()
    bias = torch.tensor(rng.normal(0.0, 0.1, 32), dtype=torch.float32, device="cuda")
    s = torch.cuda.current_stream().cuda_stream

    def convs(xs, masks):
        n = xs.shape[0]
        y0, y1 = torch.full_like(xs, float("nan")), torch.full_like(xs, float("nan"))
        _native.check(lib.prml_cnn_mid_fwd(xs.data_ptr(), w.data_ptr(), bias.data_ptr(), y0.data_ptr(), n, H, W, s), "fwd")
        _native.check(lib.prml_cnn_mid_dgrad(xs.data_ptr(), w.data_ptr(), masks.data_ptr(), y1.data_ptr(), n, H, W, s),
                      "dgrad")
        torch.cuda.synchronize()
        _native.check(lib.prml_cnn_status(), "tcgen05 status")
        return y0.view(torch.int16).cpu().numpy(), y1.view(torch.int16).cpu().numpy(), y0, y1

    b0, b1, y0, y1 = convs(x, g)
    big0, big1, _, _ = convs(x.repeat(17, 1, 1, 1), g.repeat(17, 1, 1, 1))
    assert np.array_equal(np.tile(b0, (17, 1, 1, 1)), big0) and np.array_equal(np.tile(b1, (17, 1, 1, 1)), big1)
    xf, wf, gf = (t.float().cpu().numpy().astype(np.float64) for t in (x, w, g))
    assert _rel(y0.float().cpu().numpy(), _conv_ref(xf, wf, bias=bias.cpu().numpy())) < REL
    assert _rel(y1.float().cpu().numpy(), _conv_ref(xf, wf, mask=gf)) < REL

    xp = np.zeros((B, H + 2, W + 2, 32))
    xp[:, 1:-1, 1:-1] = xf
    want = np.stack([np.einsum("bhwk,bhwn->kn", xp[:, t // 3: t // 3 + H, t % 3: t % 3 + W], gf) for t in range(9)])
    for parts in (608, 7):
        scratch = torch.empty(lib.prml_cnn_wgrad_scratch_elems(parts), dtype=torch.float32, device="cuda")
        dw = torch.full((9, 32, 32), float("nan"), dtype=torch.float32, device="cuda")
        db = torch.full((32,), float("nan"), dtype=torch.float32, device="cuda")
        _native.check(lib.prml_cnn_mid_wgrad(x.data_ptr(), g.data_ptr(), dw.data_ptr(), db.data_ptr(), parts,
                                             scratch.data_ptr(), B, H, W, s), "mid wgrad")
        torch.cuda.synchronize()
        _native.check(lib.prml_cnn_status(), "tcgen05 status")
        assert _rel(dw.cpu().numpy().astype(np.float64), want) < REL_WG
        assert _rel(db.cpu().numpy().astype(np.float64), gf.sum(axis=(0, 1, 2))) < REL_WG
