"""The tensor-core form's operand rows, certificates and list merges where
they can go wrong: widths around the runs of four columns, the eight lanes of
a row and a warp's reach, row addresses that load four values at a time or one,
the split, FP16 and unit-row forms, odd row counts (two rows share a warp).
Ids and distance bits equal the FP32 form's."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _search(lib, x, y, k, metric, precision):
    import torch

    from manifoldann_gb300 import _lib

    p = _lib.params(metric, k, precision, 0, 0)
    ids = torch.empty((len(y), k), dtype=torch.int32, device="cuda")
    d = torch.empty((len(y), k), dtype=torch.float32, device="cuda")
    _lib.check(lib.mann_knn_device(p, x.data_ptr(), len(x), y.data_ptr(), len(y), x.shape[1], ids.data_ptr(),
                                   d.data_ptr(), None, torch.cuda.current_stream().cuda_stream))
    torch.cuda.synchronize()
    return ids.cpu().numpy(), d.cpu().numpy().view(np.uint32)


@pytest.mark.parametrize("d", [4, 8, 12, 20, 36, 60, 64, 68, 100, 128, 132, 252, 256, 260, 388, 516, 1028])
@pytest.mark.parametrize("form,metric", [("bf16", 1), ("fp16", 0), ("bf16", 2), ("fp16", 2)])
@pytest.mark.parametrize("kind", ["normal", "halves"])
def test_widths_and_alignments(gpu_lib, d, form, metric, kind):
    import torch

    from manifoldann_gb300 import _lib

    prec = {"bf16": _lib.PREC_BF16, "fp16": _lib.PREC_FP16}[form]
    n, nq = 2500, 601
    rng = np.random.default_rng(d)
    X = rng.standard_normal((n + nq, d)).astype(np.float32)
    if kind == "halves":
        X = np.round(4 * X) / 4
    X[7] = 0.0  # a zero row: no unit direction
    flat = torch.from_numpy(np.ascontiguousarray(X)).cuda().reshape(-1)
    odd = torch.empty(flat.numel() + 1, device="cuda")[1:].copy_(flat)  # 4 bytes past the alignment
    want = None
    for rows in (flat, odd):
        x, y = rows[: n * d].view(n, d), rows[n * d:].view(nq, d)
        if want is None:
            want = _search(gpu_lib, x, y, 9, metric, _lib.PREC_FP32)
        got = _search(gpu_lib, x, y, 9, metric, prec)
        assert np.array_equal(got[0], want[0])
        assert np.array_equal(got[1], want[1])
