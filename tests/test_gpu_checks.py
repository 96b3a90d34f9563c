"""``dqb_state_checks`` against the same norms and traces in torch's complex128."""

import pytest
import torch

from dynamiqs_b200 import _lib

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize('n', [1, 2, 31, 32, 33, 64, 65, 130, 700])  # edges of the 32 x 32 tiles
@pytest.mark.parametrize('count', [1, 5, 2000])  # states split over blocks, or a block each
def test_state_checks(cuda_device, n, count):
    if n > 130:
        count = min(count, 5)
    g = torch.Generator(device=cuda_device).manual_seed(n)
    x = torch.randn(count, n, n, dtype=torch.complex64, device=cuda_device, generator=g)
    x[0] = x[0] + x[0].mH
    x[-1] = 0 if count > 1 else x[-1]
    lib = _lib.load()
    size = lib.dqb_state_checks_workspace_size(n, count)
    ws = torch.empty(size, dtype=torch.uint8, device=cuda_device)
    out = torch.empty(count, dtype=torch.float64, device=cuda_device)
    tr = torch.empty(count, dtype=torch.complex128, device=cuda_device)
    stream = torch.cuda.current_stream().cuda_stream
    assert lib.dqb_state_checks(x.data_ptr(), n, count, out.data_ptr(), tr.data_ptr(), ws.data_ptr(), size, stream) == 0
    st = x.to(torch.complex128)
    num = torch.linalg.norm((st - st.mH).reshape(count, -1), dim=-1)
    ref = num / torch.clamp(torch.linalg.norm(st.reshape(count, -1), dim=-1), min=1e-300)
    # FP64 sums of at most n^2 terms in another order
    assert torch.allclose(out, ref, rtol=1e-12, atol=1e-15)
    assert torch.allclose(tr, st.diagonal(dim1=-2, dim2=-1).sum(-1), rtol=1e-12, atol=1e-12)
    assert lib.dqb_state_checks(x.data_ptr(), n, count, out.data_ptr(), tr.data_ptr(), ws.data_ptr(), size - 1, stream) \
        == _lib.DQB_ERR_WORKSPACE_TOO_SMALL
