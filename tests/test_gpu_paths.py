"""Branches of the host and kernel dispatch, each at the sizes where it can go wrong, against the other entry points or
the oracle."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def pkg(lib_built):
    assert torch.cuda.is_available()
    import llama_cl_b200

    return llama_cl_b200


@pytest.mark.parametrize("rows", [1, 8, 9])
def test_host_fc_in_place_and_copied(pkg, rows):
    """Up to 8 rows the kernels work on the pinned buffers themselves, beyond that on copies: the same FC either way."""
    g = torch.Generator().manual_seed(rows)
    W = (torch.randn(1003, 640, generator=g) * 0.02).cuda()
    wq = pkg.llmops.offline_FC_quant_Q4A(W, qtype="q4_1", group_k=128)
    fc = pkg.host.HostFC(wq, 1003, max_rows=16)
    for _ in range(3):  # captured on the first call, replayed with new inputs afterwards
        x = torch.randn(1, rows, 640, generator=g)
        want = pkg.llmops.fc_Q4A(x.cuda(), wq, 1003).cpu()
        assert torch.equal(fc(x), want)
