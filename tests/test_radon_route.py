"""Which forward projection a call takes (CPU, the library calls recorded): the grouped table for scans of consecutive
angles, the per-bin table for omega subsets, whatever the size and the precision of the rows."""
from types import SimpleNamespace

import pytest
import torch

from diffractom_b200.operator import GTABLE_MIN_WARPS, SinglePhaseForwardOperator


def _operator(My, Kstride, n_batches=1):
    """The attributes of an operator that the forward projection reads, on the host."""
    op = object.__new__(SinglePhaseForwardOperator)
    one = torch.zeros(4)
    op.projector, op.My, op.Kstride, op.Ktot = "native", My, Kstride, n_batches * Kstride
    op.batches = [dict(K_batch=Kstride)] * n_batches
    op.radon_geo = SimpleNamespace(scale=1.0)
    op._ray_rp, op._ray_ent, op._ray_grp = one, one, (one, one, one)
    op.calls = []
    op._call = lambda name, *args: op.calls.append(name)
    op._s = lambda: 0
    return op


@pytest.mark.parametrize("n", [4, 45, 180, 360])
@pytest.mark.parametrize("Kstride", [512, 2048])
def test_subsets_read_the_per_bin_table(n, Kstride):
    op = _operator(263, Kstride)
    om, z = torch.zeros(n, dtype=torch.int32), torch.zeros(4, dtype=torch.bfloat16)
    many = n * 66 * (Kstride // 256) >= GTABLE_MIN_WARPS
    op._radon_fwd(0, 0, om, n, Kstride, m=1)
    op._radon_forward_bf16(0, 0, z, om, n, m=1)
    assert op.calls == ["dfx_radon_forward_table", "dfx_radon_forward_table_bf16"]
    op.calls.clear()
    op._radon_fwd(0, 0, None, n, Kstride)
    op._radon_forward_bf16(0, 0, z, om, n)
    assert op.calls == (["dfx_radon_forward_gtable", "dfx_radon_forward_gtable_bf16"] if many else
                        ["dfx_radon_forward_table", "dfx_radon_forward_table_bf16"])
