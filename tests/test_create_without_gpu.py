"""Creating a handle where no GPU is usable: an error status, and what was
created before the failure is given back (the handle's own destructor runs on
a handle that has nothing yet)."""
import pytest
import torch

from unsflow2d_gb300 import abi, mesh
from unsflow2d_gb300.solver import CCSolver, NCSolver

pytestmark = pytest.mark.skipif(torch.cuda.is_available(), reason="needs a machine without a GPU")


@pytest.mark.parametrize("kind", ["cc", "nc"])
def test_creation_fails_with_a_status(kind):
    m = (mesh.CCMesh if kind == "cc" else mesh.NCMesh).airfoil(16, 8)
    p = abi.make_params(time="lusgs", **(dict(flux="ausm", limiter="vkn") if kind == "nc" else {}))
    for _ in range(3):
        with pytest.raises(abi.UnsError, match="no usable GPU"):
            (CCSolver if kind == "cc" else NCSolver)(m, p)
