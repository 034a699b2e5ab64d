"""tm_check_finite: every position of a short or misaligned array, both value
types, and the error of the assembler call that waits for it."""
import pytest
import torch

import tensormesh_gb300 as tg
from tensormesh_gb300 import _lib
from tensormesh_gb300.validate import finite_check

pytestmark = pytest.mark.gpu
DEV = "cuda"


@pytest.mark.parametrize("dtype", [torch.float32, torch.float64])
@pytest.mark.parametrize("n", [1, 2, 3, 5, 17, 1023, 300001])
@pytest.mark.parametrize("shift", [0, 1, 3])
def test_finds_a_bad_value_anywhere(dtype, n, shift):
    good = torch.randn(n + shift, device=DEV, dtype=dtype)[shift:]
    big = torch.full_like(good, torch.finfo(dtype).max)
    with finite_check(("points", good), ("kappa", big)):
        pass
    for at in sorted({0, 1 % n, n // 2, n - 1}):
        for bad in (float("nan"), float("inf"), float("-inf")):
            x = torch.cat([good.new_zeros(shift), good])[shift:]
            x[at] = bad
            with pytest.raises(ValueError, match="points"):
                with finite_check(("points", x), ("kappa", big)):
                    pass
            with pytest.raises(ValueError, match="kappa"):
                with finite_check(("points", good), ("kappa", x)):
                    pass


def test_a_failing_body_leaves_the_next_check_clean():
    x = torch.ones(5000, device=DEV)
    x[7] = float("nan")
    with pytest.raises(RuntimeError, match="body"):
        with finite_check(("points", x)):
            raise RuntimeError("body")
    with finite_check(("points", torch.ones(5000, device=DEV))):
        pass


def test_assembler_call_raises_and_names_the_input():
    mesh = tg.Mesh.gen_unit_square(3, device=DEV)

    class KappaLaplace(tg.ElementAssembler):
        def forward(self, gradu, gradv, kappa):
            return kappa * (gradu @ gradv)

    asm = KappaLaplace.from_mesh(mesh)
    kappa = torch.ones(mesh.n_elements, dtype=torch.float64, device=DEV)
    kappa[-1] = float("inf")
    with pytest.raises(ValueError, match="the coefficient"):
        asm(mesh.points, element_data={"kappa": kappa})
    pts = mesh.points.clone()
    pts[0, 0] = float("nan")
    with pytest.raises(ValueError, match="points"):
        tg.const_node_assembler(1.0).from_mesh(mesh)(pts)


def test_rejects_bad_arguments():
    x = torch.ones(4, device=DEV)
    f = torch.zeros(2, dtype=torch.int32, device=DEV)
    for args in ((0, -1, x.data_ptr(), 0, 0, 0), (0, 4, 0, 0, 0, 0), (7, 4, x.data_ptr(), 0, 0, 0),
                 (0, 4, x.data_ptr() + 1, 0, 0, 0)):
        assert _lib.call_status("tm_check_finite", *args, f.data_ptr(), None) == _lib.TM_ERR_INVALID


def test_checks_inside_a_check_keep_their_own_answers():
    good, bad = torch.ones(5000, device=DEV), torch.ones(5000, device=DEV)
    bad[7] = float("nan")
    with pytest.raises(ValueError, match="outer"):
        with finite_check(("outer", bad)):
            torch.cuda.synchronize()
            with finite_check(("inner", good)):
                pass
    with finite_check(("outer", good)):
        with pytest.raises(ValueError, match="inner"):
            with finite_check(("inner", bad)):
                pass
    with finite_check(("points", good), ("kappa", good)):
        pass


def test_an_assembler_called_from_a_saved_tensor_hook():
    """A pack hook runs while the assembler's call is still being checked."""
    mesh = tg.Mesh.gen_unit_square(3, device=DEV)

    class KappaLaplace(tg.ElementAssembler):
        def forward(self, gradu, gradv, kappa):
            return kappa * (gradu @ gradv)

    asm, load = KappaLaplace.from_mesh(mesh), tg.const_node_assembler(1.0).from_mesh(mesh)
    kappa = torch.ones(mesh.n_elements, dtype=torch.float64, device=DEV)
    kappa[2] = float("inf")

    def pack(t):
        torch.cuda.synchronize()
        load(mesh.points)
        return t

    with pytest.raises(ValueError, match="the coefficient"):
        with torch.autograd.graph.saved_tensors_hooks(pack, lambda t: t):
            asm(mesh.points, element_data={"kappa": kappa.requires_grad_(True)})
