"""The cases of perf/cases.py: what a pass returns against the same inputs evaluated in 64 bits by
plain torch, on a small case of each kind.  Bar: the case's own tolerance, which covers the block
formats' codes that fall on the other side of a rounding behind an intermediate."""
import pytest

pytestmark = pytest.mark.gpu

SMALL = [
    {"kind": "mmvq", "k": 1024, "n": 65, "cols": 3},
    {"kind": "ffn", "hidden": 512, "inter": 1024, "layers": 2, "tokens": 1, "glu": "swiglu"},
    {"kind": "ffn", "hidden": 1280, "inter": 2048, "layers": 2, "tokens": 7, "glu": "geglu"},
    {"kind": "proj", "k": 1024, "n": 333, "layers": 3, "tokens": 2},
    {"kind": "decode_vector", "k": 1024, "n": 257, "layers": 2, "tokens": 2, "decoder": "q8_0"},
    {"kind": "decode_vector", "k": 1152, "n": 300, "layers": 2, "tokens": 1, "decoder": "bf16"},
    {"kind": "mmq", "tokens": 131, "k": 1280, "n": 520, "slab": False, "bf16": False},
    {"kind": "mmq", "tokens": 17, "k": 2304, "n": 900, "slab": True, "bf16": True},
    {"kind": "moe", "tokens": 40, "experts": 16, "used": 2, "hidden": 1024, "inter": 512, "layers": 1},
    {"kind": "moe", "tokens": 150, "experts": 16, "used": 2, "hidden": 1024, "inter": 512, "layers": 1},
]


@pytest.mark.parametrize("case", SMALL, ids=lambda c: c["kind"])
def test_a_pass_gives_what_exact_says(cuda, case):
    torch = cuda
    from perf import cases
    got, want = cases.run(cases.prepare(case, 11)), cases.exact(case, 11)
    torch.cuda.synchronize()
    for g, w in zip(got, want) if isinstance(got, list) else [(got, want)]:
        assert g.shape == w.shape
        rel = float((g.double() - w).norm() / w.norm())
        assert rel <= cases.tolerance(case)["rel"], rel
