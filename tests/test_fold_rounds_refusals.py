"""What the fold entries refuse, and that a refused call queues nothing: sizes
past a field's two-adicity, generators that are not built, shifts that are no
field elements, short or misaligned buffers. On the host, the pointers are
placeholders that no launch sees; on the GPU the transcript's state stays as it
was."""

from __future__ import annotations

import ctypes

import pytest

torch = pytest.importorskip("torch")

from zorch_gb300 import _lib  # noqa: E402
from zorch_gb300.commit import Poseidon2, koalabear16_params  # noqa: E402
from zorch_gb300.field import BABYBEAR, KOALABEAR  # noqa: E402

BAD_SHAPE, OOM, BAD_ARG, UNSUPPORTED = 1, 4, 7, 8


def _perm(orc, field):
    return (Poseidon2.builtin() if field is BABYBEAR
            else koalabear16_params(orc.load_koalabear_fixture()))


def _desc(rounds, log_n, buf, generator=0, shift=0):
    """A descriptor whose every device pointer is `buf`."""
    d = _lib.FoldRoundsDesc()
    d.rounds, d.log_n, d.beta_limbs, d.generator = rounds, log_n, 1, generator
    d.shifts_keep = (ctypes.c_uint32 * rounds)(*[shift] * rounds)
    d.shifts = ctypes.addressof(d.shifts_keep)
    for name in ("codeword", "first_tree", "layers", "trees", "final_layer", "state", "betas",
                 "roots"):
        setattr(d, name, buf)
    return d


def _refusals(field):
    p, g = field.p, field.generator
    return [
        ("two-adic", 2, field.two_adicity + 1, {}, BAD_SHAPE),
        ("generator", 2, 6, {"generator": g + 1}, UNSUPPORTED),
        ("shift", 2, 6, {"shift": p}, BAD_ARG),
        ("shift", 1, 6, {"shift": 2**32 - 1}, BAD_ARG),
    ]


@pytest.mark.parametrize("which", range(4))
@pytest.mark.parametrize("field", [BABYBEAR, KOALABEAR], ids=lambda f: f.name)
def test_fold_rounds_refuse(orc, field, which):
    text, rounds, log_n, kw, status = _refusals(field)[which]
    buf = (ctypes.c_uint32 * 1024)()
    d = _desc(rounds, log_n, (ctypes.addressof(buf) + 15) // 16 * 16, **kw)
    L = _lib.lib()
    assert L.zc_fold_rounds(_perm(orc, field).handle, ctypes.byref(d), None) == status
    assert text in L.zc_last_error().decode()


@pytest.mark.parametrize("br", [False, True])
@pytest.mark.parametrize("field", [BABYBEAR, KOALABEAR], ids=lambda f: f.name)
def test_folds_refuse_layers_past_the_two_adicity(orc, field, br):
    buf = (ctypes.c_uint32 * 64)()
    a = (ctypes.addressof(buf) + 15) // 16 * 16
    n, L = 2 << field.two_adicity, _lib.lib()
    fold = L.zc_fri_fold_bitrev if br else L.zc_fri_fold
    assert fold(field.id, a, n, 0, a, 0, 0, 0, a, None) == BAD_SHAPE


@pytest.mark.gpu
@pytest.mark.parametrize("what", ["generator", "shift", "workspace", "final_layer", "trees",
                                  "beta_limbs"])
def test_a_refused_call_leaves_the_transcript(orc, what):
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    buf = torch.zeros(1 << 14, dtype=torch.int32, device="cuda")
    state = torch.arange(34, dtype=torch.int32, device="cuda")
    d = _desc(3, 6, buf.data_ptr())
    d.state = state.data_ptr()
    want = BAD_ARG
    if what == "generator":
        d.generator, want = BABYBEAR.generator + 1, UNSUPPORTED
    elif what == "shift":
        d.shifts_keep[2] = BABYBEAR.p
    elif what == "workspace":
        for name in ("mle", "eq", "claim", "zinv", "msgs", "workspace"):
            setattr(d, name, buf.data_ptr())
        d.workspace_bytes, want = _lib.lib().zc_fold_rounds_workspace_bytes(3) - 4, OOM
    elif what == "beta_limbs":
        d.beta_limbs = 2
    else:
        setattr(d, what, buf.data_ptr() + 4)
    status = _lib.lib().zc_fold_rounds(Poseidon2.builtin().handle, ctypes.byref(d),
                                       torch.cuda.current_stream().cuda_stream)
    torch.cuda.synchronize()
    assert status == want
    assert torch.equal(state, torch.arange(34, dtype=torch.int32, device="cuda"))
    assert not buf.any()
