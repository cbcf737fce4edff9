"""The batch's actions read in place and its results written to the caller's tensors by the step's own
launches: the same bits for actions given in any form (contiguous device tensors are read in place,
all else is copied), as for the environments stepped one by one, and results that the next step
leaves alone."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

from microcosmos_b200.gym import BatchedEnv, LineEnv  # noqa: E402

FORMS = {
    "device": lambda a: torch.as_tensor(a, device="cuda"),
    "flat": lambda a: torch.as_tensor(a, device="cuda").reshape(-1),
    "strided": lambda a: torch.as_tensor(np.repeat(a, 2, axis=1), device="cuda")[:, ::2],
    "double": lambda a: torch.as_tensor(a, device="cuda").double(),
    "host": lambda a: torch.as_tensor(a),
    "numpy": lambda a: a,
}


def run(batch, steps, form, only=None):
    env = LineEnv(num_nodes=17, grid_shape=(48, 40), max_steps=2)
    be = BatchedEnv(env, batch)
    first, state = be.reset(list(range(batch)))
    E, B = state.states[0].device.E, state.states[0].device.B
    rng = np.random.default_rng(3)
    out = [first]
    for _ in range(steps):
        acts = {"d_rest_length": rng.normal(0, 0.05, (batch, E)).astype(np.float32),
                "d_bending_angle": rng.normal(0, 0.2, (batch, B)).astype(np.float32)}
        acts = {k: FORMS[form](v) for k, v in acts.items() if only in (None, k)}
        obs, state, reward, done, info = be.step(None, state, acts)
        assert done.dtype == torch.bool and info["steps"].dtype == torch.int32
        out += [obs, reward, done, info["steps"], info["energy_center"]]
    return [t.cpu().numpy() for t in out]  # read after the last step


@pytest.mark.parametrize("only", [None, "d_rest_length", "d_bending_angle"])
@pytest.mark.parametrize("form", [f for f in FORMS if f != "host"])
@pytest.mark.parametrize("batch", [1, 5])
def test_any_form_of_the_actions(batch, form, only):
    want = run(batch, 3, "host", only)
    for g, w in zip(run(batch, 3, form, only), want):
        assert g.shape == w.shape and g.tobytes() == w.tobytes()
    assert not want[3].any() and want[8].all() and want[13].all()
