"""The chains' log-probabilities around MCState.sample: its own samplers write them for the
final configurations; a call that is refused leaves those of the current ones; a sampler with
a ``sample`` of its own finds them in the state, as ``reset`` promises."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def _state(nk, sampler, alpha, **kw):
    return nk.vqs.MCState(sampler, nk.models.RBM(alpha=alpha), n_samples=sampler.n_chains * 2,
                          n_discard_per_chain=1, seed=3, **kw)


@pytest.mark.parametrize("reset_chains", [False, True])
def test_a_refused_call_leaves_log_probabilities(reset_chains):
    import netket_gb300 as nk
    hi = nk.hilbert.Spin(0.5, 4)
    vs = _state(nk, nk.sampler.MetropolisLocal(hi, n_chains=8, reset_chains=reset_chains), 1750)
    with pytest.raises(RuntimeError, match="too large"):  # M = 7,000
        vs.sample()
    st = vs.sampler_state
    assert torch.equal(st.log_prob, 2.0 * vs.log_value(st.σ))
    assert st.n_steps == 0 and st.n_accepted == 0


def test_a_sampler_of_its_own_gets_log_probabilities():
    import netket_gb300 as nk
    seen = []

    class Sampler(nk.sampler.MetropolisSampler):
        def sample(self, machine, params, *, state=None, **kw):
            seen.append((state.σ.clone(), state.log_prob.clone()))
            return super().sample(machine, params, state=state, **kw)

    hi = nk.hilbert.Spin(0.5, 6)
    vs = _state(nk, Sampler(hi, nk.sampler.LocalRule(), n_chains=8), 2)
    for _ in range(2):
        vs.sample()
    for sigma, log_prob in seen:
        assert torch.equal(log_prob, 2.0 * vs.log_value(sigma))
    st = vs.sampler_state  # and the call writes those of the final configurations
    torch.testing.assert_close(st.log_prob, 2.0 * vs.log_value(st.σ), rtol=1e-12, atol=1e-12)


def test_a_state_without_log_probabilities():
    """``sample`` needs the configurations alone, as ``reset`` does."""
    import netket_gb300 as nk
    hi = nk.hilbert.Spin(0.5, 6)
    vs = _state(nk, nk.sampler.MetropolisLocal(hi, n_chains=8), 2)
    vs.sampler_state.log_prob = None
    vs.sample()
    st = vs.sampler_state
    torch.testing.assert_close(st.log_prob, 2.0 * vs.log_value(st.σ), rtol=1e-12, atol=1e-12)
