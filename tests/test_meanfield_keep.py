"""The adjoint from kept states against the same adjoint from checkpoints:
bit for bit, where the states would not fit (N T above the budget) and where
rows have more contacts than are loaded ahead (4 and 8 pairs)."""
import numpy as np
import pytest

from replay_b200 import synthetic

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nodes,contacts", [(33, 100), (129, 4000), (1000, 9000)])
def test_kept_states_give_the_checkpointed_gradients(nodes, contacts):
    import torch
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    import replay_b200 as rb
    from replay_b200.meanfield import MeanField
    net = synthetic.tiny(seed=150, n_nodes=nodes, n_contacts=contacts)
    T = 96
    # `pad` nodes without contacts push the states of 96 steps over the 4 GB that are kept
    pad = 2_000_000
    out = []
    for n in (nodes, nodes + pad):
        g = rb.Graph.from_arrays(net["start"], net["end"], net["u"], net["v"], n)
        mf = MeanField(g, iterations=T, step_size=225.0, window=225, start_time=net["t0"], checkpoint_every=17)
        x0 = torch.zeros(4, n, device="cuda")
        x0[0, :nodes], x0[2, :nodes] = 0.9, 0.1
        x0.requires_grad_()
        sus = torch.linspace(0.5, 1.5, nodes, device="cuda")
        sus = torch.cat([sus, torch.ones(n - nodes, device="cuda")]).requires_grad_()
        beta = torch.tensor(3e-4, device="cuda", requires_grad=True)
        inc, xT = mf(x0, beta, susceptibility=sus, p_ei=0.03, p_ir=0.02, p_rs=0.01)
        grads = torch.autograd.grad(inc.square().sum() + xT[3].sum(), [x0, sus, beta])
        out.append([inc, xT[:, :nodes], grads[0][:, :nodes], grads[1][:nodes], grads[2]])
        mf.close()
        g.close()
    for a, b in zip(*out):
        np.testing.assert_allclose(a.detach().cpu().numpy(), b.detach().cpu().numpy(), rtol=2e-6, atol=0)
    for k in (1, 2, 3):  # per-node values have one order of operations
        np.testing.assert_array_equal(out[0][k].detach().cpu().numpy(), out[1][k].detach().cpu().numpy())


# networks of up to 4096 nodes run in one cluster: the same network with unconnected nodes beyond that limit
# takes a launch per step
@pytest.mark.parametrize("nodes,contacts,T,rule", [
    (1, 0, 3, {}), (32, 300, 1, {}), (257, 20_000, 2, {}), (255, 9000, 5, {"has_exposed": 0}),
    (2000, 60_000, 48, {"has_exposed": 0, "ir_to_s": 1}), (4065, 100_000, 7, {}), (4096, 30_000, 24, {})])
def test_one_cluster_agrees_with_step_launches(nodes, contacts, T, rule):
    import torch
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    import replay_b200 as rb
    from replay_b200.meanfield import MeanField
    rng = np.random.default_rng(nodes)
    t0 = synthetic.EPOCH_2000
    u = (rng.random(contacts) ** 3 * nodes).astype(np.int32)  # some nodes have hundreds of pairs
    v = ((u + rng.integers(1, max(2, nodes), contacts)) % nodes).astype(np.int32)
    start = t0 + rng.integers(0, T * 300, contacts)
    end = start + rng.integers(1, 400, contacts)
    if contacts == 0:
        start, end, u, v = np.array([t0 - 90]), np.array([t0 - 50]), np.zeros(1, np.int32), np.ones(1, np.int32)
        nodes = 2
    out = []
    for n in (nodes, nodes + 4096):
        g = rb.Graph.from_arrays(start, end, u, v, n)
        mf = MeanField(g, iterations=T, step_size=300.0, window=300, start_time=t0, ncls_cap=0, **rule)
        x0 = torch.zeros(4, n, device="cuda")
        x0[0, :nodes], x0[1, :nodes], x0[2, :nodes], x0[3, :nodes] = 0.7, 0.1, 0.15, 0.05
        x0.requires_grad_()
        sus = torch.linspace(0.5, 1.5, nodes, device="cuda")
        sus = torch.cat([sus, torch.ones(n - nodes, device="cuda")]).requires_grad_()
        beta = torch.tensor(3e-4, device="cuda", requires_grad=True)
        inc, xT = mf(x0, beta, susceptibility=sus, p_ei=0.03, p_ir=0.02, p_rs=0.01)
        loss = inc.square().sum() + (xT[3] * torch.arange(n, device="cuda").cos()).sum()
        grads = torch.autograd.grad(loss, [x0, sus, beta])
        out.append([inc, xT[:, :nodes], grads[0][:, :nodes], grads[1][:nodes], grads[2]])
        mf.close()
        g.close()
    a, b = ([x.detach().cpu().numpy() for x in o] for o in out)
    for k in (1, 2, 3):
        np.testing.assert_array_equal(a[k], b[k])
    for k in (0, 4):  # sums of the same warps' partial sums
        np.testing.assert_allclose(a[k], b[k], rtol=2e-6, atol=0)
