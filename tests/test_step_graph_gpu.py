"""The captured training step against the eager one."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("model,task", [("gpt2-tiny", "causal"), ("bert-tiny", "mlm"), ("llama-tiny", "causal")])
def test_captured_steps_equal_eager_steps(model, task):
    """Losses and weights over several steps, a learning-rate change, labels given, another shape, restored state."""
    from dynamiq_sigcomm_artifact_b200.train.engine import TrainConfig, Trainer

    cfg = dict(model=model, micro_batch=3, seq_len=65, lr=1e-3, weight_decay=0.01, task=task, total_steps=20)
    a, b = Trainer(TrainConfig(cuda_graphs=True, **cfg)), Trainer(TrainConfig(cuda_graphs=False, **cfg))
    assert a.graphed and not b.graphed
    gen = torch.Generator().manual_seed(1)
    ids = [torch.randint(0, 1024, (3, 65), generator=gen) for _ in range(4)] + [torch.randint(0, 1024, (2, 40), generator=gen)]
    for step in range(10):
        x = ids[step % 5]
        labels = x.clone() if step >= 6 else None
        if step == 4:
            for t in (a, b):
                t.opt.load_state_dict(t.opt.state_dict())
                t.opt.param_groups[0]["weight_decay"] = 0.2
        la, lb = a.train_step(x, labels), b.train_step(x, labels)
        assert abs(la - lb) < 5e-3 * abs(lb), step
    for p, q in zip(a.model.parameters(), b.model.parameters()):
        if p.dim() == 2:  # (a bias starts at zero, where the first updates follow the sign of rounding noise)
            assert float((p.detach() - q.detach()).norm()) < 2e-2 * float(q.detach().norm())
    held = a.train_step_device(ids[0].cuda())
    value = held.item()
    a.train_step_device(ids[1].cuda())
    assert held.item() == value  # the returned loss is the caller's
