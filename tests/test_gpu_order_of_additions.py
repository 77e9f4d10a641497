"""The order in which a GEMM adds does not depend on gradients being on or on the rest of the batch, wherever a loss is
taken of the result."""
import pytest
import torch

from llm_distillery_b200.collect.collector import TeacherCollector
from llm_distillery_b200.engine.trainer import DistillEngine, synthetic_batch
from llm_distillery_b200.models import llama
from llm_distillery_b200.ops import _lib

pytestmark = pytest.mark.gpu


def _model(seed=1):
    return llama.build_model(llama.preset("tinyllama-1.1b", num_hidden_layers=2), dtype=torch.bfloat16, device="cuda", seed=seed)


@pytest.mark.parametrize("loss", ["reference", "kl"])
@pytest.mark.parametrize("B,L", [(1, 93), (2, 333)])
def test_validation_loss_is_the_training_forwards_loss(loss, B, L):
    """Equal weights and batch: the bits of the loss are equal with and without gradients."""
    engine = DistillEngine(_model(), loss=loss)
    hb = synthetic_batch(32000, B, L, 100, 1, reference_fields=loss == "reference")
    without, _ = engine.eval_batch(hb)
    with_grad, _ = engine.loss_on_batch(hb.to_device(engine.device))
    assert torch.equal(without, with_grad.detach())
    assert _lib.take_device_error() == 0


@pytest.mark.parametrize("L,chunk", [(93, 0), (333, 0), (333, 128)])
def test_hidden_states_do_not_depend_on_the_rest_of_the_batch(L, chunk):
    model = _model()
    ids = torch.randint(0, 32000, (4, L), device="cuda", generator=torch.Generator("cuda").manual_seed(L))
    with torch.no_grad():
        run = (lambda x: model.hidden_states_chunked(x, chunk)) if chunk else model.hidden_states
        assert torch.equal(run(ids[:1]), run(ids)[:L])
    assert _lib.take_device_error() == 0


def test_a_teacher_may_split_unless_its_owner_chose_one_order():
    model, chosen = _model(), _model()
    chosen.ordered_sums = True
    for m in (model, chosen):
        TeacherCollector(m, topk=8, crop_to_size=32000)
    assert model.ordered_sums is False and chosen.ordered_sums is True
    engine = DistillEngine(model, loss="reference")          # the student of one run may be the teacher of another
    hb = synthetic_batch(32000, 1, 93, 100, 1, reference_fields=True)
    assert torch.equal(engine.eval_batch(hb)[0], engine.loss_on_batch(hb.to_device(engine.device))[0].detach())


def test_engines_of_two_losses_on_one_model_keep_their_orders():
    """The reference loss's backward keeps one order of additions also when an engine of another loss was made after it.
    Distinct tokens and one key block: no atomic sum has more than one term."""
    def gradient(second):
        engine = DistillEngine(_model(), loss="reference")
        if second:
            DistillEngine(engine.model, loss="kl")
        flat = engine.model.layers[0].gate_up_proj
        hb = synthetic_batch(32000, 1, 120, 100, 1, reference_fields=True)
        hb.input_ids = torch.arange(120).reshape(1, -1)
        engine.micro_step(hb.to_device(engine.device))
        return flat.grad_slot.buf.clone()
    assert torch.equal(gradient(False), gradient(True))
    assert _lib.take_device_error() == 0
