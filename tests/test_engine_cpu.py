"""What a plan of the one-call inference (flashdeberta_b200/engine.py) makes of a model, as far as that needs no GPU."""
import torch

from flashdeberta_b200 import FlashDebertaV2Model, engine
from tests.test_configs_gpu import _small_config


def test_a_model_without_registered_parameters_is_not_covered():
    """As data-parallel replicas are: their weights are plain attributes."""
    model = FlashDebertaV2Model(_small_config("b200")).eval()
    for m in model.modules():
        for name in list(m._parameters):
            m.__dict__[name] = m._parameters.pop(name)
    assert not engine._Plan(model).ok


def test_a_plan_belongs_to_one_encoder():
    a, b = (FlashDebertaV2Model(_small_config("b200")).eval() for _ in range(2))
    plan = engine._Plan(a)
    assert plan.current(a) and not plan.current(b)
