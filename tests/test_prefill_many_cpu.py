"""prefill_many: what is refused before the library is called."""
import types

import pytest

from doppler_b200.model import Runner


@pytest.mark.parametrize("prompts,seqs", [([[1], [2], [3]], [0, 1]), ([[1, 2]], [0, 1]), ([[1]], []), ([], [0])])
def test_one_sequence_for_every_prompt(prompts, seqs):
    """The library reads one sequence number per prompt: a shorter list would be read past its end."""
    def called(*args):
        raise AssertionError("the library was called")

    m = Runner()
    m.device = types.SimpleNamespace(lib=types.SimpleNamespace(dp_model_prefill_many=called), check=lambda status: None)
    with pytest.raises(ValueError):
        m.prefill_many(prompts, seqs)
