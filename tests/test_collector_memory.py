"""The bound that ``logits_chunk_bytes`` puts on the collector's logits."""
import pytest

from llm_distillery_b200.collect.collector import TeacherCollector

VOCABS = [1000, 32000, 50257, 128256, 151936, 256000]


@pytest.mark.parametrize("vocab", VOCABS)
@pytest.mark.parametrize("mb", [1, 50, 96, 100, 512, 2048])
@pytest.mark.parametrize("pairs", [0, 74])
def test_a_bound_given_by_the_caller_holds(vocab, mb, pairs):
    rows = TeacherCollector.rows_per_chunk(vocab, mb << 20, pairs)
    assert rows % 128 == 0 and (rows == 128 or 4 * rows * vocab <= mb << 20) and 4 * (rows + 128) * vocab > mb << 20


@pytest.mark.parametrize("vocab", VOCABS)
def test_the_default_stays_within_what_it_states(vocab):
    rows = TeacherCollector.rows_per_chunk(vocab, None, 74)
    assert rows >= 512 and (rows == 512 or 4 * rows * vocab <= 128 << 20)
    assert TeacherCollector.rows_per_chunk(32000, None, 74) == 1024
