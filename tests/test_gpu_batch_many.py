"""GPU: the V sum of batches by warps of 64 elements (one query head per KV head, or many sequences), at every number of query
heads per KV head, with lengths around its tiles of 32 positions, against the one-sequence operator."""
import pytest

from tests.test_gpu_batch import test_batched_attention_equals_one_sequence_attention as check

pytestmark = pytest.mark.gpu

LENS = [1, 31, 32, 33, 3, 64, 127, 500, 799, 800, 96, 130]


@pytest.mark.parametrize("hd,nh,nkv,max_seq,lens", [(64, 3, 3, 130, [1, 4, 33, 130]), (128, 2, 2, 70, [70])] +
                         [(64, 16 * rep, 16, 800, LENS) for rep in range(2, 9)] + [(128, 32, 8, 801, LENS)])
def test_many_warps_equal_one_sequence_attention(hd, nh, nkv, max_seq, lens):
    check(hd, nh, nkv, max_seq, lens)
