"""Where a prompt's product takes its activation along (`many_rows_pay`): the rule restated, at its lines."""
import pytest
import torch


def pays(rows, N, gated, sms=148):
    tiles, pairs = -(-rows // 256) * -(-N // (128 if gated else 256)), sms // 2
    return 2 * tiles >= 3 * pairs and 20 * tiles >= 17 * -(-tiles // pairs) * pairs


def test_lines_of_the_rule():
    assert pays(512, 8192, True) and pays(1024, 8192, False) and pays(6001, 8192, True) and pays(6001, 8192, False)
    assert not pays(256, 8192, True) and not pays(512, 8192, False) and not pays(65, 128256, False, 2 ** 20)
    assert not pays(768, 5000, True)           # 120 tiles: a second wave that is two thirds full


@pytest.mark.gpu
@pytest.mark.parametrize("rows,N,act", [(512, 8192, 3), (256, 8192, 3), (1024, 8192, 1), (512, 8192, 1), (1025, 7680, 3)])
def test_the_extension_follows_it(ext, device, rows, N, act):
    sms = torch.cuda.get_device_properties(device).multi_processor_count
    x, w = torch.randn(rows, 64, device=device).bfloat16(), torch.randn(N * (2 if act == 3 else 1), 64, device=device).bfloat16()
    assert (ext.many_rows(x, w, act) is not None) == pays(rows, N, act == 3, sms)
    assert ext.many_rows(x, w, 0) is None and ext.many_rows(x.float(), w.float(), act) is None
    assert ext.many_rows(x[:, :60], w[:, :60], act) is None and ext.many_rows(x[:1].expand(rows, 64), w, act) is None
