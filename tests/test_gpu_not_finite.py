"""Groups of NaNs in the block-scaled operands."""

import numpy as np
import pytest
import torch

from tests.helpers import Records, smooth_fields

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dim, query_block, dtype", [(64, 64, torch.float16), (128, 128, torch.bfloat16)])
def test_nan_groups_quantise_to_zero(native_library, dim, query_block, dtype):
    """A NaN never wins a maximum, so sixteen of them have maximum zero: scale byte and codes are zero, in
    the rows of Q and K (groups of channels) and in V (groups of keys); every other group keeps its bits."""
    from anemoi_b200 import native
    from anemoi_b200.executor import make_shape
    from anemoi_b200.layout import materialize_ragged_2d_layout

    vs = (2, 16, 16)
    q, k, v = (t.cuda() for t in smooth_fields(*vs, 2, dim, 0, seed=1, dtype=dtype))
    layout = materialize_ragged_2d_layout(q.device, frames=2, height=16, width=16, logical_block=query_block)
    shape = make_shape(q, prefix_tokens=0, video_blocks=layout.video_blocks, query_block_size=query_block,
                       active=("nvfp4",), native_prefix=False, has_maxpool=False, nvfp4_scales=(0.01, 0.01, 0.002))

    def prepared():
        store = native.allocate_operands(shape, q.device)
        for t in store.buffers.values():
            if t is not None:
                t.zero_()            # the bytes between the rows of a scale block are nobody's
        native.prepare(shape, q, k, v, layout.indices, layout.counts, store)
        torch.cuda.synchronize()
        r = Records(store, shape, 1)
        return (*r.q_nvfp4(), *r.kv_nvfp4())

    slots = layout.indices.long()
    clean = prepared()
    q[0, slots[5], 1, 16:32] = float("nan")
    k[0, slots[70], 1, :] = float("nan")
    v[0, slots[16:32], 1, 3] = float("nan")
    qc, qs, kc, ks, vc, vsf = prepared()
    for t, at in ((qc, np.s_[5, 16:32]), (qs, np.s_[5, 1]), (kc, np.s_[70]), (ks, np.s_[70]), (vc, np.s_[16:32, 3])):
        assert not t[at].any()
    changed = [np.argwhere(a != b) for a, b in zip(clean, (qc, qs, kc, ks, vc, vsf))]
    assert all((c[:, 0] == 5).all() and (c[:, 1] // 16 == 1).all() for c in changed[:1])
    assert changed[1].tolist() == [[5, 1]]
    assert (changed[2][:, 0] == 70).all() and (changed[3][:, 0] == 70).all() and len(changed[3]) == dim // 16
    assert ((changed[4][:, 0] // 16 == 1) & (changed[4][:, 1] == 3)).all() and len(changed[5]) == 1
    assert vsf[tuple(changed[5][0])] == 0
