"""The chunk kernels of the gated delta rule: forms that only long calls take."""
import numpy as np
import pytest
import torch

from raftinfer_b200 import kernels as K

from gpu_util import act_tensor, dev
from test_gated_delta_gpu import DK, HK, HV, LayerRun

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype", [K.DTYPE_BF16, K.DTYPE_F16])
def test_a_long_layer_call_equals_the_same_tokens_in_pieces(dtype):
    """Pieces of whole chunks take the image kernel with four dims a lane, the whole call the one with eight; outputs,
    recurrent states and histories are bit-identical."""
    def run(pieces):
        layer = LayerRun(0xB2006600, HK, HV, 4, dtype, K.DTYPE_F32, sum(pieces))
        if dtype == K.DTYPE_F16:
            layer.inp = layer.inp.astype(np.float16).astype(np.float32)
        outs, done, hidden = [], 0, HV * DK
        for count in pieces:
            shape = K.GatedDeltaShape(count, hidden, HK, HV, DK, DK, 4, 1.0e-6)
            nbytes = K.qwen35_gated_delta_workspace_bytes(shape)
            workspace = torch.zeros(nbytes // 4, device=dev())
            out = torch.zeros(count, hidden, device=dev(), dtype=torch.float16 if dtype == K.DTYPE_F16 else torch.bfloat16)
            K.qwen35_gated_delta(act_tensor(layer.inp[done:done + count], dtype), layer.d_conv_w, layer.d_rec_a, layer.d_dt,
                                 layer.d_norm, out, layer.d_cs, layer.d_rs, workspace, nbytes, shape, dtype, K.DTYPE_F32,
                                 torch.cuda.current_stream())
            torch.cuda.synchronize()
            outs.append(out)
            done += count
        return torch.cat(outs), layer.d_rs, layer.d_cs

    for whole, parts in zip(run([1900]), run([960, 64, 876])):
        assert torch.equal(whole, parts)
