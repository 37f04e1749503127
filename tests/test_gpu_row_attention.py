"""Attention of 2 .. 7 positions in the GEMM route, a block per query, heads of a group and share of the keys, against the decode kernel, which walks the positions one after the other: caches
around the 32 keys of a turn and the shares of a cluster, two, four and eight query heads per key head (the decode kernel has no other), both head sizes, both 16-bit types.  Behind the products both are
fp32; what is left are 16-bit roundings of the same values in another order: 2^-8 (bf16), 2^-11 (fp16) of a row, four times."""
from dataclasses import replace

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu

from xotorch_b200.synth import PRESETS, hf_config


@pytest.mark.parametrize("name", ["tiny-llama-hd64", "tiny-llama-hd128", "tiny-llama-hd64-f16", "tiny-llama-hd128-f16"])
@pytest.mark.parametrize("heads,kv_heads", [(8, 4), (8, 2), (8, 1)])
def test_against_the_decode_kernel(name, heads, kv_heads):
  from xotorch_b200.native import NativeShard
  shape = replace(PRESETS[name], name=name + "-row", n_heads=heads, n_kv_heads=kv_heads)
  eng = NativeShard(hf_config(shape), 0)
  eng.set_shard(1, 1)
  eng.init_synthetic(heads + kv_heads)
  dt = torch.float16 if shape.dtype == "float16" else torch.bfloat16
  rows = torch.randn(1600, shape.dim, generator=torch.Generator().manual_seed(heads)).to(dt).cuda()
  out = torch.empty_like(rows)
  eng.begin_request(1600)
  torch.cuda.synchronize()
  eng.forward_device(None, rows.data_ptr(), 1590, 0, out.data_ptr())
  for pos0 in (0, 1, 25, 30, 31, 57, 63, 64, 120, 126, 500, 1590):
    for n in (2, 5, 7):
      h, got = rows[pos0:pos0 + n].clone(), []
      for mode in (2, 1):
        eng.set_prefill_mode(mode)
        o = torch.empty_like(h)
        torch.cuda.synchronize()
        eng.forward_device(None, h.data_ptr(), n, pos0, o.data_ptr())
        got.append(o.double().cpu().numpy())
      eng.set_prefill_mode(0)
      err = np.sqrt(((got[0] - got[1]) ** 2).mean(-1) / (got[1] ** 2).mean(-1)).max()
      assert err < 4 * (2 ** -8 if dt == torch.bfloat16 else 2 ** -11), (pos0, n, err)
  eng.close()
