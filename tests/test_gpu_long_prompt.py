"""Prompts of the shard engine at the edges of a 4096-token prefill chunk: one call and the same prompt handed over in portions that end where the
chunks do run the same kernels on the same rows, so hidden states and logits agree bit for bit; a portion that ends elsewhere is another 16-bit
evaluation of the same model."""
import dataclasses

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

from xotorch_b200.synth import PRESETS, hf_config, synth_prompt
from tests.test_gpu_parity import ATOL, RTOL


def _logits(shape_name, prompt, cuts):
  from xotorch_b200.native import NativeShard
  shape = dataclasses.replace(PRESETS[shape_name], max_pos=8192)
  e = NativeShard(hf_config(shape), device=0)
  e.set_shard(0, shape.n_layers - 1)
  e.init_synthetic(1234)
  e.set_prefill_mode(2)
  e.begin_request(prompt.shape[1] + 8)
  pos = 0
  for n in cuts:
    out = e.forward(prompt[:, pos:pos + n].astype(np.int32), pos)[0].copy()
    pos += n
  assert pos == prompt.shape[1]
  more = e.forward(np.array([[3]], dtype=np.int32), pos)[0].copy()     # reads every cached key
  e.close()
  return np.stack([out, more])


@pytest.mark.parametrize("shape_name", ["tiny-llama-hd64", "tiny-llama-hd128"])
@pytest.mark.parametrize("n", [2701, 4095, 4096, 4097, 4096 + 130])
def test_chunks_equal_portions(shape_name, n):
  prompt = synth_prompt(PRESETS[shape_name].vocab, n)
  whole = _logits(shape_name, prompt, [n])
  if n > 4096:
    assert np.array_equal(whole, _logits(shape_name, prompt, [4096, n - 4096]))
  cut = _logits(shape_name, prompt, [1000, n - 1000])
  assert (np.abs(whole - cut) <= ATOL + RTOL * np.abs(whole)).all(), np.abs(whole - cut).max()


@pytest.mark.parametrize("shift", [0, 50, -50])
def test_output_over_the_input(shift):
  """hidden states on the device, the result laid over the input or `shift` rows beside it: as into a buffer of its own"""
  import torch
  from xotorch_b200.native import NativeShard
  shape, n = dataclasses.replace(PRESETS["tiny-llama-hd64"], max_pos=8192), 4096 + 130
  e = NativeShard(hf_config(shape), device=0)
  e.set_shard(1, 2)
  e.init_synthetic(1234)
  e.begin_request(n)
  x = torch.randn(n, shape.dim, generator=torch.Generator().manual_seed(1)).to(torch.bfloat16).cuda()
  own = torch.empty_like(x)
  e.forward_device(None, x.data_ptr(), n, 0, own.data_ptr())
  room = torch.zeros(n + 100, shape.dim, dtype=torch.bfloat16, device="cuda")
  room[50:50 + n] = x
  torch.cuda.synchronize()
  e.forward_device(None, room[50:].data_ptr(), n, 0, room[50 + shift:].data_ptr())
  assert torch.equal(room[50 + shift:50 + shift + n], own)
  e.close()
