"""Columns, windows and numbers of sequences that are no whole numbers are refused before anything is launched (an entry point
would take None for 0).  The kernel object here launches nothing: its calls end in a list."""
import types

import pytest
import torch

from zlm_b200.kernels import CudaKernels, PAGE_TOKENS


class Listed(CudaKernels):
    def __init__(self):
        self.bounds_check, self._fn, self._launches, self.calls = False, {}, 0, []
        self._join = self._shares = self._lazy = self._norm_halves = self._blank = None
        self._lane, self._scratch, self.scratch_generation = 0, {}, 0
        self.sm_count, self.decode_blocks = 148, None

    def _entry(self, name):
        return name

    def _invoke(self, name, *args):
        self.calls.append(name)
        return 0

    @staticmethod
    def _queue():
        return 0


H, D, V, T, R = 2, 8, 8, 3, 2
ints = lambda *v: torch.tensor(v, dtype=torch.int32)


def plan(**kw):
    p = dict(R=R, T=T, max_new=2, max_len=2, is_decode=False, token_pos=ints(0, 1, 0), token_slot=ints(0, 0, 1), token_seq=ints(0, 0, 1),
             seq_slot=ints(0, 1), seq_start=ints(0, 0), cu_seqlens=ints(0, 2, 3),
             scratch=lambda name, shape, dtype: torch.empty(shape, dtype=dtype))
    return types.SimpleNamespace(**{**p, **kw})


def retention(k, q_off=0, k_off=16, v_off=32, R=R):
    k.retention(torch.empty(T, H * V), torch.empty(T, 64), q_off, k_off, v_off, None, 0, torch.ones(H), torch.zeros(R or 1, H, D, V),
                plan(R=R), H, D, V, 1.0, pieces=False)


def linear_attention(k, q_off=0, k_off=16, v_off=32, R=R):
    k.linear_attention(torch.empty(T, H * V), torch.empty(T, 64), q_off, k_off, v_off, None, torch.ones(H), torch.zeros(R or 1, H, D, V),
                       plan(R=R), H, D, V, 1.0, pieces=False)


def mingru(k, z_off=0, x_off=16, g_off=32, R=R):
    k.mingru(torch.empty(T, 16), torch.empty(T, 48), z_off, x_off, g_off, None, None, torch.zeros(2, 16), plan(R=R))


def attention(k, window=0):
    k.attention(torch.empty(T, H * D), torch.empty(T, H * D), torch.zeros(2, 2, H, PAGE_TOKENS, D), ints(0, 1).view(2, 1), ints(0, 1, 0),
                ints(0, 0, 1), H, H, D, 1.0, window)


def latent_attention(k, window=0, chunk=0):
    k.latent_attention(torch.empty(T, H * D), torch.empty(T, H * (D + 4)), torch.zeros(2, PAGE_TOKENS, D + 4), ints(0, 1).view(2, 1),
                       ints(0, 1, 0), ints(0, 0, 1), H, D, 4, 1.0, window, chunk=chunk)


def sample(k, top_k=0):
    k.sample(ints(0, 0), torch.zeros(2, 9), 1.0, top_k, 1.0, 1, ints(0, 1), ints(0, 1))


CALLS = [(retention, ("q_off", "k_off", "v_off", "R")), (linear_attention, ("q_off", "k_off", "v_off", "R")),
         (mingru, ("z_off", "x_off", "g_off", "R")), (attention, ("window",)), (latent_attention, ("window", "chunk")), (sample, ("top_k",))]


@pytest.mark.parametrize("call,name", [(c, n) for c, names in CALLS for n in names])
def test_none_is_no_number(call, name):
    k = Listed()
    with pytest.raises(TypeError):
        call(k, **{name: None})
    assert not k.calls


@pytest.mark.parametrize("call", [c for c, _ in CALLS])
def test_the_same_calls_with_numbers_go_through(call):
    k = Listed()
    call(k)
    assert len(k.calls) == 1
