"""int8 mode on a flattened token batch and the paged limb-plane KV cache: the decode / prefill-row path of the
reference's plugin (src/bitexact/vllm_plugin/graph.py:69-87 `_decode_fused`, vllm_plugin/paged.py) with the model
rules of `IntLlama` (src/bitexact/int8/model.py:25-133). Nine kernels per layer: fused int8 linear (GEMM + post),
qkv, attention, attn_out, linear, add_norm, linear, silu_quant, linear, add_norm."""

import ctypes

import torch

from .. import _native as nv
from .. import attn_table
from ..engine_base import TokenRowEngine
from ..vllm_plugin import tri_fuse, tri_paged, tri_prefill
from .consts import silu_compact
from .gemm_skinny import linear_post


class IntEngine(TokenRowEngine):
    FR = 16

    def __init__(self, c, dev="cuda", n_layers=None, nl=2):
        assert nl == 2
        self.dev = torch.device(dev)
        cfg = c.get("cfg", {})
        self.D = cfg.get("hidden_size", 2048)
        self.H = cfg.get("num_attention_heads", 32)
        self.HKV = cfg.get("num_key_value_heads", 8)
        self.HD = cfg.get("head_dim") or self.D // self.H
        self.L = c["n_layers"] if n_layers is None else n_layers
        t = lambda k: c[k].to(self.dev).contiguous()
        self.emb = t("emb")
        self.V = self.emb.shape[0]
        lin = lambda k: (t(k), t(f"{k}.m"), int(c[f"{k}.fm"]) + 8 * (nl - 1) - 24)
        self.layers = [{"ga": t(f"{i}.ga"), "gm": t(f"{i}.gm"), **{n: lin(f"{i}.{n}") for n in ("wqkv", "wo", "wgu", "wd")}}
                       for i in range(self.L)]
        self.FF = self.layers[0]["wgu"][0].shape[0] // 2 if self.layers else cfg.get("intermediate_size", 8192)
        self.gf, self.lm = t("gf"), lin("lm")
        self.silu_t, self.cos, self.sin, self.ln = t("silu"), t("cos"), t("sin"), t("ln")
        self.silu_c = silu_compact(self.silu_t)              # the stage kernels' form of it
        self.ptab = tri_paged.weight_table(t("exp"))
        self.compact = attn_table.to(attn_table.int8(self.ptab), self.dev)                # the decode kernels' form of it
        self.fl = torch.zeros(1, dtype=torch.int32, device=self.dev)
        self.scr = torch.zeros(self.L, 2, dtype=torch.long, device=self.dev)
        self.timer = None                                    # optional callable(M, N, K) -> context manager

    def check(self):
        """OverflowError on a flagged integer bound; `_native.DeviceWaitError` when a device-side wait gave up."""
        nv.check_device_status()
        if bool(self.fl.item()):
            raise OverflowError("integer bound violated (int8 mode)")

    def _lin(self, pre, lin):
        """The linear directly behind the stage that made `pre`."""
        if self.timer is not None:
            with self.timer(pre[1].shape[0], lin[0].shape[0], lin[0].shape[1]):
                return linear_post(pre[0], lin[0], lin[1], lin[2], pre[1], pre[2], self.fl, True)
        return linear_post(pre[0], lin[0], lin[1], lin[2], pre[1], pre[2], self.fl, True, early=True)

    def forward(self, kvs, ids, pos, slot, bt, rmap, tiles=None):
        """Same contract as ExactEngine.forward; returns the residual stream int64 [N, D] at 16 bits."""
        fz = tri_fuse
        N, G = ids.shape[0], self.H // self.HKV
        pos = pos.long().contiguous()
        slot = torch.where(slot < 0, torch.zeros_like(slot), slot).long().contiguous()
        x = self._forward_native(kvs, ids.long(), pos, slot, bt, rmap, tiles)
        if x is not None:
            return x
        qpos = pos.view(-1, 1).expand(-1, G).contiguous()
        x, *pre = fz.embed_norm(self, ids, self.layers[0]["ga"])
        for i in range(self.L):
            ly = self.layers[i]
            q = fz.qkv(self, self._lin(pre, ly["wqkv"]), None, None, None, pos, slot, kvs[i], int32=True)
            if tiles is not None:
                num = torch.zeros(N, self.HKV, G, self.HD, dtype=torch.long, device=self.dev)
                den = torch.ones(N, self.HKV, G, 1, dtype=torch.long, device=self.dev)    # padding rows: 0 / 1
                tri_prefill.attend(q, pos, kvs[i], bt, self.ptab, tiles, num, den)
            else:
                num, den = tri_paged.attend(q, qpos, kvs[i], bt, self.ptab, rmap=rmap, compact=self.compact)
            x, *pre = fz.add_norm(self, self._lin(fz.attn_out(self, num, den), ly["wo"]), None, None, None, x, ly["gm"])
            a8, mant, e, _ = fz.silu_quant(self, self._lin(pre, ly["wgu"]), None, None, None, self.silu_t, scr=self.scr[i],
                                           compact=self.silu_c)
            nxt = self.layers[i + 1]["ga"] if i + 1 < self.L else None
            x, *pre = fz.add_norm(self, self._lin((a8, mant, e), ly["wd"]), None, None, None, x, nxt)
        fz.flag_end(self, self.scr)
        return x

    def _forward_native(self, kvs, ids, pos, slot, bt, rmap, tiles):
        if self.timer is not None or rmap is None or getattr(self._lin, "__func__", None) is not IntEngine._lin:
            return None                                          # a timer brackets every linear, another _lin is to be called for each
        rows, shapes = [], []
        for ly in self.layers[:self.L]:
            row = []
            for n in ("wqkv", "wo", "wgu", "wd"):
                w, mul, fmsh = ly[n]
                row += (w.data_ptr(), mul.data_ptr(), int(fmsh), w.shape[0], w.shape[1])
            shapes.append((row[3], row[4], row[8], row[9], row[13], row[14], row[18], row[19]))
            rows.append(row + [ly["ga"].data_ptr(), ly["gm"].data_ptr()])
        form = None if self.compact is None else attn_table.native(self.compact)       # lives until the call has read it
        fields = dict(ptab=self.ptab.data_ptr(), silu=self.silu_t.data_ptr(), silu_compact=nv.ptr(self.silu_c), scr=self.scr.data_ptr(),
                      compact=None if form is None else ctypes.addressof(form))
        return self.forward_native("bx_int8_forward", False, fields, rows, shapes, kvs, ids, pos, slot, bt, rmap, tiles)

    def logits(self, h):
        """Final residual rows [M, D] -> int64 logits [M, V] at 16 bits."""
        return self._lin(tri_fuse.pre_norm(self, h, self.gf), self.lm)
