"""What the decode loop (`decode.Session`, `generate`) asks of an engine besides `forward`, `logits` and `check`: the
per-layer cache of a session and the tile table of a prompt portion. The defaults are those of the integer engines (a
paged limb-plane KV cache in every layer, the prefill tile kernel on longer prompts)."""

import torch


class TokenRowEngine:
    """Engines with D, V, L, FR, ln, dev and forward(caches, ids, pos, slot, bt, rmap, tiles=None)."""

    page = 16               # tokens per cache page of a session
    tiles_from = 384        # prompt portions that end before this position attend row by row
    # (attention of one layer, tile kernel against row kernel, us, exact mode: 4 prompts of 16 / 64 / 128 / 256 / 383 / 1024 tokens
    # 61 : 21, 67 : 38, 83 : 81, 122 : 158, 173 : 272, 584 : 1746; one prompt of 128 / 256 / 383 / 1024 63 : 35, 78 : 56, 90 : 88,
    # 193 : 447. The lines cross between 128 tokens of four prompts and 383 of one.)

    def new_cache(self, n_seqs, n_blocks, bs):
        """The caches of a session of n_seqs sequences over n_blocks pages of bs tokens (page 0: null page), one per
        layer, as `forward` takes them."""
        return [torch.zeros(n_blocks, self.HKV, bs, 8 * self.HD, dtype=torch.int8, device=self.dev) for _ in range(self.L)]

    def tile_table(self, runs, bs):
        """Attention tiles for runs = [(table row, first token row, tokens, context length)] of a step, int32 [T, 3] on
        the host, or None when this engine has no tile kernel for its geometry."""
        from .vllm_plugin import tri_prefill
        G = self.H // self.HKV
        if self.HD != 64 or tri_prefill.BM % G or bs not in (8, 16, 32, 64, 128):
            return None
        return tri_prefill.tile_table(runs, G, tri_prefill.ROWS)

    def forward_native(self, call, exact, fields, layers, shapes, kvs, ids, pos, slot, bt, rmap, tiles):
        """All layers' kernels from one call of the library (`bx_exact_forward`, `bx_int8_forward`): fields of bx_step beside the common
        ones, layers a flat list of what a bx_*_layer holds in front of its cache, one list per layer, shapes the rows and columns of
        its four matrices. Returns the residual rows, or None where the call's geometry is not what that entry takes (the engines then run
        their own loop)."""
        import ctypes

        from . import _native as nv
        N, G, dev = ids.shape[0], self.H // self.HKV, ids.device
        if N == 0 or self.HD != 64 or G > 4 and tiles is None or len(kvs) < self.L or tiles is not None and tiles.shape[0] == 0:
            return None
        FF = shapes[0][4] // 2                                   # of the weights: a config need not name it
        if shapes.count(((self.H + 2 * self.HKV) * self.HD, self.D, self.D, self.H * self.HD, 2 * FF, self.D, self.D, FF)) < len(shapes):
            return None
        bs, flat = kvs[0].shape[2], []
        for c, layer in zip(kvs, layers):
            assert c.shape[1] == self.HKV and c.shape[3] == 8 * self.HD and c.stride(3) == 1 and c.dtype == torch.int8
            if c.shape[2] != bs:
                return None
            flat += layer
            flat += (c.data_ptr(), c.shape[0], c.stride(0), c.stride(1), c.stride(2))
        assert bt.shape[1] * bs < 43690 and bt.dtype in (torch.int32, torch.int64) and bt.stride(1) == 1
        x = torch.empty(N, self.D, dtype=torch.long, device=dev)
        n = nv.lib().bx_forward_bytes(int(exact), N, self.D, self.H, self.HKV, self.HD, FF, bt.shape[1], bs, int(tiles is not None))
        work = torch.empty(n, dtype=torch.uint8, device=dev)
        keep = [ids.contiguous(), rmap.long().contiguous()]
        s = nv.Step(ids=keep[0].data_ptr(), pos=pos.data_ptr(), slot=slot.data_ptr(), bt=bt.data_ptr(), rmap=keep[1].data_ptr(), cos=self.cos.data_ptr(),
                    sin=self.sin.data_ptr(), emb=self.emb.data_ptr(), x=x.data_ptr(), flag=self.fl.data_ptr(), work=work.data_ptr(), layers=self.L, N=N,
                    D=self.D, H=self.H, HKV=self.HKV, HD=self.HD, FF=FF, bs=bs, bt64=int(bt.dtype == torch.int64), sbt=bt.stride(0),
                    nblk=bt.shape[1], work_bytes=n, **fields)
        if tiles is None:
            keep.append(pos.view(-1, 1).expand(-1, G).contiguous())
            s.qpos = keep[-1].data_ptr()
        else:
            assert tiles.dtype == torch.int32
            keep += [tiles.contiguous(), torch.zeros(N, self.H, self.HD, dtype=torch.long, device=dev), torch.ones(N, self.H, dtype=torch.long, device=dev)]
            s.tiles, s.num, s.den, s.n_tiles = keep[-3].data_ptr(), keep[-2].data_ptr(), keep[-1].data_ptr(), tiles.shape[0]
        nv.check(getattr(nv.lib(), call)(ctypes.addressof(s), (ctypes.c_int64 * len(flat))(*flat), nv.stream()), call)
        return x

    def logits_float(self, h):
        """`logits` as float32."""
        return (self.logits(h).double() * 2.0 ** -self.FR).float()
