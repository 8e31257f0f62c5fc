"""ResNet-50 (v1.5: stride on the 3x3 convolution of each bottleneck), 25.6 M parameters.

This is the data-parallel training workload of the end-to-end benchmark: the
communication library is what is being measured, the network is the standard
consumer (the reference itself ships no model; LBANN drives it with ResNet-50,
see README.md:9-17 of the reference).  Random initialisation, no pretrained
weights.
"""
from __future__ import annotations

import torch
from torch import nn

from ..ops.activations import _bare, _modes_off, batch_norm_act, batch_norm_act_twice, max_pool
from ..ops.convolution import cast_weights, convolve, stem_applies, stem_conv


class Bottleneck(nn.Module):
    expansion = 4

    def __init__(self, c_in: int, width: int, stride: int = 1, downsample: nn.Module | None = None):
        super().__init__()
        self.conv1 = nn.Conv2d(c_in, width, 1, bias=False)
        self.bn1 = nn.BatchNorm2d(width)
        self.conv2 = nn.Conv2d(width, width, 3, stride=stride, padding=1, bias=False)
        self.bn2 = nn.BatchNorm2d(width)
        self.conv3 = nn.Conv2d(width, width * self.expansion, 1, bias=False)
        self.bn3 = nn.BatchNorm2d(width * self.expansion)
        self.relu = nn.ReLU(inplace=True)
        self.downsample = downsample

    def forward(self, x):
        if torch.jit.is_scripting():
            identity = x if self.downsample is None else self.downsample(x)
            out = self.relu(self.bn1(self.conv1(x)))
            out = self.relu(self.bn2(self.conv2(out)))
            out = self.bn3(self.conv3(out))
            return self.relu(out + identity)
        else:
            # training on the GPU: normalisation, residual addition and ReLU in one pass (the modules otherwise)
            identity = x if self.downsample is None else self.downsample(x)
            out = batch_norm_act(self.bn1, self.conv1(x), self.relu)
            out = batch_norm_act(self.bn2, self.conv2(out), self.relu)
            return batch_norm_act(self.bn3, self.conv3(out), self.relu, identity)

    def plain(self) -> bool:
        """Nothing but :meth:`forward`'s own steps happens to a block's input, and nothing in its place writes to it: :meth:`twice` may have it
        as two tensors on the same memory."""
        conv, shortcut = self._modules.get("conv1"), self.downsample
        if not (type(conv) is nn.Conv2d and _bare(conv) and _bare(self)):
            return False
        return shortcut is None or (type(shortcut) is Shortcut and _bare(shortcut) and len(shortcut) == 2 and type(shortcut[0]) is nn.Conv2d
                                    and _bare(shortcut[0]))

    def twice(self, x, same):
        """forward(x) as two tensors, for the next block's first convolution and for its end; ``same`` is x, for the end of this one."""
        convs, shortcut = [self.conv1, self.conv2, self.conv3], self.downsample
        if shortcut is not None:
            convs.append(shortcut[0])
        w = cast_weights(convs, x) or [None] * len(convs)
        if shortcut is not None:
            same = batch_norm_act(shortcut[1], convolve(shortcut[0], same, w[3]))
        out = batch_norm_act(self.bn1, convolve(self.conv1, x, w[0]), self.relu)
        out = batch_norm_act(self.bn2, convolve(self.conv2, out, w[1]), self.relu)
        return batch_norm_act_twice(self.bn3, convolve(self.conv3, out, w[2]), self.relu, same)


class Shortcut(nn.Sequential):
    """Convolution and batch norm of a block whose input and output differ in shape."""

    def forward(self, x):
        if torch.jit.is_scripting():
            for m in self:
                x = m(x)
            return x
        else:
            if len(self) != 2:   # something was added or taken out
                return super().forward(x)
            return batch_norm_act(self[1], self[0](x))


class ResNet(nn.Module):
    def __init__(self, layers=(3, 4, 6, 3), num_classes: int = 1000, width: int = 64):
        super().__init__()
        self.c = width
        self.conv1 = nn.Conv2d(3, width, 7, stride=2, padding=3, bias=False)
        self.bn1 = nn.BatchNorm2d(width)
        self.relu = nn.ReLU(inplace=True)
        self.maxpool = nn.MaxPool2d(3, stride=2, padding=1)
        self.layer1 = self._stage(width, layers[0], 1)
        self.layer2 = self._stage(width * 2, layers[1], 2)
        self.layer3 = self._stage(width * 4, layers[2], 2)
        self.layer4 = self._stage(width * 8, layers[3], 2)
        self.avgpool = nn.AdaptiveAvgPool2d(1)
        self.fc = nn.Linear(width * 8 * Bottleneck.expansion, num_classes)
        for m in self.modules():
            if isinstance(m, nn.Conv2d):
                nn.init.kaiming_normal_(m.weight, mode="fan_out", nonlinearity="relu")
            elif isinstance(m, nn.BatchNorm2d):
                nn.init.ones_(m.weight)
                nn.init.zeros_(m.bias)
        for m in self.modules():
            if isinstance(m, Bottleneck):
                nn.init.zeros_(m.bn3.weight)  # residual branches start as identity

    def _stage(self, width: int, blocks: int, stride: int) -> nn.Sequential:
        down = None
        if stride != 1 or self.c != width * Bottleneck.expansion:
            down = Shortcut(nn.Conv2d(self.c, width * Bottleneck.expansion, 1, stride=stride, bias=False),
                            nn.BatchNorm2d(width * Bottleneck.expansion))
        mods = [Bottleneck(self.c, width, stride, down)]
        self.c = width * Bottleneck.expansion
        mods += [Bottleneck(self.c, width) for _ in range(1, blocks)]
        return nn.Sequential(*mods)

    @torch.jit.unused
    def takes_any_layout(self, x) -> bool:
        """Does the first convolution lay these images out itself, so that the trainer need not?"""
        return _bare(self) and stem_applies(self.conv1, x)

    @torch.jit.unused
    def _blocks(self, x):
        """The four stages; in training block by block, each handing its output to the next one twice, so that the two gradients are
        added inside the batch norm's backward."""
        stages = (self.layer1, self.layer2, self.layer3, self.layer4)
        if _modes_off() and self.training and all(type(s) is nn.Sequential and _bare(s) and all(type(b) is Bottleneck and b.plain() for b in s) for s in stages):
            same = x
            for stage in stages:
                for block in stage:
                    x, same = block.twice(x, same)
            return x
        for stage in stages:
            x = stage(x)
        return x

    def forward(self, x):
        if torch.jit.is_scripting():
            x = self.maxpool(self.relu(self.bn1(self.conv1(x))))
        else:
            x = max_pool(self.maxpool, batch_norm_act(self.bn1, stem_conv(self.conv1, x), self.relu))
        if torch.jit.is_scripting():
            x = self.layer4(self.layer3(self.layer2(self.layer1(x))))
        else:
            x = self._blocks(x)
        return self.fc(torch.flatten(self.avgpool(x), 1))


def resnet50(num_classes: int = 1000) -> ResNet:
    return ResNet((3, 4, 6, 3), num_classes)
