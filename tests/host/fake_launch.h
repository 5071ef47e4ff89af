// fake_launch.h -- see fake_launch.cpp
#pragma once
extern int fake_fail_launches;  // n > 0: the n-th step launch from now on fails
