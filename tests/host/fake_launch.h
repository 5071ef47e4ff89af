// fake_launch.h -- see fake_launch.cpp
#pragma once
extern int fake_fail_launches;  // n > 0: the n-th step launch from now on fails
extern int fake_step_launches;  // step launches so far
extern int fake_maps;           // tensor maps encoded so far
extern bool fake_strip;         // what march_takes answers
